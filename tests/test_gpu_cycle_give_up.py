"""A launch of the one-launch multigrid cycle that gives up on a barrier is reported as that, by the solve it happens
in, and by no later one.  The give-up is set on the host (nothing waits in vain here)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ERR_CUDA, ERR_STATE = 2, 4


def _opts(U, **kw):
    return U.default_opts(mg_levels=3, schur_type=1, schur_pc=3, smoother=1, scr_rtol=1e-8, a11_rtol=1e-9,
                          back_rtol=1e-9, **kw)


def _assembled(U, W, w):
    ctx = U.Context(0)
    W.setup_context(ctx, w)
    ctx.bin_and_map(want=False)
    ctx.assemble()
    return ctx


def test_reported_once(uw):
    from earthbyte_underworld_gb300 import workloads as W
    U = uw
    with _assembled(U, W, W.grf(nel=(8, 8, 8), ppc=8, grid=32)) as ctx:
        u0, p0, rep = ctx.solve_bsscr(_opts(U))
        for _ in range(2):
            ctx.cycle_give_up()
            with pytest.raises(U.UwgpuError, match="barrier"):
                ctx.solve_bsscr(_opts(U))
            u, p, rep = ctx.solve_bsscr(_opts(U))
            assert rep.status == 0 and np.linalg.norm(u - u0) < 1e-6 * np.linalg.norm(u0)


def test_named_where_the_solve_fails_first(uw):
    """a solve that ends with another error before its own check (here: no network for the learned preconditioner)
    names the give-up, and the next solve finds no flag"""
    from earthbyte_underworld_gb300 import workloads as W
    U = uw
    with _assembled(U, W, W.grf(nel=(8, 8, 8), ppc=8, grid=32)) as ctx:
        with pytest.raises(U.UwgpuError) as plain:
            ctx.solve_bsscr(_opts(U, learned_pc=1))
        assert plain.value.code == ERR_STATE
        ctx.cycle_give_up()
        with pytest.raises(U.UwgpuError, match="barrier") as named:
            ctx.solve_bsscr(_opts(U, learned_pc=1))
        assert named.value.code == ERR_CUDA
        u, p, rep = ctx.solve_bsscr(_opts(U))
        assert rep.status == 0
