"""The one-launch multigrid cycle (csrc/cycle.cu): V-cycle solves that run it, wholly or from a coarser level
on, against W-cycle solves of the same system, which run the separate kernels."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return np.linalg.norm((a - b).reshape(-1)) / np.linalg.norm(b.reshape(-1))


# (elements, levels, smoother, precision, sweeps down, up, restart): the smallest levels, sizes beside the
# limits (2D 281^2 and 283^2 nodes, 3D 33^3 and 49^3), odd Chebyshev degrees, no pre-smoothing, a long basis
CASES = [((2, 2), 2, 0, 0, 2, 2, 30), ((10, 6), 2, 0, 0, 1, 2, 30), ((64, 48), 4, 1, 0, 3, 1, 60),
         ((280, 280), 4, 0, 0, 2, 2, 30), ((284, 284), 3, 0, 0, 2, 2, 30), ((48, 20), 3, 1, 1, 2, 2, 30),
         ((2, 4, 2), 2, 0, 0, 2, 2, 30), ((12, 8, 20), 3, 0, 0, 0, 2, 60), ((16, 16, 16), 3, 1, 1, 3, 3, 30),
         ((32, 32, 32), 4, 0, 0, 2, 2, 30), ((32, 32, 32), 4, 1, 1, 2, 2, 30), ((48, 48, 48), 4, 1, 1, 2, 2, 30)]


@pytest.mark.parametrize("nel,levels,smoother,precision,down,up,restart", CASES)
def test_cycle_solves_match_separate_kernels(uw, nel, levels, smoother, precision, down, up, restart):
    from earthbyte_underworld_gb300 import workloads as W
    U = uw
    dim = len(nel)
    w = W.rt2d(nel=nel, ppc=12) if dim == 2 else W.spheres(nel=nel, nspheres=6, seed=3)
    with U.Context(0) as ctx:
        W.setup_context(ctx, w)
        ctx.bin_and_map(want=False)
        ctx.assemble()
        out = []
        for cycle in (1, 2):
            # one Schur iteration: two velocity solves to 1e-12, each 1e-12 from the exact answer times the
            # operator's condition (here below 1e4), so 1e-8 with a margin for the sum of both
            o = U.default_opts(mg_levels=levels, smoother=smoother, precision=precision, smooth_down=down,
                               smooth_up=up, restart=restart, mg_cycle=cycle, schur_type=U.SCHUR_FGMRES,
                               max_outer=1, scr_rtol=1e-14, a11_rtol=1e-12, back_rtol=1e-12, max_inner=1000)
            u, p, rep = ctx.solve_bsscr(o, check=False)
            assert rep.vcycles > 0 and np.isfinite(u).all() and np.isfinite(p).all()
            out.append((u, p, rep))
    (u1, p1, r1), (u2, p2, r2) = out
    print(nel, "V", r1.vcycles, "W", r2.vcycles, _rel(u1, u2), _rel(p1, p2))
    assert _rel(u1, u2) < 1e-8 and _rel(p1, p2) < 1e-8
