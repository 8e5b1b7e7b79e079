"""Which form the mixed solve's BFBt inner iterations take, told by the work they count: per element and iteration 68
operations on the stencil and 110 matrix-free; the one-launch solve counts its traffic once per solve."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

STENCIL, MATRIX_FREE, ONE_LAUNCH = "stencil", "matrix-free", "one launch"
CASES = [((16, 8, 8), 0, ONE_LAUNCH), ((18, 8, 8), 0, ONE_LAUNCH), ((16, 8, 8), 2, STENCIL), ((18, 8, 8), 3, ONE_LAUNCH),
         ((16, 8, 8), 4, STENCIL), ((18, 8, 8), 4, STENCIL), ((16, 12), 0, STENCIL), ((16, 12), 3, MATRIX_FREE)]


@pytest.mark.parametrize("nel,pc,form", CASES)
def test_form_of_the_inner_solve(uw, nel, pc, form):
    from earthbyte_underworld_gb300 import workloads as W
    U = uw
    w = W.rt2d(nel=nel, ppc=12) if len(nel) == 2 else W.spheres(nel=nel, nspheres=5, seed=7)
    ne = int(np.prod(nel))
    with U.Context(0) as ctx:
        W.setup_context(ctx, w)
        ctx.bin_and_map(want=False)
        ctx.assemble()
        ctx.profile_enable()
        o = U.default_opts(mg_levels=2, schur_type=1, schur_pc=3, smoother=1, precision=1, scr_rtol=1e-6, a11_rtol=1e-7,
                           back_rtol=1e-7, bfbt_max_it=600, bfbt_inner_pc=pc)
        u, p, rep = ctx.solve_bsscr(o)
        nbytes, flops = ctx.profile_work(U.KERNEL_SCHUR_PC)
    per = flops / (ne * rep.pc_inner_its)
    if form == STENCIL:
        assert per == (68.0 if len(nel) == 3 else 32.0)
    else:
        assert per == (110.0 if len(nel) == 3 else 46.0)
        assert (nbytes < 60.0 * ne * rep.pc_inner_its / 12) == (form == ONE_LAUNCH)
