"""The BFBt inner solve in one launch: cuts into bricks from one block up, with ragged last bricks, one element
per thread up to a column of several, against the launched CG on the stencil."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nel,levels", [((4, 4, 4), 1), ((7, 5, 9), 1), ((20, 12, 28), 2), ((34, 6, 4), 2), ((2, 3, 37), 1),
                                        ((64, 40, 24), 3)])
def test_one_launch_solve_gives_the_same_solution(uw, nel, levels):
    """matrix-free form (3) against the FP32 stencil (2), solved tight: the accuracy at which two tight solves
    of this system agree, as between the forms elsewhere"""
    from earthbyte_underworld_gb300 import workloads as W
    U = uw
    w = W.spheres(nel=nel, nspheres=5, seed=7)
    with U.Context(0) as ctx:
        W.setup_context(ctx, w)
        ctx.bin_and_map(want=False)
        ctx.assemble()
        out = []
        for form in (2, 3):
            o = U.default_opts(mg_levels=levels, schur_type=1, schur_pc=3, smoother=1, precision=1, scr_rtol=1e-11,
                               a11_rtol=1e-12, back_rtol=1e-12, max_inner=2000, bfbt_max_it=2000, bfbt_inner_pc=form)
            out.append(ctx.solve_bsscr(o)[:2])
    (u2, p2), (u3, p3) = out
    assert np.linalg.norm(u3 - u2) < 1e-8 * np.linalg.norm(u2)
    assert np.linalg.norm(p3 - p2) < 1e-6 * np.linalg.norm(p2)
