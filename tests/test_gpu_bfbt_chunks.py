"""The z chunks the matrix-free BFBt direction kernel is launched with, and the forms the mixed solve picks."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nel", [(4, 3, 1), (4, 2, 2), (8, 9, 3), (36, 8, 5), (32, 16, 67), (68, 33, 20), (6, 5, 4)])
def test_matrix_free_apply_matches_stencil(uw, nel):
    """one chunk per plane up to several; the last mesh's x extent is not a multiple of 4 (the other kernel)"""
    from earthbyte_underworld_gb300 import workloads as W
    U = uw
    w = W.spheres(nel=nel, nspheres=5, seed=7)
    x = np.random.default_rng(2).standard_normal(int(np.prod(nel)))
    with U.Context(0) as ctx:
        W.setup_context(ctx, w)
        ctx.bin_and_map(want=False)
        ctx.assemble()
        ctx.solve_bsscr(U.default_opts(mg_levels=1, max_outer=1, a11_rtol=1e-2, back_rtol=1e-2), check=False)
        exact = ctx.bfbt_operator_apply(x, 0)
        free = ctx.bfbt_operator_apply(x, 1)
    # FP32 sums of 8 x 24 terms of both signs: 192 rounding errors of 2^-24 against the largest term
    assert np.abs(free - exact).max() < 192 * 2.0 ** -24 * np.abs(exact).max()


@pytest.mark.parametrize("nel", [(16, 8, 8), (18, 8, 8)])
def test_inner_forms_give_the_same_solution(uw, nel):
    """default form (matrix-free when x is a multiple of 4, else the stencil) against the forced ones, solved tight"""
    from earthbyte_underworld_gb300 import workloads as W
    U = uw
    w = W.spheres(nel=nel, nspheres=5, seed=7)
    with U.Context(0) as ctx:
        W.setup_context(ctx, w)
        ctx.bin_and_map(want=False)
        ctx.assemble()
        out = []
        for form in (0, 2, 3):
            o = U.default_opts(mg_levels=2, schur_type=1, schur_pc=3, smoother=1, precision=1, scr_rtol=1e-11,
                               a11_rtol=1e-12, back_rtol=1e-12, max_inner=2000, bfbt_max_it=2000, bfbt_inner_pc=form)
            out.append(ctx.solve_bsscr(o)[:2])
    for u, p in out[1:]:   # the accuracy at which two tight solves of this system agree
        assert np.linalg.norm(u - out[0][0]) < 1e-8 * np.linalg.norm(u)
        assert np.linalg.norm(p - out[0][1]) < 1e-6 * np.linalg.norm(p)
