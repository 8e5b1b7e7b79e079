"""The inner CG of the scaled BFBt preconditioner by itself (uwgpu_bfbt_inner_solve): range of its sums, and its
four forms against the FP64 stencil."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _uniform(U, nel):
    """a context with one material of viscosity 1 and a built operator"""
    dim = len(nel)
    e = np.arange(int(np.prod(nel)))
    c = []
    for n in nel:
        c.append((e % n + 0.5) / n)
        e = e // n
    ctx = U.Context(0)
    ctx.mesh_q1(dim, nel)
    ctx.bc_set(U.free_slip_mask(dim, nel))
    ctx.materials_set([U.make_material([(U.LAW_MATERIAL_VISCOSITY, [1.0])], density=1.0)])
    ctx.fields_set(None, 1.0, dim - 1)
    ctx.particles_upload(*(c + [None] * (3 - dim)))
    _build(U, ctx)
    return ctx


def _build(U, ctx):
    ctx.bin_and_map(want=False)
    ctx.assemble()
    ctx.solve_bsscr(U.default_opts(mg_levels=1, max_outer=1, a11_rtol=1e-2, back_rtol=1e-2), check=False)


def test_one_launch_sums_have_the_range_of_fp64(uw):
    """A right-hand side scaled by a power of two gives the solution scaled by it, bit for bit, as long as the FP32
    values and the FP32 sums of one warp stay in range; the sums over all warps may pass the largest FP32."""
    nel = (24, 24, 24)
    with _uniform(uw, nel) as ctx:
        b = np.random.default_rng(3).choice([-1.0, 1.0], int(np.prod(nel)))
        b -= b.mean()
        x, its = ctx.bfbt_inner_solve(b, form=1, rtol=1e-5)
        d = float(b @ ctx.bfbt_operator_apply(b) / (b @ b))
        # r.z of the whole mesh at twice the largest FP32: 13,824 like terms, of which a warp adds at most 256
        most = float((b @ b) * max(1.0, 1.0 / d))
        scale = 2.0 ** np.ceil(0.5 * np.log2(2.0 * 3.4e38 / most))
        big, its_big = ctx.bfbt_inner_solve(b * scale, form=1, rtol=1e-5)
    assert 24 <= its == its_big and np.isfinite(x).all() and np.abs(x).max() > 0
    assert np.array_equal(big, x * scale)


@pytest.mark.parametrize("nel,form", [((16, 12), 2), ((10, 9, 8), 2), ((16, 12), 3), ((12, 9, 8), 3), ((10, 9, 8), 3),
                                      ((68, 19, 21), 3), ((30, 31, 21), 3), ((12, 9, 8), 1), ((10, 9, 8), 0)])
def test_inner_solve_stops_where_its_test_is_met(uw, nel, form):
    """x meets the tolerance, and twelve iterations before the end it did not: each form, the two-kernel matrix-free
    one with both of its direction kernels (x extents that are a multiple of 4 and not).  Tolerances that FP32
    meets (the recurrence's residual is then that of x to a few 2^-24, so cases within 5% are left out)."""
    seen = 0
    with _uniform(uw, nel) as ctx:
        b = np.random.default_rng(5).standard_normal(int(np.prod(nel)))
        b = ctx.bfbt_operator_apply(b - b.mean())
        for rtol in 10.0 ** -np.arange(1.0, 4.5, 0.125):
            x, its = ctx.bfbt_inner_solve(b, form=form, rtol=rtol, max_it=480)
            if its < 24:
                continue
            y, before = ctx.bfbt_inner_solve(b, form=form, rtol=rtol, max_it=its - 12)
            res = [np.linalg.norm(b - ctx.bfbt_operator_apply(v)) / np.linalg.norm(b) / rtol for v in (x, y)]
            assert before == its - 12 and res[0] < 1.05
            if abs(res[1] - 1.0) > 0.05:
                seen += 1
                assert res[1] > 1.0, (rtol, its, res)
    assert seen > 0
