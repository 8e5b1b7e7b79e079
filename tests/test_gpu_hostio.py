"""Layout changes at the host boundary (csrc/hostio.cu): ranges and sizes around the 32-element tiles and the
64 MB staging pieces give the same bytes as fetching elements in other ranges."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nel,ranges", [((5, 3), [(0, 1), (1, 14), (7, 8), (15, 0)]),
                                        ((33, 9), [(0, 297), (31, 2), (32, 33), (296, 1)]),
                                        ((5, 3, 4), [(0, 60), (59, 1), (3, 31)]),
                                        ((28, 27, 20), [(14500, 200), (14563, 1), (15119, 1)])])
def test_element_matrix_ranges(uw, nel, ranges):
    from earthbyte_underworld_gb300 import workloads as W
    U = uw
    w = W.rt2d(nel=nel, ppc=12) if len(nel) == 2 else W.spheres(nel=nel, nspheres=6, seed=3)
    with U.Context(0) as ctx:
        W.setup_context(ctx, w)
        ctx.bin_and_map(want=False)
        ctx.assemble()
        full = ctx.element_matrices()   # the last mesh: 70 MB, two pieces
        assert np.array_equal(full[0], full[0].transpose(0, 2, 1)) and (full[3] > 0).all()
        for first, count in ranges:
            part = ctx.element_matrices(first, count)
            for a, b in zip(part, full):
                assert np.array_equal(a, b[first:first + count])


@pytest.mark.parametrize("nel", [(3, 2), (17, 30), (2, 3, 2), (120, 117, 110)])
def test_nodal_vectors_round_trip(uw, nel):
    """the operator's identity rows return the fixed entries of x unchanged, node by node (the last mesh's
    vector is 111 MB: two pieces)"""
    from earthbyte_underworld_gb300 import uwgpu as U
    dim = len(nel)
    nodes = int(np.prod([n + 1 for n in nel]))
    rng = np.random.default_rng(1)
    x = rng.standard_normal(nodes * dim)
    E = int(np.prod(nel))
    with U.Context(0) as ctx:
        ctx.mesh_q1(dim, nel)
        ctx.bc_set(np.ones(nodes * dim, np.uint8))
        ctx.materials_set([U.make_material([(U.LAW_MATERIAL_VISCOSITY, [1.0])], density=1.0)])
        ctx.fields_set(None, 1.0, dim - 1)
        e = np.arange(E)
        c = []
        for n in nel:
            c.append((e % n + 0.5) / n)
            e = e // n
        ctx.particles_upload(*(c + [None] * (3 - dim)))
        perm, offsets, xi = ctx.bin_and_map()
        assert np.array_equal(perm, np.arange(E)) and xi.shape == (E, 3) and np.abs(xi).max() < 1e-9
        ctx.assemble()
        assert np.array_equal(ctx.operator_apply(x, U.PREC_FP64), x)
        assert np.array_equal(ctx.operator_apply(x, U.PREC_MIXED), x.astype(np.float32).astype(np.float64))
        if E < 1000:
            ctx.solution_set(x, np.zeros(E))
