"""k_dvc's FP32 contests and its limit of points per element: ties and near ties between points, and elements of
64, 65 and mixed counts, bit for bit against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _layout(kind, dim, nel, rng):
    """points as element-local coordinates in (0, 1)^dim per element"""
    E = int(np.prod(nel))
    if kind == "lattice":   # symmetric: many cells are equidistant from several points
        g = (np.arange(4) + 0.5) / 4
        base = np.stack(np.meshgrid(*[g] * dim, indexing="ij"), -1).reshape(-1, dim)
        return [base for _ in range(E)]
    if kind == "near":      # pairs of points a few ulps to 1e-5 apart: contests near zero
        out = []
        for e in range(E):
            a = rng.uniform(0.05, 0.95, (10, dim))
            out.append(np.concatenate([a, a + rng.choice([1e-16, 1e-12, 1e-8, 1e-5], (10, dim)) * rng.choice([-1, 1], (10, dim))]))
        return out
    return [rng.uniform(0, 1, (n, dim)) for n in rng.choice([1, 2, 31, 32, 33, 64, 65, 100], E)]


@pytest.mark.parametrize("kind", ["lattice", "near", "counts"])
@pytest.mark.parametrize("dim,nel,res", [(2, (5, 4), (10, 10)), (2, (3, 4), (32, 32)), (3, (3, 4, 3), (10, 10, 10)),
                                         (3, (3, 3, 2), (1, 7, 32))])
def test_contests_match_oracle(oracle, uw, kind, dim, nel, res):
    O, U = oracle, uw
    rng = np.random.default_rng(3)
    pts = []
    for e, loc in enumerate(_layout(kind, dim, nel, rng)):
        idx = [e % nel[0], e // nel[0] % nel[1]] + ([e // (nel[0] * nel[1])] if dim == 3 else [])
        pts.append((np.array(idx) + loc) / np.array(nel))
    pts = np.concatenate(pts)[rng.permutation(sum(len(p) for p in pts))]
    with U.Context(0) as ctx:
        ctx.mesh_q1(dim, nel)
        ctx.bc_set(U.free_slip_mask(dim, nel))
        ctx.materials_set([U.make_material([(U.LAW_MATERIAL_VISCOSITY, [1.0])], density=1.0)])
        ctx.fields_set(None, 1.0, dim - 1)
        ctx.particles_upload(pts[:, 0], pts[:, 1], pts[:, 2] if dim == 3 else None)
        perm, offsets, xi = ctx.bin_and_map()
        ctx.weights_set(U.WEIGHTS_DVC, res)
        ctx.assemble()
        gxi, gw = ctx.integration_points()
    cxi, cw = O.dvc_weights(O.make_mesh(dim, nel), res, offsets, xi)
    assert np.array_equal(gxi, cxi) and np.array_equal(gw, cw)
