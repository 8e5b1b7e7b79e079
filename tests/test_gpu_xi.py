"""Local coordinates of the mapping, bit for bit: xi = RN((2 (x - x0) - h) / h).  The kernel multiplies by RN(1/h) and
corrects the quotient once; here the same with a division."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# element counts whose widths have significands from just above 1 to just below 2, where a rounded reciprocal is
# worst; boxes from 0, whose node coordinates have one rounding more than the quotient i / nel whatever the compiler
# does with the product and the sum
@pytest.mark.parametrize("nel,mx", [((65, 33, 17), (1.0, 1.0, 1.0)), ((64, 63, 31), (1.0, 7.0 / 3.0, 1e-3)),
                                    ((1025, 1023), (1.0, 1.0)), ((4099, 3), (1e7 / 3.0, 0.1))])
def test_local_coordinates_are_the_rounded_quotients(uw, nel, mx):
    U = uw
    dim, N = len(nel), 400_000
    rng = np.random.default_rng(9)
    pts = [rng.uniform(0.0, m, N) for m in mx]
    for d in range(dim):   # some on nodes and element centres, and a rounding beside them
        k = rng.integers(0, 2 * nel[d] + 1, N // 8)
        pts[d][:N // 8] = np.minimum(np.abs(k / (2 * nel[d]) * mx[d] * (1.0 + rng.choice([0.0, 2.0 ** -52, -(2.0 ** -53)], N // 8))),
                                     mx[d])
    with U.Context(0) as ctx:
        ctx.mesh_q1(dim, nel, (0.0,) * dim, mx)
        ctx.particles_upload(*(pts + [None] * (3 - dim)))
        perm, offsets, xi = ctx.bin_and_map()
    e = np.repeat(np.arange(len(offsets) - 1), np.diff(offsets))
    for d in range(dim):
        nodes = np.arange(nel[d] + 1) / nel[d] * mx[d]
        nodes[-1] = mx[d]
        i = e % nel[d]
        e = e // nel[d]
        x0 = nodes[i]
        h = nodes[i + 1] - x0
        assert np.array_equal(xi[:, d], (2.0 * (pts[d][perm] - x0) - h) / h)
