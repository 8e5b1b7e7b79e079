"""Element search (csrc/locate.cuh): the fixed-point form against the reference rule, at cell edges and inside."""
import struct
from fractions import Fraction

import numpy as np
import pytest

AXES = [(0.0, 1.0, 1), (0.0, 1.0, 64), (0.0, 1.0, 7), (-3.7, 12.9, 45), (1.0e3, 1.0e3 + 2.0, 999), (0.0, 1e-3, 130),
        (-0.5, 2.5, 262144), (0.0, 1.0, 262145), (-1e6, 1e6, 333), (5.0, 5.0 + 1e-9, 12)]


def _points(mn, mx, nel, rng, count):
    sep = (mx - mn) / nel
    k = rng.integers(0, nel + 1, count)
    edge = mn + k * sep
    ulp = np.spacing(np.maximum(np.abs(edge), sep))
    off = rng.choice([0.0, 1.0, -1.0, 3.0, -3.0], count) * ulp
    off += rng.choice([0.0, 0.0, 1.0, -1.0], count) * sep * 2.0 ** -rng.integers(25, 36, count)
    off += rng.choice([0.0, 0.0, 1e-12, -1e-12, 9e-13, -1.1e-12], count)
    x = np.concatenate([edge + off, mn + (mx - mn) * rng.uniform(-0.01, 1.01, count)])
    return np.concatenate([x, [mn, mx, np.nan, np.inf, -np.inf, 1e300, -1e300, 0.0, -0.0]])


def _rule(mn, mx, nel, x):
    sep = (mx - mn) / nel
    if not np.isfinite(x):
        return None
    if -1e-12 <= x - mx <= 1e-12:
        return nel - 1
    if x < mn or x > mx:
        return None
    out = (x - mn) / sep
    i = int(out)
    if i > 0 and out - i <= 1e-12:
        i -= 1
    return min(i, nel - 1)


def _fixed_point(mn, mx, nel, x):
    """the FMA form of axis_index; False where it leaves the point to the rule"""
    inv = 1.0 / ((mx - mn) / nel)
    shift = mn * inv
    if not (nel <= 1 << 18 and abs(shift) <= 262144.0 and 1e-12 * inv < 0.25) or not np.isfinite(x):
        return False
    try:
        m = float(Fraction(x) * Fraction(inv) + Fraction(1572864.0 - shift))
    except OverflowError:
        return False
    hi, lo = struct.unpack(">iI", struct.pack(">d", m))
    i = hi - 0x41380000
    return i if 0 <= i < nel and 8 <= lo < 0xfffffff8 else False


@pytest.mark.parametrize("mn,mx,nel", AXES)
def test_fixed_point_search_agrees_with_the_rule(mn, mx, nel):
    taken = 0
    xs = _points(mn, mx, nel, np.random.default_rng(nel), 2000)
    for x in xs.tolist():
        i = _fixed_point(mn, mx, nel, x)
        if i is not False:
            taken += 1
            assert i == _rule(mn, mx, nel, x), x
    shift_ok = abs(mn / ((mx - mn) / nel)) <= 262144.0
    assert (taken > 1000) == (nel <= 1 << 18 and shift_ok and 1e-12 * nel / (mx - mn) < 0.25)


@pytest.mark.gpu
@pytest.mark.parametrize("mn,mx,nel", AXES)
def test_mapping_at_cell_edges_matches_the_rule(uw, mn, mx, nel):
    """every point of the mapping, and the outside count, against the rule on the host"""
    U = uw
    rng = np.random.default_rng(nel + 1)
    x = _points(mn, mx, nel, rng, 3000)
    ref = [_rule(mn, mx, nel, v) for v in x.tolist()]
    y = np.full(x.size, 0.25)
    with U.Context(0) as ctx:
        ctx.mesh_q1(2, (nel, 2), (mn, 0.0, 0.0), (mx, 1.0, 1.0))
        ctx.particles_upload(x, y)
        with pytest.raises(U.UwgpuError) as err:   # the points that are not finite lie outside
            ctx.bin_and_map(want=False)
        assert err.value.code == U.ERR_DOMAIN and str(sum(r is None for r in ref)) in str(err.value)
        keep = np.array([r is not None for r in ref])
        ctx.particles_upload(x[keep], y[keep])
        perm, offsets, xi = ctx.bin_and_map()
    cell = np.array([r for r in ref if r is not None])
    assert np.array_equal(perm, np.argsort(cell, kind="stable"))
    assert np.array_equal(offsets[:-1], np.searchsorted(np.sort(cell), np.arange(2 * nel)))


@pytest.mark.gpu
@pytest.mark.parametrize("ppc,nel", [(31, (3, 2)), (33, (3, 2)), (65, (5, 4, 3)), (400, (2, 2)), (3, (91, 91))])
def test_permutation_of_full_elements(uw, ppc, nel):
    """points per element around the warp's 32 and several times it; the last mesh has more elements than the
    one-block scan takes"""
    U = uw
    dim, E = len(nel), int(np.prod(nel))
    rng = np.random.default_rng(ppc)
    c = [rng.uniform(0, 1, E * ppc) for _ in nel]
    cell, mul = np.zeros(E * ppc, np.int64), 1
    for x, n in zip(c, nel):
        cell += mul * np.minimum((x * n).astype(np.int64), n - 1)
        mul *= n
    with U.Context(0) as ctx:
        ctx.mesh_q1(dim, nel)
        ctx.particles_upload(*(c + [None] * (3 - dim)))
        perm, offsets, xi = ctx.bin_and_map()
    assert np.array_equal(perm, np.argsort(cell, kind="stable"))
    assert np.array_equal(np.diff(offsets), np.bincount(cell, minlength=E))
    for d, (x, n) in enumerate(zip(c, nel)):
        i = cell[perm] // int(np.prod(nel[:d])) % n
        assert np.abs(xi[:, d] - ((x[perm] * n - i) * 2 - 1)).max() < 1e-12
