"""Device memory that uploads of nodal vectors take besides the vector: one staging piece, whatever the mesh."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MB = 1 << 20


def _used(U):
    free, total = ctypes.c_size_t(), ctypes.c_size_t()
    lib = U.load()
    assert lib.cudaMemGetInfo(ctypes.byref(free), ctypes.byref(total)) == 0
    return total.value - free.value


def test_staging_is_one_piece(uw):
    U = uw
    nel = (199, 199, 199)
    u = np.random.default_rng(0).standard_normal((200 ** 3, 3))   # 192 MB
    p = np.zeros(199 ** 3)
    with U.Context(0) as ctx:
        ctx.mesh_q1(3, (2, 2, 2))
        ctx.solution_set(np.zeros((27, 3)), np.zeros(8))
        before = _used(U)
        ctx.mesh_q1(3, nel)
        ctx.solution_set(u, p)
        grown = _used(U) - before
    # the solution itself, a piece of 64 MB, and what the allocator rounds three blocks up by
    assert grown <= u.nbytes + p.nbytes + 64 * MB + 3 * 2 * MB, grown / MB


def test_vector_of_two_pieces_round_trips(uw):
    """the operator's identity rows return the fixed entries of x unchanged, node by node; 4.3M nodes are 69 MB"""
    U = uw
    nel = (2100, 2050)
    nodes, E = 2101 * 2051, 2100 * 2050
    x = np.random.default_rng(1).standard_normal(nodes * 2)
    e = np.arange(E)
    with U.Context(0) as ctx:
        ctx.mesh_q1(2, nel)
        ctx.bc_set(np.ones(nodes * 2, np.uint8))
        ctx.materials_set([U.make_material([(U.LAW_MATERIAL_VISCOSITY, [1.0])], density=1.0)])
        ctx.fields_set(None, 1.0, 1)
        ctx.particles_upload((e % 2100 + 0.5) / 2100, (e // 2100 + 0.5) / 2050, None)
        ctx.bin_and_map(want=False)
        ctx.assemble()
        assert np.array_equal(ctx.operator_apply(x, U.PREC_FP64), x)
        assert np.array_equal(ctx.operator_apply(x, U.PREC_MIXED), x.astype(np.float32).astype(np.float64))
