"""Convolutions of the learned preconditioner at the edges of their tiles and plans: grids that are no
multiple of the 8 x 16 voxel tile, one or few tiles (output channels shared between blocks), and channel
counts that reach each form of the kernels (weights resident or streamed, nine or three taps per stage,
27, 9 or 3 taps per gradient block, input and output channels in chunks)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from test_learned import _gpu_pass, _quantized_params, _rel  # noqa: E402


@pytest.mark.gpu
@pytest.mark.parametrize("nel,levels,base", [
    ((19, 32, 8), 1, 8),     # 20 x 33 x 9 voxels: three tiles in y, the last one row; 27 taps per gradient block
    ((2, 1, 20), 2, 16),     # extents below one tile
    ((8, 16, 6), 2, 24),     # 24 / 48 / 72 channels: padded chunks, nine and three taps
    ((31, 30, 33), 3, 16),   # more tiles than SMs: resident weights, persistent blocks
    ((6, 16, 5), 1, 128),    # 128 channels: output channels in two chunks, both gradient parts streamed
    ((5, 8, 3), 2, 72),      # 216 input channels in two chunks, 144 output channels in three
])
def test_convolution_tiles(uw, nel, levels, base):
    """Data as in the quantized part of test_learned: the FP32 sums of the first layers are exact.  Where
    later sums round, an activation at a BF16 tie may flip: a sum of n terms is off by about sqrt(n) 2^-24
    of its size, so that sqrt(n) 2^-16 of the activations flip by 2^-9, which for n = 27 x 216 is 7e-5 of a
    layer's norm; six layers stay below 5e-4.  The gradients see the flips of both passes and ReLU's edge:
    2e-3.  A wrong row, tap or channel is off by 1e-2 and more."""
    from oracle import unet_ref as R
    nodes = tuple(n + 1 for n in nel)
    nn = int(np.prod(nodes))
    rng = np.random.default_rng(5)
    params = _quantized_params(R, levels, base, rng)
    inp = (rng.integers(-3, 4, (7, nn)) / 2.0).astype(np.float32)
    gout = (rng.integers(-3, 4, (3, nn)) / 4.0).astype(np.float32)
    _, out, gp, gi = _gpu_pass(uw, nel, levels, base, params, inp, gout)
    rout, rgp, rgi = R.value_and_grads(params, inp, gout, nodes, levels, base, emulate_bf16=True)
    assert _rel(out, rout) < 5e-4
    assert _rel(gi, rgi) < 2e-3
    off = 0
    for cin, cout in R.layer_shapes(levels, base)[1]:
        n = 27 * cin * cout + cout
        assert _rel(gp[off:off + n], rgp[off:off + n]) < 2e-3, (cin, cout)
        off += n
