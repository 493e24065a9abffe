"""Weight-gradient kernel at the edges of its row chunks, stages, splits and channel slices.

Gradients and activations are whole numbers in [-3, 3], so every product and every partial sum is a
whole number far below 2**24 (at most 9 x 16,000 voxels): FP32 accumulation is exact in any order and
the kernel has to give the oracle's weights exactly, on top of what the buffer held before."""
import numpy as np
import pytest

from oracle import unet as ou

pytestmark = pytest.mark.gpu

# one voxel; rows shorter than a core matrix; interiors of one chunk to within a row; several CTAs with a
# ragged last range (2048 rows each); long z rows
SHAPES = [(1, 1, 1), (3, 2, 5), (1, 7, 126), (9, 5, 14), (11, 13, 17), (20, 25, 32)]
COMBOS = [(16, 16), (16, 32), (32, 16), (32, 32), (32, 64), (64, 16), (64, 32), (64, 64), (16, 64)]


@pytest.mark.parametrize("taps", [27, 9])
@pytest.mark.parametrize("cout,cin", COMBOS)
def test_weight_gradient_is_exact_on_whole_numbers(gpu, cout, cin, taps):
    import torch
    from bug_defense_b200 import denoise
    rng = np.random.default_rng(1000 * cout + 10 * cin + taps)
    for shape in SHAPES:
        g = rng.integers(-3, 4, size=(cout,) + shape).astype(np.float64)
        x = rng.integers(-3, 4, size=(cin,) + shape).astype(np.float64)
        was = rng.integers(-3, 4, size=(taps, cout, cin)).astype(np.float64)
        dw = torch.from_numpy(was).to("cuda", torch.float32)
        planes = [denoise.to_planes(torch.from_numpy(a).to("cuda", torch.float32)) for a in (g, x)]
        denoise.conv3d_wgrad(planes[0], planes[1], dw, shape, cin, cout, taps=taps)
        np.testing.assert_array_equal(dw.double().cpu().numpy(), was + ou.conv_wgrad(g, x, taps), err_msg=str(shape))


@pytest.mark.parametrize("cout,cin,taps", [(16, 16, 27), (32, 64, 27), (64, 32, 27), (16, 16, 9)])
def test_long_rows_and_unaligned_weights(gpu, cout, cin, taps):
    """z rows longer than a chunk (the dy rows then come as copies of their own), chunks of each length, and
    a weight buffer that is not 16-byte aligned (single additions instead of four at a time)."""
    import torch
    from bug_defense_b200 import denoise
    rng = np.random.default_rng(7 * cout + cin + taps)
    for shape in [(1, 2, 500), (2, 3, 300), (2, 5, 190), (3, 4, 96), (4, 4, 62)]:
        g = rng.integers(-3, 4, size=(cout,) + shape).astype(np.float64)
        x = rng.integers(-3, 4, size=(cin,) + shape).astype(np.float64)
        buf = torch.zeros(taps * cout * cin + 1, device="cuda")
        dw = buf[1:].view(taps, cout, cin)
        planes = [denoise.to_planes(torch.from_numpy(a).to("cuda", torch.float32)) for a in (g, x)]
        denoise.conv3d_wgrad(planes[0], planes[1], dw, shape, cin, cout, taps=taps)
        np.testing.assert_array_equal(dw.double().cpu().numpy(), ou.conv_wgrad(g, x, taps), err_msg=str(shape))
        assert float(buf[0]) == 0.0
