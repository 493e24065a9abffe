"""Convolution kernel at the edges of its tiles, units and row windows.

Inputs, weights and biases are whole numbers of which three in four are zero, so that every sum is a whole
number of at most 256 (checked on the oracle's result): exact in FP32 in any order and in the bf16 of the
stored output, and the kernel has to give the oracle's values exactly."""
import numpy as np
import pytest

from oracle import unet as ou

pytestmark = pytest.mark.gpu

# one voxel; a plane of less than a tile; two and three tiles with ragged ends; many units to a CTA; z rows longer
# than a unit's rows (the dy rows then come as copies of their own); a single plane of many tiles
SHAPES = [(1, 1, 1), (7, 3, 9), (5, 9, 25), (3, 11, 34), (90, 60, 30), (2, 3, 500), (1, 40, 66)]
RELU, RAW = 0, 3        # relu(conv + bias), and the plain data gradient


def _sparse(rng, shape):
    return rng.integers(-1, 2, size=shape) * (rng.random(shape) < 0.375)


@pytest.mark.parametrize("taps", [27, 9])
@pytest.mark.parametrize("cin,cout", [(16, 16), (16, 64), (32, 32), (32, 16), (64, 32), (32, 64)])
def test_convolution_is_exact_on_whole_numbers(gpu, cin, cout, taps):
    import torch
    from bug_defense_b200 import denoise
    rng = np.random.default_rng(100 * cin + cout + taps)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a, np.float32)).cuda()
    for shape in SHAPES:
        x = _sparse(rng, (cin,) + shape).astype(np.float64)
        w = _sparse(rng, (taps, cout, cin)).astype(np.float64)
        b = rng.integers(-3, 4, size=cout).astype(np.float64)
        img = denoise.pack_weights(dev(w), taps, cin, cout)
        xp = denoise.to_planes(dev(x))
        ref = ou.conv(x, w, taps)
        assert np.abs(ref).max() + 3 <= 256
        for mode in (RELU, RAW):
            out = denoise.zeros_planes(cout, shape)
            denoise.conv3d(mode, xp, img, shape, cin, cout, taps=taps, bias=dev(b), out=out)
            want = np.maximum(ref + b[:, None, None, None], 0.0) if mode == RELU else ref
            np.testing.assert_array_equal(denoise.from_planes(out, shape).double().cpu().numpy(), want,
                                          err_msg=f"{shape} mode {mode}")
