"""The blur at sides that its groups of four outputs and 32 columns divide unevenly,
with taps over part of the line and over the whole circle, masked voxels included,
against the FFT in FP64 (FP32 sums of at most 65 taps that add to one: 65 x 6e-8 of the
largest value; 1e-5)."""
import numpy as np
import pytest
import torch

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sigma", [0.4, 1.0, 6.0])
@pytest.mark.parametrize("side", [2, 3, 5, 31, 33, 64, 65])
def test_blur(ctx, cuda, side, sigma):
    rng = np.random.default_rng(side)
    m = rng.uniform(0.0, 2.0, size=side ** 3).astype(np.float32)
    m[rng.random(side ** 3) < 0.05] = -1.0
    t = torch.as_tensor(m, device=cuda)
    ctx.blur_model(t, side, sigma)
    got = t.cpu().numpy()
    want = O.blur_fft_fp64(m, side, sigma)
    assert np.array_equal(got == -1.0, m < 0)
    assert np.abs(got - want)[m >= 0].max() < 1e-5
