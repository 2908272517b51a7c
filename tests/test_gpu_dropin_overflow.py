"""The drop-in likelihood where a pair's sum of squares leaves the FP32 range: -inf,
as the reference's FP64 terms give, not NaN."""
import numpy as np
import pytest
import torch

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count,phi,s", [(1e9, 1e-9, 1e-10), (3e7, 3e-8, 1e-10), (0.0, 1.0, 1e18),
                                         (1e9, 1e-9, 1e18), (1e3, 1e-9, 1e-3)])
def test_sum_beyond_fp32(ctx, cuda, count, phi, s):
    side, N, R = 96, 5, 3
    n2 = side * side
    images = np.full((N, n2), count, np.float32)
    images[1] = 1.0
    slices = np.full((R, n2), s, np.float32)
    slices[1] = 0.7
    mask = np.ones(n2, np.int32)
    scal, w = np.full((R, N), phi, np.float32), np.full(R, 0.25, np.float32)
    want = np.zeros((R, N), np.float32)
    with np.errstate(all="ignore"):
        O.calculate_responsabilities(slices, images, mask, np.float32(0.3), scal, want, w, 0, 1)
    t = lambda a, dt=torch.float32: torch.as_tensor(a, dtype=dt, device=cuda)
    got = torch.zeros((R, N), device=cuda)
    ctx.calculate_responsabilities(t(slices), t(images), t(mask, torch.int32), 0.3, t(scal), got, t(w),
                                   n2, N, 0, R, 1)
    ctx.sync()
    np.testing.assert_allclose(got.cpu().numpy(), want, rtol=2.4e-7, equal_nan=True)
