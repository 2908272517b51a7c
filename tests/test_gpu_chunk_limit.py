"""Chunks of rotations of the drop-in scaling and likelihood: all that the entry
points accept (524,280) run, also where one launch's grid does not hold them; longer
ones are refused."""
import numpy as np
import pytest
import torch

import emc_gb300 as E
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("chunk", [262140, 262141, 524280])
def test_long_chunks(ctx, cuda, chunk):
    rng = np.random.default_rng(chunk)
    n2, N, start = 6, 3, 5
    images = rng.poisson(3.0, (N, n2)).astype(np.float32)
    slices = rng.gamma(2.0, 2.0, (chunk, n2)).astype(np.float32)
    mask = np.ones(n2, np.int32)
    t = lambda a, dt=torch.float32: torch.as_tensor(a, dtype=dt, device=cuda)
    got, want = torch.full((start + chunk, N), 7.0, device=cuda), np.full((start + chunk, N), 7.0, np.float32)
    ctx.update_scaling_full(t(images), t(slices), t(mask, torch.int32), got, n2, N, start, chunk)
    O.update_scaling_full(images, slices, mask, want, start)
    ctx.sync()
    np.testing.assert_array_equal(got.cpu().numpy(), want)
    w = np.full(start + chunk, 0.5, np.float32)
    res, want_r = torch.full_like(got, 7.0), np.full_like(want, 7.0)
    ctx.calculate_responsabilities(t(slices), t(images), t(mask, torch.int32), 0.3, got, res, t(w), n2,
                                   N, start, chunk, E.DIFF_POISSON)
    with np.errstate(all="ignore"):
        O.calculate_responsabilities(slices, images, mask, np.float32(0.3), want, want_r, w, start, 1)
    ctx.sync()
    np.testing.assert_allclose(res.cpu().numpy(), want_r, rtol=2.4e-7, equal_nan=True)


def test_longer_chunks_are_refused(ctx, cuda):
    t = torch.zeros(8, device=cuda)
    i = torch.zeros(8, device=cuda, dtype=torch.int32)
    with pytest.raises(E.EmcError):
        ctx.update_scaling_full(t, t, i, t, 1, 1, 0, 524281)
    with pytest.raises(E.EmcError):
        ctx.calculate_responsabilities(t, t, i, 0.3, t, t, t, 1, 1, 0, 524281, E.DIFF_POISSON)
