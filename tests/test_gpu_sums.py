"""The plan's sums over rotation tiles, patterns and voxels at the edges of the
blocks that share them: fewer tiles than warps, one more than a whole share, one
pattern, a block of 32 and one more; models of less than one block and of many.
The normaliser against FP64 on the plan's own log-likelihoods (recovered from the
responsibilities: they sum to one per pattern; FP32 exponentials, 1e-5), the mean
against numpy's FP64 sum (one FP32 rounding, 1e-6)."""
import numpy as np
import pytest
import torch

import emc_gb300 as E
from emc_gb300 import synthetic as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("R", [1, 100, 1025, 1200])  # 1, 1, 9 and 10 tiles of 128
@pytest.mark.parametrize("N", [1, 33, 64])
def test_responsibilities_sum_to_one(ctx, cuda, R, N):
    prob = S.make_problem(S.tiny(side=16, n_images=N, rot_n=3, photons=300, n_atoms=40, radius=3.0))
    quats, wts = prob.quats[:R], prob.weights[:R]
    assert quats.shape[0] == R
    f = lambda a, dt=torch.float32: torch.as_tensor(np.ascontiguousarray(a), dtype=dt, device=cuda)
    plan = E.Plan(ctx, 16, N, R, precision=E.PREC_MIXED)
    plan.bind(f(prob.images), f(prob.mask, torch.int32), f(prob.x), f(prob.y), f(prob.z), f(quats),
              f(wts))
    m = f(prob.init_model)
    st = plan.iterate(m, torch.empty_like(m), 0.6)
    P = ctx.copy_real_to_host(plan.results()[0], R * N).reshape(R, N).astype(np.float64)
    plan.close()
    assert np.abs(P.sum(0) - 1.0).max() < 1e-5
    assert np.isfinite(st.total_loglik)
    got = m.cpu().numpy().astype(np.float64)
    assert abs(got[got > 0].mean() - 1.0) < 1e-6


@pytest.mark.parametrize("side", [2, 9, 64, 150])
def test_positive_mean(ctx, cuda, side):
    x = np.random.default_rng(side).normal(size=side ** 3).astype(np.float32)
    t = torch.as_tensor(x, device=cuda)
    mean = ctx.normalize_model(side, t)
    want = x[x > 0].astype(np.float64).mean()
    assert abs(mean - want) <= 1e-6 * want
    np.testing.assert_allclose(t.cpu().numpy(), x / want, rtol=1e-6)
