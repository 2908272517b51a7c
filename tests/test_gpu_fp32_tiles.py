"""The FP32 likelihood and M-step at the edges of their 128 x 128 tiles and 16-step
stages: one row, a full tile, one more; with stages in which every rotation covers
every pixel, stages in which some do not, and slices of zeros.  Likelihood, scaling
and inserted sums against FP64 restatements from the same slices (FP32 sums of up to
400 terms in order: 400 x 6e-8 = 2.4e-5 of the terms' magnitude; the model 1e-4
relative L2, the FP32 path's tolerance)."""
import numpy as np
import pytest
import torch

import emc_gb300 as E
from emc_gb300 import synthetic as S
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("known", [False, True])
@pytest.mark.parametrize("R,N", [(1, 1), (128, 129), (130, 128), (300, 37)])
@pytest.mark.parametrize("diff", [E.DIFF_POISSON, E.DIFF_TRUE_POISSON], ids=["poisson", "true"])
def test_fp32_against_fp64(ctx, cuda, R, N, diff, known):
    side = 20
    prob = S.make_problem(S.tiny(side=side, n_images=N, rot_n=2, photons=900, n_atoms=60,
                                 radius=4.0))
    quats, wts = prob.quats[:R], prob.weights[:R]
    assert quats.shape[0] == R
    f = lambda a, dt=torch.float32: torch.as_tensor(np.ascontiguousarray(a), dtype=dt, device=cuda)
    model = prob.init_model.reshape(side, side, side).copy()
    model[:, :, :4] = 0.0  # some rotations see zeros at some pixels
    plan = E.Plan(ctx, side, N, R, precision=E.PREC_FP32, diff=diff, known_intensity=known,
                  insert_mode=E.INSERT_DETERMINISTIC)
    plan.bind(f(prob.images), f(prob.mask, torch.int32), f(prob.x), f(prob.y), f(prob.z), f(quats),
              f(wts))
    m, w = f(model.reshape(-1)), torch.empty(side ** 3, device=cuda)
    st = plan.iterate(m, w, 0.5)
    P = ctx.copy_real_to_host(plan.results()[0], R * N).reshape(R, N).astype(np.float64)
    phi = ctx.copy_real_to_host(plan.results()[1], R * N).reshape(R, N).astype(np.float64)
    plan.close()
    on = prob.mask == 1
    x, y, z = prob.x[on], prob.y[on], prob.z[on]
    K = O.compacted_counts(prob.images, prob.mask, side).astype(np.float64)
    ref = O.fused_iteration_fp64(model.reshape(-1).astype(np.float32), prob.images, prob.mask,
                                 prob.x, prob.y, prob.z, quats, wts, 0.5, side,
                                 1 if diff == E.DIFF_POISSON else 0, known_intensity=known)
    np.testing.assert_allclose(phi, ref["phi"], rtol=5e-5)
    # the terms: squared differences (each sum a few times the result), or K |log s|
    size = 4 * np.abs(ref["lse"]).sum() if diff == E.DIFF_POISSON else 8 * K.sum()
    assert abs(st.total_loglik - ref["total_loglik"]) <= 2.4e-5 * size
    assert np.abs(P.sum(0) - 1.0).max() < 1e-5
    want = O.mstep_fp64(P, phi, K, x, y, z, quats, side, 0)
    got_m, got_w = m.cpu().numpy().astype(np.float64), w.cpu().numpy().astype(np.float64)
    assert np.linalg.norm(got_w - want["weight"]) <= 1e-4 * np.linalg.norm(want["weight"])
    ref_m = want["model"] * want["mean_before"]
    assert np.linalg.norm(got_m * st.model_mean_before - ref_m) <= 1e-4 * np.linalg.norm(ref_m)
