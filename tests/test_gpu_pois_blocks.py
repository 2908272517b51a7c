"""The tensor-core true-Poisson likelihood over the 64-pixel blocks with counts:
pattern tiles with blocks without counts, one without any count, edges of the 128-
and 256-row tiles, more tiles than the chip runs at once, CTA pairs and single CTAs.

Against the FP64 iteration on the same slices.  A pattern's log-likelihood is a sum
of 2 x ceil(P / 16) products accumulated in FP32, each step within 2^-23 of the
running sum, which K max|log s| bounds; a responsibility in [0, 1] moves by at most
twice that."""
import numpy as np
import pytest
import torch

import emc_gb300 as E
from emc_gb300 import synthetic as S
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pair", [1, 0], ids=["pairs", "single"])
@pytest.mark.parametrize("N,R,known", [(5, 3, False), (129, 128, True), (300, 257, False),
                                       (128, 384, False), (3900, 1380, False)])
def test_against_fp64(ctx, cuda, N, R, known, pair):
    side = 20
    prob = S.make_problem(S.tiny(side=side, n_images=N, rot_n=3, photons=200, n_atoms=60,
                                 radius=4.0))
    quats, wts = prob.quats[:R], prob.weights[:R]
    assert quats.shape[0] == R
    r = np.hypot(*np.meshgrid(np.arange(side) - side / 2 + 0.5,
                              np.arange(side) - side / 2 + 0.5)).reshape(-1)
    im = prob.images.copy()
    im[:, r > 8] = 0.0  # the outer pixels: no counts in any pattern
    if N >= 300:
        im[128:256] = 0.0  # and a tile of patterns with none at all
    f = lambda a, dt=torch.float32: torch.as_tensor(np.ascontiguousarray(a), dtype=dt, device=cuda)
    plan = E.Plan(ctx, side, N, R, precision=E.PREC_MIXED, diff=E.DIFF_TRUE_POISSON,
                  known_intensity=known)
    plan.set_option(E.Plan.OPT_ESTEP_PAIR, pair)
    plan.bind(f(im), f(prob.mask, torch.int32), f(prob.x), f(prob.y), f(prob.z), f(quats), f(wts))
    m = f(prob.init_model)
    st = plan.iterate(m, torch.empty_like(m), 0.5)
    got_P = ctx.copy_real_to_host(plan.results()[0], R * N).reshape(R, N).astype(np.float64)
    got_phi = ctx.copy_real_to_host(plan.results()[1], R * N).reshape(R, N).astype(np.float64)
    plan.close()
    want = O.fused_iteration_fp64(prob.init_model, im, prob.mask, prob.x, prob.y, prob.z, quats,
                                  wts, 0.5, side, diff=3, known_intensity=known)
    K = O.compacted_counts(im, prob.mask, side).sum(1).astype(np.float64)
    steps = 2 * -(-int((prob.mask == 1).sum()) // 16)
    tol = 1e-5 + steps * 2.0 ** -23 * K * 14.0  # |log s| <= -log(1e-6)
    assert (np.abs(got_P - want["respons"]) <= 2 * tol[None, :]).all()
    np.testing.assert_allclose(got_phi, want["phi"], rtol=1e-5)
    assert abs(st.total_loglik - want["total_loglik"]) <= tol.sum()
