"""The pruned M-step on CTA pairs (true Poisson: a pair's rotation tiles have one list
of pattern blocks) against single CTAs: an odd number of rotation tiles, pixel tiles
without counts, lists of more than 32 entries.  Both multiply the same blocks in the
same order, so only the FP32 rounding inside a product may differ: 1e-5 of the model
(whose sums are fixed-point); the reference likelihood stays on single CTAs and must
not change at all."""
import numpy as np
import pytest
import torch

import emc_gb300 as E
from emc_gb300 import synthetic as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("diff", [E.DIFF_TRUE_POISSON, E.DIFF_POISSON], ids=["true", "poisson"])
def test_pairs_and_singles(ctx, cuda, diff):
    # 32 pattern tiles, 201 rotation tiles (the last partial)
    cfg = S.Config("prune64", 64, 400, 1.5, 12, 4000, 3000, (0.5, 1.5), 4, 8, 1, seed=3)
    prob = S.make_problem(cfg, device="cuda")
    N, R = prob.images.shape[0], prob.quats.shape[0]
    f = lambda a, dt=torch.float32: torch.as_tensor(np.ascontiguousarray(a), dtype=dt, device=cuda)
    im = prob.images.copy()
    r = np.hypot(prob.x, prob.y)
    im[:, r > np.quantile(r, 0.8)] = 0.0  # the outer pixel tiles: none
    out = {}
    for pair in (1, 0):
        plan = E.Plan(ctx, 64, N, R, diff=diff, precision=E.PREC_MIXED,
                      insert_mode=E.INSERT_DETERMINISTIC)
        keep = (f(im), f(prob.mask, torch.int32), f(prob.x), f(prob.y), f(prob.z),
                f(prob.quats[:R]), f(prob.weights[:R]))
        plan.bind(*keep)
        plan.set_pruning(True, min_mass=0.999, dilate=1.0)
        m = f(prob.true_model)
        ctx.normalize_model(64, m)
        sigma = 0.4 if diff == E.DIFF_TRUE_POISSON else 0.02
        w = torch.empty_like(m)
        plan.iterate(m, w, sigma)  # the full scan that builds the lists, the same in both
        plan.set_option(E.Plan.OPT_MSTEP_PAIR, pair)
        plan.iterate(m, w, sigma)
        out[pair] = (m.cpu().numpy().astype(np.float64), w.cpu().numpy().astype(np.float64),
                     plan.prune_info()["pruned"])
        plan.close()
    assert out[1][2] == out[0][2]
    if diff == E.DIFF_TRUE_POISSON:
        assert out[1][2] == 1
    tol = 1e-5 if diff == E.DIFF_TRUE_POISSON or not out[1][2] else 0.0  # full scans use pairs
    for k in range(2):
        assert np.linalg.norm(out[1][k] - out[0][k]) <= tol * np.linalg.norm(out[0][k]) + 1e-300
