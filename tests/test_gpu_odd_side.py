"""A detector with an odd number of pixels: the pattern pass keeps FP64 sums behind a
row of that many floats in shared memory.  The sums K_i are whole numbers, so with one
rotation, where phi_i = K_i / S, the ratios of phi are the ratios of the counts."""
import numpy as np
import pytest
import torch

import emc_gb300 as E

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [E.PREC_FP32, E.PREC_MIXED], ids=["fp32", "mixed"])
@pytest.mark.parametrize("side", [9, 21])
def test_pattern_sums(ctx, cuda, side, prec):
    rng = np.random.default_rng(side)
    im = rng.poisson(2.0, size=(17, side * side)).astype(np.float32)
    f = lambda a, dt=torch.float32: torch.as_tensor(np.ascontiguousarray(a), dtype=dt, device=cuda)
    px = np.arange(side * side)
    plan = E.Plan(ctx, side, 17, 1, precision=prec, diff=E.DIFF_TRUE_POISSON)
    plan.bind(f(im), f(np.ones(side * side), torch.int32), f(px % side - side / 2 + 0.5),
              f(px // side - side / 2 + 0.5), f(np.zeros(side * side)), f([[1, 0, 0, 0]]), f([1.0]))
    m = f(np.ones(side ** 3))
    plan.iterate(m, torch.empty_like(m), 0.5)
    phi = ctx.copy_real_to_host(plan.results()[1], 17).astype(np.float64)
    plan.close()
    np.testing.assert_allclose(phi / phi[0], im.sum(1) / im[0].sum(), rtol=1e-6)
