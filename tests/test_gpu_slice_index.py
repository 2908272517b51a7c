"""The expand's index arithmetic: coordinates on voxel boundaries (exact halves, both
signs), at the rims the reference leaves out, outside and far outside the volume, and
the block sizes of short and long rows; unknown and zero voxels.  The scaling of every
pair against the FP64 iteration on slices that the oracle takes with roundf and floorf:
a wrong voxel changes it by parts in ten (voxels differ by that much), FP32 sums by
5e-5, the tensor path's FP16 slices by 2^-12 each (1e-3 allowed)."""
import numpy as np
import pytest
import torch

import emc_gb300 as E
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def rotations():
    h = np.sqrt(0.5)
    exact = [(1, 0, 0, 0), (0, 1, 0, 0), (0, 0, 1, 0), (0, 0, 0, 1), (0.5, 0.5, 0.5, 0.5),
             (0.5, -0.5, 0.5, 0.5), (0.5, 0.5, -0.5, 0.5), (h, h, 0, 0), (h, 0, 0, h)]
    q = np.random.default_rng(1).normal(size=(124, 4))
    q /= np.linalg.norm(q, axis=1, keepdims=True)
    return np.concatenate([np.array(exact), q]).astype(np.float32)


@pytest.mark.parametrize("prec", [E.PREC_FP32, E.PREC_MIXED], ids=["fp32", "mixed"])
@pytest.mark.parametrize("interp", [E.INTERP_NEAREST, E.INTERP_TRILINEAR], ids=["near", "tri"])
@pytest.mark.parametrize("diff", [E.DIFF_POISSON, E.DIFF_TRUE_POISSON], ids=["poisson", "true"])
@pytest.mark.parametrize("side", [11, 12, 41])
def test_scaling(ctx, cuda, side, diff, interp, prec):
    rng = np.random.default_rng(side)
    n2, N = side * side, 30
    xyz = np.round(rng.uniform(-side, side, size=(3, n2))) / 2
    xyz += rng.choice([0.0, 0.25, 0.5], size=(3, n2))
    xyz[:, :4] = [[1e9, -1e9, 3e8, 0.5]] * 3
    x, y, z = xyz.astype(np.float32)
    model = rng.uniform(0.5, 2.0, size=side ** 3).astype(np.float32)
    model[rng.random(side ** 3) < 0.1] = 0.0
    model[rng.random(side ** 3) < 0.1] = -1.0
    images = rng.poisson(1.0, size=(N, n2)).astype(np.float32)
    mask = (rng.random(n2) < 0.9).astype(np.int32)
    quats = rotations()
    R = quats.shape[0]
    wts = np.full(R, 1.0 / R, np.float32)
    f = lambda a, dt=torch.float32: torch.as_tensor(np.ascontiguousarray(a), dtype=dt, device=cuda)
    plan = E.Plan(ctx, side, N, R, precision=prec, diff=diff, interp=interp)
    plan.bind(f(images), f(mask, torch.int32), f(x), f(y), f(z), f(quats), f(wts))
    m = f(model)
    plan.iterate(m, torch.empty_like(m), 0.5)
    phi = ctx.copy_real_to_host(plan.results()[1], R * N).reshape(R, N).astype(np.float64)
    plan.close()
    want = O.fused_iteration_fp64(model, images, mask, x, y, z, quats, wts, 0.5, side, diff=diff,
                                  interp=0 if interp == E.INTERP_NEAREST else 1)
    np.testing.assert_allclose(phi, want["phi"], rtol=5e-5 if prec == E.PREC_FP32 else 1e-3)
