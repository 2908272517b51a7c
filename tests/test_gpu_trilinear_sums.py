"""Trilinear insertion through the sums by x edges: even and odd sides (an edge starts
at an even or odd voxel of its row's storage), cells at every rim of the volume, all
insertion modes of the path.  Against the FP64 M-step of the plan's own
responsibilities and scaling (5e-4 relative L2); with fixed-point sums two runs give
the same bits."""
import numpy as np
import pytest
import torch

import emc_gb300 as E
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("insert", [E.INSERT_DETERMINISTIC, E.INSERT_ATOMIC], ids=["fixed", "float"])
@pytest.mark.parametrize("side", [9, 10])
def test_edges(ctx, cuda, side, insert):
    rng = np.random.default_rng(side)
    n2, N, R = side * side, 40, 140
    xyz = rng.uniform(-side / 2 - 1, side / 2 + 1, size=(3, n2))
    x, y, z = xyz.astype(np.float32)
    images = rng.poisson(1.0, size=(N, n2)).astype(np.float32)
    q = rng.normal(size=(R, 4))
    q = (q / np.linalg.norm(q, axis=1, keepdims=True)).astype(np.float32)
    f = lambda a, dt=torch.float32: torch.as_tensor(np.ascontiguousarray(a), dtype=dt, device=cuda)
    model = rng.uniform(0.5, 2.0, size=side ** 3).astype(np.float32)
    plan = E.Plan(ctx, side, N, R, precision=E.PREC_MIXED, interp=E.INTERP_TRILINEAR,
                  insert_mode=insert)
    plan.bind(f(images), f(np.ones(n2), torch.int32), f(x), f(y), f(z), f(q), f(np.full(R, 1 / R)))
    runs = []
    for _ in range(2):
        m, w = f(model), torch.empty(side ** 3, device=cuda)
        st = plan.iterate(m, w, 0.5)
        runs.append((m.cpu().numpy(), w.cpu().numpy()))
    P = ctx.copy_real_to_host(plan.results()[0], R * N).reshape(R, N).astype(np.float64)
    phi = ctx.copy_real_to_host(plan.results()[1], R * N).reshape(R, N).astype(np.float64)
    plan.close()
    want = O.mstep_fp64(P, phi, images.astype(np.float64), x, y, z, q, side, 1)
    got_m, got_w = runs[1]
    assert np.linalg.norm(got_w - want["weight"]) <= 5e-4 * np.linalg.norm(want["weight"])
    # voxels that hardly any weight reaches are ratios of rounding errors
    big = want["weight"] > 1e-3 * want["weight"].max()
    ref = want["model"] * want["mean_before"]
    err = (got_m * st.model_mean_before - ref)[big]
    assert np.linalg.norm(err) <= 5e-4 * np.linalg.norm(ref[big])
    if insert == E.INSERT_DETERMINISTIC:
        assert np.array_equal(runs[0][0], runs[1][0]) and np.array_equal(runs[0][1], runs[1][1])
