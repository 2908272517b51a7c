"""The drop-in scaling, likelihood and slice update where their FP32 forms hand
over to the general operations: infinite, zero and NaN scalings, operands near and
beyond the range that the forms check, counts that truncate, integer sums beyond
2^24, ragged image and rotation counts.  Against the oracle, bit for bit where no
transcendental function is involved."""
import numpy as np
import pytest
import torch

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def T(a, dev, dt=torch.float32):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=dt, device=dev)


def problem(side, N, R, seed):
    rng = np.random.default_rng(seed)
    n2 = side * side
    images = rng.poisson(1.5, (N, n2)).astype(np.float32)
    slices = rng.gamma(0.5, 2.0, (R, n2)).astype(np.float32)
    slices[rng.random((R, n2)) < 0.1] = -1.0
    slices[rng.random((R, n2)) < 0.05] = 0.0
    mask = (rng.random(n2) < 0.8).astype(np.int32)
    return rng, images, slices, mask


def scaled(ctx, dev, images, slices, mask):
    N, R, n2 = images.shape[0], slices.shape[0], images.shape[1]
    got = torch.ones((R, N), device=dev)
    ctx.update_scaling_full(T(images, dev), T(slices, dev), T(mask, dev, torch.int32), got, n2, N, 0, R)
    want = np.ones((R, N), np.float32)
    O.update_scaling_full(images, slices, mask, want, 0)
    ctx.sync()
    return got.cpu().numpy(), want


# side 23: 529 pixels, one past the 512 partials; N, R not multiples of 4 or 8
@pytest.mark.parametrize("side,N,R", [(5, 1, 1), (23, 9, 5), (40, 13, 7)])
@pytest.mark.parametrize("kscale", [1.0, 1e-3, 3e6, 1e-30, 1e30])
def test_scaling(ctx, cuda, side, N, R, kscale):
    _, images, slices, mask = problem(side, N, R, side)
    with np.errstate(all="ignore"):
        got, want = scaled(ctx, cuda, (images * np.float32(kscale)).astype(np.float32), slices, mask)
    np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("diff", [0, 1, 2])
@pytest.mark.parametrize("kscale,sscale", [(1.0, 1.0), (1e-25, 1.0), (1e12, 1.0), (1.0, 1e-20),
                                           (1.0, 1e20)])
def test_likelihood(ctx, cuda, diff, kscale, sscale):
    side, N, R = 23, 13, 7
    rng, images, slices, mask = problem(side, N, R, 3)
    images = (images * np.float32(kscale)).astype(np.float32)
    slices = np.where(slices > 0, slices * np.float32(sscale), slices).astype(np.float32)
    phi = rng.uniform(0.2, 5.0, (R, N)).astype(np.float32)
    phi[0, 0], phi[1, 1], phi[2, 2], phi[3, 3] = np.inf, 1e-35, 1e25, np.nan
    phi[4, 9], phi[5, 10] = 0.0, -2.0
    w = np.full(R, 1.0 / R, np.float32)
    n2 = side * side
    want = np.zeros((R, N), np.float32)
    with np.errstate(all="ignore"):
        O.calculate_responsabilities(slices, images, mask, np.float32(0.3), phi, want, w, 0, diff)
    got = torch.zeros((R, N), device=cuda)
    ctx.calculate_responsabilities(T(slices, cuda), T(images, cuda), T(mask, cuda, torch.int32), 0.3,
                                   T(phi, cuda), got, T(w, cuda), n2, N, 0, R, diff)
    ctx.sync()
    np.testing.assert_allclose(got.cpu().numpy(), want, rtol=2.4e-7, equal_nan=True)


@pytest.mark.parametrize("case", ["plain", "wide", "special"])
def test_slice_update(ctx, cuda, case):
    side, N, R = 23, 70, 11
    rng, images, slices, mask = problem(side, N, R, 11)
    n2 = side * side
    resp = rng.dirichlet(np.ones(R), N).T.astype(np.float32)
    phi = rng.uniform(0.2, 5.0, (R, N)).astype(np.float32)
    active = (rng.random(N) < 0.9).astype(np.int32)
    images[:, : n2 // 2] *= (rng.random((N, n2 // 2)) < 0.02)  # warps without counts
    if case != "plain":
        resp *= (10.0 ** rng.uniform(-40, 0, (R, N))).astype(np.float32)
        images[3] *= np.float32(1e-20)
        phi[:, 5] = np.float32(1e-12)
    if case == "special":
        phi[2, 7], phi[3, 8], resp[4, 9], images[11, 100] = np.nan, 0.0, np.nan, np.inf
    x = rng.uniform(-side / 2, side / 2, (3, n2)).astype(np.float32)
    quats = rng.standard_normal((R, 4)).astype(np.float32)
    quats /= np.linalg.norm(quats, axis=1, keepdims=True)
    out = torch.zeros((R, n2), device=cuda)
    m, w = torch.zeros(side ** 3, device=cuda), torch.zeros(side ** 3, device=cuda)
    ctx.update_slices(T(images, cuda), out, T(mask, cuda, torch.int32), T(resp, cuda), T(phi, cuda),
                      T(active, cuda, torch.int32), N, 0, R, n2, side, m, T(x[0], cuda),
                      T(x[1], cuda), T(x[2], cuda), T(quats, cuda), w)
    ctx.sync()
    with np.errstate(all="ignore"):
        want, _ = O.update_slices(images, mask, resp, phi, active, 0, R)
    np.testing.assert_array_equal(out.cpu().numpy(), want)
