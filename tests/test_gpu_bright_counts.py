"""Bright counts at pixels that no rotation covers (detector corners outside the
volume) beside dim counts at the covered ones.  The scaling phi = sum k^2 / sum k s
runs over the covered pixels only, so a pattern's sum of squares may exceed what it
has there by any factor; sums of squares of 2^24 and more are not whole numbers in
FP32, and k (k - 1) of a count above 2,048 does not fit two FP16 terms.  Against the
FP64 oracle, with the tolerances of the mixed path's parity tests."""
import numpy as np
import pytest
import torch

import emc_gb300 as E
from emc_gb300 import synthetic as S
from oracle import oracle as O

pytestmark = pytest.mark.gpu

TOL_LL, TOL_PHI, TOL_RESP = 2e-5, 5e-4, 1e-3


def T(a, dev, dt=torch.float32):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=dt, device=dev)


@pytest.fixture(scope="module")
def prob():
    # three pattern tiles, the last ragged
    return S.make_problem(S.tiny(side=32, n_images=300, rot_n=2, photons=3000, n_atoms=120,
                                 radius=7.0))


def radius(prob, values):
    s = prob.cfg.side
    q = np.arange(s) - s / 2.0 + 0.5
    return np.sqrt(sum(np.square(v) for v in np.meshgrid(*[q] * values, indexing="ij"))).reshape(-1)


@pytest.mark.parametrize("pair", [1, 0], ids=["pairs", "single"])
@pytest.mark.parametrize("outside", [-1.0, 0.0, 5e-11], ids=["unknown", "zeros", "tiny"])
@pytest.mark.parametrize("pixels,count,ghlo", [(1, 60000, -1), (1, 30000, -1), (4, 60000, -1),
                                               (1, 3001, -1), (5, 2000, -1), (40, 2000, -1),
                                               (4, 60000, 3), (40, 2000, 0)])
def test_scaling_over_covered_pixels(ctx, cuda, prob, pixels, count, ghlo, outside, pair):
    s, R, N = prob.cfg.side, prob.quats.shape[0], prob.images.shape[0]
    rng = np.random.default_rng(pixels * count)
    r2 = radius(prob, 2)
    im = np.where(r2 < 12.0, rng.poisson(0.4, (N, s * s)), 0).astype(np.float32)
    corner = np.nonzero(r2 > 15.5)[0]
    hot = np.r_[0:9, 140, 290:N]  # patterns of every tile; the others stay dim
    for n in hot:
        im[n, rng.choice(corner, pixels, replace=False)] = count
    mask = np.ones(s * s, np.int32)
    m0 = (prob.init_model + 0.05).astype(np.float32)
    m0[radius(prob, 3) > 14.0] = outside
    plan = E.Plan(ctx, s, N, R, precision=E.PREC_MIXED)
    plan.set_option(E.Plan.OPT_ESTEP_PAIR, pair)
    plan.set_option(E.Plan.OPT_ESTEP_GHLO, ghlo)
    if count > 2048:
        plan.set_option(E.Plan.OPT_COUNTS_ROUND, 1)
        im = im.astype(np.float16).astype(np.float32)  # the counts that the plan takes
    plan.bind(T(im, cuda), T(mask, cuda, torch.int32), T(prob.x, cuda), T(prob.y, cuda),
              T(prob.z, cuda), T(prob.quats, cuda), T(prob.weights, cuda))
    m, w = T(m0, cuda), torch.empty(s ** 3, device=cuda)
    st = plan.iterate(m, w, 0.4)
    r_ptr, s_ptr, _ = plan.results()
    P = ctx.copy_real_to_host(r_ptr, R * N).reshape(R, N)
    phi = ctx.copy_real_to_host(s_ptr, R * N).reshape(R, N)
    plan.close()
    want = O.fused_iteration_fp64(m0, im, mask, prob.x, prob.y, prob.z, prob.quats, prob.weights,
                                  0.4, s)
    np.testing.assert_allclose(phi, want["phi"], rtol=TOL_PHI)
    assert st.bad_pairs == int((~np.isfinite(want["loglik"])).sum())
    assert abs(st.total_loglik - want["total_loglik"]) <= TOL_LL * abs(want["total_loglik"])
    if outside <= 0.0:  # (under a tiny s the bright counts make the responsibilities one-hot)
        assert np.abs(P - want["respons"]).max() < TOL_RESP


@pytest.mark.parametrize("pair", [1, 0], ids=["pairs", "single"])
@pytest.mark.parametrize("outside", [-1.0, 5e-11], ids=["unknown", "tiny"])
def test_known_intensity(ctx, cuda, prob, outside, pair):
    """phi = 1: the sums over the covered pixels stay exact beside 60,000 counts at every
    pixel outside the volume (single CTAs with a tiny s: the largest stage, one slot)."""
    s, R, N = prob.cfg.side, prob.quats.shape[0], prob.images.shape[0]
    rng = np.random.default_rng(4)
    r2 = radius(prob, 2)
    im = np.where(r2 < 12.0, rng.poisson(0.4, (N, s * s)), 0).astype(np.float32)
    im[:, r2 > 15.5] = 60000.0
    if outside > 0.0:
        im[:, r2 > 15.5] = 2000.0
    mask = np.ones(s * s, np.int32)
    m0 = (prob.init_model + 0.05).astype(np.float32)
    m0[radius(prob, 3) > 14.0] = outside
    plan = E.Plan(ctx, s, N, R, precision=E.PREC_MIXED, known_intensity=1)
    plan.set_option(E.Plan.OPT_ESTEP_PAIR, pair)
    plan.set_option(E.Plan.OPT_COUNTS_ROUND, 1)
    plan.bind(T(im, cuda), T(mask, cuda, torch.int32), T(prob.x, cuda), T(prob.y, cuda),
              T(prob.z, cuda), T(prob.quats, cuda), T(prob.weights, cuda))
    m, w = T(m0, cuda), torch.empty(s ** 3, device=cuda)
    st = plan.iterate(m, w, 0.4)
    plan.close()
    want = O.fused_iteration_fp64(m0, im, mask, prob.x, prob.y, prob.z, prob.quats, prob.weights,
                                  0.4, s, known_intensity=True)
    assert st.bad_pairs == 0
    assert abs(st.total_loglik - want["total_loglik"]) <= TOL_LL * abs(want["total_loglik"])


def test_rebind_from_bright_to_dim(ctx, cuda, prob):
    """A binding of dim counts after one of bright counts gives what a new plan gives."""
    s, N, R = prob.cfg.side, prob.images.shape[0], prob.quats.shape[0]
    bright = prob.images.copy()
    bright[7, :40] = 2000.0
    m0 = (prob.init_model + 0.05).astype(np.float32)
    m0[radius(prob, 3) > 12.0] = -1.0
    rest = (torch.ones(s * s, device=cuda, dtype=torch.int32), T(prob.x, cuda), T(prob.y, cuda),
            T(prob.z, cuda), T(prob.quats, cuda), T(prob.weights, cuda))
    out = []
    for first in (bright, None):
        plan = E.Plan(ctx, s, N, R, precision=E.PREC_MIXED, insert_mode=E.INSERT_DETERMINISTIC)
        images = T(prob.images, cuda)
        if first is not None:
            other = T(first, cuda)
            plan.bind(other, *rest)
            plan.iterate(T(m0, cuda), torch.empty(s ** 3, device=cuda), 0.4)
        plan.bind(images, *rest)
        m, w = T(m0, cuda), torch.empty(s ** 3, device=cuda)
        st = plan.iterate(m, w, 0.4)
        out.append((st.total_loglik, st.bad_pairs, m.cpu().numpy(), w.cpu().numpy()))
        plan.close()
    assert out[0][:2] == out[1][:2]
    np.testing.assert_array_equal(out[0][2], out[1][2])
    np.testing.assert_array_equal(out[0][3], out[1][3])
