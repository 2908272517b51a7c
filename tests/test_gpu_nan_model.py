"""A model that holds NaN: a NaN sample is no value of the slice, as a voxel of -1 is
not, on the tensor-core paths.  Both count as uncovered for the reference likelihood
and as the floor for the true-Poisson one, so every result is the same bit for bit."""
import numpy as np
import pytest
import torch

import emc_gb300 as E
from emc_gb300 import synthetic as S

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def prob():
    return S.make_problem(S.tiny(side=32, n_images=300, rot_n=2, photons=3000, n_atoms=120,
                                 radius=7.0))


def T(a, dev, dt=torch.float32):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=dt, device=dev)


def iterate(ctx, dev, prob, model, weights=None, **kw):
    s, R, N = prob.cfg.side, prob.quats.shape[0], prob.images.shape[0]
    pair = kw.pop("pair", 1)
    plan = E.Plan(ctx, s, N, R, precision=E.PREC_MIXED, insert_mode=E.INSERT_DETERMINISTIC, **kw)
    plan.set_option(E.Plan.OPT_ESTEP_PAIR, pair)
    plan.bind(T(prob.images, dev), T(prob.mask, dev, torch.int32), T(prob.x, dev), T(prob.y, dev),
              T(prob.z, dev), T(prob.quats, dev), T(prob.weights if weights is None else weights, dev))
    m, w = T(model, dev), torch.empty(s ** 3, device=dev)
    st = plan.iterate(m, w, 0.3)
    r_ptr, s_ptr, _ = plan.results()
    P = ctx.copy_real_to_host(r_ptr, R * N)
    phi = ctx.copy_real_to_host(s_ptr, R * N)
    plan.close()
    return st, P, phi, m.cpu().numpy(), w.cpu().numpy()


# one voxel: a quadruple of samples with a single NaN; 5 % and 60 %: two, three and all four
@pytest.mark.parametrize("share", [0.0, 0.05, 0.6])
@pytest.mark.parametrize("kw", [dict(), dict(pair=0), dict(known_intensity=1),
                                dict(diff=E.DIFF_TRUE_POISSON)],
                         ids=["pairs", "single", "known", "poisson"])
def test_nan_voxels_are_uncovered(ctx, cuda, prob, share, kw):
    rng = np.random.default_rng(11)
    model = (prob.init_model + 0.05).astype(np.float32)
    c = prob.cfg.side // 2
    pick = rng.random(model.size) < share
    pick[(c * prob.cfg.side + c) * prob.cfg.side + c + 5] = True
    holed, other = model.copy(), model.copy()
    holed[pick], other[pick] = np.nan, -1.0
    got = iterate(ctx, cuda, prob, holed, **kw)
    want = iterate(ctx, cuda, prob, other, **kw)
    assert np.isfinite(want[0].total_loglik)
    assert got[0].total_loglik == want[0].total_loglik
    assert got[0].bad_pairs == want[0].bad_pairs
    assert got[0].captured_mass == want[0].captured_mass
    for g, w in zip(got[1:], want[1:]):
        np.testing.assert_array_equal(g, w)


@pytest.mark.parametrize("bad", [np.nan, -1.0], ids=["nan", "negative"])
@pytest.mark.parametrize("kw", [dict(), dict(pair=0), dict(known_intensity=1),
                                dict(diff=E.DIFF_TRUE_POISSON),
                                dict(diff=E.DIFF_TRUE_POISSON, pair=0)],
                         ids=["pairs", "single", "known", "poisson", "poisson-single"])
def test_nan_loglik_has_no_responsibility(ctx, cuda, prob, bad, kw):
    """The log-likelihoods of a rotation whose weight has no logarithm are NaN: it is left
    out of the normaliser and of the model, as one of weight 0 is."""
    weights = prob.weights.copy()
    weights[3], weights[140] = bad, bad
    zero = np.where(weights > 0, weights, 0.0).astype(np.float32)
    got = iterate(ctx, cuda, prob, prob.init_model, weights=weights, **kw)
    want = iterate(ctx, cuda, prob, prob.init_model, weights=zero, **kw)
    assert abs(want[0].captured_mass - 1.0) < 1e-4
    assert got[0].total_loglik == want[0].total_loglik
    assert got[0].captured_mass == want[0].captured_mass
    for g, w in zip(got[1:], want[1:]):
        np.testing.assert_array_equal(g, w)
