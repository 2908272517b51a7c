"""EMC_OPT_ESTEP_GHLO with bit 1 (lo terms in every product): the scaling's denominator
sums s as FP16 hi + lo.  s 2^-8 of a model of values in (0.25, 1) lies above 2^-10, where
the lo half's spacing (2^-24) leaves at most 2^-25 of it: relative 2^-15 = 3.1e-5 a
pixel, and hi alone 2^-12 = 2.4e-4.  Over the thousand counts of a pattern the errors
average out: 1e-5 is the FP32 path's tolerance for the scaling, which hi alone exceeds."""
import numpy as np
import pytest
import torch

import emc_gb300 as E
from emc_gb300 import synthetic as S
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def T(a, dev, dt=torch.float32):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=dt, device=dev)


@pytest.fixture(scope="module")
def prob():
    return S.make_problem(S.tiny(side=32, n_images=300, rot_n=2, photons=3000, n_atoms=120,
                                 radius=7.0))


@pytest.mark.parametrize("pair", [1, 0], ids=["pairs", "single"])
@pytest.mark.parametrize("holes", [0.0, 0.05])
@pytest.mark.parametrize("bright", [0, 1], ids=["dim", "bright"])
def test_scaling_with_every_lo_term(ctx, cuda, prob, pair, holes, bright):
    s, R, N = prob.cfg.side, prob.quats.shape[0], prob.images.shape[0]
    rng = np.random.default_rng(2)
    m0 = (0.25 + 0.75 * rng.random(s ** 3)).astype(np.float32)
    m0[rng.random(m0.size) < holes] = -1.0
    im = prob.images.copy()
    if bright:  # sums over the covered pixels
        im[5, np.flatnonzero(prob.mask)[:40]] = 2000.0
    args = (T(im, cuda), T(prob.mask, cuda, torch.int32), T(prob.x, cuda), T(prob.y, cuda),
            T(prob.z, cuda), T(prob.quats, cuda), T(prob.weights, cuda))
    want = O.fused_iteration_fp64(m0, im, prob.mask, prob.x, prob.y, prob.z, prob.quats,
                                  prob.weights, 0.4, s)
    out = []
    for before in (True, False):  # the option set before or after the binding
        plan = E.Plan(ctx, s, N, R, precision=E.PREC_MIXED)
        plan.set_option(E.Plan.OPT_ESTEP_PAIR, pair)
        if before:
            plan.set_option(E.Plan.OPT_ESTEP_GHLO, 3)
        plan.bind(*args)
        m, w = T(m0, cuda), torch.empty(s ** 3, device=cuda)
        if not before:
            plan.iterate(m, w, 0.4)
            plan.set_option(E.Plan.OPT_ESTEP_GHLO, 3)
            m = T(m0, cuda)
        st = plan.iterate(m, w, 0.4)
        phi = ctx.copy_real_to_host(plan.results()[1], R * N).reshape(R, N)
        np.testing.assert_allclose(phi, want["phi"], rtol=1e-5)
        assert abs(st.total_loglik - want["total_loglik"]) <= 1e-5 * abs(want["total_loglik"])
        out.append(phi)
        # and back
        plan.set_option(E.Plan.OPT_ESTEP_GHLO, -1)
        plan.iterate(T(m0, cuda), w, 0.4)
        phi = ctx.copy_real_to_host(plan.results()[1], R * N).reshape(R, N)
        np.testing.assert_allclose(phi, want["phi"], rtol=5e-4)
        assert np.abs(phi / want["phi"] - 1).max() > 1e-5
        plan.close()
    np.testing.assert_array_equal(out[0], out[1])
