"""The tensor-core M-step over the (256-pixel, 64-pattern) blocks that hold counts:
pixel tiles with no counts at all, with counts in one block of patterns only, and
full ones, for both tile shapes, both interpolations and the three insertions.  The
model and the weight against the FP64 M-step of the plan's own responsibilities and
scaling (the mixed path's model tolerance, relative L2 5e-4)."""
import numpy as np
import pytest
import torch

import emc_gb300 as E
from emc_gb300 import synthetic as S
from oracle import oracle as O

pytestmark = pytest.mark.gpu

TOL = 5e-4


def T(a, dev, dt=torch.float32):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=dt, device=dev)


def rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


@pytest.mark.parametrize("pair", [1, 0], ids=["pairs", "single"])
@pytest.mark.parametrize("interp,insert", [
    (E.INTERP_NEAREST, E.INSERT_ATOMIC), (E.INTERP_NEAREST, E.INSERT_DETERMINISTIC),
    (E.INTERP_NEAREST, E.INSERT_SORTED), (E.INTERP_TRILINEAR, E.INSERT_ATOMIC),
    (E.INTERP_TRILINEAR, E.INSERT_DETERMINISTIC)])
def test_blocks_with_counts(ctx, cuda, interp, insert, pair):
    prob = S.make_problem(S.tiny(side=48, n_images=200, rot_n=2, photons=1500, n_atoms=120,
                                 radius=9.0))
    s, R, N = prob.cfg.side, prob.quats.shape[0], prob.images.shape[0]
    r = np.hypot(*np.meshgrid(np.arange(s) - s / 2 + 0.5, np.arange(s) - s / 2 + 0.5)).reshape(-1)
    im = prob.images.copy()
    im[:, r > 20] = 0.0  # the outermost pixel tiles: none
    im[:64, (r > 14) & (r <= 20)] = 0.0  # then: the second block of patterns only
    im[128:, (r > 14) & (r <= 20)] = 0.0
    assert im.sum(1).min() > 0
    plan = E.Plan(ctx, s, N, R, precision=E.PREC_MIXED, interp=interp, insert_mode=insert)
    plan.set_option(E.Plan.OPT_MSTEP_PAIR, pair)
    plan.bind(T(im, cuda), T(prob.mask, cuda, torch.int32), T(prob.x, cuda), T(prob.y, cuda),
              T(prob.z, cuda), T(prob.quats, cuda), T(prob.weights, cuda))
    m, w = T(prob.init_model, cuda), torch.empty(s ** 3, device=cuda)
    st = plan.iterate(m, w, 0.4)
    r_ptr, s_ptr, _ = plan.results()
    P = ctx.copy_real_to_host(r_ptr, R * N).reshape(R, N)
    phi = ctx.copy_real_to_host(s_ptr, R * N).reshape(R, N)
    plan.close()
    on = prob.mask == 1
    want = O.mstep_fp64(P, phi, O.compacted_counts(im, prob.mask, s), prob.x[on], prob.y[on],
                        prob.z[on], prob.quats, s, interp)
    got_m, got_w = m.cpu().numpy().astype(np.float64), w.cpu().numpy().astype(np.float64)
    assert rel(got_w, want["weight"]) < TOL
    assert rel(got_m * st.model_mean_before, want["model"] * want["mean_before"]) < TOL
    big = want["weight"] > 1e-6 * want["weight"].max()
    assert (got_w[big] > 0).all() and (got_w[want["weight"] == 0] == 0).all()
