"""The rows of the FP32 and of the hi + lo M-step operand at the lengths where their
loads change: whole 16-byte tuples and not, one, two and more turns of 512 threads, with
and without per-pattern normalisation and the mass bound of the deterministic insertion.
The model and the weight against the FP64 M-step of the plan's own responsibilities and
scaling (the mixed path's model tolerance, relative L2 5e-4), the responsibilities
against their sum (FP32 exponentials, 1e-5)."""
import numpy as np
import pytest
import torch

import emc_gb300 as E
from emc_gb300 import synthetic as S
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [E.PREC_FP32, E.PREC_MIXED], ids=["fp32", "hi-lo"])
@pytest.mark.parametrize("N,norm,insert", [
    (1, 0, E.INSERT_ATOMIC), (4, 0, E.INSERT_DETERMINISTIC), (7, 1, E.INSERT_ATOMIC),
    (2049, 0, E.INSERT_DETERMINISTIC), (2052, 1, E.INSERT_ATOMIC), (4092, 0, E.INSERT_ATOMIC),
    (4100, 1, E.INSERT_DETERMINISTIC), (4101, 0, E.INSERT_ATOMIC)])
def test_rows(ctx, cuda, N, norm, insert, precision):
    prob = S.make_problem(S.tiny(side=16, n_images=N, rot_n=2, photons=60, n_atoms=40, radius=3.0))
    R = 40
    quats, wts = prob.quats[:R], prob.weights[:R]
    im = prob.images.copy()
    im[:, np.flatnonzero(prob.mask)[0]] += 1.0  # no empty pattern
    f = lambda a, dt=torch.float32: torch.as_tensor(np.ascontiguousarray(a), dtype=dt, device=cuda)
    plan = E.Plan(ctx, 16, N, R, precision=precision, insert_mode=insert, normalize_images=norm)
    plan.set_option(E.Plan.OPT_MSTEP_QLO, 1)
    plan.bind(f(im), f(prob.mask, torch.int32), f(prob.x), f(prob.y), f(prob.z), f(quats), f(wts))
    m, w = f(prob.init_model), torch.empty(16 ** 3, device=cuda)
    st = plan.iterate(m, w, 0.4)
    P = ctx.copy_real_to_host(plan.results()[0], R * N).reshape(R, N).astype(np.float64)
    phi = ctx.copy_real_to_host(plan.results()[1], R * N).reshape(R, N).astype(np.float64)
    plan.close()
    assert np.abs(P.sum(0) - 1.0).max() < 1e-5
    on = prob.mask == 1
    want = O.mstep_fp64(P, phi, O.compacted_counts(im, prob.mask, 16, bool(norm)), prob.x[on],
                        prob.y[on], prob.z[on], quats, 16, 0)
    got_m, got_w = m.cpu().numpy().astype(np.float64), w.cpu().numpy().astype(np.float64)
    assert np.linalg.norm(got_w - want["weight"]) <= 5e-4 * np.linalg.norm(want["weight"])
    ref = want["model"] * want["mean_before"]
    assert np.linalg.norm(got_m * st.model_mean_before - ref) <= 5e-4 * np.linalg.norm(ref)
