"""Plan.results after graph replays and captures: what the buffer holds, the
log-likelihoods of the last iteration or its responsibilities, follows the work that
ran, not the work that was recorded."""
import numpy as np
import pytest
import torch

import emc_gb300 as E
from emc_gb300 import synthetic as S

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def prob():
    return S.make_problem(S.tiny(side=24, n_images=200, rot_n=2))


def bound(ctx, prob, dev, precision):
    T = lambda a, dt=torch.float32: torch.as_tensor(np.ascontiguousarray(a), dtype=dt, device=dev)
    s, R, N = prob.cfg.side, prob.quats.shape[0], prob.images.shape[0]
    plan = E.Plan(ctx, s, N, R, precision=precision, insert_mode=E.INSERT_DETERMINISTIC)
    plan._inputs = (T(prob.images), T(prob.mask, torch.int32), T(prob.x), T(prob.y), T(prob.z),
                    T(prob.quats), T(prob.weights))
    plan.bind(*plan._inputs)
    return plan, T(prob.init_model)


def respons(ctx, plan, prob):
    R, N = prob.quats.shape[0], prob.images.shape[0]
    return ctx.copy_real_to_host(plan.results()[0], R * N).reshape(R, N).copy()


@pytest.fixture(scope="module", params=[E.PREC_FP32, E.PREC_MIXED], ids=["fp32", "mixed"])
def direct(ctx, cuda, prob, request):
    plan, m = bound(ctx, prob, cuda, request.param)
    w = torch.empty_like(m)
    out = []
    for sg in (0.4, 0.3):
        plan.iterate(m, w, sg)
        out.append(respons(ctx, plan, prob))
    plan.close()
    np.testing.assert_allclose(out[0].sum(0), 1.0, atol=1e-4)
    assert not np.array_equal(out[0], out[1])
    return request.param, out


def test_results_after_each_replay(ctx, cuda, prob, direct):
    precision, want = direct
    plan, m = bound(ctx, prob, cuda, precision)
    w = torch.empty_like(m)
    plan.capture(m, w)
    for sg, P in zip((0.4, 0.3), want):
        plan.replay(sg)
        plan.wait()
        for _ in range(2):  # a second reading changes nothing
            np.testing.assert_array_equal(respons(ctx, plan, prob), P)
    plan.close()


def test_results_after_a_capture(ctx, cuda, prob, direct):
    """Recording an iteration runs nothing: the responsibilities are still the last
    iteration's, read before or only after the capture."""
    precision, want = direct
    for read_first in (True, False):
        plan, m = bound(ctx, prob, cuda, precision)
        w = torch.empty_like(m)
        plan.iterate(m, w, 0.4)
        if read_first:
            np.testing.assert_array_equal(respons(ctx, plan, prob), want[0])
        plan.capture(m, w)
        np.testing.assert_array_equal(respons(ctx, plan, prob), want[0])
        plan.replay(0.3)
        plan.wait()
        np.testing.assert_array_equal(respons(ctx, plan, prob), want[1])
        plan.close()


def test_results_after_batch_runs(ctx, cuda, prob, direct):
    precision, want = direct
    plan, m = bound(ctx, prob, cuda, precision)
    w = torch.empty_like(m)
    batch = E.Batch([plan], [m], [w])
    for sg, P in zip((0.4, 0.3), want):
        batch.run([sg])
        batch.wait()
        np.testing.assert_array_equal(respons(ctx, plan, prob), P)
    batch.close()
    plan.close()


def test_replay_after_eager_with_pruning_written(ctx, cuda, prob):
    """A graph recorded while pruning is on writes the responsibilities itself; the
    reading after its replay must not form them again."""
    plan, m = bound(ctx, prob, cuda, E.PREC_MIXED)
    plan.set_pruning(True)
    w = torch.empty_like(m)
    plan.capture(m, w)
    plan.iterate(m.clone(), w.clone(), 0.4)
    plan.replay(0.4)
    plan.wait()
    a = respons(ctx, plan, prob)
    np.testing.assert_allclose(a.sum(0), 1.0, atol=1e-4)
    np.testing.assert_array_equal(respons(ctx, plan, prob), a)
    plan.close()


def test_stats_of_a_rank_after_a_capture(ctx, cuda, prob):
    """The log-likelihood of a rank's M-step is still reported after a capture."""
    plan, m = bound(ctx, prob, cuda, E.PREC_MIXED)
    N = prob.images.shape[0]
    dmax, dsum = torch.empty(N, device=cuda), torch.empty(N, device=cuda, dtype=torch.float64)
    plan.rank_estep(m, 0.4, dmax, dsum)
    lse = dmax.double() + torch.log(dsum) + 3.0  # as if other ranks had a share
    ms, ws = torch.empty_like(m), torch.empty_like(m)
    plan.rank_mstep(lse, ms, ws)
    before = plan.wait().total_loglik
    np.testing.assert_allclose(before, float(lse.sum()), rtol=1e-12)
    plan.capture(m, torch.empty_like(m))
    assert plan.wait().total_loglik == before
    plan.close()
