"""The tensor-core likelihood's block kinds: what a 64-pixel block of a pattern
tile multiplies follows from its counts (none, all 0 or 1, larger ones, k (k - 1)
beyond one FP16 term) and from the slices (invalid pixels, values in (0, 1e-10)
that count in the likelihood but not in the scaling).  Each mix against the FP64
oracle, with the tolerances of the mixed path's parity tests."""
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
    # three pattern tiles (an odd number: the last pair's second half is empty), the last ragged
    return S.make_problem(S.tiny(side=32, n_images=300, rot_n=2, photons=3000, n_atoms=120,
                                 radius=7.0))


def counts(prob, kind):
    im = prob.images.copy()
    if kind == "binary":
        im = np.minimum(im, 1.0)
    elif kind == "mixed":  # tiles: none counted in one half, 0 / 1, bright
        im[:128] = 0.0
        im[0] = prob.images[0]
        im[128:256] = np.minimum(im[128:256], 1.0)
        im[256:] = np.minimum(im[256:] * 9.0, 2048.0)
    return im.astype(np.float32)


def start(prob, kind):
    m = prob.init_model.copy() + np.float32(0.05)
    pick = np.random.default_rng(5).random(m.size) < 0.05
    m[pick] = {"valid": m[pick], "zeros": 0.0, "unknown": -1.0, "tiny": 5e-11}[kind]
    return m.astype(np.float32)


@pytest.mark.parametrize("pair", [1, 0], ids=["pairs", "single"])
@pytest.mark.parametrize("count_kind,model_kind,opts,known", [
    ("drawn", "valid", {}, 0),
    ("binary", "valid", {}, 0),
    ("binary", "zeros", {}, 0),
    ("mixed", "valid", {}, 0),
    ("mixed", "unknown", {}, 0),
    ("mixed", "tiny", {}, 0),
    ("binary", "tiny", {}, 0),
    ("mixed", "zeros", {E.Plan.OPT_ESTEP_GHLO: 3}, 0),
    ("mixed", "zeros", {E.Plan.OPT_ESTEP_GHLO: 0}, 0),
    ("mixed", "zeros", {E.Plan.OPT_GLO_TAIL: 0}, 0),
    ("drawn", "unknown", {}, 1),
    ("binary", "tiny", {}, 1),
])
def test_block_kinds_match_oracle(ctx, cuda, prob, count_kind, model_kind, opts, known, pair):
    im, m0 = counts(prob, count_kind), start(prob, model_kind)
    s, R, N = prob.cfg.side, prob.quats.shape[0], im.shape[0]
    plan = E.Plan(ctx, s, N, R, precision=E.PREC_MIXED, known_intensity=known)
    for o, v in {**opts, E.Plan.OPT_ESTEP_PAIR: pair}.items():
        plan.set_option(o, v)
    args = (T(im, cuda), T(prob.mask, cuda, torch.int32), T(prob.x, cuda), T(prob.y, cuda),
            T(prob.z, cuda), T(prob.quats, cuda), T(prob.weights, cuda))
    # an earlier binding's blocks must leave nothing behind
    plan.bind(T(counts(prob, "mixed")[::-1], cuda), *args[1:])
    plan.bind(*args)
    m, w = T(m0, cuda), torch.empty(s ** 3, device=cuda)
    st = plan.iterate(m, w, 0.4)
    r_ptr, s_ptr, _ = plan.results()
    P = ctx.copy_real_to_host(r_ptr, R * N).reshape(R, N)
    phi = ctx.copy_real_to_host(s_ptr, R * N).reshape(R, N)
    plan.close()
    want = O.fused_iteration_fp64(m0, im, prob.mask, prob.x, prob.y, prob.z, prob.quats,
                                  prob.weights, 0.4, s, known_intensity=bool(known))
    bad = ~np.isfinite(want["loglik"])
    assert st.bad_pairs == int(bad.sum())
    assert abs(st.total_loglik - want["total_loglik"]) <= TOL_LL * abs(want["total_loglik"])
    np.testing.assert_allclose(phi, want["phi"], rtol=TOL_PHI)
    if not known:  # phi = 1 gives near one-hot responsibilities on these counts
        assert np.abs(P - want["respons"]).max() < TOL_RESP


def test_more_blocks_than_the_shared_list(ctx, cuda):
    """1,118 blocks of 64 pixels: the last are read from the list in global memory."""
    side, N = 302, 130
    quats, weights = E.generate_rotations(2)
    R = 140
    assert quats.shape[0] >= R
    rng = np.random.default_rng(3)
    x, y, z = E.calculate_coordinates(side, S.PIXEL_SIZE, S.DISTANCE, S.WAVELENGTH)
    mask = S.detector_mask(side, 2.0, 0.0, rng)
    assert -(-int(mask.sum()) // 64) > 1100
    im = rng.poisson(0.4, (N, side * side)).astype(np.float32)
    m0 = rng.random(side ** 3).astype(np.float32)
    plan = E.Plan(ctx, side, N, R, precision=E.PREC_MIXED)
    plan.bind(T(im, cuda), T(mask, cuda, torch.int32), T(x, cuda), T(y, cuda), T(z, cuda),
              T(quats[:R], cuda), T(weights[:R], cuda))
    m, w = T(m0, cuda), torch.empty(side ** 3, device=cuda)
    st = plan.iterate(m, w, 0.4)
    _, s_ptr, _ = plan.results()
    phi = ctx.copy_real_to_host(s_ptr, R * N).reshape(R, N)
    plan.close()
    S1 = O.get_slices(m0, side, quats[:R], x, y, z).astype(np.float64)
    on = np.nonzero(mask)[0]
    Sv, K = S1[:, on], im[:, on].astype(np.float64)
    M = Sv > 1e-10
    np.testing.assert_allclose(phi, (M @ (K * K).T) / ((Sv * M) @ K.T), rtol=TOL_PHI)
    assert st.bad_pairs == 0
