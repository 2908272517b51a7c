"""The workloads this library is measured on, as calls of its public interface.

A case is a dict of plain values; `listed` names the fixed ones, `draw` makes
more of the same ranges.  `prepare` builds what a program holds before the call
(patterns, detector, rotations, a start model and the plan or network), `run`
makes one pass, `exact` restates the pass in 64-bit torch arithmetic.

The kinds of pass:

* "iterate": one fused EMC iteration (`Plan.iterate`, or a captured iteration
  replayed as a CUDA graph) from a given model: expand, scaling, likelihood,
  normalisation, M-step, insertion, model normalisation and blur;
* "pruned": the same with pruning on, seeded by the previous iteration's
  responsibilities (the late iterations of a true-Poisson reconstruction);
* "split": one rank of a rotation split (`rank_estep`, `rank_mstep`,
  `model_from_sums`), with the intensity known;
* "dropin": an iteration through the reference's own entry points, in slice
  chunks;
* "proposal": the rotation-proposal network's loss and gradients for one batch,
  and its predictions for every pattern.

The synthetic data have the shapes, photon counts, scale spread and beamstop of
the library's benchmark configurations: |F|^2 of Gaussian atoms in a sphere,
patterns that are Poisson-sampled slices of it.  `atom_sigma` sets how far out
counts reach (1.5 as the configurations; 0.7: to the detector's edge).  A
"random" start is the U(0, 1) model of a first iteration, a "late" one the true
intensity as that many photons determine it (Poisson noise per voxel, unvisited
voxels -1).
"""
import math

import numpy as np
import torch

import emc_gb300 as E

WAVELENGTH, PIXEL_SIZE, DISTANCE = 1.03e-9, 75.0e-6, 740.0e-3  # emc.conf's detector
POIS_C, SLICE_FLOOR = 0.02, 1e-6  # constants of the two likelihoods
DEV = "cuda"

INSERT = {"atomic": E.INSERT_ATOMIC, "fixed": E.INSERT_DETERMINISTIC, "sorted": E.INSERT_SORTED}
INTERP = {"nearest": E.INTERP_NEAREST, "trilinear": E.INTERP_TRILINEAR}
DIFF = {"poisson": E.DIFF_POISSON, "true_poisson": E.DIFF_TRUE_POISSON}
PRECISION = {"mixed": E.PREC_MIXED, "fp32": E.PREC_FP32}


def _case(kind, side, images, level, photons, **more):
    c = {"kind": kind, "side": side, "images": images, "level": level, "photons": photons,
         "atom_sigma": 1.5, "beamstop": max(2.0, round(side / 21.0, 1)), "masked": 0.0,
         "scale_lo": 0.5, "scale_hi": 1.5, "sigma": 0.4, "start": "random", "diff": "poisson",
         "interp": "nearest", "insert": "atomic", "precision": "mixed", "blur": 0.0,
         "graph": False, "normalize": False}
    c.update(more)
    return c


def listed():
    return [
        # the smallest problem of the batched configuration: a few rotations and
        # patterns, where launches and waits count
        dict(_case("iterate", 48, 500, 3, 1000.0), name="iterate_48"),
        # the small configuration as a loop of graph replays: blurred model, no
        # wait between iterations
        dict(_case("iterate", 64, 2000, 4, 1000.0, blur=1.0, graph=True), name="replay_64_blur"),
        # trilinear slicing and splatting with bit-reproducible insertion, a
        # ragged pattern count, and atoms sharp enough to count at the rim
        dict(_case("iterate", 96, 4999, 6, 3000.0, atom_sigma=0.7, interp="trilinear",
                   insert="fixed", start="late", sigma=0.35), name="iterate_96_trilinear"),
        # the low-count configuration: 80 photons a pattern, half the detector
        # masked, bit-reproducible sorted-voxel insertion
        dict(_case("iterate", 128, 50000, 6, 80.0, beamstop=6.0, masked=0.5, scale_lo=0.2,
                   scale_hi=2.0, insert="sorted", start="late", sigma=0.35),
             name="iterate_128_lowcount"),
        # the headline configuration
        dict(_case("iterate", 128, 20000, 8, 5000.0, beamstop=6.0, start="late"),
             name="iterate_128_mid"),
        # the counts x log-slice likelihood at a middle size of the batched configuration
        dict(_case("iterate", 112, 10000, 6, 1000.0, diff="true_poisson"), name="poisson_112"),
        # the plain FP32 path on per-pattern normalised (non-integer) intensities
        dict(_case("iterate", 64, 2000, 4, 1000.0, precision="fp32", normalize=True),
             name="fp32_64"),
        # a late iteration of the fifth-size mid configuration, pruned to the
        # tiles that hold the responsibilities
        dict(_case("pruned", 128, 4000, 8, 5000.0, beamstop=6.0, diff="true_poisson",
                   start="late"), name="pruned_128"),
        # half of the rotations of a middle-sized problem, as one rank of two
        # takes them, with known beam intensity (phi = 1)
        dict(_case("split", 80, 2500, 5, 1000.0, scale_lo=1.0, scale_hi=1.0,
                   rotations=3150), name="split_80_known"),
        # the reference's entry points in its own order, two slice chunks, the last ragged
        dict(_case("dropin", 64, 2000, 4, 1000.0, rotations=180, chunk=100), name="dropin_64"),
        # the proposal network on the small configuration's patterns
        dict(_case("proposal", 64, 2000, 4, 1000.0, batch=250), name="proposal_64"),
    ]


# the mid configuration's rotation x pattern x pixel count: no drawn case costs more
_MOST = 25680 * 20000 * 12756.0


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["iterate", "iterate", "iterate", "iterate", "fp32", "pruned", "split",
                       "dropin", "proposal"])
    atom = rng.choice([0.7, 1.0, 1.5])
    if kind == "proposal":
        return _case("proposal", rng.choice([64, 128]), log(500, 4000), 4, rng.choice([300.0, 1000.0]),
                     atom_sigma=atom, batch=log(64, 256))
    if kind == "dropin":
        return _case("dropin", 2 * log(20, 32), log(300, 2000), 4, rng.choice([300.0, 1000.0]),
                     atom_sigma=atom, rotations=log(60, 180), chunk=rng.choice([50, 64, 100]),
                     sigma=rng.uniform(0.3, 0.4))
    while True:
        side, images, level = 2 * log(24, 80), log(500, 50000), rng.randint(3, 8)
        photons = float(log(80, 5000))
        rot = E.rotation_count(level)
        pairs, cost = rot * images, rot * images * 0.785 * side * side
        if cost > 0.9 * _MOST or images * side * side > 1.0e9:
            continue
        sigma, start = rng.uniform(0.3, 0.4), rng.choice(["random", "late"])
        if kind == "fp32":
            if cost > _MOST / 60:
                continue
            return _case("iterate", side, images, level, photons, atom_sigma=atom, sigma=sigma,
                         start=start, precision="fp32", normalize=rng.random() < 0.5,
                         diff=rng.choice(["poisson", "true_poisson"]))
        if kind == "pruned":
            if pairs < 2e7 or cost > 0.3 * _MOST:
                continue
            return _case("pruned", side, images, level, max(photons, 1000.0), atom_sigma=atom,
                         diff="true_poisson", start="late")
        if kind == "split":
            return _case("split", side, images, level, photons, atom_sigma=atom, scale_lo=1.0,
                         scale_hi=1.0, sigma=sigma, start=start,
                         rotations=rot // rng.choice([1, 2, 3]))
        interp = rng.choice(["nearest", "nearest", "nearest", "trilinear"])
        insert = rng.choice(["atomic", "atomic", "fixed"] + (["sorted"] if interp == "nearest" else []))
        return _case("iterate", side, images, level, photons, atom_sigma=atom, sigma=sigma,
                     start=start, interp=interp, insert=insert,
                     diff=rng.choice(["poisson", "poisson", "true_poisson"]),
                     blur=rng.choice([0.0, 0.0, 1.0]), graph=rng.random() < 0.3,
                     masked=rng.choice([0.0, 0.0, 0.5]))


# ------------------------------------------------------------- inputs ----
def _detector_mask(c):
    """Circle of radius side / 2 minus the beamstop, minus panel gaps (the gaps
    are the instrument's: the same for every seed)."""
    s = c["side"]
    q = np.arange(s) - s / 2.0 + 0.5
    r = np.sqrt(q[None, :] ** 2 + q[:, None] ** 2)
    m = (r <= s / 2.0) & (r >= c["beamstop"])
    rng = np.random.default_rng(7)
    target = (1.0 - c["masked"]) * m.sum()
    while m.sum() > target:
        o, w = rng.integers(0, s), rng.integers(1, max(2, s // 24))
        if rng.random() < 0.5:
            m[:, o:o + w] = False
        else:
            m[o:o + w, :] = False
    return m.reshape(-1)


def _pixels(c):
    return int(_detector_mask(c).sum())


def _rotation_count(c):
    return int(c.get("rotations") or E.rotation_count(c["level"]))


def _particle(c, gen):
    """|F|^2 at the voxel centres of Gaussian atoms uniform in a ball, mean 1."""
    s = c["side"]
    atoms = max(60, int(3000 * (s / 128.0) ** 3))
    pos = torch.randn(atoms, 3, generator=gen, device=DEV)
    pos *= (s * 0.2 * torch.rand(atoms, generator=gen, device=DEV) ** (1 / 3) / pos.norm(dim=1))[:, None]
    q = torch.arange(s, device=DEV) - s / 2.0 + 0.5
    e = [torch.polar(torch.ones(atoms, s, device=DEV), -2 * math.pi / s * torch.outer(pos[:, k], q))
         for k in range(3)]
    out = torch.empty(s, s, s, device=DEV)
    g = torch.exp(-2 * math.pi ** 2 * c["atom_sigma"] ** 2 * q * q / s ** 2)
    for z in range(s):
        f = (e[1] * e[2][:, z:z + 1]).T @ e[0]
        out[z] = (f.abs() * g[:, None] * g[None, :] * g[z]) ** 2
    return out / out.mean()


def _rotation_matrices(q):
    a, b, c, d = q.unbind(1)
    return torch.stack([a * a + b * b - c * c - d * d, 2 * b * c - 2 * a * d, 2 * b * d + 2 * a * c,
                        2 * b * c + 2 * a * d, a * a - b * b + c * c - d * d, 2 * c * d - 2 * a * b,
                        2 * b * d - 2 * a * c, 2 * c * d + 2 * a * b, a * a - b * b - c * c + d * d],
                       1).view(-1, 3, 3)


def _patterns(c, true, pts, mask, gen):
    """Poisson counts of randomly oriented, randomly scaled slices, and the mean
    count per unit of model intensity."""
    s, n = c["side"], c["images"]
    q = torch.randn(n, 4, generator=gen, device=DEV)
    q /= q.norm(dim=1, keepdim=True)
    scale = c["scale_lo"] + (c["scale_hi"] - c["scale_lo"]) * torch.rand(n, 1, generator=gen, device=DEV)
    lam = torch.empty(n, s * s, device=DEV)
    step = max(1, 16_000_000 // (s * s))
    for i in range(0, n, step):
        p = torch.einsum("nij,pj->npi", _rotation_matrices(q[i:i + step]), pts) + (s / 2 - 0.5)
        g = ((p + 0.5) / s * 2 - 1)[None, :, :, None, :]
        lam[i:i + step] = torch.nn.functional.grid_sample(
            true[None, None], g, mode="bilinear", padding_mode="zeros",
            align_corners=False)[0, 0, :, :, 0] * mask
    unit = c["photons"] / float(lam.sum(1).mean())
    for i in range(0, n, step):
        lam[i:i + step] = torch.poisson(lam[i:i + step] * (unit * scale[i:i + step]), generator=gen)
    return lam, unit


def _start_model(c, true, unit, gen):
    s = c["side"]
    if c["start"] == "random":
        return torch.rand(s ** 3, generator=gen, device=DEV)
    q = torch.arange(s, device=DEV) - s / 2.0 + 0.5
    rho = (q[:, None, None] ** 2 + q[None, :, None] ** 2 + q[None, None, :] ** 2).sqrt()
    # a voxel at radius rho is met by about 1 / (2 rho) of the patterns
    seen = c["images"] * unit / (2.0 * rho.clamp(min=1.0))
    m = torch.poisson(true * seen, generator=gen) / seen
    m[rho > s / 2.0 - 0.5] = -1.0
    m = m.reshape(-1)
    return torch.where(m > 0, m / m[m > 0].mean(), m)


def _inputs(c, seed):
    gen = torch.Generator(device=DEV)
    gen.manual_seed(int(seed) + 1)
    s, R = c["side"], _rotation_count(c)
    x, y, z = (torch.as_tensor(v, device=DEV) for v in
               E.calculate_coordinates(s, PIXEL_SIZE, DISTANCE, WAVELENGTH))
    quats, weights = E.generate_rotations(c["level"])
    mask = torch.as_tensor(_detector_mask(c), device=DEV)
    true = _particle(c, gen)
    images, unit = _patterns(c, true, torch.stack([x, y, z], 1), mask.float(), gen)
    return {"x": x, "y": y, "z": z, "mask": mask.to(torch.int32), "images": images,
            "rot": torch.as_tensor(quats[:R], device=DEV).contiguous(),
            "rotw": torch.as_tensor(weights[:R], device=DEV).contiguous(),
            "model0": _start_model(c, true, unit, gen), "gen": gen}


def _params(gen):
    """He-uniform weights and zero biases, in the network's parameter order."""
    parts = []
    for cin in (1, 64, 64, 64):
        b = math.sqrt(6.0 / (9 * cin))
        parts += [(2 * torch.rand(64 * cin * 9, generator=gen, device=DEV) - 1) * b,
                  torch.zeros(64, device=DEV)]
    parts += [(2 * torch.rand(6 * 1024, generator=gen, device=DEV) - 1) * math.sqrt(3.0 / 1024),
              torch.zeros(6, device=DEV)]
    return torch.cat(parts)


def _network_inputs(c, d):
    q = torch.randn(c["images"], 4, generator=d["gen"], device=DEV)
    q /= q.norm(dim=1, keepdim=True)
    rows = torch.randperm(c["images"], generator=d["gen"], device=DEV)[:c["batch"]]
    return q.contiguous(), rows.to(torch.int32).cpu().numpy(), _params(d["gen"])


def prepare(case, seed):
    c, d = case, _inputs(case, seed)
    ctx = E.Context(0)
    st = {"case": c, "ctx": ctx, **d}
    if c["kind"] == "proposal":
        st["quats"], st["rows"], p = _network_inputs(c, d)
        st["net"] = E.Proposal(ctx, seed=0)
        st["net"].set_params(p.cpu().numpy())
        st["net"].set_data(d["images"], d["mask"], c["side"])
        st["out"] = torch.empty(c["images"], 2, 4, device=DEV)
        return st
    n3, R, N = c["side"] ** 3, d["rot"].shape[0], c["images"]
    st["model"] = torch.empty(n3, device=DEV)
    st["weight"] = torch.empty(n3, device=DEV)
    if c["kind"] == "dropin":
        st["slices"] = torch.empty(c["chunk"], c["side"] ** 2, device=DEV)
        st["scaling"] = torch.empty(R, N, device=DEV)
        st["respons"] = torch.empty(R, N, device=DEV)
        for k in ("maxr", "sums", "lse"):
            st[k] = torch.empty(N, device=DEV)
        st["active"] = torch.ones(N, dtype=torch.int32, device=DEV)
        return st
    plan = st["plan"] = E.Plan(
        ctx, c["side"], N, R, diff=DIFF[c["diff"]], interp=INTERP[c["interp"]],
        precision=PRECISION[c["precision"]], insert_mode=INSERT[c["insert"]],
        known_intensity=1 if c["kind"] == "split" else 0,
        normalize_images=1 if c["normalize"] else 0, blur_sigma=c["blur"])
    plan.bind(d["images"], d["mask"], d["x"], d["y"], d["z"], d["rot"], d["rotw"])
    if c["kind"] == "split":
        st["dmax"] = torch.empty(N, device=DEV)
        st["dsum"] = torch.empty(N, dtype=torch.float64, device=DEV)
        st["model_sum"] = torch.empty(n3, device=DEV)
        st["weight_sum"] = torch.empty(n3, device=DEV)
        return st
    if c["kind"] == "pruned":
        plan.set_pruning(True)
        for _ in range(2):  # responsibilities of this model, then its tiles
            st["model"].copy_(d["model0"])
            plan.iterate(st["model"], st["weight"], c["sigma"])
    if c["graph"]:
        st["model"].copy_(d["model0"])
        plan.iterate(st["model"], st["weight"], c["sigma"])
        plan.capture(st["model"], st["weight"])
    return st


# --------------------------------------------------------------- pass ----
def run(st):
    c = st["case"]
    if c["kind"] == "proposal":
        loss, grads = st["net"].loss_grad(st["rows"], st["quats"])
        return {"loss": loss, "grads": grads, "quats": st["net"].predict(st["out"])}
    if c["kind"] == "dropin":
        return _run_dropin(st)
    plan, model, weight = st["plan"], st["model"], st["weight"]
    if c["kind"] == "split":
        plan.rank_estep(st["model0"], c["sigma"], st["dmax"], st["dsum"])
        # the exchange of the normaliser; this rank's part stands for all ranks'
        lse = st["dmax"].double() + torch.log(st["dsum"])
        plan.rank_mstep(lse, st["model_sum"], st["weight_sum"])
        plan.model_from_sums(st["model_sum"], st["weight_sum"], 2, model, weight)
        return {"lse": lse.float(), "model_sum": st["model_sum"], "weight_sum": st["weight_sum"],
                "model": model, "weight": weight}
    model.copy_(st["model0"])  # an iteration works in place
    if c["graph"]:
        plan.replay(c["sigma"])
        return {"model": model, "weight": weight}
    stats = plan.iterate(model, weight, c["sigma"])
    return {"model": model, "weight": weight, "loglik": stats.total_loglik}


def _run_dropin(st):
    c, ctx = st["case"], st["ctx"]
    s, n2, N, R = c["side"], c["side"] ** 2, c["images"], st["rot"].shape[0]
    sl, img, mask, resp, scal = st["slices"], st["images"], st["mask"], st["respons"], st["scaling"]
    for r0 in range(0, R, c["chunk"]):
        n = min(c["chunk"], R - r0)
        ctx.get_slices(st["model0"], s, sl, st["rot"], st["x"], st["y"], st["z"], r0, n)
        ctx.update_scaling_full(img, sl, mask, scal, n2, N, r0, n)
        ctx.calculate_responsabilities(sl, img, mask, c["sigma"], scal, resp, st["rotw"], n2, N, r0, n)
    ctx.max_vector(resp, N, R, st["maxr"])
    ctx.respons_max_expf(resp, st["maxr"], N, R, st["sums"])
    ctx.log_sum_max(st["sums"], st["maxr"], st["lse"], N)
    ctx.norm_respons_sumexpf(resp, st["lse"], st["maxr"], N, R)
    ctx.reset_real(st["model"])
    ctx.reset_real(st["weight"])
    for r0 in range(0, R, c["chunk"]):
        n = min(c["chunk"], R - r0)
        ctx.update_slices(img, sl, mask, resp, scal, st["active"], N, r0, n, n2, s, st["model"],
                          st["x"], st["y"], st["z"], st["rot"][r0:], st["weight"])
    ctx.divide_model_by_weight(s, st["model"], st["weight"])
    mean = ctx.normalize_model(s, st["model"])
    return {"scaling": scal, "respons": resp, "model": st["model"], "weight": st["weight"],
            "mean": mean}


def work(case):
    c = case
    s, N, R, P = c["side"], c["images"], _rotation_count(c), _pixels(c)
    pairs, n3 = float(R) * N, s ** 3
    if c["kind"] == "proposal":
        # 26 MFLOP a pattern forward, three times that with the gradients
        return {"bytes": 4.0 * (4096 * (N + c["batch"]) + 2 * 117574 + 8 * N),
                "flops": 26.2e6 * (N + 3 * c["batch"])}
    if c["kind"] == "dropin":
        # scaling 4, likelihood 6 and slice average 3 operations a pixel of a pair
        return {"bytes": 4.0 * (N * s * s + 4 * pairs + R * P + 3 * n3), "flops": 13.0 * pairs * P}
    # four contractions (scaling numerator and denominator, the two likelihood
    # terms) and the M-step's; the true-Poisson likelihood has one, a known
    # intensity needs no scaling; the counts once at their size in the plan
    terms = 2 if c["diff"] == "true_poisson" else (3 if c["kind"] == "split" else 5)
    share = 0.3 if c["kind"] == "pruned" else 1.0
    return {"bytes": (4.0 if c["precision"] == "fp32" else 2.0) * N * P + 12.0 * n3,
            "flops": 2.0 * terms * pairs * P * share}


# ------------------------------------------------- 64-bit restatement ----
def _fma(a, b, c):
    """float32 a * b + c with one rounding (the product is exact in 64 bits)."""
    return (a.double() * b.double() + c.double()).float()


def _matrices32(q):
    a, b, c, d = q.float().unbind(1)
    a2, b2, c2 = 2 * a, 2 * b, 2 * c
    return [_fma(-d, d, _fma(-c, c, _fma(b, b, a * a))), _fma(-a2, d, b2 * c), _fma(a2, c, b2 * d),
            _fma(a2, d, b2 * c), _fma(-d, d, _fma(c, c, _fma(-b, b, a * a))), _fma(-a2, b, c2 * d),
            _fma(-a2, c, b2 * d), _fma(a2, b, c2 * d), _fma(d, d, _fma(-c, c, _fma(-b, b, a * a)))]


def _coords(rot, d, pix, side):
    """Fractional voxel coordinates [3][R][P] in the library's float32 geometry
    (which voxel a pixel falls into is decided there)."""
    m = [v[:, None] for v in _matrices32(rot)]
    x, y, z = (d[k][pix][None, :] for k in ("x", "y", "z"))
    return [(side / 2.0 - 0.5) + _fma(m[3 * k + 2], z, _fma(m[3 * k + 1], y, m[3 * k] * x))
            for k in range(3)]


def _nearest(co, side, lo):
    i = [torch.where(v >= 0, torch.floor(v.double() + 0.5), torch.ceil(v.double() - 0.5)).long()
         for v in co]
    ok = (i[0] >= lo) & (i[0] < side) & (i[1] >= lo) & (i[1] < side) & (i[2] >= lo) & (i[2] < side)
    return torch.where(ok, (i[2] * side + i[1]) * side + i[0], -1)


def _corners(co, side):
    f = [torch.floor(v) for v in co]
    t = [(v - w).double() for v, w in zip(co, f)]
    for k in range(8):
        i = [f[a].long() + ((k >> a) & 1) for a in range(3)]
        w = 1.0
        for a in range(3):
            w = w * (t[a] if (k >> a) & 1 else 1.0 - t[a])
        ok = w > 0
        for a in range(3):
            ok = ok & (i[a] >= 0) & (i[a] < side)
        yield torch.where(ok, (i[2] * side + i[1]) * side + i[0], -1), torch.where(ok, w, 0.0)


def _slices(c, model, co):
    if c["interp"] == "nearest":
        v = _nearest(co, c["side"], 1)
        return torch.where(v >= 0, model[v.clamp(min=0)].double(), -1.0)
    acc, ws = 0.0, 0.0
    for v, w in _corners(co, c["side"]):
        val = model[v.clamp(min=0)].double()
        w = torch.where((v >= 0) & (val >= 0), w, 0.0)
        acc, ws = acc + w * val, ws + w
    return torch.where(ws > 1e-6, acc / ws.clamp(min=1e-30), -1.0)


def _insert(c, co, U, T, msum, wsum):
    """T (U / T) and T at the pixels' voxels, rotations with T > 1e-10."""
    live = (T.float() > 1e-10)[:, None]
    parts = ([(_nearest(co, c["side"], 0), 1.0)] if c["interp"] == "nearest"
             else _corners(co, c["side"]))
    for v, w in parts:
        on = (v >= 0) & live
        msum.index_add_(0, v[on], (U * w)[on])
        wsum.index_add_(0, v[on], (T[:, None] * w).expand_as(U)[on])


def _blurred(m, side, sigma):
    keep = ~(m < 0)
    k = torch.arange(side, device=DEV)
    k = torch.minimum(k, side - k).double()
    g = torch.exp(-2 * math.pi ** 2 * sigma ** 2 * k ** 2 / side ** 2)
    f = torch.fft.fftn(torch.where(keep, m, 0.0).view(side, side, side))
    b = torch.fft.ifftn(f * g[:, None, None] * g[None, :, None] * g[None, None, :]).real
    return torch.where(keep, b.reshape(-1), -1.0)


def _finished(c, msum, wsum):
    m = torch.where(wsum > 0, msum / torch.where(wsum > 0, wsum, 1.0), -1.0)
    m = m / m[m > 0].mean()
    return _blurred(m, c["side"], c["blur"]) if c["blur"] > 0 else m


def exact(case, seed):
    c = case
    s, N, R, P = c["side"], c["images"], _rotation_count(c), _pixels(c)
    if c["kind"] == "proposal":
        return _exact_proposal(c, seed)
    if c["kind"] == "dropin":
        return _exact_dropin(c, _inputs(c, seed))
    if float(R) * N * P > 1.4e12 or float(R) * N > 3e8:
        return None  # half a minute and more of 64-bit products
    d = _inputs(c, seed)
    pix = torch.nonzero(d["mask"]).reshape(-1)
    K = d["images"][:, pix].double()
    if c["normalize"]:
        K = (d["images"][:, pix] * (s * s / K.sum(1, keepdim=True)).float()).double()
    logw, model = torch.log(d["rotw"].double()), d["model0"]
    known, pois = c["kind"] == "split", c["diff"] == "poisson"
    L = torch.empty(R, N, dtype=torch.float64, device=DEV)
    phi = torch.ones(R, N, dtype=torch.float64, device=DEV)
    Ksum = K.sum(1)
    for a in range(0, R, 512):
        S = _slices(c, model, _coords(d["rot"][a:a + 512], d, pix, s))
        lw, f = logw[a:a + 512, None], phi[a:a + 512]
        if pois:
            M = (S > 0).double()
            ok = (M.sum(1) > 0)[:, None].expand(-1, N)
            if not known:
                num, den = (S >= 1e-10).double() @ (K * K).T, (S * (S >= 1e-10)) @ K.T
                ok = ok & (num > 0) & (den > 0)
                f.copy_(torch.where(ok, num / torch.where(ok, den, 1.0), 1.0))
            G, H = M * S / (S + POIS_C), M / (S + POIS_C)
            sig = (G * S).sum(1)[:, None] - 2 * (G @ K.T) / f + (H @ (K * K).T) / f ** 2
            L[a:a + 512] = torch.where(
                ok, lw - sig / (2 * M.sum(1).clamp(min=1)[:, None] * c["sigma"] ** 2), -math.inf)
        else:
            S = S.clamp(min=SLICE_FLOOR)
            sr, ll = S.sum(1)[:, None], torch.log(S) @ K.T
            if known:
                L[a:a + 512] = lw + ll - sr
            else:
                f.copy_(Ksum[None, :] / sr)
                L[a:a + 512] = torch.where(
                    Ksum[None, :] > 0,
                    lw + ll + Ksum[None, :] * torch.log(f.clamp(min=1e-300)) - Ksum[None, :], lw)
    lse = torch.logsumexp(L, 0)
    msum = torch.zeros(s ** 3, dtype=torch.float64, device=DEV)
    wsum = torch.zeros_like(msum)
    for a in range(0, R, 512):
        Pr = torch.where(torch.isfinite(lse)[None, :], torch.exp(L[a:a + 512] - lse[None, :]), 0.0)
        Q = torch.where(phi[a:a + 512] > 0, Pr / phi[a:a + 512].clamp(min=1e-300), 0.0)
        _insert(c, _coords(d["rot"][a:a + 512], d, pix, s), Q @ K, Pr.sum(1), msum, wsum)
    if known:
        return {"lse": lse, "model_sum": msum, "weight_sum": wsum,
                "model": _finished(c, msum / 2, wsum / 2), "weight": wsum / 2}
    # counts x log-slices peak so sharply that outer voxels are reached only by
    # responsibilities below the smallest float: positive in 64 bits, 0 in the
    # library's, they change the number of voxels that the mean is taken over
    out = {"model": _finished(c, msum, wsum) if pois else None, "weight": wsum}
    return out if c["graph"] else {**out, "loglik": lse[torch.isfinite(lse)].sum().reshape(())}


def _exact_dropin(c, d):
    s, n2, N, R = c["side"], c["side"] ** 2, c["images"], d["rot"].shape[0]
    allp = torch.arange(n2, device=DEV)
    on = d["mask"] > 0
    K32 = d["images"]
    K = K32.double()
    phi = torch.empty(R, N, dtype=torch.float64, device=DEV)
    L = torch.empty_like(phi)
    S_all = torch.empty(R, n2, dtype=torch.float64, device=DEV)
    for a in range(0, R, 64):
        S_all[a:a + 64] = _slices(c, d["model0"], _coords(d["rot"][a:a + 64], d, allp, s))
    steps = -(-n2 // 512)
    pad = steps * 512 - n2
    for r in range(R):
        S = S_all[r]
        use = (on & (S > 1e-10))[None, :] & (K > 1e-10)
        # the reference's denominator: 512 integer partial sums, truncated at every term
        t = torch.nn.functional.pad(torch.where(use, K * S[None, :], 0.0), (0, pad)).view(N, steps, 512)
        den = torch.zeros(N, 512, dtype=torch.float64, device=DEV)
        for j in range(steps):
            den = torch.trunc((den + t[:, j]).float().double())
        num = torch.where(use, K * K, 0.0).sum(1)
        phi[r] = num / den.sum(1)
        m = on & (S > 0)
        Sm = S[m]
        diff = (Sm[None, :] - K[:, m] / phi[r][:, None]) ** 2 / (Sm + POIS_C)[None, :]
        L[r] = math.log(float(d["rotw"][r])) - diff.sum(1) / (2.0 * int(m.sum()) * c["sigma"] ** 2)
    resp = torch.exp(L - torch.logsumexp(L, 0)[None, :])
    T = resp.sum(1)
    U = (resp / phi) @ torch.where(on[None, :], K, 0.0)
    msum = torch.zeros(s ** 3, dtype=torch.float64, device=DEV)
    wsum = torch.zeros_like(msum)
    pix = torch.nonzero(on).reshape(-1)
    _insert(c, _coords(d["rot"], d, pix, s), U[:, pix], T, msum, wsum)
    m = torch.where(wsum > 0, msum / torch.where(wsum > 0, wsum, 1.0), -1.0)
    mean = m[m > 0].mean()
    return {"scaling": phi, "respons": resp, "model": m / mean, "weight": wsum,
            "mean": mean.reshape(())}


def _exact_proposal(c, seed):
    d = _inputs(c, seed)
    quats, rows, p = _network_inputs(c, d)
    b = c["side"] // 64
    v = (d["images"] * (d["mask"] > 0)).double().clamp(min=0).view(-1, 64, b, 64, b).sum((2, 4))
    v = v.reshape(-1, 4096)
    X = torch.log1p(v * 4096.0 / v.sum(1, keepdim=True).clamp(min=1.0))
    X = (X - X.mean(0)) / torch.sqrt(X.var(0, unbiased=False) + 1e-4)
    p = p.double().requires_grad_(True)
    at, w = 0, []
    for shape in [(64, 1, 3, 3), (64,), (64, 64, 3, 3), (64,), (64, 64, 3, 3), (64,),
                  (64, 64, 3, 3), (64,), (6, 1024), (6,)]:
        n = math.prod(shape)
        w.append(p[at:at + n].view(shape))
        at += n

    def net(x):
        x = x.view(-1, 1, 64, 64)
        for k in range(4):  # 3x3, stride 2, padding 1, as products of unfolded columns
            h = x.shape[2] // 2
            cols = torch.nn.functional.unfold(x, 3, padding=1, stride=2)
            x = torch.relu(w[2 * k].view(64, -1) @ cols + w[2 * k + 1][:, None]).view(-1, 64, h, h)
        return x.reshape(-1, 1024) @ w[8].T + w[9]

    idx = torch.as_tensor(rows, device=DEV).long()
    o = net(X[idx])
    M = _rotation_matrices(quats[idx].double())
    t = torch.cat([M[:, :, 0], M[:, :, 1]], 1)
    loss = torch.minimum(((o - t) ** 2).sum(1), ((o + t) ** 2).sum(1)).mean()
    loss.backward()
    with torch.no_grad():
        o = torch.cat([net(X[i:i + 256]) for i in range(0, X.shape[0], 256)])
        a = o[:, :3] / o[:, :3].norm(dim=1, keepdim=True)
        e = o[:, 3:] - (a * o[:, 3:]).sum(1, keepdim=True) * a
        e = e / e.norm(dim=1, keepdim=True)
        f = torch.linalg.cross(a, e)
        tr = [1 + a[:, 0] + e[:, 1] + f[:, 2], 1 + a[:, 0] - e[:, 1] - f[:, 2],
              1 - a[:, 0] + e[:, 1] - f[:, 2], 1 - a[:, 0] - e[:, 1] + f[:, 2]]
        q = torch.stack([u.clamp(min=0).sqrt() / 2 for u in tr], 1)
        sign = torch.stack([torch.ones_like(q[:, 0]), e[:, 2] - f[:, 1], f[:, 0] - a[:, 2],
                            a[:, 1] - e[:, 0]], 1)
        q = torch.copysign(q, sign)
        q = q / q.norm(dim=1, keepdim=True)
        mate = torch.stack([-q[:, 3], q[:, 2], -q[:, 1], q[:, 0]], 1)
        mate = torch.where(mate[:, :1] < 0, -mate, mate)
    return {"loss": loss.detach().reshape(()), "grads": p.grad.detach(),
            "quats": torch.stack([q, mate], 1)}
