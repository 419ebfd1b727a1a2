"""What a program that uses this framework has it do, as cases to time.

The work is the matvec of the directional Helmholtz FMM: an operator is built
once from points, order, leaf size and wavenumber (``IBFMM_Mat.prcmpt``), then
applied to charge vector after charge vector.  The cases cover

* sizes from the smallest problems of a ragged batch (5,000 points) to a
  sphere of 600,000 points, with odd counts among them;
* both precisions: FP64 on complex128 vectors (the drop-in), and mixed
  precision on complex64 vectors (how the many-right-hand-side and large
  workloads hold theirs), widened to the entry point's complex128 on the way
  in and narrowed on the way out;
* device vectors, host vectors, blocks of right-hand sides, one graph launch
  over a ragged batch of operators, and a whole build-and-apply on new points;
* surfaces and volumes, equal and distinct source and target sets, high
  frequency and the zero-wavenumber (Laplace) operator, orders 4 to 7.

A case is a dict of plain values:

  flow       "apply" (device vectors), "host" (numpy vectors), "once" (build
             from new points and apply), "batch" (many operators, one launch)
  geometry   "sphere", "cube", "blobs", "spheroid", or "apart" (sources in
             blobs, targets on a sphere inside them)
  n, nt      sources (and targets; nt differs only for "apart")
  waves      wavelengths across the geometry's diameter (0: Laplace)
  order, ncrit, precision
  nrhs       right-hand sides per call; groups: direction groups of a block
             (0: as memory needs)
  count, hi  "batch": number of operators, largest one (n: smallest one)
"""
from __future__ import annotations

import math

import numpy as np
import torch

from defmm_b200 import Batch, IBFMM_Mat, gemv
from defmm_b200 import workloads as W


def _case(name, flow, geometry, n, waves, order, ncrit, precision, nrhs=1, groups=0, nt=0, count=0, hi=0):
    c = {"flow": flow, "geometry": geometry, "n": n, "nt": nt or n, "waves": waves, "order": order, "ncrit": ncrit,
         "precision": precision, "nrhs": nrhs, "groups": groups, "count": count, "hi": hi}
    return {"name": name, **c} if name else c


def listed():
    return [
        # the smallest problem of a ragged batch by itself: launches and latency
        _case("sphere_fp64_5k", "apply", "sphere", 5003, 7.9, 4, 64, "fp64"),
        # the drop-in call of the small CPU-runnable workload, numpy in and out
        _case("cube_fp64_20k_host", "host", "cube", 20000, 16.0, 4, 64, "fp64"),
        # a field evaluated away from its sources, a few right-hand sides
        _case("apart_fp64_block3", "apply", "apart", 15001, 6.0, 4, 40, "fp64", nrhs=3, nt=7999),
        # the Laplace operator (every level low-frequency), order 5
        _case("laplace_fp64_60k", "apply", "cube", 60001, 0.0, 5, 64, "fp64"),
        # the like-for-like sample of the large sphere, mixed precision
        _case("sphere_mixed_31k", "apply", "sphere", 31250, 16.0, 5, 64, "mixed"),
        # a volume: dense near field, long far lists, order 6
        _case("blobs_mixed_60k", "apply", "blobs", 59999, 24.0, 6, 64, "mixed"),
        # the drop-in at scale: the large sphere's points per square wavelength
        _case("sphere_fp64_250k", "apply", "sphere", 250000, 45.25, 5, 64, "fp64"),
        # the order-6 spheroid at half a million points
        _case("spheroid_mixed_500k", "apply", "spheroid", 500000, 90.5, 6, 96, "mixed"),
        # the large sphere in mixed precision, the largest call
        _case("sphere_mixed_600k", "apply", "sphere", 600001, 70.1, 5, 64, "mixed"),
        # eight right-hand sides per pass, expansions streamed in direction groups
        _case("sphere_mixed_block8", "apply", "sphere", 250000, 45.25, 5, 64, "mixed", nrhs=8, groups=3),
        # independent problems of uneven size in one graph launch
        _case("ragged_mixed_12", "batch", "ragged", 5000, 8.0, 4, 64, "mixed", count=12, hi=60000),
        # one solve on new points: plan, upload, matvec
        _case("once_fp64_50k", "once", "sphere", 50021, 20.0, 5, 64, "fp64"),
    ]


def draw(rng):
    flow = rng.choice(["apply"] * 7 + ["host", "batch", "once"])
    if flow == "batch":
        lo = int(round(math.exp(rng.uniform(math.log(5000), math.log(12000)))))
        hi = int(round(lo * math.exp(rng.uniform(math.log(2.0), math.log(5.0)))))
        return _case("", flow, "ragged", lo, 8.0, 4, 64, rng.choice(["fp64", "mixed"]),
                     count=rng.randint(4, 12), hi=hi)
    order = rng.choice([4, 4, 5, 5, 5, 6, 6, 7])
    precision = rng.choice(["fp64", "mixed"])
    top = 120e3 if order >= 6 else 250e3
    nrhs = 1
    if flow == "apply" and rng.random() < 0.25:
        nrhs, top = rng.randint(2, 8), 50e3
    n = int(round(math.exp(rng.uniform(math.log(5e3), math.log(top)))))
    waves = math.exp(rng.uniform(math.log(4.0), math.log(64.0)))
    waves = round(max(2.0, min(waves, math.sqrt(n / (25.0 * math.pi)))), 3)
    geometry = rng.choice(["sphere", "cube", "blobs", "spheroid", "apart"])
    if geometry == "cube" and flow == "apply" and rng.random() < 0.25:
        waves = 0.0
    ncrit = rng.choice([48, 64]) if n < 20000 else rng.choice([48, 64, 96])
    nt = n if geometry != "apart" else int(round(n * rng.uniform(0.4, 1.0)))
    return _case("", flow, geometry, n, waves, order, ncrit, precision, nrhs=nrhs, nt=nt)


# ------------------------------------------------------------------- inputs
def _points(case, seed):
    """(sources, targets, wavenumber)"""
    g, n, waves = case["geometry"], case["n"], case["waves"]
    if g == "sphere":
        p = W.sphere_surface(n, seed=seed).points
        return p, p, 2.0 * math.pi * waves / 2.0
    if g == "cube":
        p = W.cube_surface(n, seed=seed).points
    elif g == "blobs":
        p = W.gaussian_blobs(n, seed=seed).points
    elif g == "spheroid":
        p = W.spheroid(n, seed=seed).points
        return p, p, 2.0 * math.pi * waves / 2.0
    else:
        p = W.gaussian_blobs(n, seed=seed).points
        return p, W.sphere_surface(case["nt"], seed=seed + 1).points * 0.45, 2.0 * math.pi * waves / math.sqrt(3.0)
    return p, p, 2.0 * math.pi * waves / math.sqrt(3.0)


def _ragged(case, seed):
    """The batch's members as single cases: sizes log-spaced, geometries and
    orders cycling, 25 points per square wavelength at most."""
    out = []
    for i in range(case["count"]):
        n = int(round(case["n"] * (case["hi"] / case["n"]) ** (i / max(1, case["count"] - 1)))) + i % 2
        waves = max(2.0, min(8.0 * 1.15 ** i, math.sqrt(n / (25.0 * math.pi))))
        out.append((_case("", "apply", ("cube", "sphere", "blobs")[i % 3], n, waves, 4 + i % 3, case["ncrit"],
                          case["precision"]), seed + 7919 * i))
    return out


def _charges(case, seed):
    q = W.charges(case["n"], seed + 1, None if case["nrhs"] == 1 else case["nrhs"])
    return q if case["precision"] == "fp64" else q.astype(np.complex64)


def _operator(case, src, trg, kappa):
    A = IBFMM_Mat()
    A.set_precision(case["precision"])
    A.addSourceParticles(src)
    A.addTargetParticles(trg)
    A.prcmpt(case["order"], case["ncrit"], kappa)
    return A


def _vectors(case, seed):
    """The user's charges and potentials on the device, and the complex128
    vectors of the entry point (the same ones in FP64)."""
    shape = (case["nt"],) if case["nrhs"] == 1 else (case["nrhs"], case["nt"])
    q = torch.from_numpy(_charges(case, seed)).cuda()
    p = torch.empty(shape, dtype=q.dtype, device="cuda")
    if case["precision"] == "fp64":
        return q, p, q, p
    return q, p, torch.empty_like(q, dtype=torch.complex128), torch.empty_like(p, dtype=torch.complex128)


def prepare(case, seed):
    if case["flow"] == "batch":
        members = _ragged(case, seed)
        ops = [_operator(c, *_points(c, s)) for c, s in members]
        vec = [_vectors(c, s) for c, s in members]
        stream = torch.cuda.Stream()
        torch.cuda.synchronize()
        batch = Batch(ops, [v[2].data_ptr() for v in vec], [v[3].data_ptr() for v in vec])
        return {"case": case, "batch": batch, "vec": vec, "stream": stream}
    src, trg, kappa = _points(case, seed)
    if case["flow"] == "once":
        return {"case": case, "src": src, "trg": trg, "kappa": kappa, "q": _charges(case, seed)}
    A = _operator(case, src, trg, kappa)
    if case["nrhs"] > 1:
        A.set_blocking(case["nrhs"], case["groups"])
    else:
        A.autotune()
    if case["flow"] == "host":
        q = _charges(case, seed)
        return {"case": case, "A": A, "q": q, "p": np.empty(case["nt"], dtype=q.dtype)}
    stream = torch.cuda.Stream()
    vec = _vectors(case, seed)
    torch.cuda.synchronize()
    return {"case": case, "A": A, "vec": vec, "stream": stream}


# --------------------------------------------------------------------- pass
def run(state):
    case = state["case"]
    if case["flow"] == "once":
        A = _operator(case, state["src"], state["trg"], state["kappa"])
        return A.matvec(state["q"])
    if case["flow"] == "host":
        gemv(state["A"], state["q"], state["p"])
        return state["p"]
    with torch.cuda.stream(state["stream"]):
        sid = state["stream"].cuda_stream
        if case["flow"] == "batch":
            for q, p, dq, dp in state["vec"]:
                if dq is not q:
                    dq.copy_(q)
            state["batch"].launch(sid)
            for q, p, dq, dp in state["vec"]:
                if dp is not p:
                    p.copy_(dp)
            return [v[1] for v in state["vec"]]
        q, p, dq, dp = state["vec"]
        if dq is not q:
            dq.copy_(q)
        state["A"].matvec_device(dq.data_ptr(), dp.data_ptr(), case["nrhs"], sid)
        if dp is not p:
            p.copy_(dp)
        return p


# --------------------------------------------------------------------- work
def work(case):
    """Bytes: points read, charges read and potentials written once.  Flops:
    one complex multiply-add per spectrum entry of every far pair and per
    particle interaction (whose kernel value, about 20 flops, serves both
    points of a pair when sources and targets are the same set), the
    separable transfers and the leaf interpolations, by the plan's counts."""
    total = {"bytes": 0.0, "flops": 0.0}
    for c, s in (_ragged(case, 1) if case["flow"] == "batch" else [(case, 1)]):
        src, trg, kappa = _points(c, s)
        A = _operator(c, src, trg, kappa)
        i, L, R = A.info(), c["order"], c["nrhs"]
        same = c["geometry"] != "apart"
        item = 16 if c["precision"] == "fp64" else 8
        total["bytes"] += (24 + item * R) * (c["n"] + c["nt"])
        total["flops"] += (20.0 * i["i_near"] * (0.5 if same else 1.0) + R * (
            8.0 * i["i_near"] + 8.0 * (2 * L - 1) ** 3 * (i["far_hf"] + i["far_lf"])
            + 12.0 * L ** 4 * (i["m2m_entries"] + i["l2l_entries"])
            + 4.0 * L ** 3 * (i["p2m_point_slots"] + i["l2p_point_slots"])))
    return total


# -------------------------------------------------------------------- exact
def _direct(case, src, trg, kappa, q):
    """sum_j exp(i k r) / (4 pi r) q_j in FP64 (0 at r = 0), all targets."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    s = torch.from_numpy(src).to(dev)
    t = torch.from_numpy(trg).to(dev)
    z = torch.from_numpy(np.atleast_2d(q.astype(np.complex128))).to(dev).T
    z = torch.cat([z.real, z.imag], dim=1).contiguous()
    R = z.shape[1] // 2
    out = torch.empty((len(trg), R), dtype=torch.complex128, device=dev)
    step = max(1, int(2e8) // len(src))
    for a in range(0, len(trg), step):
        x = t[a:a + step]
        r = (x[:, 0:1] - s[None, :, 0]).square_()
        r += (x[:, 1:2] - s[None, :, 1]).square_()
        r += (x[:, 2:3] - s[None, :, 2]).square_()
        r.sqrt_()
        g = r.reciprocal().mul_(1.0 / (4.0 * math.pi))
        g.masked_fill_(r < 1e-8, 0.0)
        r *= kappa
        c = torch.cos(r).mul_(g) @ z
        e = r.sin_().mul_(g) @ z
        out[a:a + step] = torch.complex(c[:, :R] - e[:, R:], c[:, R:] + e[:, :R])
    out = out.T.contiguous()
    return out[0] if q.ndim == 1 else out


def exact(case, seed):
    if case["flow"] == "batch":
        members = _ragged(case, seed)
        return [_direct(c, *_points(c, s), _charges(c, s)) for c, s in members]
    if case["n"] * case["nt"] > 1e11:
        return None
    src, trg, kappa = _points(case, seed)
    p = _direct(case, src, trg, kappa, _charges(case, seed))
    return p.cpu().numpy() if case["flow"] in ("host", "once") else p
