"""Performance cases: what users of the magnetization-and-force library have it do.

``listed()`` names the cases, ``draw()`` gives more of the same ranges,
``prepare()`` makes a case's inputs and handles, ``run()`` is one pass through
the public entry points (the Python binding of ``include/mf.h``), ``work()``
what a pass cannot do without and ``exact()`` its outputs in plain FP64 torch.

Kinds
-----
object   One object from scratch, as a caller of the reference's class has it:
         construct, solve, force, read M, B and F back to the host.
step     One timestep of a resident object: the caller's moved positions in
         (device memory), the warm-started solve, the Kelvin force, B and F out
         (device memory).  The last step's b meets the tolerance, as it does at
         the timesteps such simulations run at.
sweep    A resident body in the field of a permanent magnet (external dipoles)
         and a uniform field that turns: for each of two directions the external
         field and its gradient, a solve, the force.
batch    A few graph-replayed timesteps of many independent objects, then B and F
         of every object read back.
probe    Field and force tensor of given dipoles at separate probe points, on
         device arrays, direct summation.
matrix   The same through the FMM matrix, host arrays.
"""
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_PKG = os.path.join(ROOT, "magnetic-force_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import mfgb  # noqa: E402

DEV = "cuda"
MU0 = 1.25663706e-6


def listed():
    return [
        # A small object through the reference's class with its default solver
        # (NLCG): the size of the reference's own demo grids.  Launches, host
        # round trips and allocations count here.
        {"name": "object_1k", "kind": "object", "n": 1000, "shape": "sphere", "precision": "fp32", "chi": 2.0},
        # The FP64 configuration: 4,096 uniformly random particles, CG to 1e-8.
        {"name": "object_fp64_4k", "kind": "object", "n": 4096, "shape": "cube", "precision": "fp64", "chi": 1.0},
        # Timesteps of resident objects: a small one, a mid-sized one of an odd
        # count, and the benchmark's 65,536-particle sphere.
        {"name": "step_3k", "kind": "step", "n": 3001, "shape": "sphere", "chi": 2.0},
        {"name": "step_16k", "kind": "step", "n": 16411, "shape": "sphere", "chi": 1.0},
        {"name": "step_65k", "kind": "step", "n": 65536, "shape": "sphere", "chi": 2.0},
        # A body between the poles of a magnet: solves that iterate, and the
        # external dipoles' field and gradient tensor.
        {"name": "sweep_12k", "kind": "sweep", "n": 12289, "n_ext": 6000, "shape": "cylinder", "chi": 1.5},
        # Many objects together: a small mixed batch and the 256-scene one.
        {"name": "batch_24", "kind": "batch", "scenes": 24, "lo": 512, "hi": 8192},
        {"name": "batch_256", "kind": "batch", "scenes": 256, "lo": 512, "hi": 32768},
        # Field maps around a body: more sources than probe points, odd counts.
        {"name": "probe_10k", "kind": "probe", "n": 40001, "nt": 9973, "shape": "sphere"},
        {"name": "matrix_150k", "kind": "matrix", "n": 150000, "nt": 30011, "shape": "cylinder"},
        # Timesteps of large objects (FMM): the served stream's large requests
        # and the 1,048,576-particle cylinder.
        {"name": "step_200k", "kind": "step", "n": 200003, "shape": "sphere", "chi": 1.5},
        {"name": "step_1m", "kind": "step", "n": 1048576, "shape": "cylinder", "chi": 1.5},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["object", "object", "step", "step", "step", "step", "sweep", "batch", "probe", "matrix"])
    shape = rng.choice(["sphere", "cylinder"])
    if kind == "object":
        if rng.random() < 0.5:
            return {"kind": kind, "n": _log(rng, 700, 4096), "shape": rng.choice(["cube", "sphere"]),
                    "precision": "fp64", "chi": round(rng.uniform(0.5, 1.5), 3)}
        return {"kind": kind, "n": _log(rng, 250, 6000), "shape": shape, "precision": "fp32",
                "chi": round(rng.uniform(0.5, 3.0), 3)}
    if kind == "step":
        return {"kind": kind, "n": _log(rng, 800, 350000), "shape": shape, "chi": round(rng.uniform(0.5, 3.0), 3)}
    if kind == "sweep":
        return {"kind": kind, "n": _log(rng, 1000, 20000), "n_ext": _log(rng, 100, 12000), "shape": shape,
                "chi": round(rng.uniform(0.5, 2.0), 3)}
    if kind == "batch":
        lo = rng.choice([512, 1024])
        return {"kind": kind, "scenes": rng.randint(8, 96), "lo": lo, "hi": _log(rng, 4096, 24000)}
    if kind == "probe":
        return {"kind": kind, "n": _log(rng, 1500, 60000), "nt": _log(rng, 700, 40000), "shape": shape}
    return {"kind": kind, "n": _log(rng, 50000, 300000), "nt": _log(rng, 5000, 60000), "shape": shape}


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _cloud(n, shape, radius, height, seed):
    """A cubic lattice jittered by a quarter of its spacing and clipped to a
    sphere (radius) or a cylinder (radius, height), exactly n points (the ones
    farthest out are dropped).  Returns float32 [n, 3] on the GPU, the spacing
    and the particle volume."""
    vs = 4.0 / 3.0 * math.pi * radius ** 3 if shape == "sphere" else math.pi * radius ** 2 * height
    s = (vs / n) ** (1.0 / 3.0)
    ext = (radius, radius, radius if shape == "sphere" else 0.5 * height)
    while True:
        s *= 0.985
        g = torch.Generator(device=DEV)
        g.manual_seed(seed)
        ax = [torch.arange(-math.ceil(e / s) - 1, math.ceil(e / s) + 2, device=DEV, dtype=torch.float64) * s
              for e in ext]
        p = torch.stack(torch.meshgrid(*ax, indexing="ij"), dim=-1).reshape(-1, 3)
        p = p + (torch.rand(p.shape, generator=g, device=DEV, dtype=torch.float64) - 0.5) * (0.5 * s)
        if shape == "sphere":
            key = p.norm(dim=1) / radius
        else:
            key = torch.maximum(p[:, :2].norm(dim=1) / radius, p[:, 2].abs() / (0.5 * height))
        if int((key <= 1.0).sum()) >= n:
            keep = torch.sort(torch.argsort(key, stable=True)[:n]).values
            return p[keep].to(torch.float32).contiguous(), s, vs / n


def _body(case, seed):
    """Positions (GPU float32), h and particle volume of a single-object case."""
    n, shape = case["n"], case["shape"]
    if shape == "cube":
        g = torch.Generator(device=DEV)
        g.manual_seed(seed)
        vol = 1.0 / n
        return torch.rand((n, 3), generator=g, device=DEV), 2.0 * vol ** (1.0 / 3.0), vol
    radius, height = (0.5, 0.0) if shape == "sphere" else (0.3, 1.0)
    p, s, vol = _cloud(n, shape, radius, height, seed)
    return p, 2.0 * s, vol


def _moments(p, vol, seed):
    """Magnetization of a body in a field along z: near-uniform, with spread."""
    g = torch.Generator(device=DEV)
    g.manual_seed(seed + 7)
    m = 0.3 * torch.randn(p.shape, generator=g, device=DEV)
    m[:, 2] += 1.0
    return (m * vol).contiguous()


def _probe_points(case, p, seed):
    """Probe points in a box a little larger than the body."""
    g = torch.Generator(device=DEV)
    g.manual_seed(seed + 13)
    lo, hi = p.min(dim=0).values, p.max(dim=0).values
    u = torch.rand((case["nt"], 3), generator=g, device=DEV)
    return (lo - 0.1 * (hi - lo) + u * (1.2 * (hi - lo))).contiguous()


def _sweep_magnet(case, seed):
    """Two blocks of dipoles (poles of a magnet) beyond the body's ends."""
    rng = np.random.default_rng(seed + 3)
    k = case["n_ext"]
    pos = rng.uniform(-0.4, 0.4, size=(k, 3))
    pos[:, 2] = np.where(np.arange(k) % 2 == 0, 1.0, -1.0) * rng.uniform(0.7, 1.0, size=k)
    mom = rng.normal(scale=0.1, size=(k, 3)) + np.array([0.0, 0.0, 1.0])
    return pos.astype(np.float32), (mom * (0.4 / k)).astype(np.float32)


def _sweep_fields(seed):
    a = 0.3 + 0.1 * (seed % 7)
    return [(math.sin(t), 0.0, math.cos(t)) for t in (a, a + 0.6)]


class _Scene:
    def __init__(self, pos, h, volume, chi, H0):
        self.pos, self.h, self.volume, self.chi, self.H0 = pos, h, volume, chi, H0


def _batch_scenes(case, seed):
    # counts log-uniform, the same for every seed: outputs keep their shape
    sizes = np.random.default_rng(case["scenes"]).uniform(math.log(case["lo"]), math.log(case["hi"]), case["scenes"])
    rng = np.random.default_rng(seed)
    out = []
    for i in range(case["scenes"]):
        n = int(round(math.exp(sizes[i])))
        radius, chi = float(rng.uniform(0.2, 0.5)), float(rng.uniform(0.5, 3.0))
        H = rng.normal(size=3)
        H /= np.linalg.norm(H)
        p, s, vol = _cloud(n, "sphere", radius, 0.0, seed + i)
        out.append(_Scene(p.cpu().numpy(), 2.0 * s, vol, chi, tuple(float(v) for v in H)))
    return out


BATCH_DT, BATCH_STEPS = 1e-6, 4


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        scenes = _batch_scenes(case, seed)
        b = mfgb.Batch(scenes)
        b.solve(200, 3e-7)
        b.advance(BATCH_DT, BATCH_STEPS, iters_per_step=4, rel_tol=1e-6, graph=True)
        return {"kind": kind, "batch": b}
    p, h, vol = _body(case, seed)
    n = case["n"]
    if kind == "object":
        return {"kind": kind, "pos": p.cpu().numpy(), "h": h, "vol": vol, "chi": case["chi"],
                "precision": case["precision"]}
    if kind == "step":
        s = mfgb.Solver(n, h, h, vol, case["chi"], (0.0, 0.0, 1.0), None, None, p.cpu().numpy())
        s.set_option("solver", mfgb.SOLVER_CG)
        s.set_option("rel_tol", 3e-7)
        s.solve(200)
        s.set_option("rel_tol", 1e-6)
        return {"kind": kind, "solver": s, "pos": p, "B": torch.empty_like(p), "F": torch.empty_like(p)}
    if kind == "sweep":
        sp, sm = _sweep_magnet(case, seed)
        fields = _sweep_fields(seed)
        s = mfgb.Solver(n, h, 2.0 * h, vol, case["chi"], fields[-1], sp, sm, p.cpu().numpy())
        s.set_option("solver", mfgb.SOLVER_CG)
        s.solve(200)
        return {"kind": kind, "solver": s, "fields": fields, "sp": sp, "sm": sm, "ext_h": 2.0 * h,
                "B": [torch.empty_like(p) for _ in fields], "F": [torch.empty_like(p) for _ in fields]}
    m = _moments(p, vol, seed)
    t = _probe_points(case, p, seed)
    if kind == "probe":
        return {"kind": kind, "t": t, "p": p, "m": m, "h": h}
    a = mfgb.FmmMatrix(p.cpu().numpy(), h, targets=t.cpu().numpy())
    return {"kind": kind, "matrix": a, "m": m.cpu().numpy()}


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------
def run(state):
    kind = state["kind"]
    if kind == "object":
        fp64 = state["precision"] == "fp64"
        s = mfgb.Solver(len(state["pos"]), state["h"], state["h"], state["vol"], state["chi"], (0.0, 0.0, 1.0), None,
                        None, state["pos"], precision=state["precision"])
        if fp64:
            s.set_option("solver", mfgb.SOLVER_CG)
        else:
            s.tolerance = 1e-4
        s.solve(200)
        s.evaluate_fitted_near_foece()
        out = {"M": s.get("M", f64=fp64), "B": s.get("total_B_over_mu0", f64=fp64),
               "F": s.get("magnetic_bodyforce", f64=fp64)}
        s.close()
        return out
    if kind == "step":
        s = state["solver"]
        s.set_positions_device(state["pos"].data_ptr(), state["pos"].shape[0])
        s.solve(200)
        s.evaluate_fitted_near_foece()
        s.get_into_device("total_B_over_mu0", state["B"].data_ptr())
        s.get_into_device("magnetic_bodyforce", state["F"].data_ptr())
        return {"B": state["B"], "F": state["F"]}
    if kind == "sweep":
        s = state["solver"]
        for k, H0 in enumerate(state["fields"]):
            s.setHext(H0, state["sp"], state["sm"], state["ext_h"])
            s.solve(200)
            s.evaluate_fitted_near_foece()
            s.get_into_device("total_B_over_mu0", state["B"][k].data_ptr())
            s.get_into_device("magnetic_bodyforce", state["F"][k].data_ptr())
        return {"B": state["B"], "F": state["F"]}
    if kind == "batch":
        b = state["batch"]
        b.advance(BATCH_DT, BATCH_STEPS, iters_per_step=4, rel_tol=1e-6, graph=True)
        k = range(len(b.sizes))
        return {"B": np.concatenate([b.get(i, "total_B_over_mu0") for i in k]),
                "F": np.concatenate([b.get(i, "magnetic_bodyforce") for i in k])}
    if kind == "probe":
        return {"field": mfgb.direct_field(state["t"], state["p"], state["m"], state["h"]),
                "tensor": mfgb.direct_force_tensor(state["t"], state["p"], state["m"], state["h"])}
    a = state["matrix"]
    return {"field": a.field(state["m"]), "tensor": a.hessian(state["m"])}


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------
# FLOP per unordered pair of one set: the field 49, the force 55, both from
# one evaluation 86; per target-source pair: field 32, tensor 49.  Large sets
# (hierarchical): per particle the pairs inside the kernel's support (4 h, about
# 2,100 at h = 2 spacings, once per unordered pair) and one expansion's upkeep.
_FMM_PER_PARTICLE = 0.5 * 2100 * 86 + 2.0e4


def work(case):
    kind = case["kind"]
    if kind == "batch":
        a, b = math.log(case["lo"]), math.log(case["hi"])
        mean_n = (case["hi"] - case["lo"]) / (b - a)
        mean_n2 = (case["hi"] ** 2 - case["lo"] ** 2) / (2.0 * (b - a))
        return {"bytes": case["scenes"] * mean_n * 60.0, "flops": BATCH_STEPS * case["scenes"] * 0.5 * mean_n2 * 86.0}
    n = case["n"]
    if kind == "object":
        size = 8.0 if case["precision"] == "fp64" else 4.0
        iters = 12  # CG iterations of a cold solve: one field product each
        return {"bytes": n * (12.0 + 9.0 * size), "flops": 0.5 * n * n * (iters * 49.0 + 55.0)}
    if kind == "step":
        return {"bytes": n * 36.0, "flops": 0.5 * n * n * 86.0 if n <= 65536 else n * _FMM_PER_PARTICLE}
    if kind == "sweep":
        iters = 8
        return {"bytes": 2.0 * (n * 36.0 + case["n_ext"] * 24.0),
                "flops": 2.0 * (0.5 * n * n * (iters * 49.0 + 55.0) + n * case["n_ext"] * 70.0)}
    nt = case["nt"]
    flops = nt * n * (32.0 + 49.0) if kind == "probe" else (n + nt) * _FMM_PER_PARTICLE
    return {"bytes": n * 24.0 + nt * 60.0, "flops": flops}


# ---------------------------------------------------------------------------
# The outputs in FP64
# ---------------------------------------------------------------------------
_CURVES = [
    [9.97813616438174e-09, -2.97897856524718e-08, 2.38918644566813e-09, 4.53199938857366e-08, 2.44617454752747e-11,
     6.69550479838731e-08, -1.61753307173877e-07, 1.68213714992711e-08, 1.34558143036838e-07, 1.10976027980100e-10],
    [-2.76473728643294e-09, 2.86975546540539e-08, -9.94582836806651e-08, 1.25129924573675e-07, -2.37010166723652e-08,
     -3.08460139955194e-08, 2.29192245602275e-07, -5.88399621128587e-07, 5.61170054591844e-07, -1.14421132829680e-07],
    [-1.09679990621465e-09, 9.77055663264614e-09, -2.54781238661150e-08, 2.65020634884934e-09, 5.00787562417835e-08,
     3.50477408060213e-09, -5.25956271895141e-08, 2.78876509535747e-07, -6.24199554212217e-07, 4.91807818904985e-07],
    [3.79927162333632e-10, -6.26368404962679e-09, 3.94760528277489e-08, -1.13580541622200e-07, 1.27491333574323e-07,
     7.33485346367840e-10, -9.58855788627803e-09, 4.37085309763591e-08, -7.48004594092261e-08, 2.34161209605651e-08],
]
_CHUNK = 1 << 25


def _pairs(t, p):
    """Offsets and squared distances of a chunk of targets to all sources."""
    d = [t[:, k, None] - p[None, :, k] for k in range(3)]
    return d, d[0] * d[0] + d[1] * d[1] + d[2] * d[2]


def _h32(h):
    return float(np.float32(h))


def _field_coeffs(r2, h):
    """(alpha, beta) of B/mu0 = (3 d (d.m) alpha - m beta) / 4 pi."""
    near = (r2 < 4.0 * h * h).nonzero(as_tuple=True)
    rn = r2[near].sqrt()
    beta = r2.clamp_min(1e-300).pow_(-1.5)
    alpha = beta / r2.clamp_min(1e-300)
    q = rn / h
    tmq3 = (2.0 - q) ** 3
    hi = q >= 1.0
    q3 = q ** 3
    P = q ** 6 / 6.0 - 6.0 * q ** 5 / 5.0 + 3.0 * q ** 4 - 8.0 * q3 / 3.0 + 1.0 / 15.0
    wa = torch.where(hi, -3.0 * P / q3.clamp_min(1e-300), (15.0 * q3 - 36.0 * q * q + 40.0) / 10.0)
    wd = torch.where(hi, tmq3, tmq3 - 4.0 * (1.0 - q) ** 3)
    beta[near] = (wa / 3.0 - wd) / h ** 3
    alpha[near] = torch.where(rn > 0, (wa - wd) / (3.0 * h ** 3 * (rn * rn).clamp_min(1e-300)), torch.zeros_like(rn))
    return alpha, beta


def _field(t, p, m, h):
    out = torch.empty_like(t)
    step = max(1, _CHUNK // len(p))
    for i in range(0, len(t), step):
        d, r2 = _pairs(t[i:i + step], p)
        alpha, beta = _field_coeffs(r2, h)
        w = (d[0] * m[:, 0] + d[1] * m[:, 1] + d[2] * m[:, 2]) * alpha
        s2 = beta @ m
        for k in range(3):
            out[i:i + step, k] = (3.0 * (d[k] * w).sum(dim=1) - s2[:, k]) / (4.0 * math.pi)
    return out


def _tensor_terms(r2, h):
    """(P, Q) of T = P ((d.s) I + s d^T + d s^T) + Q (d.s) d d^T."""
    K = 3.0 * MU0 / (4.0 * math.pi)
    near = (r2 <= 16.0 * h * h).nonzero(as_tuple=True)
    rn = r2[near].sqrt()
    P = K * r2.clamp_min(1e-300).pow_(-2.5)
    Q = -5.0 * P / r2.clamp_min(1e-300)
    q = (rn / h).clamp_max(4.0)
    piece = (q.ceil().long() - 1).clamp_(0, 3)
    tab = torch.tensor(_CURVES, dtype=torch.float64, device=r2.device)
    c1, c2 = torch.zeros_like(q), torch.zeros_like(q)
    for k in range(5):
        c1 = c1 * q + tab[:, k][piece]
        c2 = c2 * q + tab[:, 5 + k][piece]
    r = rn.clamp_min(1e-300)
    zero = torch.zeros_like(rn)
    P[near] = torch.where(rn > 0, c1 / (h ** 4 * r), zero)
    Q[near] = torch.where(rn > 0, (c2 - 3.0 * c1) / (h ** 4 * r ** 3), zero)
    return P, Q


def _tensor(t, p, m, h):
    """[nt, 9]: the symmetric 3 x 3 force tensor at each target."""
    out = torch.empty((len(t), 9), dtype=torch.float64, device=t.device)
    step = max(1, _CHUNK // len(p))
    for i in range(0, len(t), step):
        d, r2 = _pairs(t[i:i + step], p)
        P, Q = _tensor_terms(r2, h)
        ds = d[0] * m[:, 0] + d[1] * m[:, 1] + d[2] * m[:, 2]
        pd = (P * ds).sum(dim=1)
        qd = Q * ds
        Pd = [P * d[k] for k in range(3)]
        for a in range(3):
            for b in range(a, 3):
                v = Pd[b] @ m[:, a] + Pd[a] @ m[:, b] + (qd * d[a] * d[b]).sum(dim=1)
                if a == b:
                    v = v + pd
                out[i:i + step, 3 * a + b] = v
                out[i:i + step, 3 * b + a] = v
    return out


def _contract(T, m):
    return (T.reshape(-1, 3, 3) @ m.unsqueeze(-1)).squeeze(-1)


def _solution(p, h, c, hext):
    """b of (I - c G) b = hext by conjugate gradients to 1e-11."""
    b = hext.clone()
    r = hext - (b - c * _field(p, p, b, h))
    d = r.clone()
    rr = (r * r).sum()
    for _ in range(80):
        if rr.sqrt() <= 1e-11 * hext.norm():
            break
        q = d - c * _field(p, p, d, h)
        a = rr / (d * q).sum()
        b = b + a * d
        r = r - a * q
        new = (r * r).sum()
        d = r + (new / rr) * d
        rr = new
    return b


def _coef(vol, chi):
    v, x = float(np.float32(vol)), float(np.float32(chi))
    return v * x / (x + 1.0)


def _uniform(n, H0):
    return torch.tensor([float(np.float32(v)) for v in H0], dtype=torch.float64, device=DEV).expand(n, 3).clone()


def _solved(p, h, vol, chi, hext, rext=None):
    p, h, c = p.double(), _h32(h), _coef(vol, chi)
    b = _solution(p, h, c, hext)
    m = c * b
    T = _tensor(p, p, m, h)
    return b, m, _contract(T if rext is None else T + rext, m)


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        # the sum of squared counts decides the time
        if work(case)["flops"] > 6.0e11:
            return None
        B, F = [], []
        for sc in _batch_scenes(case, seed):
            b, _, f = _solved(torch.from_numpy(sc.pos).to(DEV), sc.h, sc.volume, sc.chi, _uniform(len(sc.pos), sc.H0))
            B.append(b)
            F.append(f)
        return {"B": torch.cat(B), "F": torch.cat(F)}
    if kind == "step" and case["n"] > 65536:
        return None
    p, h, vol = _body(case, seed)
    n = case["n"]
    if kind == "object":
        b, m, f = _solved(p, h, vol, case["chi"], _uniform(n, (0.0, 0.0, 1.0)))
        return {"M": m, "B": b, "F": f}
    if kind == "step":
        b, _, f = _solved(p, h, vol, case["chi"], _uniform(n, (0.0, 0.0, 1.0)))
        return {"B": b, "F": f}
    if kind == "sweep":
        sp, sm = (torch.from_numpy(v).to(DEV).double() for v in _sweep_magnet(case, seed))
        eh = _h32(2.0 * h)
        ext, rext = _field(p.double(), sp, sm, eh), _tensor(p.double(), sp, sm, eh)
        B, F = [], []
        for H0 in _sweep_fields(seed):
            b, _, f = _solved(p, h, vol, case["chi"], _uniform(n, H0) + ext, rext)
            B.append(b)
            F.append(f)
        return {"B": B, "F": F}
    m, t = _moments(p, vol, seed).double(), _probe_points(case, p, seed).double()
    p, h = p.double(), _h32(h)
    if kind == "matrix":
        # both products stay within a few seconds up to this size
        if n * case["nt"] > 1.0e10:
            return None
    return {"field": _field(t, p, m, h), "tensor": _tensor(t, p, m, h)}
