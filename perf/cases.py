"""The work that programs on this library give it, as measurable cases.

A case is a dict of plain values:

  kind       solve     tree build + plan set-up + evaluation on device arrays (one time step of a
                       particle code: the points moved, so everything is new)
             evaluate  evaluation alone with the tree and plan kept (an iterative solver: fixed
                       points, new charges every call)
             dropin    the reference library's own call sequence on host arrays
                       (Box, OctreePartitioner.refine, FMM3D, evaluate)
             batch     several small independent point sets in one call (host arrays)
             serve     a burst of requests of mixed size to the serving loop (host arrays)
             direct    direct sums at sampled targets, the accuracy check every user runs
  dist       uniform | plummer | shell | gauss2, the distributions of simplefmm_b200.workloads
  n, p       points, expansion order
  leaf       most points in a leaf
  qdim       1: scalar charges, field sum q R/|R|^3; 3: vector charges, Biot-Savart field
  precision  fp64 | mixed
  pot, field which outputs are wanted
  sets       batch / serve: number of point sets or requests; their sizes lie between `n_min` and `n`, the
             same for every seed
  targets    direct: number of targets
"""
from __future__ import annotations

import math

import numpy as np
import torch

import simplefmm_b200 as sf


def _case(name=None, **kw):
    c = dict(kind="solve", dist="plummer", n=100_000, p=10, leaf=64, qdim=1, precision="fp64", pot=True, field=True)
    c.update(kw)
    if name:
        c = dict(name=name, **c)
    return c


def listed():
    return [
        # the smallest drop-in call: a few thousand points in host memory, where latency and launches count
        _case("dropin_2k_p10", kind="dropin", n=2_000, p=10),
        # a batch of small sets that share a plan, ragged sizes
        _case("batch_8x10k_p10", kind="batch", sets=8, n=12_000, n_min=6_000, p=10),
        # the reference's own CPU-sized problem: 100k uniform points, p = 8
        _case("solve_100k_uniform_p8", dist="uniform", n=100_000, p=8),
        # one time step of a small particle run in mixed precision at low order, a ragged size
        _case("solve_50k_shell_p6_mixed", dist="shell", n=50_021, p=6, precision="mixed"),
        # an iterative solver: points fixed, evaluation with new charges, an odd size
        _case("evaluate_300k_p10", kind="evaluate", n=300_007, p=10),
        # vortex / magnetostatics: vector charges, vector potential and Biot-Savart field
        _case("solve_60k_biot_savart_p8", dist="shell", n=60_013, p=8, qdim=3),
        # potential alone (energies) of a clustered set at low order
        _case("solve_400k_gauss2_p6_pot", dist="gauss2", n=400_000, p=6, field=False),
        # the headline workload: 4M Plummer points, p = 10, FP64
        _case("solve_4M_plummer_p10", n=4_000_000, p=10),
        # a mid-sized mixed-precision step
        _case("solve_1M_plummer_p10_mixed", n=1_000_003, p=10, precision="mixed"),
        # the large mixed-precision workload: 16M uniform points, p = 12, its best leaf size
        _case("solve_16M_uniform_p12_mixed", dist="uniform", n=16_000_000, p=12, leaf=128, precision="mixed"),
        # the serving loop: a burst of requests of mixed size, distribution and order
        _case("serve_24_mixed", kind="serve", sets=24, n_min=1_000, n=300_000, precision="mixed"),
        # the accuracy check against direct sums at 10,000 sampled targets
        _case("direct_400k_10k", kind="direct", n=400_000, targets=10_000),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "solve", "evaluate", "evaluate", "dropin", "batch", "serve", "direct"])
    dist = rng.choice(["uniform", "plummer", "shell", "gauss2"])
    p = rng.choice([4, 5, 6, 7, 8, 9, 10, 11, 12])
    leaf = rng.choice([32, 64, 64, 128])
    precision = rng.choice(["fp64", "fp64", "mixed"])
    qdim = 3 if kind in ("solve", "evaluate", "dropin") and rng.random() < 0.2 else 1
    outs = rng.choice([(True, True), (True, True), (True, False), (False, True)])
    c = dict(dist=dist, p=p, leaf=leaf, qdim=qdim, precision=precision, pot=outs[0], field=outs[1])
    if kind in ("solve", "evaluate"):
        top = 4_000_000 if precision == "mixed" else 1_200_000
        return _case(kind=kind, n=_log(rng, 1_000, top // 4 if qdim == 3 or leaf == 32 else top), **c)
    if kind == "dropin":
        return _case(kind=kind, n=_log(rng, 1_000, 250_000), **c)
    c.update(pot=True, field=True)
    if kind == "batch":
        return _case(kind=kind, sets=rng.randint(2, 16), n_min=1_000, n=_log(rng, 2_000, 40_000), **c)
    if kind == "serve":
        return _case(kind=kind, sets=rng.randint(6, 30), n_min=1_000, n=_log(rng, 20_000, 300_000), **c)
    return _case(kind=kind, n=_log(rng, 10_000, 800_000), targets=rng.randint(500, 10_000), **c)


# ------------------------------------------------------------------ inputs
def _points(dist, n, g):
    """n x 3 positions on the GPU; the distributions of simplefmm_b200.workloads."""
    def u(*shape):
        return torch.rand(*shape, generator=g, device="cuda", dtype=torch.float64)

    if dist == "uniform":
        return u(n, 3)
    if dist == "gauss2":                                     # sigma 0.05, centres 0.5 apart in the unit cube
        x = 0.5 + 0.05 * torch.randn(n, 3, generator=g, device="cuda", dtype=torch.float64)
        x[: n // 2, 0] -= 0.25
        x[n // 2:, 0] += 0.25
        return x.clamp_(0.0, 1.0)
    if dist == "plummer":                                    # scale radius 1, radii up to 10
        top = (1.0 + 1.0 / 100.0) ** -1.5
        r = ((u(n).clamp_min_(1e-12) * top) ** (-2.0 / 3.0) - 1.0) ** -0.5
    elif dist == "shell":                                    # radius 1, thickness 0.01, uniform in volume
        a, b = 0.995 ** 3, 1.005 ** 3
        r = (a + (b - a) * u(n)) ** (1.0 / 3.0)
    else:
        raise ValueError(dist)
    ct = 2.0 * u(n) - 1.0
    ph = (2.0 * math.pi) * u(n)
    st = (1.0 - ct * ct).sqrt()
    return torch.stack([r * st * ph.cos(), r * st * ph.sin(), r * ct], dim=1).contiguous()


def _charges(n, qdim, g):
    q = 2.0 * torch.rand(n, qdim, generator=g, device="cuda", dtype=torch.float64) - 1.0
    return q[:, 0].contiguous() if qdim == 1 else q


def _sizes(case):
    """Sizes of a batch's or burst's sets: spread over n_min .. n on a log scale, in a fixed mixed order."""
    k, lo, hi = case["sets"], math.log(case["n_min"]), math.log(max(case["n"], case["n_min"]))
    return [int(math.exp(lo + (hi - lo) * ((0.37 + 0.618034 * i) % 1.0))) for i in range(k)]


def _members(case, g):
    """(positions, charges, order) of each set, on the GPU."""
    out = []
    for i, n in enumerate(_sizes(case)):
        dist, p = case["dist"], case["p"]
        if case["kind"] == "serve":
            dist, p = ("uniform", "plummer", "shell")[i % 3], (6, 10)[i % 2]
        out.append((_points(dist, n, g), _charges(n, 1, g), p))
    return out


def _inputs(case, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    if case["kind"] in ("batch", "serve"):
        return _members(case, g)
    pos, q = _points(case["dist"], case["n"], g), _charges(case["n"], case["qdim"], g)
    if case["kind"] == "direct":
        t = torch.randint(case["n"], (case["targets"],), generator=g, device="cuda")
        return pos, q, t
    return pos, q


_contexts = {}


def _context(host):
    """The process's contexts: one on torch's current stream for device arrays, one on its own stream for host arrays."""
    if host not in _contexts:
        _contexts[host] = sf.Context(0)
        if not host:
            _contexts[host].set_stream(torch.cuda.current_stream().cuda_stream)
    return _contexts[host]


def prepare(case, seed):
    kind, inputs = case["kind"], _inputs(case, seed)
    ctx = _context(kind not in ("solve", "evaluate"))
    s = dict(case=case, kind=kind, ctx=ctx)
    if kind in ("batch", "serve"):
        s["sets"] = [(x.cpu().numpy(), q.cpu().numpy(), p) for x, q, p in inputs]
        if kind == "serve":
            s["server"] = sf.Server(0, slots=4, memory_budget=32 << 30)
        return s
    if kind == "direct":
        s["pos"], s["q"], s["t"] = (x.cpu().numpy() for x in inputs)
        return s
    if kind == "dropin":
        s["pos"], s["q"] = (x.cpu().numpy() for x in inputs)
        return s
    s["pos"], s["q"] = inputs
    n, qd = case["n"], case["qdim"]
    s["pot"] = torch.zeros((n,) if qd == 1 else (n, qd), dtype=torch.float64, device="cuda") if case["pot"] else None
    s["field"] = torch.zeros((n, 3), dtype=torch.float64, device="cuda") if case["field"] else None
    if kind == "evaluate":
        s["tree"] = sf.Tree(s["pos"], 20, case["leaf"], ctx=ctx)
        s["plan"] = sf.Plan(s["tree"], case["p"], qd, precision=case["precision"])
    return s


def run(s):
    c, kind = s["case"], s["kind"]
    if kind in ("solve", "evaluate"):
        for u in (s["pot"], s["field"]):                      # the library accumulates
            if u is not None:
                u.zero_()
        if kind == "solve":
            tree = sf.Tree(s["pos"], 20, c["leaf"], ctx=s["ctx"])
            plan = sf.Plan(tree, c["p"], c["qdim"], precision=c["precision"])
            plan.evaluate(s["q"], s["pot"], s["field"])
            plan.close()
            tree.close()
        else:
            s["plan"].evaluate(s["q"], s["pot"], s["field"])
        return [u for u in (s["pot"], s["field"]) if u is not None]
    if kind == "dropin":
        n, qd = c["n"], c["qdim"]
        part = sf.OctreePartitioner(s["pos"], sf.Box(s["pos"]), ctx=s["ctx"]).refine(20, c["leaf"])
        fmm = sf.FMM3D(part, c["p"], qd, precision=c["precision"])
        pot = np.zeros((n,) if qd == 1 else (n, qd)) if c["pot"] else None
        field = np.zeros((n, 3)) if c["field"] else None
        fmm.evaluate(s["q"], pot, field)
        return [u for u in (pot, field) if u is not None]
    if kind == "batch":
        return sf.solve_batch([(x, q) for x, q, _ in s["sets"]], c["p"], 1, precision=c["precision"], leaf=c["leaf"],
                              ctx=s["ctx"])
    if kind == "serve":
        ids = [s["server"].submit(x, q, p, precision=c["precision"], leaf=c["leaf"]) for x, q, p in s["sets"]]
        return [s["server"].wait(i)[:2] for i in ids]
    return sf.direct(s["pos"], s["q"], s["t"], ctx=s["ctx"])


# ------------------------------------------------------------------ exact values
def _direct64(pos, q, pot, field, targets=None):
    """Direct sums in 64 bits: pot_i = sum q_j / r, field_i = sum q_j R / r^3 (scalar charges) or
    sum q_j x R / r^3 (vector charges), R = x_i - x_j."""
    n = pos.shape[0]
    idx = torch.arange(n, device="cuda") if targets is None else targets
    vec = q.dim() == 2
    xs = [pos[:, k].contiguous() for k in range(3)]
    chunk = max(1, (1 << 28) // n)
    ps, fs = [], []
    for t in idx.split(chunk):
        d = [xs[k][t][:, None] - xs[k][None, :] for k in range(3)]
        w = (d[0] * d[0] + d[1] * d[1] + d[2] * d[2]).rsqrt()
        w[torch.arange(t.numel(), device="cuda"), t] = 0.0
        if pot:
            ps.append(w @ q)
        if field:
            w = w * w * w
            if vec:
                f = [[(w * d[k]) @ q[:, b] for k in range(3)] for b in range(3)]      # f[b][k] = sum q_b R_k / r^3
                fs.append(torch.stack([f[1][2] - f[2][1], f[2][0] - f[0][2], f[0][1] - f[1][0]], dim=1))
            else:
                fs.append(torch.stack([(w * d[k]) @ q for k in range(3)], dim=1))
    return (torch.cat(ps) if pot else None), (torch.cat(fs) if field else None)


def _pairs(case):
    if case["kind"] in ("batch", "serve"):
        return sum(n * n for n in _sizes(case))
    return case["n"] * case.get("targets", case["n"])


def exact(case, seed):
    if _pairs(case) > 2.5e11:                                 # the direct sum of all targets would take too long
        return None
    inputs = _inputs(case, seed)
    if case["kind"] in ("batch", "serve"):
        return [tuple(v.cpu().numpy() for v in _direct64(x, q, True, True)) for x, q, _ in inputs]
    if case["kind"] == "direct":
        return tuple(v.cpu().numpy() for v in _direct64(inputs[0], inputs[1], True, True, inputs[2]))
    out = [v for v in _direct64(inputs[0], inputs[1], case["pot"], case["field"]) if v is not None]
    return [v.cpu().numpy() for v in out] if case["kind"] == "dropin" else out


# ------------------------------------------------------------------ what a pass cannot do without
def _solve_work(n, p, leaf, qdim, pot, field):
    """Inputs and outputs once; near-field pairs and interaction-list translations of a tree whose leaves are a third
    full: 27 neighbour boxes a target (11 flops a pair for the potential, 9 for the field), 160 translations a box, each
    rotated, translated along z and rotated back."""
    fill = max(1.0, 0.33 * leaf)
    boxes = 1.15 * n / fill
    out = (qdim if pot else 0) + (3 if field else 0)
    near = n * min(n, 27 * fill) * qdim * ((11 if pot else 6) + (9 if field else 0))
    rot = 2 * sum((k + 1) ** 2 for k in range(p + 1))
    tz = 2 * sum((p + 1 - k) ** 2 for k in range(p + 1))
    back = rot * (int(pot) + int(field))
    far = 160 * boxes * qdim * 2 * (rot + tz + back) if n > 64 * leaf else 0
    return 8 * n * (3 + qdim + out), near + far


def work(case):
    k = case["kind"]
    if k == "direct":
        t = case["targets"]
        return {"bytes": 8 * (4 * case["n"] + 5 * t), "flops": 20.0 * t * case["n"]}
    if k in ("batch", "serve"):
        orders = [case["p"] if k == "batch" else (6, 10)[i % 2] for i in range(case["sets"])]
        w = [_solve_work(n, p, case["leaf"], 1, True, True) for n, p in zip(_sizes(case), orders)]
        return {"bytes": sum(a for a, _ in w), "flops": float(sum(b for _, b in w))}
    b, f = _solve_work(case["n"], case["p"], case["leaf"], case["qdim"], case["pot"], case["field"])
    return {"bytes": b, "flops": float(f)}
