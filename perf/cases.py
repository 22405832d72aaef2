"""What this framework's speed is measured on: one pass of each thing that a user has it do.

A case is a dict of plain values. `kind` names the call; the sizes, the distribution and the options
are its parameters. Inputs are the seeded synthetic distributions that the benchmark and the tests use
(uniform cube, truncated Plummer sphere, mixture of Plummer subclusters). Two ways in are
used, as users use them: the numpy frontends (host arrays in and out) for the interactive sizes and
for the contexts that return float32, and the C ABI on device arrays where a simulation keeps its particles in
GPU memory. A tree is built from the positions in every pass except by the resident contexts, since
the particles have moved.
"""

import ctypes
import math

import numpy as np
import torch

import pytreegrav_gb300 as tg
from pytreegrav_gb300 import _lib
from pytreegrav_gb300 import cuda as tg_cuda
from pytreegrav_gb300 import theta as tg_theta

FIELD_BITS = {"potential": 1, "accel": 2, "tidal": 4}
FIELD_WIDTH = {"potential": 1, "accel": 3, "tidal": 9}
# algorithmic flops of one point-mass interaction, and what a quadrupole adds to it (add, sub, mul = 1,
# FMA = 2, rsqrt = 1)
FLOPS_MONO = {"potential": 11, "accel": 18, "tidal": 32}
FLOPS_QUAD = {"potential": 27, "accel": 38, "tidal": 80}
FUNCTIONS = {"potential": tg.Potential, "accel": tg.Accel, "tidal": tg.TidalTensor}
TARGET_FUNCTIONS = {"potential": tg.PotentialTarget, "accel": tg.AccelTarget, "tidal": tg.TidalTensorTarget}


def listed():
    return [
        # a few hundred bodies, host arrays, default arguments: the adaptive method takes the exact
        # direct sum (a star cluster's or a planetary system's step; latency is what the user feels)
        {"name": "accel_700", "kind": "direct", "nt": 700, "ns": 700, "mutual": True, "field": "accel", "dist": "plummer"},
        # a tree call at the size of a notebook or of a small simulation, default arguments, host arrays
        {"name": "accel_12k", "kind": "frontend", "n": 12345, "field": "accel", "dist": "plummer", "quadrupole": False,
         "theta": 0.7, "precision": "fp32", "h": 0.01},
        # the benchmark's plain configuration: 1e5 in the unit cube, potential and acceleration of one
        # field object from host arrays, default grouping
        {"name": "field_100k", "kind": "field", "n": 100000, "fields": "potential,accel", "dist": "uniform",
         "quadrupole": False, "theta": 0.7, "precision": "fp32", "h": 0.01},
        # the same object at the precision that a convergence check asks for
        {"name": "field_fp64_50k", "kind": "field", "n": 50000, "fields": "accel", "dist": "plummer",
         "quadrupole": True, "theta": 0.7, "precision": "fp64", "h": 0.01},
        # exact float32 sums against resident sources (the numba-cuda brute-force context's role)
        {"name": "direct_f32_50k", "kind": "direct_f32", "ns": 50001, "nt": 50001, "field": "accel", "dist": "plummer"},
        # a resident tree evaluated at new points, float32 (the numba-cuda tree context's role), its
        # default per-target opening test
        {"name": "context_f32_300k", "kind": "context", "ns": 300000, "nt": 100003, "field": "accel",
         "dist": "clustered", "group_size": 1},
        # the benchmark's headline step on device arrays: build and learned walk of a 1e6 Plummer sphere
        {"name": "learned_1m", "kind": "device", "n": 1000000, "fields": "accel", "dist": "plummer",
         "quadrupole": True, "theta": 0.7, "learned": True, "h": 0.005},
        # every field from one plain walk at 1e6 (the benchmark's precision configuration)
        {"name": "all_fields_1m", "kind": "device", "n": 1000000, "fields": "potential,accel,tidal", "dist": "plummer",
         "quadrupole": True, "theta": 0.7, "learned": False, "h": 0.005},
        # many external points in the field of many more sources, learned walk (a quarter of the
        # benchmark's largest configuration)
        {"name": "targets_8m", "kind": "targets", "ns": 8000000, "nt": 500009, "fields": "potential,accel",
         "quadrupole": True, "theta": 0.7, "learned": True},
        # many independent systems of uneven sizes in one arena: segmented build, walk in a CUDA graph
        {"name": "batched_1024", "kind": "batched", "systems": 1024, "n_min": 256, "n_max": 16384, "theta": 0.7},
        # six axis rays from every particle through spheres of their radii
        {"name": "column_60k", "kind": "column", "n": 60000, "dist": "plummer", "radius": 0.01},
        # the velocity structure function with its default bins, jitter and opening angle
        {"name": "structure_200k", "kind": "structure", "n": 200000, "dist": "plummer"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["direct", "direct", "frontend", "frontend", "field", "direct_f32", "context", "device", "device",
                       "targets", "batched", "column", "structure"])
    dist = rng.choice(["plummer", "plummer", "uniform", "clustered"])
    field = rng.choice(["potential", "accel", "accel", "tidal"])
    quadrupole = rng.random() < 0.5
    theta = rng.choice([0.5, 0.7, 0.7, 1.0])
    if kind == "direct":  # up to where the adaptive method leaves the direct sum
        if rng.random() < 0.5:
            n = _log_int(rng, 20, 1000)
            return {"kind": kind, "nt": n, "ns": n, "mutual": True, "field": field, "dist": dist}
        nt = _log_int(rng, 20, 20000)
        return {"kind": kind, "nt": nt, "ns": _log_int(rng, 20, 1000000 // nt), "mutual": False, "field": field,
                "dist": dist}
    if kind == "frontend":
        return {"kind": kind, "n": _log_int(rng, 1001, 100000), "field": field, "dist": dist, "quadrupole": quadrupole,
                "theta": theta, "precision": "fp32", "h": 0.01}
    if kind == "field":
        precision = rng.choice(["fp32", "fp32", "fp64"])
        return {"kind": kind, "n": _log_int(rng, 2000, 100000 if precision == "fp32" else 50000),
                "fields": rng.choice(["potential,accel", "accel", "potential"]), "dist": dist,
                "quadrupole": quadrupole, "theta": theta, "precision": precision, "h": 0.01}
    if kind == "direct_f32":
        return {"kind": kind, "ns": _log_int(rng, 1000, 50000), "nt": _log_int(rng, 1000, 50000),
                "field": rng.choice(["potential", "accel"]), "dist": dist}
    if kind == "context":
        return {"kind": kind, "ns": _log_int(rng, 10000, 300000), "nt": _log_int(rng, 1000, 100000),
                "field": rng.choice(["potential", "accel"]), "dist": dist, "group_size": rng.choice([1, 1, 8, 32])}
    if kind == "device":
        learned = rng.random() < 0.5
        return {"kind": kind, "n": _log_int(rng, 50000, 1000000), "dist": dist, "quadrupole": quadrupole, "theta": 0.7,
                "fields": "accel" if learned else rng.choice(["accel", "potential,accel", "potential,accel,tidal"]),
                "learned": learned, "h": 0.005}
    if kind == "targets":
        return {"kind": kind, "ns": _log_int(rng, 200000, 8000000), "nt": _log_int(rng, 20000, 500000),
                "fields": rng.choice(["accel", "potential,accel"]), "quadrupole": quadrupole, "theta": 0.7,
                "learned": rng.random() < 0.5}
    if kind == "batched":
        return {"kind": kind, "systems": _log_int(rng, 64, 1024), "n_min": 256, "n_max": rng.choice([2048, 8192, 16384]),
                "theta": rng.choice([0.5, 0.7])}
    if kind == "column":
        return {"kind": kind, "n": _log_int(rng, 2000, 60000), "dist": dist, "radius": rng.choice([0.003, 0.01])}
    return {"kind": "structure", "n": _log_int(rng, 5000, 200000), "dist": dist}


# ---------------------------------------------------------------------------------------------
# Inputs, made on the GPU from the seed.


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(1000003 * int(seed) + 17)
    return g


def _rand(g, *shape):
    return torch.rand(*shape, generator=g, device="cuda", dtype=torch.float64)


def _plummer(g, n):
    """Plummer sphere, a = 1, truncated at r < 50 (by the range of the uniform variate)."""
    u = _rand(g, n) * (1.0 + 50.0 ** -2) ** -1.5
    r = 1.0 / torch.sqrt(u.clamp_min(1e-12) ** (-2.0 / 3.0) - 1.0)
    d = torch.randn(n, 3, generator=g, device="cuda", dtype=torch.float64)
    return (d / d.norm(dim=1, keepdim=True) * r[:, None]).contiguous()


def _positions(g, dist, n):
    if dist == "plummer":
        return _plummer(g, n)
    if dist == "uniform":
        return _rand(g, n, 3)
    # 64 Plummer subclusters: centres in a cube of side 20, lognormal radii, uneven member counts
    weight = -torch.log(_rand(g, 64).clamp_min(1e-12))
    centre = 20.0 * (_rand(g, 64, 3) - 0.5)
    radius = torch.exp(math.log(0.3) + 0.5 * torch.randn(64, generator=g, device="cuda", dtype=torch.float64))
    member = torch.multinomial(weight, n, replacement=True, generator=g)
    return (centre[member] + radius[member][:, None] * _plummer(g, n)).contiguous()


def _masses(n):
    return torch.full((n,), 1.0 / n, dtype=torch.float64, device="cuda")


def _const(n, value):
    return torch.full((n,), value, dtype=torch.float64, device="cuda")


def _host(t):
    return t.cpu().numpy()


def _vp(t):
    return ctypes.c_void_p(t.data_ptr())


def _stream():
    return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)


def _names(case):
    return [case["field"]] if "field" in case else case["fields"].split(",")


def _inputs(case, seed):
    """The particles of a case, on the GPU: what prepare() hands on and what exact() sums over."""
    g = _generator(seed)
    kind = case["kind"]
    if kind == "direct":
        ns, nt = case["ns"], case["nt"]
        x = _positions(g, case["dist"], ns)
        s = {"x": x, "m": _masses(ns), "h": _const(ns, 0.02)}
        if not case["mutual"]:
            s["xt"] = _positions(g, case["dist"], nt)
            s["ht"] = _const(nt, 0.0)
        return s
    if kind in ("direct_f32", "context"):  # float32 positions, as these contexts take them
        ns, nt = case["ns"], case["nt"]
        x = _positions(g, case["dist"], ns).float().double()
        s = {"x": x, "m": _masses(ns).float().double(), "h": _const(ns, 0.01).float().double()}
        s["xt"] = x[:nt].contiguous() if nt <= ns and kind == "direct_f32" else _positions(g, case["dist"], nt).float().double()
        s["ht"] = _const(nt, 0.01).float().double()
        return s
    if kind == "targets":
        ns, nt = case["ns"], case["nt"]
        x = _plummer(g, ns).float().double()
        h = torch.exp(math.log(0.003) + 0.7 * torch.randn(ns, generator=g, device="cuda", dtype=torch.float64))
        d = torch.randn(nt, 3, generator=g, device="cuda", dtype=torch.float64)
        xt = d / d.norm(dim=1, keepdim=True) * (5.0 * _rand(g, nt) ** (1.0 / 3.0))[:, None]
        return {"x": x, "m": _masses(ns), "h": h, "xt": xt.contiguous(), "ht": _const(nt, 0.0)}
    if kind == "batched":  # even systems uniform cubes, odd ones Plummer spheres, float32 positions
        lo, hi = math.log(case["n_min"]), math.log(case["n_max"])
        k = torch.arange(case["systems"], device="cuda", dtype=torch.float64)
        counts = torch.exp(lo + (hi - lo) * (k + 0.5) / case["systems"]).round().long()  # log-uniform sizes,
        counts = counts[torch.randperm(case["systems"], generator=g, device="cuda")]     # in any order
        n = int(counts.sum())
        system = torch.repeat_interleave(torch.arange(case["systems"], device="cuda"), counts)
        x = torch.where((system % 2 == 0)[:, None], _rand(g, n, 3), _plummer(g, n)).float().double().contiguous()
        off = np.concatenate([[0], np.cumsum(_host(counts))]).astype(np.int64)
        return {"x": x, "m": (1.0 / counts.double())[system].contiguous(), "h": _const(n, 0.01), "off": off}
    n = case["n"]
    s = {"x": _positions(g, case["dist"], n), "m": _masses(n)}
    s["h"] = _const(n, case.get("h", case.get("radius", 0.0)))
    if kind == "structure":
        s["v"] = 0.3 * s["x"] + torch.randn(n, 3, generator=g, device="cuda", dtype=torch.float64)
    return s


HOST_KINDS = ("direct", "frontend", "field", "column", "structure")


def prepare(case, seed):
    s = _inputs(case, seed)
    kind = case["kind"]
    if kind in HOST_KINDS:  # numpy users: host arrays
        s = {k: _host(v) for k, v in s.items()}
    elif kind == "direct_f32":
        s = {k: _host(v).astype(np.float32) for k, v in s.items()}
        s["context"] = (tg_cuda.CudaAccelBruteforce if case["field"] == "accel" else tg_cuda.CudaPotentialBruteforce)(
            s["x"], s["m"], s["h"])
    elif kind == "context":
        tree = tg.ConstructTree(_host(s["x"]), _host(s["m"]), _host(s["h"]))
        s = {"xt": _host(s["xt"]).astype(np.float32), "ht": _host(s["ht"]).astype(np.float32),
             "context": (tg_cuda.CudaAccel if case["field"] == "accel" else tg_cuda.CudaPotential)(tree)}
    else:
        n = case["nt"] if kind == "targets" else len(s["m"])
        width = 3 if kind == "batched" else sum(FIELD_WIDTH[f] for f in _names(case))
        s["out"] = torch.zeros((n, width), dtype=torch.float64, device="cuda")
        if case.get("learned"):
            s["model"] = tg_theta.ThetaModel.load()
            s["model"].handle()
            s["log10_lambda"] = tg_theta.default_lambda(s["model"], case["quadrupole"], kind == "targets")
    s["case"] = dict(case)
    torch.cuda.synchronize()
    return s


# ---------------------------------------------------------------------------------------------


def run(s):
    return _RUN[s["case"]["kind"]](s, s["case"])


def _run_direct(s, c):
    if c["mutual"]:
        return FUNCTIONS[c["field"]](s["x"], s["m"], s["h"])
    return TARGET_FUNCTIONS[c["field"]](s["xt"], s["x"], s["m"], softening_target=s["ht"], softening_source=s["h"])


def _run_frontend(s, c):
    return FUNCTIONS[c["field"]](s["x"], s["m"], s["h"], theta=c["theta"], quadrupole=c["quadrupole"],
                                 precision=c["precision"])


def _run_field(s, c):
    f = tg.Field(s["x"], s["m"], s["h"], theta=c["theta"], quadrupole=c["quadrupole"], precision=c["precision"])
    return f.evaluate(**{k: True for k in _names(c)})


def _run_direct_f32(s, c):
    return s["context"](s["xt"], s["ht"])


def _run_context(s, c):
    return s["context"](s["xt"], s["ht"], theta=0.7, group_size=c["group_size"])


def _columns(out, names):
    res, o = {}, 0
    for f in ("potential", "accel", "tidal"):
        if f in names:
            w = FIELD_WIDTH[f]
            res[f] = out[:, o:o + w]
            o += w
    return res


def _build(L, s, quadrupole):
    tree = ctypes.c_void_p()
    _lib.check(L.tg_tree_build(_vp(s["x"]), _vp(s["m"]), _vp(s["h"]), len(s["m"]), int(quadrupole), 1,
                               _lib.TG_MEM_DEVICE, _stream(), ctypes.byref(tree)), "build")
    return tree


def _run_device(s, c):
    L = _lib.load()
    names, quad, n, st = _names(c), int(c["quadrupole"]), len(s["m"]), _stream()
    bits = sum(FIELD_BITS[f] for f in names)
    tree = _build(L, s, quad)
    if c["learned"]:
        _lib.check(L.tg_tree_fields_learned(tree, bits, quad, 1.0, 32, s["model"].handle(), float(s["log10_lambda"]),
                                            c["theta"], _lib.TG_MEM_DEVICE, _vp(s["out"]), st), "learned walk")
    else:
        _lib.check(L.tg_tree_fields(tree, None, None, n, bits, quad, c["theta"], 1.0, 32, _lib.TG_GROUP_TREE,
                                    _lib.TG_ORDER_TREE, _lib.TG_FP32, None, _lib.TG_MEM_DEVICE, _vp(s["out"]), st),
                   "walk")
    L.tg_tree_free(tree)
    return _columns(s["out"], names)


def _run_targets(s, c):
    L = _lib.load()
    names, quad, st = _names(c), int(c["quadrupole"]), _stream()
    bits = sum(FIELD_BITS[f] for f in names)
    tree = _build(L, s, quad)
    targets = ctypes.c_void_p()
    _lib.check(L.tg_targets_create(tree, _vp(s["xt"]), _vp(s["ht"]), c["nt"], 32, _lib.TG_MEM_DEVICE, st,
                                   ctypes.byref(targets)), "targets")
    if c["learned"]:
        _lib.check(L.tg_targets_fields_learned(targets, bits, quad, 1.0, s["model"].handle(), float(s["log10_lambda"]),
                                               c["theta"], _lib.TG_MEM_DEVICE, _vp(s["out"]), st), "learned walk")
    else:
        _lib.check(L.tg_targets_fields(targets, bits, quad, c["theta"], 1.0, _lib.TG_FP32, None, _lib.TG_MEM_DEVICE,
                                       _vp(s["out"]), st), "walk")
    L.tg_targets_free(targets)
    L.tg_tree_free(tree)
    return _columns(s["out"], names)


def _run_batched(s, c):
    L = _lib.load()
    st, tree, graph = _stream(), ctypes.c_void_p(), ctypes.c_void_p()
    _lib.check(L.tg_tree_build_batched(_vp(s["x"]), _vp(s["m"]), _vp(s["h"]), _lib.ptr(s["off"]), c["systems"], 0,
                                       _lib.TG_MEM_DEVICE, st, ctypes.byref(tree)), "batched build")
    # the launch shape that the autotuner picks for this workload
    _lib.check(L.tg_tree_set_walk_config(tree, 8, 1024), "walk shape")
    _lib.check(L.tg_walk_graph_create(tree, _lib.TG_FIELD_ACCEL, 0, c["theta"], 1.0, 32, _lib.TG_GROUP_TREE,
                                      _vp(s["out"]), ctypes.byref(graph)), "walk graph")
    _lib.check(L.tg_walk_graph_launch(graph, st), "launch")
    _lib.check(L.tg_walk_graph_status(graph, st), "walk")
    L.tg_walk_graph_free(graph)
    L.tg_tree_free(tree)
    return s["out"]


def _run_column(s, c):
    return tg.ColumnDensity(s["x"], s["m"], s["h"], rays=6)


def _run_structure(s, c):
    rbins, sv = tg.VelocityStructFunc(s["x"], s["m"], s["v"], seed=12345)
    return {"rbins": rbins, "sv": sv}


_RUN = {"direct": _run_direct, "frontend": _run_frontend, "field": _run_field, "direct_f32": _run_direct_f32,
        "context": _run_context, "device": _run_device, "targets": _run_targets, "batched": _run_batched,
        "column": _run_column, "structure": _run_structure}


# ---------------------------------------------------------------------------------------------


def _walk_interactions(n, theta, learned):
    """List entries per target of a walk that accepts at theta, from the walks' counters: about 1950
    at 1e6 particles and theta = 0.7 (the count grows with log N and as theta^-2), half of them learned."""
    return min(n, 1950.0 * (math.log(max(n, 8)) / math.log(1e6)) * (0.7 / theta) ** 2 * (0.52 if learned else 1.0))


def _flops(case, names, quadrupole):
    return max(FLOPS_MONO[f] + (FLOPS_QUAD[f] if quadrupole else 0) for f in names) + 2 * (len(names) - 1)


def work(case):
    kind = case["kind"]
    if kind == "direct":
        ns, nt = case["ns"], case["nt"]
        w = FIELD_WIDTH[case["field"]]
        return {"bytes": 8 * (5 * ns + (0 if case["mutual"] else 4 * nt) + w * nt),
                "flops": ns * nt * FLOPS_MONO[case["field"]]}
    if kind == "direct_f32":
        ns, nt = case["ns"], case["nt"]
        return {"bytes": 4 * (5 * ns + (4 + FIELD_WIDTH[case["field"]]) * nt), "flops": ns * nt * FLOPS_MONO[case["field"]]}
    if kind == "context":
        ns, nt = case["ns"], case["nt"]
        return {"bytes": 4 * (8 * ns + (4 + FIELD_WIDTH[case["field"]]) * nt),
                "flops": int(nt * _walk_interactions(ns, 0.7, False) * FLOPS_MONO[case["field"]])}
    if kind == "batched":
        mean = (case["n_max"] - case["n_min"]) / math.log(case["n_max"] / case["n_min"])
        n = int(case["systems"] * mean)
        return {"bytes": 8 * (5 + 3) * n,
                "flops": int(n * _walk_interactions(mean, case["theta"], False) * FLOPS_MONO["accel"])}
    if kind == "column":  # per ray: the spheres and cells met on the way, about 2 N^(1/3) log2 N of them
        n = case["n"]
        return {"bytes": 8 * (5 + 6) * n, "flops": int(6 * n * 20 * 2 * n ** (1.0 / 3.0) * math.log2(n))}
    if kind == "structure":
        n = case["n"]
        return {"bytes": 8 * 7 * n + 16 * int(n ** (1.0 / 3.0)),
                "flops": int(n * _walk_interactions(n, 1.0, False) * 20)}
    names = _names(case)
    width = sum(FIELD_WIDTH[f] for f in names)
    ns = case["ns"] if kind == "targets" else case["n"]
    nt = case["nt"] if kind == "targets" else ns
    per = _walk_interactions(ns, case["theta"], case.get("learned", False))
    return {"bytes": 8 * (5 * ns + (4 * nt if kind == "targets" else 0) + width * nt),
            "flops": int(nt * per * _flops(case, names, case["quadrupole"]))}


# ---------------------------------------------------------------------------------------------
# The direct sums in 64 bits (plain torch).


def _pair_sums(xt, ht, x, m, h, names):
    """Potential, acceleration and tidal tensor of the sources at the targets: point masses outside
    the larger of the two softening lengths, the cubic spline inside; pairs at zero distance drop out."""
    nt, ns = len(xt), len(x)
    out = {f: torch.zeros((nt, FIELD_WIDTH[f]), dtype=torch.float64, device="cuda") for f in names}
    rows = max(1, (1 << 26) // max(ns, 1))
    for a in range(0, nt, rows):
        b = min(nt, a + rows)
        d = [x[None, :, k] - xt[a:b, None, k] for k in range(3)]
        r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2]
        zero = r2 == 0
        r = torch.sqrt(torch.where(zero, 1.0, r2))
        inv = torch.where(zero, 0.0, 1.0 / r)
        force = m[None, :] * inv ** 3
        near = ((r < torch.maximum(h[None, :], ht[a:b, None])) & ~zero).nonzero(as_tuple=True)
        rn = r[near]
        hn = torch.maximum(h[near[1]], ht[a:b][near[0]])
        mn = m[near[1]]
        q = rn / hn
        inner = q <= 0.5
        force[near] = mn / hn ** 3 * torch.where(
            inner, 32.0 / 3.0 + q * q * (32.0 * q - 38.4),
            64.0 / 3.0 - 48.0 * q + 38.4 * q * q - 32.0 / 3.0 * q ** 3 - 1.0 / 15.0 / q ** 3)
        if "potential" in names:
            phi = -m[None, :] * inv
            phi[near] = mn / hn * torch.where(
                inner, -2.8 + q * q * (16.0 / 3.0 + q * q * (6.4 * q - 9.6)),
                -3.2 + 1.0 / 15.0 / q + q * q * (32.0 / 3.0 + q * (-16.0 + q * (9.6 - 32.0 / 15.0 * q))))
            out["potential"][a:b, 0] = phi.sum(1)
        if "accel" in names:
            for k in range(3):
                out["accel"][a:b, k] = (force * d[k]).sum(1)
        if "tidal" in names:
            quad = 3.0 * m[None, :] * inv ** 5
            quad[near] = mn / hn ** 5 * torch.where(inner, 76.8 - 96.0 * q, 48.0 / q - 76.8 + 32.0 * q - 0.2 / q ** 5)
            for i in range(3):
                for j in range(i, 3):
                    t = (quad * d[i] * d[j]).sum(1) - (force.sum(1) if i == j else 0.0)
                    out["tidal"][a:b, 3 * i + j] = t
                    out["tidal"][a:b, 3 * j + i] = t
    return out


def _shaped(v, field):
    v = _host(v)
    return v[:, 0] if field == "potential" else v.reshape(-1, 3, 3) if field == "tidal" else v


def _column_sums(x, m, radius):
    """Mass per area of the uniform spheres along the six axis rays from every particle to infinity."""
    n = len(x)
    out = np.empty((n, 6))
    rows = max(1, (1 << 26) // n)
    for a in range(0, n, rows):
        b = min(n, a + rows)
        d = [x[None, :, k] - x[a:b, None, k] for k in range(3)]
        inside = d[0] * d[0] + d[1] * d[1] + d[2] * d[2] <= radius[None, :] ** 2
        for axis in range(3):
            z, u, w = d[axis], d[(axis + 1) % 3], d[(axis + 2) % 3]
            half2 = radius[None, :] ** 2 - (u * u + w * w)
            half = torch.sqrt(half2.clamp_min(0.0))
            rho = (3.0 / (4.0 * math.pi)) * m[None, :] / radius[None, :] ** 3
            for sign, col in ((1.0, axis), (-1.0, axis + 3)):
                length = torch.where(inside, sign * z + half, torch.where(sign * z > 0, 2.0 * half, 0.0))
                out[a:b, col] = _host((rho * torch.where(half2 > 0, length, 0.0)).sum(1))
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "structure":  # the bin edges; the binned sums are jittered at random
        x = _host(_inputs(case, seed)["x"])
        r = np.sort(np.sqrt(((x - np.median(x, axis=0)) ** 2).sum(axis=1)))
        return {"rbins": 10 ** np.linspace(np.log10(r[10]), np.log10(r[-1]), int(len(r) ** (1.0 / 3.0))), "sv": None}
    if kind == "batched":
        s = _inputs(case, seed)
        out = torch.empty((len(s["m"]), 3), dtype=torch.float64, device="cuda")
        for a, b in zip(s["off"][:-1], s["off"][1:]):
            p = [s[k][a:b] for k in ("x", "h", "x", "m", "h")]
            out[a:b] = _pair_sums(*p, ["accel"])["accel"]
        return out
    ns = case["ns"] if "ns" in case else case["n"]
    nt = case["nt"] if "nt" in case else case["n"]
    if ns * nt > 4e10:  # the direct sum would take over 20 s
        return None
    s = _inputs(case, seed)
    if kind == "column":
        return _column_sums(s["x"], s["m"], s["h"])
    names = _names(case)
    sums = _pair_sums(s.get("xt", s["x"]), s.get("ht", s["h"]), s["x"], s["m"], s["h"], names)
    if kind == "field":
        return {f: _shaped(sums[f], f) for f in names}
    if kind in ("device", "targets"):
        return {f: sums[f] for f in names}
    return _shaped(sums[names[0]], names[0])
