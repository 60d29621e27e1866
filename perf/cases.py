"""The calls that a user of this framework makes, as measurable cases.

Five kinds, each through the C ABI / package entry points on device buffers:

* ``query``  closest-point queries (n2w_bvh_query_device, plain and masked);
* ``walk``   per-point Walk-on-Spheres estimates (n2w_wos_estimate): Laplace and
             Poisson problems, one or several source samples per ball;
* ``batch``  uneven instances on several meshes, one captured graph replayed;
* ``infer`` / ``train``  the neural cache: inference, and a training step split
             as the data-parallel trainer runs it (gradients, then Adam);
* ``nc2lmc`` the whole two-level estimate with a cache.

A case holds sizes and options only; meshes, points, walk seeds and weights come
from the seed that ``prepare`` is given.
"""
import ctypes as C
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "n2wos-cuda_b200"))

import n2w  # noqa: E402
from n2w import nc, workloads  # noqa: E402
from n2w._lib import BatchItem, PointStats, call  # noqa: E402

DEV = "cuda"

# The mesh sizes of the repository's own workloads, by name (triangles):
# displaced icospheres of level 4..6 and bumpy spheres of the batched workload,
# and the reference's bumpy sphere of the published figure run.
MESHES = {"ico4": 5120, "ico5": 20480, "ico6": 81920, "bumpy32": 3968, "bumpy64": 16128, "bumpy128": 65024,
          "bumpy256": 261120, "figure": 65024}

# Cache configurations of the library default and of the evaluation tool's presets.
NETS = {"default": dict(),
        "heavy": dict(n_levels=16, log2_hashmap_size=19, base_resolution=8.0, per_level_scale=1.4, n_neurons=64,
                      n_hidden_layers=3),
        "baseline": dict(n_levels=12, log2_hashmap_size=18, base_resolution=8.0, per_level_scale=1.5, n_neurons=32,
                         n_hidden_layers=2),
        "light": dict(n_levels=8, log2_hashmap_size=15, base_resolution=8.0, per_level_scale=1.5, n_neurons=16,
                      n_hidden_layers=1),
        "nano": dict(n_levels=6, log2_hashmap_size=13, base_resolution=8.0, per_level_scale=1.5, n_neurons=16,
                     n_hidden_layers=1)}


def listed():
    return [
        # A probe of a few points, as an interactive caller or a test makes it: launch latency.
        {"name": "query_small", "kind": "query", "mesh": "ico4", "n": 1000, "points": "uniform", "masked": False},
        # The benchmark's query set: uniform in the grown box of the 65k-triangle bumpy sphere.
        {"name": "query_uniform", "kind": "query", "mesh": "bumpy128", "n": 262144, "points": "uniform",
         "masked": False},
        # A wavefront caller's step: walk positions near the surface, finished slots masked off, a ragged count.
        {"name": "query_masked", "kind": "query", "mesh": "ico6", "n": 1000003, "points": "surface", "masked": True},
        # The largest query set of the benchmark's range: throughput.
        {"name": "query_large", "kind": "query", "mesh": "ico6", "n": 4194304, "points": "uniform", "masked": False},
        # A handful of probe points solved at once, as a serving request's first sweep.
        {"name": "walk_small", "kind": "walk", "mesh": "bumpy32", "problem": "charges", "n": 37, "walks": 64,
         "eps": 1e-3},
        # Laplace solve with the seeded charge boundary at interior points, ragged counts.
        {"name": "walk_laplace", "kind": "walk", "mesh": "bumpy128", "problem": "charges", "n": 20011, "walks": 101,
         "eps": 1e-3},
        # The published figure run's problem, walk count and shell (a thin epsilon shell, analytic boundary).
        {"name": "walk_figure", "kind": "walk", "mesh": "figure", "problem": "zebra", "n": 40000, "walks": 64,
         "eps": 1e-4},
        # The headline slice: Poisson, one Green's-function source sample per ball.
        {"name": "walk_poisson", "kind": "walk", "mesh": "ico6", "problem": "sinprod", "n": 40000, "walks": 128,
         "eps": 5e-4},
        # The time-to-error setting: 16 source samples per ball.
        {"name": "walk_poisson16", "kind": "walk", "mesh": "ico6", "problem": "sinprod16", "n": 10000, "walks": 128,
         "eps": 5e-4},
        # Many small instances on four meshes, a replayed graph (the batched workload at an eighth of its points).
        {"name": "batch", "kind": "batch", "instances": 48, "points_lo": 64, "points_hi": 8192, "walks_lo": 32,
         "walks_hi": 256, "eps": 1e-3},
        # One online-training step at the default batch and network.
        {"name": "train", "kind": "train", "net": "default", "n": 65536},
        # The two-level estimate with the evaluation tool's walk counts (its inference is the cache's forward path).
        {"name": "nc2lmc", "kind": "nc2lmc", "mesh": "bumpy128", "problem": "sinprod", "net": "default", "n": 8192,
         "coarse": 256, "residual": 16, "depth": 8, "eps": 1e-3},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["query", "query", "walk", "walk", "batch", "infer", "train", "nc2lmc"])
    mesh = rng.choice(["ico4", "ico5", "ico6", "bumpy32", "bumpy64", "bumpy128", "figure"])
    if kind == "query":
        return {"kind": kind, "mesh": mesh, "n": _log_int(rng, 1, 2000000), "points": rng.choice(["uniform", "surface"]),
                "masked": rng.random() < 0.3}
    if kind == "walk":
        n = _log_int(rng, 1, 30000)
        return {"kind": kind, "mesh": mesh, "problem": rng.choice(["charges", "zebra", "sinprod", "sinprod16",
                                                                    "multiscale"]),
                "n": n, "walks": _log_int(rng, 1, max(2, min(1024, 2000000 // n))),
                "eps": rng.choice([1e-4, 5e-4, 1e-3])}
    if kind == "batch":
        return {"kind": kind, "instances": _log_int(rng, 1, 48), "points_lo": 1, "points_hi": _log_int(rng, 16, 4096),
                "walks_lo": 1, "walks_hi": _log_int(rng, 8, 256), "eps": 1e-3}
    if kind == "infer":
        return {"kind": kind, "net": rng.choice(sorted(NETS)), "n": _log_int(rng, 1, 4000000)}
    if kind == "train":
        return {"kind": kind, "net": rng.choice(sorted(NETS)), "n": _log_int(rng, 64, 131072)}
    return {"kind": kind, "mesh": mesh, "problem": rng.choice(["charges", "sinprod"]), "net": rng.choice(sorted(NETS)),
            "n": _log_int(rng, 1, 8192), "coarse": _log_int(rng, 8, 256), "residual": _log_int(rng, 1, 32),
            "depth": rng.choice([1, 2, 4, 8]), "eps": 1e-3}


# ---- inputs -----------------------------------------------------------------------
def _mesh(name, seed):
    if name.startswith("ico"):
        m = n2w.Mesh.icosphere_displaced(int(name[3:]), 0.12, 3.0, 4, 0.5, 12345 + seed)
    elif name == "figure":
        m = n2w.Mesh.bumpy_sphere_ref(128, 256, 0.15)
    else:
        s = int(name[5:])
        m = n2w.Mesh.bumpy_sphere_trig(s, 2 * s, 0.08, 6, 8)
    m.normalize()
    return m


def _problem(name, seed):
    if name == "charges":
        return n2w.problem_charges_seeded(8, 1.6, 2.0, 12345 + seed)
    if name == "zebra":
        return n2w.problem_from_name("harmonic_zebra_k8")
    if name == "multiscale":  # a reference mode with a source, by the reference's centre rule
        return n2w.problem_from_name("poisson_multiscale", n2w.N2W_SOURCE_CENTER)
    p = n2w.problem_sinprod(3.0 * math.pi)
    p.source_samples = 16 if name == "sinprod16" else 1
    return p


def _query_points(case, mesh, seed):
    rng = np.random.default_rng(seed)
    n = case["n"]
    if case["points"] == "uniform":
        return rng.uniform(-1.2, 1.2, (n, 3)).astype(np.float32)
    # near the surface: a point of a random triangle moved by a log-uniform distance
    v, t = mesh.arrays()
    tri = v[t[rng.integers(0, len(t), n)]]
    w = rng.dirichlet((1.0, 1.0, 1.0), n).astype(np.float32)
    d = rng.normal(size=(n, 3))
    d *= (np.exp(rng.uniform(math.log(5e-4), math.log(0.5), n)) / np.linalg.norm(d, axis=1))[:, None]
    return ((w[:, :, None] * tri).sum(1) + d).astype(np.float32)


def _interior(bvh, n, seed):
    return workloads.interior_ball_points(bvh, n, np.random.default_rng(seed), 0.9)


class _Stats:
    """Per-point accumulators in torch memory, in the library's layout."""

    def __init__(self, n):
        self.out = {"sum": torch.zeros(n, dtype=torch.float64, device=DEV),
                    "sum_sq": torch.zeros(n, dtype=torch.float64, device=DEV),
                    "count": torch.zeros(n, dtype=torch.int32, device=DEV),
                    "steps": torch.zeros(n, dtype=torch.int64, device=DEV),
                    "forced": torch.zeros(n, dtype=torch.int32, device=DEV)}

    def struct(self, first=0):
        o = self.out
        return PointStats(o["sum"].data_ptr() + 8 * first, o["sum_sq"].data_ptr() + 8 * first,
                          o["count"].data_ptr() + 4 * first, o["steps"].data_ptr() + 8 * first,
                          o["forced"].data_ptr() + 4 * first)


class _DeviceArray:
    """A float32 device buffer of the library for torch.as_tensor (no copy); keeps the buffer's owner alive."""

    def __init__(self, ptr, count, owner):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (count,), "typestr": "<f4", "data": (ptr, False), "version": 3}


def _net_params(net, seed):
    """Weights of a trained network's size: features of a few tenths, MLP weights at their initial scale."""
    d = n2w.cache_describe(n2w.cache_config(**NETS[net]))
    cfg = n2w.cache_config(**NETS[net])
    rng = np.random.default_rng(7000 + seed)
    g, m = d["grid_params"], d["mlp_params"]
    p = np.empty(g + m, np.float32)
    p[:g] = 0.2 * rng.standard_normal(g, dtype=np.float32)
    fan = cfg.n_neurons + (16 if 2 * cfg.n_levels <= 16 else 32)
    p[g:] = rng.uniform(-1.0, 1.0, m).astype(np.float32) * math.sqrt(6.0 / fan)
    return p


def _unit_inputs(n, seed):
    """Interior points of the unit ball, mapped to the unit cube as the trainer maps them, and smooth noisy labels."""
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    d = torch.randn(n, 3, generator=g, device=DEV, dtype=torch.float32)
    r = torch.rand(n, 1, generator=g, device=DEV, dtype=torch.float32) ** (1.0 / 3.0)
    x = (0.5 + 0.45 * r * d / d.norm(dim=1, keepdim=True)).clamp(0.0, 1.0).contiguous()
    t = torch.sin(9.0 * x).prod(1) + 0.3 * torch.randn(n, generator=g, device=DEV, dtype=torch.float32)
    return x, t.contiguous()


def _cache(net, seed):
    c = n2w.Cache(n2w.cache_config(**NETS[net]))
    c.set_params(_net_params(net, seed))
    return c


def prepare(case, seed):
    k = case["kind"]
    s = {"case": case}
    if k in ("infer", "train"):
        s["cache"] = _cache(case["net"], seed)
        s["x"], s["t"] = _unit_inputs(case["n"], seed)
        s["y"] = torch.empty(case["n"], dtype=torch.float32, device=DEV)
        if k == "train":
            ptr, cnt, loss = C.c_void_p(), C.c_int64(), C.c_void_p()
            call("n2w_cache_gradient_buffer", s["cache"].handle, C.byref(ptr), C.byref(cnt), C.byref(loss))
            s["grad"] = torch.as_tensor(_DeviceArray(ptr.value, cnt.value, s["cache"]), device=DEV)
            s["loss"] = torch.as_tensor(_DeviceArray(loss.value, 1, s["cache"]), device=DEV)
        return s
    if k == "batch":
        return _prepare_batch(case, seed, s)
    s["mesh"] = _mesh(case["mesh"], seed)
    s["bvh"] = n2w.Bvh(s["mesh"], 4, "sah")
    n = case["n"]
    if k == "query":
        s["pts"] = torch.from_numpy(_query_points(case, s["mesh"], seed)).to(DEV)
        s["d2"] = torch.empty(n, dtype=torch.float32, device=DEV)
        s["cp"] = torch.empty(n, 3, dtype=torch.float32, device=DEV)
        s["id"] = torch.empty(n, dtype=torch.int32, device=DEV)
        s["ov"] = torch.empty(n, dtype=torch.int32, device=DEV)
        s["active"] = None
        if case["masked"]:
            s["active"] = torch.from_numpy((np.random.default_rng(seed + 1).random(n) < 0.6).astype(np.uint8)).to(DEV)
        return s
    s["problem"] = _problem(case["problem"], seed)
    s["pts"] = torch.from_numpy(_interior(s["bvh"], n, seed)).to(DEV)
    if k == "walk":
        s["options"] = n2w.walk_options(walks_per_point=case["walks"], max_steps=256, epsilon=case["eps"],
                                        seed=99 + seed)
        s["stats"] = _Stats(n)
    else:
        s["cache"] = _cache(case["net"], seed)
        s["options"] = nc.nc2lmc_options(s["mesh"], case["coarse"], case["residual"], case["depth"], 256, case["eps"],
                                         0.999, 99 + seed)
        s["coarse"], s["residual"] = _Stats(n), _Stats(n)
    return s


def _instances(case, seed):
    rng = np.random.default_rng(seed)
    return [(k % len(workloads.BATCH_MESHES), workloads.log_uniform_int(rng, case["points_lo"], case["points_hi"]),
             workloads.log_uniform_int(rng, case["walks_lo"], case["walks_hi"]), int(rng.integers(1, 2**62)))
            for k in range(case["instances"])]


def _prepare_batch(case, seed, s):
    # instance sizes belong to the case (they set the work), the points and walks to the seed
    inst = _instances(case, 2024)
    s["meshes"] = [workloads.bumpy_sphere(n2w, a, b) for a, b in workloads.BATCH_MESHES]
    s["bvhs"] = [n2w.Bvh(m, 4, "sah") for m in s["meshes"]]
    s["scene"] = n2w.Scene(s["bvhs"])
    problems = [n2w.problem_charges_seeded(8, 1.6, 2.0, 500 + seed + k) for k in range(len(inst))]
    s["problems"] = (type(problems[0]) * len(problems))(*problems)
    total = sum(i[1] for i in inst)
    s["stats"] = _Stats(total)
    items = (BatchItem * len(inst))()
    s["pts"] = []
    first = 0
    for k, (m, n, w, key) in enumerate(inst):
        p = torch.from_numpy(_interior(s["bvhs"][m], n, 31 * seed + k)).to(DEV)
        s["pts"].append(p)
        items[k].mesh, items[k].problem, items[k].d_points = m, k, p.data_ptr()
        items[k].point_count, items[k].walks_per_point, items[k].seed = n, w, key + seed
        items[k].stats = s["stats"].struct(first)
        first += n
    torch.cuda.synchronize()
    o = n2w.walk_options(max_steps=256, epsilon=case["eps"])
    s["batch"] = _Batch(s["scene"], s["problems"], items, o)
    return s


class _Batch(n2w.Batch):
    """n2w.Batch over caller-owned point and statistics buffers."""

    def __init__(self, scene, problems, items, options):
        self.scene, self.options, self.points, self.stats = scene, options, [], []
        h = C.c_void_p()
        call("n2w_batch_create", scene.handle, problems, len(problems), items, len(items), C.byref(options),
             C.byref(h))
        self._h = h
        self.counters = n2w.DeviceBuffer(64)
        self.stream = n2w.Stream()
        self.capture_graph(self.stream)


# ---- one pass -----------------------------------------------------------------------
def run(s):
    case = s["case"]
    k = case["kind"]
    if k == "query":
        s["bvh"].query_device(s["pts"].data_ptr(), case["n"], s["d2"].data_ptr(), s["cp"].data_ptr(),
                              s["id"].data_ptr(), s["ov"].data_ptr(),
                              d_active=None if s["active"] is None else s["active"].data_ptr())
        return {"d2": s["d2"], "cp": s["cp"], "id": s["id"], "overflow": s["ov"]}
    if k == "walk":
        call("n2w_wos_estimate", s["bvh"].handle, C.byref(s["problem"]), s["pts"].data_ptr(), case["n"],
             C.byref(s["options"]), s["stats"].struct(), None, None, None)
        return s["stats"].out
    if k == "batch":
        s["batch"].graph_launch(s["batch"].stream)
        return s["stats"].out
    if k == "infer":
        call("n2w_cache_infer", s["cache"].handle, s["x"].data_ptr(), case["n"], s["y"].data_ptr(), None)
        return s["y"]
    if k == "train":
        h = s["cache"].handle
        call("n2w_cache_gradients", h, s["x"].data_ptr(), s["t"].data_ptr(), case["n"], s["y"].data_ptr(), None)
        grad = s["grad"].clone()  # Adam clears the buffer
        call("n2w_cache_apply_gradients", h, C.c_float(1.0), None)
        return {"grad": grad, "outputs": s["y"], "loss_sum": s["loss"].clone()}
    call("n2w_nc2lmc_estimate", s["bvh"].handle, C.byref(s["problem"]), s["cache"].handle, s["pts"].data_ptr(),
         case["n"], C.byref(s["options"]), s["coarse"].struct(), s["residual"].struct(), None)
    return {"coarse": s["coarse"].out, "residual": s["residual"].out}


# ---- what one pass cannot do without --------------------------------------------------
def _net_size(net):
    d = n2w.cache_describe(n2w.cache_config(**NETS[net]))
    return d["grid_params"], d["mlp_params"]


def _walk_work(points, walks, triangles):
    # a walk takes ~20 steps, each at least one closest-point query (a triangle test
    # of ~60 operations) and one move (~80 operations); the mesh is read once
    steps = 20.0 * points * walks
    return {"bytes": 44.0 * points + 48.0 * triangles, "flops": 140.0 * steps}


def work(case):
    k = case["kind"]
    if k == "query":
        n = case["n"]
        return {"bytes": (12 + 24 + (1 if case["masked"] else 0)) * n + 48.0 * MESHES[case["mesh"]],
                "flops": 60.0 * n}
    if k == "walk":
        return _walk_work(case["n"], case["walks"], MESHES[case["mesh"]])
    if k == "batch":
        w = [_walk_work(n, wk, 0) for _, n, wk, _ in _instances(case, 2024)]
        tris = sum(2 * b * (a - 1) for a, b in workloads.BATCH_MESHES)
        return {"bytes": sum(x["bytes"] for x in w) + 48.0 * tris, "flops": sum(x["flops"] for x in w)}
    grid, mlp = _net_size(case["net"])
    if k == "infer":
        return {"bytes": 16.0 * case["n"] + 2.0 * (grid + mlp), "flops": 2.0 * mlp * case["n"]}
    if k == "train":
        # gradients out (4 B), then Adam: gradient and moments and master in, master, moments and fp16 copy out
        return {"bytes": 20.0 * case["n"] + (4.0 + 2.0 + 4.0 + 16.0 + 14.0) * (grid + mlp), "flops": 6.0 * mlp * case["n"]}
    a = _walk_work(case["n"], case["coarse"], MESHES[case["mesh"]])
    b = _walk_work(case["n"], case["residual"], 0)
    samples = case["n"] * (case["coarse"] + case["residual"])
    return {"bytes": a["bytes"] + b["bytes"] + 2.0 * (grid + mlp), "flops": a["flops"] + b["flops"] + 2.0 * mlp * samples}


# ---- the same in 64 bits -----------------------------------------------------------------
def _closest(p, a, b, c):
    """Closest point of triangles abc to p, all [k, 3] float64: the nearest of the face point and the three edges'."""
    def edge(u, v):
        e = v - u
        t = (((p - u) * e).sum(1) / (e * e).sum(1).clamp_min(1e-300)).clamp(0.0, 1.0)
        return u + t[:, None] * e

    best = edge(a, b)
    for q in (edge(b, c), edge(c, a)):
        best = torch.where((((q - p) ** 2).sum(1) < ((best - p) ** 2).sum(1))[:, None], q, best)
    nrm = torch.linalg.cross(b - a, c - a)
    nn = (nrm * nrm).sum(1).clamp_min(1e-300)
    q = p - (((p - a) * nrm).sum(1) / nn)[:, None] * nrm
    inside = torch.ones(len(p), dtype=torch.bool, device=p.device)
    for u, v in ((a, b), (b, c), (c, a)):
        inside &= (torch.linalg.cross(v - u, q - u) * nrm).sum(1) >= 0.0
    return torch.where(inside[:, None], q, best)


def _exact_query(case, seed):
    n = case["n"]
    if n * MESHES[case["mesh"]] > 2.5e9:
        return None
    mesh = _mesh(case["mesh"], seed)
    v, t = mesh.arrays()
    tri = torch.from_numpy(v.astype(np.float64)).to(DEV)[torch.from_numpy(t.astype(np.int64)).to(DEV)]
    pts = torch.from_numpy(_query_points(case, mesh, seed).astype(np.float64)).to(DEV)
    cen = tri.mean(1)
    rad = (tri - cen[:, None]).norm(dim=2).amax(1)
    d2 = torch.empty(n, dtype=torch.float64, device=DEV)
    cp = torch.empty(n, 3, dtype=torch.float64, device=DEV)
    for i in range(0, n, 512):
        p = pts[i:i + 512]
        d = torch.cdist(p, cen, compute_mode="donot_use_mm_for_euclid_dist")
        near = d - rad <= (d + rad).amin(1, keepdim=True)
        q, j = near.nonzero(as_tuple=True)
        c = _closest(p[q], tri[j, 0], tri[j, 1], tri[j, 2])
        dd = ((c - p[q]) ** 2).sum(1)
        low = torch.full((len(p),), math.inf, dtype=torch.float64, device=DEV).scatter_reduce(0, q, dd, "amin")
        first = torch.full((len(p),), len(q), dtype=torch.int64, device=DEV)
        at = torch.arange(len(q), device=DEV)
        first.scatter_reduce_(0, q, torch.where(dd == low[q], at, len(q)), "amin")
        d2[i:i + 512], cp[i:i + 512] = low, c[first]
    if case["masked"]:
        off = torch.from_numpy(np.random.default_rng(seed + 1).random(n) >= 0.6).to(DEV)
        d2[off] = 0.0
        cp[off] = pts[off]
    return {"d2": d2, "cp": cp, "id": None, "overflow": None}


def _exact_net(case, seed):
    d = n2w.cache_describe(n2w.cache_config(**NETS[case["net"]]))
    cfg = n2w.cache_config(**NETS[case["net"]])
    w, dim = cfg.n_neurons, 16 if 2 * cfg.n_levels <= 16 else 32
    grid_n = d["grid_params"]
    par = torch.from_numpy(_net_params(case["net"], seed)).to(DEV).double()
    x, t = _unit_inputs(case["n"], seed)
    grad = case["kind"] == "train"
    par.requires_grad_(grad)
    out, total = [], None
    for i in range(0, case["n"], 1 << 16):
        u, off, feats = x[i:i + (1 << 16)], 0, []
        for res, size in zip(d["resolution"].tolist(), d["table_size"].tolist()):
            p = (u * float(res)).double()  # the input of a level is rounded to 32 bits
            base = p.floor().clamp(0, res - 1)
            f, base, acc = p - base, base.long(), 0.0
            for k in range(8):
                o = [k & 1, (k >> 1) & 1, (k >> 2) & 1]
                c = [base[:, a] + o[a] for a in range(3)]
                wt = math.prod(f[:, a] if o[a] else 1.0 - f[:, a] for a in range(3))
                if (res + 1) ** 3 <= 1 << cfg.log2_hashmap_size:
                    idx = c[0] + (res + 1) * (c[1] + (res + 1) * c[2])
                else:
                    idx = ((c[0] ^ c[1] * 2654435761 ^ c[2] * 805459861) & 0xFFFFFFFF) % size
                acc = acc + wt[:, None] * par[:grid_n].view(-1, 2)[off + idx]
            feats.append(acc)
            off += size
        h = torch.cat(feats, 1)
        h = torch.nn.functional.pad(h, (0, dim - h.shape[1]))
        at = grid_n
        for layer in range(cfg.n_hidden_layers):
            cols = dim if layer == 0 else w
            h = torch.relu(h @ par[at:at + w * cols].view(w, cols).T)
            at += w * cols
        y = h @ par[at:at + w]
        out.append(y.detach())
        if grad:
            e = ((y - t[i:i + (1 << 16)].double()) ** 2).sum()
            (e / case["n"]).backward()
            total = e.detach() if total is None else total + e.detach()
    y = torch.cat(out)
    return {"grad": par.grad, "outputs": y, "loss_sum": total.reshape(1)} if grad else y


def exact(case, seed):
    if case["kind"] == "query":
        return _exact_query(case, seed)
    if case["kind"] in ("infer", "train"):
        return _exact_net(case, seed)
    return None  # Monte Carlo estimates: their value is set by the random walks
