"""The work that users of this framework give it, as cases that can be timed.

A case is a dict of plain values.  ``listed()`` holds the named ones, ``draw(rng)``
makes one more of the same ranges; ``prepare`` makes what a program holds before the
call (points in device memory, the AppData and its scratch), ``run`` makes one pass
through the package's public entry points and returns what it leaves, ``work`` says
which bytes and operations the pass cannot do without, and ``exact`` computes the
floating outputs in 64 bits with plain torch.

Kinds:
  pipeline  one cloud in device memory, all seven stages fused (run_pipeline)
  stages    the reference's own call sequence, run_stage1 .. run_stage7
  batch     many clouds of uneven size in one go (Batch.run)
  host      one cloud from host memory and its octree back to it (run_host)
  learned   run_pipeline with the learned-CDF sort in stage 2
  train     one optimiser step of the learned sort's boundary network
"""
import importlib.util
import math
import os
import random
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
RANGE = 1024.0  # the box of AppData: [0, 1024) on every axis
TOP = float(np.nextafter(np.float32(RANGE), np.float32(0)))
ROWS = 1.0  # octree rows a point: room for every cloud (AppData's 0.6 is too little for some small ones)
MLP_SIZES = (("w1", 64 * 16), ("b1", 64), ("w2", 64 * 64), ("b2", 64), ("w3", 64), ("b3", 1))
BETA1, BETA2, EPS, LR, STEP = 0.9, 0.999, 1e-8, 1e-3, 500


def _package():
    """The package's folder name is not an identifier: it is loaded by its place."""
    name = "redwood_comp_b200"
    if name not in sys.modules:
        at = os.path.join(ROOT, "redwood-comp_b200")
        spec = importlib.util.spec_from_file_location(
            name, os.path.join(at, "__init__.py"), submodule_search_locations=[at])
        mod = importlib.util.module_from_spec(spec)
        sys.modules[name] = mod
        spec.loader.exec_module(mod)
    return sys.modules[name]


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _cloud(name, kind, n, dist="uniform", bits=32, **more):
    return dict({"name": name} if name else {}, kind=kind, n=n, dist=dist, bits=bits, **more)


def listed():
    return [
        # the smallest clouds that are built one at a time (a frame's region, a chunk of a
        # scan): latency and the number of launches are all that counts
        _cloud("pipeline_3k_u32", "pipeline", 3001),
        # the reference's demo: its default cloud size
        _cloud("pipeline_307k_u32", "pipeline", 307200),
        # an odd-sized lidar-like cloud, with exact geometry and linked leaves: the two
        # options that change the reference's outputs on purpose
        _cloud("pipeline_1m_mixture_u32_options", "pipeline", 1000003, "mixture", options=3),
        # the benchmark's cloud, and its clustered form (half of the keys are duplicates)
        _cloud("pipeline_16m_u32", "pipeline", 16777216),
        _cloud("pipeline_16m_mixture_u32", "pipeline", 16777216, "mixture"),
        # 21 bits an axis, ragged size
        _cloud("pipeline_5m_mixture_u64", "pipeline", 5000011, "mixture", 64),
        # the reference's callers: seven calls, each waited for
        _cloud("stages_2m_u32", "stages", 2000003),
        # the batched form: sizes log-uniform, uniform and clustered clouds mixed
        dict(name="batch_256_u32", kind="batch", clouds=256, lo=1024, hi=262144, bits=32),
        # fewer, larger clouds with wide keys
        dict(name="batch_16_u64", kind="batch", clouds=16, lo=131072, hi=1048576, bits=64),
        # points in pinned host memory, the octree back in pinned host memory
        _cloud("host_1m_u32", "host", 1048576),
        # a large clustered cloud with the learned sort in stage 2
        _cloud("learned_33m_mixture_u32", "learned", 33554432, "mixture"),
        # the boundary network's training batch (its trainer's own size)
        dict(name="train_8192", kind="train", rows=8192),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["pipeline"] * 6 + ["stages", "batch", "batch", "host", "learned", "train"])
    if kind == "train":
        return {"kind": kind, "rows": _log_int(rng, 512, 32768)}
    bits = 32 if kind == "learned" or rng.random() < 0.65 else 64
    if kind == "batch":
        lo = _log_int(rng, 1024, 65536)
        hi = _log_int(rng, 2 * lo, 1 << 20)
        most = max(8, min(256, (12 << 20) // (2 * (lo + hi) // 3 + 1)))  # points in all stay below a large cloud's
        return {"kind": kind, "clouds": rng.randint(8, most), "lo": lo, "hi": hi, "bits": bits}
    dist = rng.choice(["uniform", "mixture"])
    lo, hi = {"pipeline": (2000, (16 << 20) if bits == 32 else (8 << 20)), "stages": (2000, 4 << 20),
              "host": (10000, 2 << 20), "learned": (8 << 20, (16 if dist == "uniform" else 32) << 20)}[kind]
    case = _cloud(None, kind, _log_int(rng, lo, hi), dist, bits)
    if kind == "pipeline" and rng.random() < 0.25:
        case["options"] = rng.choice([1, 2, 3])
    return case


# ---- inputs ------------------------------------------------------------------

def _generator(seed):
    g = torch.Generator(device=_device())
    g.manual_seed(int(seed) * 7919 + 17)
    return g


def _points(n, dist, g, components=32):
    """[n, 4] points in the box, w = 1: uniform, or an isotropic Gaussian mixture with
    sigma 4 to 40, clamped into the box."""
    dev = _device()
    p = torch.empty(n, 4, device=dev)
    if dist == "uniform":
        p[:, :3] = torch.rand(n, 3, device=dev, generator=g) * RANGE
    else:
        centre = torch.rand(components, 3, device=dev, generator=g) * RANGE
        sigma = 4.0 + 36.0 * torch.rand(components, 1, device=dev, generator=g)
        k = torch.randint(0, components, (n,), device=dev, generator=g)
        p[:, :3] = centre[k] + sigma[k] * torch.randn(n, 3, device=dev, generator=g)
    p[:, 3] = 1.0
    p[:, :3].clamp_(0.0, TOP)
    return p


def _clouds(case, seed):
    # the sizes belong to the case, the points to the seed
    r, g = random.Random(case["clouds"] * 31 + case["lo"] * 7 + case["hi"]), _generator(seed)
    out = []
    for _ in range(case["clouds"]):
        n = _log_int(r, case["lo"], case["hi"])
        out.append(_points(n, r.choice(["uniform", "mixture"]), g, r.randint(8, 64)))
    return out


def _training(case, seed):
    """Rows of a training batch, and parameters and Adam moments of a run under way."""
    g, dev, rows = _generator(seed), _device(), case["rows"]
    n = sum(s for _, s in MLP_SIZES)
    rand = lambda *shape: torch.randn(*shape, device=dev, generator=g)  # noqa: E731
    p = torch.cat([rand(64 * 16) * math.sqrt(2 / 16), 0.1 * rand(64), rand(64 * 64) * math.sqrt(2 / 64),
                   0.1 * rand(64), rand(64) * math.sqrt(1 / 64), 0.1 * rand(1)])
    x = torch.sort(2 * torch.rand(rows, 16, device=dev, generator=g) - 1, dim=1).values.contiguous()
    t = 0.2 * rand(rows)
    return p, x, t, 1e-2 * rand(n), 1e-4 * torch.rand(n, device=dev, generator=g) + 1e-6


def prepare(case, seed):
    rw = _package()
    kind = case["kind"]
    if kind == "train":
        p, x, t, m, v = _training(case, seed)
        return {"kind": kind, "rw": rw, "rows": case["rows"], "p": p, "x": x, "t": t, "m": m, "v": v,
                "grad": torch.zeros_like(p), "loss": torch.zeros(1, device=p.device)}
    if kind == "batch":
        return {"kind": kind, "batch": rw.Batch([c.cpu().numpy() for c in _clouds(case, seed)],
                                                case["bits"], octree_ratio=ROWS)}
    n = case["n"]
    points = _points(n, case["dist"], _generator(seed))
    app = rw.AppData(n, case["bits"], points=np.zeros((n, 4), np.float32), octree_ratio=ROWS)
    im = rw.ImStorage(n, case["bits"])
    if case.get("options"):
        im.set_options(case["options"])
    s = {"kind": kind, "rw": rw, "app": app, "im": im}
    if kind == "host":
        pin = lambda *shape, dtype: torch.zeros(*shape, dtype=dtype, pin_memory=True)  # noqa: E731
        s["points"] = pin(n, 4, dtype=torch.float32)
        s["points"].copy_(points)
        rows = app.oct_capacity
        s["out"] = {"children": pin(rows, 8, dtype=torch.int32), "corner": pin(rows, 4, dtype=torch.float32),
                    "cell_size": pin(rows, dtype=torch.float32), "child_node_mask": pin(rows, dtype=torch.int32),
                    "child_leaf_mask": pin(rows, dtype=torch.int32)}
        return s
    app.u_input_points.copy_(points)
    if kind == "learned":
        s["learned"] = rw.Learned(n)
        im.set_learned(s["learned"], rw.LEARNED_MLP)
    return s


# ---- one pass ----------------------------------------------------------------

def _tree(app):
    """What a pass leaves in AppData: its buffers, and the counts that say how much of
    them is filled."""
    return {"n_unique": app.get_n_unique(), "n_octree_nodes": app.get_n_octree_nodes(),
            "sorted_keys": app.u_morton_keys_alt, "unique_keys": app.u_morton_keys,
            "prefix_n": app.brt_prefix_n, "has_leaf_left": app.brt_has_leaf_left,
            "has_leaf_right": app.brt_has_leaf_right, "left_child": app.brt_left_child,
            "parents": app.brt_parents, "edge_count": app.u_edge_count,
            "edge_offset": app.u_edge_offset, "children": app.oct_children,
            "corner": app.oct_corner, "cell_size": app.oct_cell_size,
            "child_node_mask": app.oct_child_node_mask, "child_leaf_mask": app.oct_child_leaf_mask}


def run(s):
    kind = s["kind"]
    if kind == "train":
        rw = s["rw"]
        s["grad"].zero_()
        s["loss"].zero_()
        rw.mlp_grad(s["p"], s["x"], s["t"], s["rows"], s["grad"], s["loss"])
        rw.mlp_adam(s["p"], s["grad"], s["m"], s["v"], LR, STEP, BETA1, BETA2, EPS)
        return {k: s[k] for k in ("grad", "loss", "p", "m", "v")}
    if kind == "batch":
        b = s["batch"]
        b.run()
        return {"sorted_keys": b.morton_keys_alt, "unique_keys": b.morton_keys, "n_unique": b.n_unique,
                "n_octree_nodes": b.n_octree_nodes, "status": b.status, "prefix_n": b.prefix_n,
                "has_leaf_left": b.has_leaf_left, "has_leaf_right": b.has_leaf_right,
                "left_child": b.left_child, "parents": b.parents, "edge_count": b.edge_count,
                "edge_offset": b.edge_offset, "children": b.children, "corner": b.corner,
                "cell_size": b.cell_size, "child_node_mask": b.child_node_mask,
                "child_leaf_mask": b.child_leaf_mask}
    rw, app, im = s["rw"], s["app"], s["im"]
    if kind == "host":
        rw.run_host(app, im, s["points"].numpy(), s["out"])
        return dict(s["out"], n_octree_nodes=app.get_n_octree_nodes())
    if kind == "stages":
        for stage in (rw.run_stage1, rw.run_stage2, rw.run_stage3, rw.run_stage4, rw.run_stage5,
                      rw.run_stage6, rw.run_stage7):
            stage(app, im)
    else:
        rw.run_pipeline(app, im)
    return _tree(app)


# ---- what a pass cannot do without --------------------------------------------

def _tree_bytes(n, bits, dist):
    """Points read; sorted and unique keys, 19 bytes a radix-tree node and 60 bytes an
    octree row written.  Distinct keys and rows by the distribution (measured: 16.8M
    uniform points have 0.99 n distinct 30-bit keys, mixtures 0.49 n; 0.44 to 0.5 rows
    a key)."""
    k = bits // 8
    cells = 2.0 ** 30
    if bits == 64:
        u = n
    elif dist == "uniform":
        u = cells * -math.expm1(-n / cells)
    else:
        u = n / (1.0 + n / 16.8e6)
    return 16 * n + k * n + k * u + 19 * u + 60 * 0.47 * u


def work(case):
    kind = case["kind"]
    if kind == "train":
        rows, n = case["rows"], sum(s for _, s in MLP_SIZES)
        # x and t read; parameters and moments read and written, the gradient written
        return {"bytes": 68 * rows + 4 * 7 * n, "flops": 6 * rows * (16 * 64 + 64 * 64 + 64)}
    if kind == "batch":
        mean = (case["hi"] - case["lo"]) / math.log(case["hi"] / case["lo"])
        return {"bytes": case["clouds"] * _tree_bytes(mean, case["bits"], "uniform"), "flops": 0}
    total = _tree_bytes(case["n"], case["bits"], case["dist"])
    if kind == "host":
        # the points come over the link to device memory, the rows go back over it
        total += 2 * 16 * case["n"] + 2 * 60 * 0.47 * case["n"]
    return {"bytes": total, "flops": 0}


# ---- floating outputs in 64 bits ------------------------------------------------

def _spread(v, bits):
    out = torch.zeros_like(v)
    for b in range(bits):
        out |= ((v >> b) & 1) << (3 * b)
    return out


def _gather(v, bits):
    out = torch.zeros_like(v)
    for b in range(bits):
        out |= ((v >> (3 * b)) & 1) << b
    return out


def _bit_length(x):
    """Bits of positive int64 values, by the exponent of their halves as doubles."""
    hi, lo = x >> 32, x & 0xFFFFFFFF
    eh = torch.frexp(hi.double()).exponent
    el = torch.frexp(lo.double()).exponent
    return torch.where(hi > 0, eh + 32, el).long()


def _octree(points, key_bits, geometric=False):
    """(corner [m, 4], cell_size [m]) of the octree rows, in doubles: the radix tree's
    nodes as ranges of equal prefix found by search, then every row's cell."""
    word, axis = key_bits, (10 if key_bits == 32 else 21)
    code_bits = 3 * axis
    q = (points[:, :3].double() / RANGE * (1 << axis)).long()
    keys = _spread(q[:, 0], axis) | _spread(q[:, 1], axis) << 1 | _spread(q[:, 2], axis) << 2
    keys = torch.unique(keys)
    n = keys.numel() - 1  # gaps and nodes
    delta = lambda a, b: word - _bit_length(a ^ b) - 1  # noqa: E731
    d = delta(keys[:-1], keys[1:])
    # gap g splits the keys that share its prefix of d[g] bits (after the sign bit)
    low = word - 1 - d
    base = (keys[:-1] >> low) << low
    first = torch.searchsorted(keys, base)
    last = torch.searchsorted(keys, base + (torch.ones_like(low) << low) - 1, right=True) - 1
    dl = torch.where(first > 0, d[(first - 1).clamp(min=0)], -1)
    dr = torch.where(last < n, d[last.clamp(max=n - 1)], -1)
    node = torch.where(dr > dl, last, first)
    inner = (first > 0) | (last < n)
    # the root is computed over all keys but the last
    root_true, root = int(delta(keys[:1], keys[-1:])), int(delta(keys[:1], keys[-2:-1]))
    parent = torch.maximum(dl, dr)
    parent = torch.where(parent == root_true, torch.full_like(parent, root), parent)
    less = 1 if geometric and key_bits == 32 else 0
    prefix = torch.zeros(n, dtype=torch.long, device=keys.device)
    count = torch.zeros_like(prefix)
    prefix[0] = root - less
    prefix[node[inner]] = d[inner] - less
    count[node[inner]] = ((d - less) // 3 - (parent - less) // 3)[inner]
    if int(count.min()) < 0:
        return None  # rows that are written twice: left to the order of the nodes
    off = torch.cumsum(count, 0) - count
    owner = torch.repeat_interleave(torch.arange(n, device=keys.device), count)
    k = torch.arange(owner.numel(), device=keys.device) - off[owner]
    level = prefix[owner] // 3 - k
    cut = code_bits - 3 * level
    code = (keys[owner] >> cut) << cut
    corner = torch.ones(owner.numel(), 4, dtype=torch.float64, device=keys.device)
    for a in range(3):
        corner[:, a] = _gather(code >> a, axis).double() / (1 << axis) * RANGE
    return corner, RANGE / torch.exp2((level - int(prefix[0]) // 3).double())


def _exact_train(case, seed):
    p, x, t, m, v = (a.double() for a in _training(case, seed))
    q, at = {}, 0
    for name, size in MLP_SIZES:
        q[name], at = p[at:at + size], at + size
    half = lambda w: w.float().bfloat16().double()  # noqa: E731  weights are used rounded to BF16
    w1, w2, w3 = half(q["w1"]).view(64, 16), half(q["w2"]).view(64, 64), half(q["w3"])
    z1 = x @ w1.T + q["b1"]
    h1 = z1.clamp(min=0)
    z2 = h1 @ w2.T + q["b2"]
    h2 = z2.clamp(min=0)
    e = h2 @ w3 + q["b3"] - t
    dy = 2.0 * e / case["rows"]
    dz2 = dy[:, None] * w3 * (z2 > 0)
    dz1 = (dz2 @ w2) * (z1 > 0)
    g = torch.cat([(dz1.T @ x).reshape(-1), dz1.sum(0), (dz2.T @ h1).reshape(-1), dz2.sum(0), h2.T @ dy,
                   dy.sum().reshape(1)])
    m = BETA1 * m + (1 - BETA1) * g
    v = BETA2 * v + (1 - BETA2) * g * g
    p = p - LR * (m / (1 - BETA1 ** STEP)) / ((v / (1 - BETA2 ** STEP)).sqrt() + EPS)
    return {"grad": g, "loss": (e * e).sum().reshape(1), "p": p, "m": m, "v": v}


def exact(case, seed):
    kind = case["kind"]
    if kind == "train":
        return _exact_train(case, seed)
    if kind == "batch":
        clouds, bits, geometric = _clouds(case, seed), case["bits"], False
    else:
        clouds = [_points(case["n"], case["dist"], _generator(seed))]
        bits, geometric = case["bits"], bool(case.get("options", 0) & 1)
    # the buffers as they are filled: rows past a cloud's own stay zero
    rows = [max(1, int(np.float32(c.shape[0]) * np.float32(ROWS))) for c in clouds]
    corner = torch.zeros(sum(rows), 4, dtype=torch.float64, device=_device())
    cell = torch.zeros(sum(rows), dtype=torch.float64, device=_device())
    at = 0
    for c, r in zip(clouds, rows):
        tree = _octree(c, bits, geometric)
        if tree is None or tree[1].numel() + 1 > r:
            return None
        m = tree[1].numel()
        corner[at:at + m], cell[at:at + m] = tree
        at += r
    return {"corner": corner, "cell_size": cell}
