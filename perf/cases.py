"""The partitioner's workloads as its users run them, for timing.

Every case goes through the Python binding of the C ABI (the package
``dac_g-kway_b200``): one graph resident on the GPU, one graph in host memory,
one graph for several part counts, a batch of small graphs, or a METIS file.
The graphs are made on the GPU from the seed, with the shapes, degrees and
weights of the workloads in ``bench.py`` and ``generators.py``:

* ``mesh``     planar triangulation (mean degree 6, unit weights; weighted on
               request), vertices in random order like a point cloud's
               triangulation (``shuffled``) or in row order like a mesher's;
* ``grid27``   3D grid of the 27-point stencil with 1% of the stencil's edges
               missing, unit weights, natural order;
* ``road``     spanning tree plus 8% of the remaining short edges (mean degree
               2.3), vertices in random order;
* ``circuit``  levelised netlist: Poisson fan-in from the five levels before,
               0.1% of vertices with power-law fan-out up to 10k, edge weights
               1..8, vertex weights 1..4.

Outputs are whole numbers (part ids and cuts).
"""
import importlib
import math
import os
import random
import tempfile

import numpy as np
import torch

pkg = importlib.import_module("dac_g-kway_b200")

_kept = {}


def _handle():
    """The handle a program keeps for all its partitions."""
    if "handle" not in _kept:
        _kept["handle"] = pkg.Handle(0)
    return _kept["handle"]


def _server():
    """The server a program keeps for its batches."""
    if "server" not in _kept:
        _kept["server"] = pkg.Server(0)
    return _kept["server"]


# ---------------------------------------------------------------- graphs ----
def _csr(n, lo, hi, gen, dev, weighted):
    """Symmetric CSR (int32) of undirected edges lo < hi; duplicates merge."""
    key = torch.unique(lo * n + hi)
    lo, hi = key // n, key % n
    ne = key.numel()
    w = (torch.randint(1, 9, (ne,), generator=gen, device=dev, dtype=torch.int32) if weighted
         else torch.ones(ne, dtype=torch.int32, device=dev))
    vw = (torch.randint(1, 5, (n,), generator=gen, device=dev, dtype=torch.int32) if weighted
          else torch.ones(n, dtype=torch.int32, device=dev))
    full, order = torch.sort(torch.cat([key, hi * n + lo]))
    adj = (full % n).to(torch.int32)
    deg = torch.bincount(full // n, minlength=n)
    xadj = torch.zeros(n + 1, dtype=torch.int32, device=dev)
    xadj[1:] = torch.cumsum(deg, 0)
    return xadj, adj, torch.cat([w, w])[order], vw


def _renumber(n, lo, hi, gen, dev):
    p = torch.randperm(n, generator=gen, device=dev)
    a, b = p[lo], p[hi]
    return torch.minimum(a, b), torch.maximum(a, b)


def _mesh_edges(n, gen, dev):
    """Right, down and one diagonal per cell of a grid of n points."""
    nx = max(2, int(round(math.sqrt(n))))
    v = torch.arange(n, device=dev)
    x = v % nx
    right = v[(x < nx - 1) & (v + 1 < n)]
    down = v[v + nx < n]
    cell = v[(x < nx - 1) & (v + nx + 1 < n)]
    flip = torch.rand(cell.numel(), generator=gen, device=dev) < 0.5
    dlo = torch.where(flip, cell + 1, cell)
    dhi = torch.where(flip, cell + nx, cell + nx + 1)
    return torch.cat([right, down, dlo]), torch.cat([right + 1, down + nx, dhi])


def _mesh(n, gen, dev, shuffled, weighted):
    lo, hi = _mesh_edges(n, gen, dev)
    if shuffled:
        lo, hi = _renumber(n, lo, hi, gen, dev)
    return _csr(n, lo, hi, gen, dev, weighted)


def _grid27(nx, ny, nz, gen, dev):
    n = nx * ny * nz
    v = torch.arange(n, device=dev)
    x, y, z = v % nx, (v // nx) % ny, v // (nx * ny)
    los, his = [], []
    for dz in (-1, 0, 1):
        for dy in (-1, 0, 1):
            for dx in (-1, 0, 1):
                if (dz, dy, dx) <= (0, 0, 0):
                    continue
                ok = (x + dx >= 0) & (x + dx < nx) & (y + dy >= 0) & (y + dy < ny) & (z + dz < nz)
                ok &= torch.rand(n, generator=gen, device=dev) >= 0.01
                a = v[ok]
                los.append(a)
                his.append(a + dx + nx * (dy + ny * dz))
    return _csr(n, torch.cat(los), torch.cat(his), gen, dev, False)


def _road(n, gen, dev):
    nx = max(2, int(round(math.sqrt(n))))
    v = torch.arange(1, n, device=dev)
    # every vertex joins its left or upper neighbour: a spanning tree
    left = (v % nx != 0) & ((v < nx) | (torch.rand(n - 1, generator=gen, device=dev) < 0.5))
    tree = torch.where(left, v - 1, torch.clamp(v - nx, min=0))
    lo, hi = _mesh_edges(n, gen, dev)
    extra = torch.rand(lo.numel(), generator=gen, device=dev) < 0.08
    lo, hi = _renumber(n, torch.cat([tree, lo[extra]]), torch.cat([v, hi[extra]]), gen, dev)
    return _csr(n, lo, hi, gen, dev, False)


def _circuit(n, gen, dev):
    levels = min(200, max(8, n // 200))
    hub_max = max(16, min(10000, n // 10))
    per = max(1, n // levels)
    fan = torch.poisson(torch.full((n,), 2.5, device=dev), generator=gen).to(torch.int64)
    fan[:per] = 0
    src = torch.repeat_interleave(torch.arange(n, device=dev), fan)
    m0 = src.numel()
    lv = torch.clamp(src // per, max=levels - 1)
    back = torch.randint(1, 6, (m0,), generator=gen, device=dev)
    lo = torch.clamp(lv - back, min=0) * per
    hi = lv * per
    span = torch.clamp(hi - lo, min=1)
    rel = (src - lv * per).to(torch.float64) / per
    width = torch.clamp(span // 20, min=1)
    off = ((torch.rand(m0, generator=gen, device=dev) * 2 - 1) * width).to(torch.int64)
    near = torch.minimum(torch.clamp(lo + (rel * span).to(torch.int64) + off, min=0), lo + span - 1)
    near = torch.maximum(near, lo)
    far = lo + (torch.rand(m0, generator=gen, device=dev, dtype=torch.float64) * span).to(torch.int64)
    dst = torch.where(torch.rand(m0, generator=gen, device=dev) < 0.9, near, far)
    n_hub = max(1, round(0.001 * n))
    hubs = torch.randperm(n, generator=gen, device=dev)[:n_hub]
    u = torch.rand(n_hub, generator=gen, device=dev, dtype=torch.float64).clamp(min=1e-12)
    fo = torch.clamp(((u ** (-1.0 / 1.2) - 1.0) * 20 + 10).to(torch.int64), max=hub_max)
    hs = torch.repeat_interleave(hubs, fo)
    hd = torch.randint(0, n, (hs.numel(),), generator=gen, device=dev)
    a, b = torch.cat([src, hs]), torch.cat([dst, hd])
    keep = a != b
    a, b = a[keep], b[keep]
    return _csr(n, torch.minimum(a, b), torch.maximum(a, b), gen, dev, True)


def _graph(kind, n, gen, dev, shuffled=True, weighted=False):
    if kind == "mesh":
        return _mesh(n, gen, dev, shuffled, weighted)
    if kind == "grid27":
        nx, ny, nz = _box(n)
        return _grid27(nx, ny, nz, gen, dev)
    if kind == "road":
        return _road(n, gen, dev)
    return _circuit(n, gen, dev)


def _box(n):
    """Sides of a 27-point grid of about n points (960000: 100 x 100 x 96)."""
    if n == 960000:
        return 100, 100, 96
    a = max(2, int(round(n ** (1 / 3))))
    return a, a, max(2, int(round(n / (a * a))))


# ----------------------------------------------------------------- cases ----
def listed():
    return [
        # the smallest graphs a program partitions: the 2048-point fixture's
        # size, where launches and round trips count
        {"name": "mesh_2k_k8", "entry": "device", "kind": "mesh", "n": 2048, "k": 8, "shuffled": True,
         "weighted": False, "balanced": True},
        # a block of a netlist with weights, hubs and an odd part count
        {"name": "circuit_30k_k24", "entry": "device", "kind": "circuit", "n": 30011, "k": 24, "balanced": True},
        # an ordinary mesh from a mesher, in its own vertex order
        {"name": "mesh_100k_k32", "entry": "device", "kind": "mesh", "n": 99991, "k": 32, "shuffled": False,
         "weighted": False, "balanced": True},
        # a weighted mesh in the reference's own mode (no balance rounds)
        {"name": "mesh_260k_k128_refmode", "entry": "device", "kind": "mesh", "n": 262144, "k": 128,
         "shuffled": True, "weighted": True, "balanced": False},
        # the benchmark's headline: a million-point triangulation on the GPU
        {"name": "mesh_1m_k64", "entry": "device", "kind": "mesh", "n": 1 << 20, "k": 64, "shuffled": True,
         "weighted": False, "balanced": True},
        # the same size from host memory and back, as a C caller has it
        {"name": "mesh_1m_k64_host", "entry": "host", "kind": "mesh", "n": 1 << 20, "k": 64, "shuffled": False,
         "weighted": False, "balanced": True},
        # a volume mesh: the 27-point grid of the large configurations
        {"name": "grid27_960k_k64", "entry": "device", "kind": "grid27", "n": 960000, "k": 64, "balanced": True},
        # a continental road network, many parts
        {"name": "road_12m_k256", "entry": "device", "kind": "road", "n": 12000000, "k": 256, "balanced": True},
        # a whole chip's timing graph: the largest work
        {"name": "circuit_4m_k256", "entry": "device", "kind": "circuit", "n": 4000000, "k": 256,
         "balanced": True},
        # many small independent graphs in one call
        {"name": "batch_256", "entry": "batch", "graphs": 256, "n_min": 1000, "n_max": 64000},
        # one graph for a sweep of part counts
        {"name": "mesh_200k_ks", "entry": "multi_k", "kind": "mesh", "n": 200003, "k": 128, "shuffled": True,
         "weighted": False},
        # the command line's path: METIS file in, part file out
        {"name": "file_100k_k16", "entry": "file", "kind": "mesh", "n": 100000, "k": 16, "shuffled": True,
         "weighted": False},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _parts(rng, n, most):
    ks = [k for k in (2, 3, 4, 6, 8, 12, 16, 24, 32, 48, 64, 100, 128, 200, 256) if k <= most and n >= 100 * k]
    return rng.choice(ks)


def draw(rng: random.Random):
    entry = rng.choice(["device"] * 6 + ["host", "batch", "multi_k", "file"])
    if entry == "batch":
        return {"entry": "batch", "graphs": _log_int(rng, 8, 256), "n_min": 1000, "n_max": _log_int(rng, 4000, 64000)}
    if entry == "file":
        n = _log_int(rng, 2000, 100000)
        return {"entry": "file", "kind": "mesh", "n": n, "k": _parts(rng, n, 64), "shuffled": rng.random() < 0.5,
                "weighted": rng.random() < 0.3}
    if entry == "multi_k":
        n = _log_int(rng, 20000, 400000)
        return {"entry": "multi_k", "kind": "mesh", "n": n, "k": rng.choice([k for k in (16, 64, 128) if n >= 100 * k]),
                "shuffled": rng.random() < 0.5, "weighted": rng.random() < 0.3}
    kind = rng.choice(["mesh", "mesh", "grid27", "road", "circuit"])
    n = _log_int(rng, 2000, {"mesh": 2000000, "grid27": 960000, "road": 6000000, "circuit": 2000000}[kind])
    c = {"entry": entry, "kind": kind, "n": n, "k": _parts(rng, n, 256), "balanced": rng.random() < 0.75}
    if kind == "mesh":
        c["shuffled"] = rng.random() < 0.6
        c["weighted"] = rng.random() < 0.3
    return c


def _sweep(k):
    """Part counts of a sweep up to k: powers of two."""
    ks = []
    while k >= 2:
        ks.append(k)
        k //= 2
    return ks[::-1]


def _batch_plan(case, seed):
    """(kind, n, k) of each graph of a batch; the sizes belong to the case."""
    r = random.Random(case["graphs"] * 1000003 + case["n_max"])
    return [(("mesh", "grid27", "circuit")[i % 3], _log_int(r, case["n_min"], case["n_max"]),
             r.choice([2, 4, 8, 16, 32])) for i in range(case["graphs"])]


class _HostGraph:
    def __init__(self, g):
        self.xadj, self.adjncy, self.adjwgt, self.vwgt = (a.cpu().numpy() for a in g)


def _pinned(a):
    t = torch.empty(a.shape, dtype=torch.int32, pin_memory=True)
    t.copy_(torch.as_tensor(a))
    return t.numpy()


def _metis_text(g, weighted):
    x, a, w, vw = (t.cpu().numpy() for t in g)
    n = x.shape[0] - 1
    head = "%d %d%s\n" % (n, a.shape[0] // 2, " 011" if weighted else "")
    if weighted:
        tok = list(map("%d %d".__mod__, zip((a + 1).tolist(), w.tolist())))
        vws = vw.tolist()
    else:
        tok = list(map(str, (a + 1).tolist()))
    xs = x.tolist()
    lines = [" ".join(([str(vws[v])] if weighted else []) + tok[xs[v]:xs[v + 1]]) for v in range(n)]
    return head + "\n".join(lines) + "\n"


def prepare(case, seed):
    dev = torch.device("cuda", 0)
    gen = torch.Generator(device=dev)
    gen.manual_seed(int(seed) * 7919 + 17)
    entry = case["entry"]
    state = {"entry": entry}
    if entry == "batch":
        plan = _batch_plan(case, seed)
        graphs = [_HostGraph(_graph(kind, n, gen, dev)) for kind, n, _ in plan]
        *arrays, ptr = pkg.concat_graphs(graphs)
        state.update(server=_server(), arrays=arrays, ptr=ptr, ks=np.array([k for _, _, k in plan], np.int32))
        return state
    state["handle"] = _handle()
    g = _graph(case["kind"], case["n"], gen, dev, case.get("shuffled", True), case.get("weighted", False))
    n = g[0].numel() - 1
    state["k"] = case["k"]
    if entry == "device":
        state.update(graph=g, part=torch.empty(n, dtype=torch.int32, device=dev),
                     opts=pkg.default_options(enforce_balance=1 if case["balanced"] else 0))
    elif entry == "host":
        state.update(graph=[_pinned(a.cpu()) for a in g], part=_pinned(np.zeros(n, np.int32)),
                     opts=pkg.default_options(enforce_balance=1 if case["balanced"] else 0))
    elif entry == "multi_k":
        state.update(graph=[_pinned(a.cpu()) for a in g], ks=_sweep(case["k"]))
    else:
        tmp = tempfile.TemporaryDirectory(prefix="gkw_cases_")
        path = os.path.join(tmp.name, "in.graph")
        with open(path, "w") as f:
            f.write(_metis_text(g, case["weighted"]))
        state.update(tmp=tmp, path=path, out=os.path.join(tmp.name, "out.part"))
    torch.cuda.synchronize()   # the handle's stream does not wait for torch's
    return state


def run(state):
    entry = state["entry"]
    if entry == "device":
        cut, _ = state["handle"].partition_device(*state["graph"], state["k"], state["part"], opts=state["opts"])
        return {"part": state["part"], "cut": cut}
    if entry == "host":
        part, cut, _ = state["handle"].partition(*state["graph"], state["k"], opts=state["opts"],
                                                 part_out=state["part"])
        return {"part": part, "cut": cut}
    if entry == "batch":
        part, cuts, status = state["server"].partition_batch(*state["arrays"], state["ptr"], state["ks"])
        return {"part": part, "cuts": cuts, "status": status}
    if entry == "multi_k":
        parts, cuts = state["handle"].partition_multi_k(*state["graph"], state["ks"])
        return {"parts": parts, "cuts": cuts}
    g = state["handle"].read_metis_device(state["path"])
    part = torch.empty(g[0].numel() - 1, dtype=torch.int32, device=g[0].device)
    cut, _ = state["handle"].partition_device(*g, state["k"], part)
    state["handle"].write_partition_device(state["out"], part)
    return {"part": part, "cut": cut}


def _entries(kind, n):
    """About how many CSR entries a graph of the kind has."""
    if kind == "mesh":
        return 6.0 * n
    if kind == "grid27":
        x, y, z = _box(n)
        return 0.99 * ((3 * x - 2.0) * (3 * y - 2.0) * (3 * z - 2.0) - x * y * z)
    if kind == "road":
        return 2.3 * n
    return 5.2 * n


def work(case):
    """The graph read once (row offsets, ids, edge and vertex weights), the
    part ids written once; for a file, its text instead of the arrays."""
    if case["entry"] == "batch":
        plan = _batch_plan(case, 0)
        return {"bytes": sum(12.0 * n + 8.0 * _entries(kind, n) for kind, n, _ in plan), "flops": 0}
    n = case["n"]
    m = _entries(case["kind"], n)
    if case["entry"] == "file":
        digits = 1 + math.log10(max(n, 10))
        return {"bytes": m * digits * (1.3 if case["weighted"] else 1.0) + 3.0 * n, "flops": 0}
    outs = len(_sweep(case["k"])) if case["entry"] == "multi_k" else 1
    return {"bytes": 8.0 * n + 8.0 * m + 4.0 * n * outs, "flops": 0}


def exact(case, seed):
    """Every output is a whole number: nothing has a value in 64 bits."""
    return None
