"""The work whose speed is measured: colorings through the library's public entry points.

A case is one coloring job, as a program that uses the library runs it: priorities by a heuristic,
Jones-Plassmann, and often Culberson rounds, on a CSR that already lives on the device ("graph"),
on a batch of graphs ("batch"), or on host buffers through the reference-named drop-in call
("drop-in").  The graph families, sizes, degrees and heuristics are those of the benchmark and the
tests: Erdos-Renyi, R-MAT (power law), random geometric graphs and 27-point stencils (meshes),
from a thousand to sixteen million vertices.

Graphs are made from the seed alone, on the device with torch, so that preparing the largest case
takes seconds.  The model weights are the benchmark's synthetic ones for each layer count: a program
loads one model and colors many graphs with it.
"""
import ctypes as C
import math
import os
import random
import sys
import tempfile

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "gnn-coloring_b200"))
import gnn_coloring as gcn  # noqa: E402

DEV = "cuda"
STENCIL = [(dx, dy, dz) for dz in (-1, 0, 1) for dy in (-1, 0, 1) for dx in (-1, 0, 1) if (dx, dy, dz) != (0, 0, 0)]


def listed():
    return [
        # the smallest graphs of a mixed stream, one call each: launches and latency are all there is
        dict(name="er_1k_ff", kind="graph", family="er", n=1000, degree=16.0, heuristic="FF", recolor=0),
        # the benchmark's Erdos-Renyi configuration (n = 65,536, m = 524,288): a plain heuristic, the
        # GNN, and the peeling heuristic with its many rounds
        dict(name="er_65k_lf", kind="graph", family="er", n=65536, degree=16.0, heuristic="LF", recolor=0),
        dict(name="er_65k_gnn3", kind="graph", family="er", n=65536, degree=16.0, heuristic="GNN3", recolor=0),
        dict(name="er_65k_sl", kind="graph", family="er", n=65536, degree=16.0, heuristic="SL", recolor=0),
        # a medium power-law graph of odd size, polished by two Culberson rounds
        dict(name="rmat_100003_llf_c2", kind="graph", family="rmat", n=100003, degree=16.0, heuristic="LLF", recolor=2),
        # smallest degree last on a large power-law graph: hundreds of peeling rounds
        dict(name="rmat_1m_sl", kind="graph", family="rmat", n=1 << 20, degree=32.0, heuristic="SL", recolor=0),
        # the benchmark's headline: GNN3 + Jones-Plassmann on R-MAT scale 22, edge factor 16
        dict(name="rmat_4m_gnn3", kind="graph", family="rmat", n=1 << 22, degree=32.0, heuristic="GNN3", recolor=0),
        # the benchmark's mesh configurations with the reference's `-c 10` (the first coloring and nine
        # Culberson rounds): a random geometric graph and the largest job, a 256^3 stencil
        dict(name="rgg_8m_gnn4_c9", kind="graph", family="rgg", n=1 << 23, degree=12.0, heuristic="GNN4", recolor=9),
        dict(name="stencil_256_gnn4_c9", kind="graph", family="stencil", nx=256, ny=256, nz=256, holes=8,
             heuristic="GNN4", recolor=9),
        # a ragged mesh with cut-outs in its natural vertex order, first fit: the cheapest way to color a
        # matrix or a simulation grid
        dict(name="stencil_97x61x113_ff", kind="graph", family="stencil", nx=97, ny=61, nz=113, holes=8,
             heuristic="FF", recolor=0),
        # a batch of mixed ER / R-MAT graphs of 1,000 to 200,000 vertices, one replayed pass
        dict(name="batch_64_gnn2", kind="batch", graphs=64, n_min=1000, n_max=200000, heuristic="GNN2", recolor=0),
        # the reference-named call from page-locked host buffers: upload, GNN3, coloring, both results back
        dict(name="dropin_rmat_300007_gnn3", kind="drop-in", family="rmat", n=300007, degree=32.0, heuristic="GNN3",
             recolor=0),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    heuristics = ["FF", "LF", "LLF", "SL", "SLL", "GNN2", "GNN3", "GNN4"]
    rounds = [0, 0, 0, 1, 2, 4, 9]
    kind = rng.choices(["graph", "batch", "drop-in"], [10, 2, 1])[0]
    if kind == "batch":
        hi = _log_uniform(rng, 4000, 200000)
        return dict(kind="batch", graphs=_log_uniform(rng, 2, 96), n_min=1000, n_max=hi,
                    heuristic=rng.choice(["FF", "LF", "LLF", "GNN2", "GNN3"]), recolor=rng.choice([0, 0, 1]))
    if kind == "drop-in":
        return dict(kind="drop-in", family=rng.choice(["er", "rmat"]), n=_log_uniform(rng, 1000, 1 << 19),
                    degree=round(rng.uniform(8.0, 32.0), 2), heuristic=rng.choice(["LF", "GNN3"]), recolor=0)
    family = rng.choice(["er", "rmat", "rgg", "stencil"])
    case = dict(kind="graph", family=family)
    if family == "er":
        case.update(n=_log_uniform(rng, 1000, 1 << 21), degree=round(rng.uniform(8.0, 32.0), 2))
    elif family == "rmat":
        case.update(n=_log_uniform(rng, 1000, 1 << 22), degree=round(rng.uniform(8.0, 32.0), 2))
    elif family == "rgg":
        case.update(n=_log_uniform(rng, 10000, 1 << 22), degree=round(rng.uniform(8.0, 16.0), 2))
    else:
        case.update(nx=rng.randint(20, 160), ny=rng.randint(20, 160), nz=rng.randint(20, 160), holes=rng.randint(1, 12))
    case.update(heuristic=rng.choice(heuristics), recolor=rng.choice(rounds))
    return case


# ---- graphs on the device --------------------------------------------------------------------------


def _generator(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _csr(n, i, j):
    """Simple, symmetric, sorted CSR (int32 tensors) of the undirected pairs (i, j)."""
    keep = i != j
    i, j = i[keep], j[keep]
    key = torch.cat([i * n + j, j * n + i])
    del i, j, keep
    return _csr_from_keys(n, torch.unique(key))


def _csr_from_keys(n, key):
    """CSR of the directed entries row * n + column, given sorted and distinct."""
    E = (key % n).to(torch.int32)
    V = torch.searchsorted(key, torch.arange(n + 1, device=DEV) * n).to(torch.int32)
    return V, E


def _er(n, degree, gen):
    m = int(round(n * degree / 2))
    return _csr(n, torch.randint(n, (m,), device=DEV, generator=gen), torch.randint(n, (m,), device=DEV, generator=gen))


def _rmat(n, degree, gen):
    """R-MAT with (a, b, c) = (0.57, 0.19, 0.19) over 2^ceil(log2 n) ids, samples outside n dropped."""
    m = int(round(n * degree / 2))
    i = torch.zeros(m, dtype=torch.int64, device=DEV)
    j = torch.zeros(m, dtype=torch.int64, device=DEV)
    for _ in range(max(1, (n - 1).bit_length())):
        u = torch.rand(m, device=DEV, generator=gen)
        down = u >= 0.76
        right = ((u >= 0.57) & (u < 0.76)) | (u >= 0.95)
        i = (i << 1) + down
        j = (j << 1) + right
    keep = (i < n) & (j < n)
    return _csr(n, i[keep], j[keep])


def _rgg(n, degree, gen):
    """n uniform points of the unit square, joined when closer than the radius for this mean degree."""
    r = math.sqrt(degree / (math.pi * n))
    g = max(1, int(1.0 / r))  # cells at least r wide
    x = torch.rand(n, dtype=torch.float64, device=DEV, generator=gen)
    y = torch.rand(n, dtype=torch.float64, device=DEV, generator=gen)
    cx, cy = (x * g).long().clamp_(max=g - 1), (y * g).long().clamp_(max=g - 1)
    cell, order = torch.sort(cy * g + cx)
    first = torch.searchsorted(cell, torch.arange(g * g + 1, device=DEV))
    keys = []
    for a in range(0, n, 1 << 20):
        p = torch.arange(a, min(n, a + (1 << 20)), device=DEV)
        for dy in (-1, 0, 1):  # the three cells of a row are one run of the sorted points
            row = cy[p] + dy
            inside = (row >= 0) & (row < g)
            row = row.clamp(0, g - 1)
            beg = first[row * g + (cx[p] - 1).clamp(min=0)]
            cnt = torch.where(inside, first[row * g + (cx[p] + 1).clamp(max=g - 1) + 1] - beg, 0)
            src = torch.repeat_interleave(p, cnt)
            off = torch.arange(src.numel(), device=DEV) - torch.repeat_interleave(torch.cumsum(cnt, 0) - cnt, cnt)
            dst = order[torch.repeat_interleave(beg, cnt) + off]
            near = ((x[src] - x[dst]) ** 2 + (y[src] - y[dst]) ** 2 < r * r) & (src != dst)
            keys.append(src[near] * n + dst[near])
    return _csr_from_keys(n, torch.sort(torch.cat(keys))[0])


def _stencil(nx, ny, nz, holes, gen):
    """27-point stencil in natural order; `holes` seeded boxes of cells (up to an eighth of each side
    long) have no neighbours, as cells outside the domain."""
    n = nx * ny * nz
    active = torch.ones((nz, ny, nx), dtype=torch.bool, device=DEV)
    at = torch.rand((holes, 6), generator=gen, device=DEV).cpu().tolist()
    for b in at:
        lo = [int(b[k] * s) for k, s in enumerate((nz, ny, nx))]
        ln = [1 + int(b[3 + k] * s / 8) for k, s in enumerate((nz, ny, nx))]
        active[lo[0]:lo[0] + ln[0], lo[1]:lo[1] + ln[1], lo[2]:lo[2] + ln[2]] = False
    ids = torch.arange(n, dtype=torch.int32, device=DEV)
    act = active.view(-1)
    cols, oks = [], []
    ix, iy, iz = ids % nx, (ids // nx) % ny, ids // (nx * ny)
    for dx, dy, dz in STENCIL:  # ascending neighbour id
        ok = (ix + dx >= 0) & (ix + dx < nx) & (iy + dy >= 0) & (iy + dy < ny) & (iz + dz >= 0) & (iz + dz < nz)
        v = ids + (dx + dy * nx + dz * nx * ny)
        oks.append(ok & act & act[torch.where(ok, v, ids).long()])
        cols.append(v)
    mask = torch.stack(oks, 1)
    V = torch.zeros(n + 1, dtype=torch.int32, device=DEV)
    V[1:] = torch.cumsum(mask.sum(1), 0)
    return V, torch.stack(cols, 1)[mask]


def _graph(case, seed):
    """(n, V, E) of a case on the device."""
    gen = _generator(seed)
    if case["family"] == "stencil":
        V, E = _stencil(case["nx"], case["ny"], case["nz"], case["holes"], gen)
        return V.numel() - 1, V, E
    V, E = {"er": _er, "rmat": _rmat, "rgg": _rgg}[case["family"]](case["n"], case["degree"], gen)
    return case["n"], V, E


def _batch_sizes(case):
    """The batch's vertex counts: log-uniform in [n_min, n_max], the same for every seed."""
    rng = random.Random(case["graphs"])
    return [_log_uniform(rng, case["n_min"], case["n_max"]) for _ in range(case["graphs"])]


def _batch(case, seed):
    """(voff, V with global row offsets, E with local ids): ER (mean degree 8 to 32) and R-MAT (edge
    factor 8) graphs in turn."""
    gen = _generator(seed)
    sizes = _batch_sizes(case)
    rng = random.Random(case["graphs"] + 1)
    Vs, Es, base = [torch.zeros(1, dtype=torch.int32, device=DEV)], [], 0
    for k, n in enumerate(sizes):
        V, E = _er(n, rng.uniform(8.0, 32.0), gen) if k % 2 == 0 else _rmat(n, 16.0, gen)
        Vs.append(V[1:] + base)
        Es.append(E)
        base += E.numel()
    return np.cumsum([0] + sizes, dtype=np.uint32), torch.cat(Vs), torch.cat(Es)


def _model(case):
    """(params, md) of the case's GNN: the benchmark's synthetic weights."""
    return gcn.synthetic_model(_layers(case), 1000 + _layers(case))


def _layers(case):
    return int(case["heuristic"][3:]) if case["heuristic"].startswith("GNN") else 0


# ---- states ------------------------------------------------------------------------------------------

_context = None


def _ctx():
    """The program's one context, as every program that uses the library holds."""
    global _context
    if _context is None:
        _context = gcn.Context(0)
    return _context


class _View:
    """A device buffer of the library, for torch (no copy); it keeps the buffer's owner alive."""

    def __init__(self, owner, ptr, n, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = dict(shape=(n,), typestr=typestr, data=(ptr, False), version=2)


def _tensor(owner, ptr, n, typestr="<i4"):
    return torch.as_tensor(_View(owner, C.cast(ptr, C.c_void_p).value, n, typestr), device=DEV)


class _DeviceGraph(gcn.Graph):
    """A graph over a CSR that already lives on the device (gc_graph_wrap_device)."""

    def __init__(self, ctx, n, V, E):
        self.ctx, self.N, self.V, self.E = ctx, n, V, E
        h = gcn.vp()
        ctx.check(gcn.lib.gc_graph_wrap_device(ctx.h, n, E.numel(), V.data_ptr(), E.data_ptr(), C.byref(h)), "wrap")
        self.h = h
        gcn._live_objects.add(self)


class _Job:
    pass


def _prepare_graph(case, seed):
    s = _Job()
    n, V, E = _graph(case, seed)
    torch.cuda.synchronize()
    L = _layers(case)
    s.model = gcn.Model(_ctx(), *_model(case)) if L else None
    s.graph = _DeviceGraph(_ctx(), n, V, E)
    s.heuristic, s.recolor = ("GNN" if L else case["heuristic"]), case["recolor"]
    s.out = {"color": _tensor(s.graph, gcn.lib.gc_graph_device_colors(s.graph.h), n)}
    if not s.recolor:  # (a Culberson round replaces the priorities by the colors before it)
        s.out["priority"] = _tensor(s.graph, gcn.lib.gc_graph_device_keys(s.graph.h), n, "<f4" if L else "<i4")
    return s


def _run_graph(s):
    s.graph.priority(s.heuristic, s.model)
    count = s.graph.color(s.recolor)
    return dict(s.out, colors=count)


def _prepare_batch(case, seed):
    s = _Job()
    L = _layers(case)
    voff, V, E = _batch(case, seed)
    s.model = gcn.Model(_ctx(), *_model(case)) if L else None
    s.batch = gcn.Batch(_ctx(), voff, V.cpu().numpy().view(np.uint32), E.cpu().numpy().view(np.uint32))
    s.heuristic, s.recolor = ("GNN" if L else case["heuristic"]), case["recolor"]
    g = gcn.vp(gcn.lib.gc_batch_graph(s.batch.h))
    n = s.batch.N
    s.out = {"color": _tensor(s.batch, gcn.lib.gc_graph_device_colors(g), n)}
    if not s.recolor:
        s.out["priority"] = _tensor(s.batch, gcn.lib.gc_graph_device_keys(g), n, "<f4" if L else "<i4")
    return s


def _run_batch(s):
    counts = s.batch.color(s.heuristic, s.model, s.recolor)
    return dict(s.out, colors=counts)


class _DropIn(_Job):
    """The reference's calls: X_setup, jones_plassmann_setup once, then X_internal_par per graph."""

    def __del__(self):
        gcn.lib.jones_plassmann_cleanup(self.jp)
        (gcn.lib.gnn_cleanup if self.gnn else gcn.lib.largest_degree_first_cleanup)(self.heur)


for _name in ("largest_degree_first_setup",):
    gcn._sig(_name, gcn.vp, C.c_uint32, C.c_uint32)
gcn._sig("largest_degree_first_cleanup", None, gcn.vp)
gcn._sig("largest_degree_first_internal_par", None, C.c_uint32, gcn.u32p, gcn.u32p, gcn.vp, gcn.vp, gcn.f64p, gcn.i32p)


def _prepare_dropin(case, seed):
    s = _DropIn()
    n, V, E = _graph(case, seed)
    L = _layers(case)
    s.n, s.m, s.gnn = n, E.numel(), bool(L)
    s.V, s.E = V.cpu().pin_memory(), E.cpu().pin_memory()
    s.p = torch.zeros(n + 8, dtype=torch.float64).pin_memory()
    s.color = torch.zeros(n, dtype=torch.int32).pin_memory()
    if s.gnn:
        with tempfile.TemporaryDirectory() as d:
            gcn.model_write(os.path.join(d, "m%d.gnn" % L), *_model(case))
            os.environ["GC_MODEL_DIR"] = d
            C.c_int.in_dll(gcn.lib, "layers").value = L
            s.heur = gcn.lib.gnn_setup(n, s.m)
    else:
        s.heur = gcn.lib.largest_degree_first_setup(n, s.m)
    s.jp = gcn.lib.jones_plassmann_setup(n, s.m)
    u32 = lambda t: C.cast(t.data_ptr(), gcn.u32p)  # noqa: E731
    s.call = gcn.lib.gnn_internal_par if s.gnn else gcn.lib.largest_degree_first_internal_par
    s.args = (n, u32(s.V), u32(s.E), s.heur, s.jp, C.cast(s.p.data_ptr(), gcn.f64p), C.cast(s.color.data_ptr(), gcn.i32p))
    return s


def _run_dropin(s):
    s.call(*s.args)
    return {"color": s.color, "priority": s.p[:s.n]}


def prepare(case, seed):
    s = {"graph": _prepare_graph, "batch": _prepare_batch, "drop-in": _prepare_dropin}[case["kind"]](case, seed)
    s.pass_ = {"graph": _run_graph, "batch": _run_batch, "drop-in": _run_dropin}[case["kind"]]
    return s


def run(state):
    return state.pass_(state)


# ---- what a pass cannot do without ---------------------------------------------------------------------


def _size(case):
    """(vertices, directed edges) of a case, R-MAT and batches by expectation."""
    if case["kind"] == "batch":
        n = sum(_batch_sizes(case))
        return n, n * 17
    if case["family"] == "stencil":
        n = case["nx"] * case["ny"] * case["nz"]
        return n, (3 * case["nx"] - 2) * (3 * case["ny"] - 2) * (3 * case["nz"] - 2) - n
    return case["n"], int(case["n"] * case["degree"] * (0.94 if case["family"] == "rmat" else 1.0))


def work(case):
    """The CSR read once, colors (and priorities) written once; the GNN's sums and dense layers."""
    n, m = _size(case)
    L = _layers(case)
    priority = 8 if case["kind"] == "drop-in" else (4 if not case["recolor"] else 0)
    flops = 0.0
    if L:
        flops = 2.0 * m + 16.0 * m * (L - 1) + 1024.0 * n * L
    return {"bytes": 4.0 * (n + 1) + 4.0 * m + (4.0 + priority) * n, "flops": flops}


# ---- the GNN's priorities in 64 bits --------------------------------------------------------------------


def _sage64(n, V, E, params, md, first=None, size=None):
    """GraphSAGE-16 with mean aggregation in float64; `first` and `size`: each vertex's first id and
    vertex count of its own graph (a batch)."""
    deg = (V[1:] - V[:-1]).double()
    A = torch.sparse_csr_tensor(V, E, torch.ones(E.numel(), dtype=torch.float64, device=DEV), size=(n, n))
    ids = torch.arange(n, dtype=torch.float64, device=DEV)
    ids = ids / n if first is None else (ids - first) / size
    P = torch.from_numpy(np.asarray(params, np.float64)).to(DEV).view(-1, 528)
    x = torch.stack([deg / md, ids], 1)
    for k in range(P.shape[0]):
        mean = (A @ x) / deg.clamp(min=1.0)[:, None]
        a = torch.cat([mean, x], 1)
        if k == 0:
            a = a.repeat_interleave(8, 1)
        x = torch.relu(a @ P[k, :512].view(32, 16) + P[k, 512:])
    return x.sum(1)


def exact(case, seed):
    L = _layers(case)
    if not L or case["recolor"]:
        return None
    params, md = _model(case)
    if case["kind"] == "batch":
        voff, V, E = _batch(case, seed)
        voff = torch.from_numpy(voff.astype(np.int64)).to(DEV)
        n = V.numel() - 1
        size = voff[1:] - voff[:-1]
        first = torch.repeat_interleave(voff[:-1], size)
        E = (E + torch.repeat_interleave(first, (V[1:] - V[:-1]).long())).to(torch.int32)
        p = _sage64(n, V, E, params, md, first.double(), torch.repeat_interleave(size, size).double())
        return {"color": None, "priority": p, "colors": None}
    n, V, E = _graph(case, seed)
    p = _sage64(n, V, E, params, md)
    return {"color": None, "priority": p} if case["kind"] == "drop-in" else {"color": None, "priority": p, "colors": None}
