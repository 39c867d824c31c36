"""The dataflow coloring (graphs of small maximum degree) against the oracle and the ticket kernels:
at the edges of its neighbour-mask words (maximum degree 31/32, 63/64, 127/128), around its number of
queue arrays (31 vertices), on wavefronts, on long chains, and after Culberson rounds."""
import os

import numpy as np
import pytest

import gnn_coloring as gcn
from oracle import restatement as O

pytestmark = pytest.mark.gpu


def _clique(n):
    i, j = np.triu_indices(n, 1)
    return gcn.csr_from_pairs(n, i.astype(np.uint32), j.astype(np.uint32))


def _star(n):
    return gcn.csr_from_pairs(n, np.zeros(n - 1, np.uint32), np.arange(1, n, dtype=np.uint32))


def _path(n):
    i = np.arange(n - 1, dtype=np.uint32)
    return gcn.csr_from_pairs(n, i, i + 1)


GRAPHS = {
    "one": lambda: gcn.csr_from_pairs(1, np.zeros(0, np.uint32), np.zeros(0, np.uint32)),
    "edgeless": lambda: gcn.csr_from_pairs(777, np.zeros(0, np.uint32), np.zeros(0, np.uint32)),
    "path30": lambda: _path(30),
    "path31": lambda: _path(31),
    "path32": lambda: _path(32),
    "path5000": lambda: _path(5000),
    **{f"clique{n}": (lambda n=n: _clique(n)) for n in (31, 32, 33, 64, 65, 128, 129)},
    **{f"star{n}": (lambda n=n: _star(n)) for n in (32, 33, 64, 65, 128, 129)},
    "er_small": lambda: gcn.gen_er(1000, 8000, 3),
    "er_deg40": lambda: gcn.gen_er(30001, 600000, 5),
    "rgg": lambda: gcn.gen_rgg2d(100003, 0.006, 2),
    "stencil": lambda: gcn.gen_stencil27(40, 33, 57),
    "bar": lambda: gcn.gen_stencil27(3, 2, 3001),
}


@pytest.fixture(scope="module")
def contexts():
    """A context with the dataflow kernels and one without; small graphs have no kernel of their own."""
    device = int(os.environ.get("GC_DEVICE", "0"))
    os.environ["GC_JP_SMALL"] = "0"
    try:
        flow = gcn.Context(device)
        os.environ["GC_JP_FLOW"] = "0"
        tickets = gcn.Context(device)
    finally:
        os.environ.pop("GC_JP_FLOW", None)
        del os.environ["GC_JP_SMALL"]
    models = [gcn.Model(c, *gcn.synthetic_model(3, 1003)) for c in (flow, tickets)]
    yield list(zip((flow, tickets), models))
    for m in models:
        m.close()
    flow.close()
    tickets.close()


@pytest.mark.parametrize("name", list(GRAPHS))
def test_flow_colors_match_oracle_and_tickets(contexts, name):
    N, V, E = GRAPHS[name]()
    for heur in ("FF", "LF", "LLF", "SL", "GNN"):
        results = []
        for ctx, model in contexts:
            g = gcn.Graph(ctx, N, V, E)
            g.priority(heur, model if heur == "GNN" else None)
            count = g.color()
            p, c = g.priorities(), g.colors()
            uncounted = g.color(count=False)
            assert uncounted == 0 and np.array_equal(g.colors(), c), (name, heur, "colors without a count")
            after = g.recolor(2)
            results.append((count, c, p, after, g.colors()))
            g.close()
        ref, _ = O.greedy_color(N, V, E, results[0][2])
        assert np.array_equal(results[0][1], ref), (name, heur, "oracle")
        assert results[0][0] == O.validate(N, V, E, ref), (name, heur, "count")
        for a, b in zip(*results):
            assert np.array_equal(a, b), (name, heur, "tickets")


def test_flow_on_user_priorities_and_a_reused_graph(contexts):
    """Caller priorities with ties and negatives; then the same graph object holds a graph whose hubs
    send it to the ticket kernels, and a small one again."""
    ctx, _ = contexts[0]
    rng = np.random.default_rng(1)
    sizes = [gcn.gen_stencil27(20, 21, 22), gcn.gen_rmat(1 << 13, 8, 3), gcn.gen_er(5000, 40000, 4)]
    h = gcn.vp()
    import ctypes as C
    ctx.check(gcn.lib.gc_graph_create(ctx.h, max(s[0] for s in sizes), max(len(s[2]) for s in sizes), C.byref(h)))
    g = gcn.Graph.__new__(gcn.Graph)
    g.ctx, g.h = ctx, h
    for N, V, E in sizes:
        V, E = np.ascontiguousarray(V, np.uint32), np.ascontiguousarray(E, np.uint32)
        ctx.check(gcn.lib.gc_graph_reupload(ctx.h, h, N, V.ctypes.data_as(gcn.u32p), E.ctypes.data_as(gcn.u32p)))
        g.N = N
        for p in (rng.normal(size=N), rng.integers(0, 4, N).astype(np.float64)):
            g.set_priority(p)
            g.color()
            assert np.array_equal(g.colors(), O.greedy_color(N, V, E, p)[0])
    g.close()
