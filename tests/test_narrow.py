"""Colorings in which few vertices become ready at a time (paths, bands, strips, caterpillars): begun by dataflow or by
tickets, found narrow, and colored by tickets with most of them in one cluster.  Colors, counts and rounds are the
oracle's; wavefronts that only start narrow stay with the dataflow kernel."""
import ctypes as C
import os

import numpy as np
import pytest

import gnn_coloring as gcn
from oracle import restatement as O

pytestmark = pytest.mark.gpu


def _pairs(n, i, j):
    return gcn.csr_from_pairs(n, np.asarray(i, np.uint32), np.asarray(j, np.uint32))


def _band(n, w):
    i = np.concatenate([np.arange(n - d) for d in range(1, w + 1)])
    return _pairs(n, i, np.concatenate([np.arange(n - d) + d for d in range(1, w + 1)]))


def _strip(n, w):
    x = np.arange(n * w).reshape(n, w)
    return _pairs(n * w, np.concatenate([x[:-1].ravel(), x[:, :-1].ravel()]), np.concatenate([x[1:].ravel(), x[:, 1:].ravel()]))


def _caterpillar(n, leaves):
    sp = np.arange(n - 1)
    return _pairs(n * (1 + leaves), np.concatenate([sp, np.repeat(np.arange(n), leaves)]),
                  np.concatenate([sp + 1, n + np.arange(n * leaves)]))


def _kernels(ctx, call):
    """The names of the kernel groups that `call` ran, and its result."""
    gcn.lib.gc_prof_read.argtypes = [C.c_void_p, C.c_void_p, C.c_void_p, C.c_void_p, C.c_int]
    names, total, launches = (C.c_char_p * 64)(), (C.c_double * 64)(), (C.c_uint64 * 64)()
    ctx.check(gcn.lib.gc_prof_enable(ctx.h, 1))
    result = call()
    n = gcn.lib.gc_prof_read(ctx.h, names, total, launches, 64)
    ctx.check(gcn.lib.gc_prof_enable(ctx.h, 0))
    return {names[i].decode() for i in range(n)}, result


def _context(**env):
    os.environ.update(env)
    try:
        return gcn.Context(int(os.environ.get("GC_DEVICE", "0")))
    finally:
        for k in env:
            del os.environ[k]


NARROW = {
    "path": lambda: _band(20000, 1),
    "path_long": lambda: _band(60000, 1),
    "band15": lambda: _band(6000, 15),
    "band60": lambda: _band(40000, 60),
    "strip": lambda: _strip(5000, 4),
    "caterpillar": lambda: _caterpillar(8000, 50),
    "bar": lambda: gcn.gen_stencil27(4, 4, 2000),
}


@pytest.mark.parametrize("name", list(NARROW))
def test_narrow_graphs_match_oracle(gpu_ctx, name):
    N, V, E = NARROW[name]()
    g = gcn.Graph(gpu_ctx, N, V, E)
    for heur in ("FF", "LF"):
        g.priority(heur)
        ref, _ = O.greedy_color(N, V, E, g.priorities())
        for rounds, count in ((0, True), (0, False), (2, True)):
            want = O.culberson(N, V, E, ref, rounds) if rounds else ref
            g.priority(heur)
            names, got = _kernels(gpu_ctx, lambda: g.color(rounds, count=count))
            assert {"jp_flow", "jp_core"} <= names, (name, heur, names)
            assert got == (O.validate(N, V, E, want) if count else 0)
            assert np.array_equal(g.colors(), want), (name, heur, rounds)
    g.close()


def test_wavefronts_stay_with_the_dataflow_kernel(gpu_ctx):
    for N, V, E in (gcn.gen_stencil27(60, 60, 60), _strip(400, 400)):
        g = gcn.Graph(gpu_ctx, N, V, E)
        g.priority("FF")
        names, _ = _kernels(gpu_ctx, g.color)
        assert "jp_flow" in names and "jp_color" not in names
        assert np.array_equal(g.colors(), O.greedy_color(N, V, E, g.priorities())[0])
        g.close()


def test_narrow_off():
    ctx = _context(GC_JP_NARROW="0")
    N, V, E = NARROW["path"]()
    g = gcn.Graph(ctx, N, V, E)
    g.priority("FF")
    names, _ = _kernels(ctx, g.color)
    assert "jp_color" not in names
    assert np.array_equal(g.colors(), O.greedy_color(N, V, E, g.priorities())[0])
    g.close()
    ctx.close()


def _wheel(n):
    i = np.arange(1, n)
    return _pairs(n, np.concatenate([i, np.zeros(n - 1, int)]), np.concatenate([np.where(i + 1 < n, i + 1, 1), i]))


@pytest.mark.parametrize("name", ["wheel", "band100", "band200"])
def test_narrow_tickets_match_oracle(gpu_ctx, name):
    N, V, E = {"wheel": lambda: _wheel(12000), "band100": lambda: _band(20000, 100), "band200": lambda: _band(30000, 200)}[name]()
    g = gcn.Graph(gpu_ctx, N, V, E)
    for heur in ("FF", "SL"):
        g.priority(heur)
        ref, _ = O.greedy_color(N, V, E, g.priorities())
        for rounds, count in ((0, True), (0, False), (2, True)):
            want = O.culberson(N, V, E, ref, rounds) if rounds else ref
            g.priority(heur)
            names, got = _kernels(gpu_ctx, lambda: g.color(rounds, count=count))
            assert "jp_core" in names and "jp_flow" not in names, names
            assert got == (O.validate(N, V, E, want) if count else 0)
            assert np.array_equal(g.colors(), want), (name, heur, rounds)
    g.close()


@pytest.mark.parametrize("classes", ["0", "1"])
def test_narrow_batches_match_oracle(classes):
    """The first pass is found narrow and runs again; the captured one starts with the cluster.  A batch pass with
    streams is stopped like one without."""
    graphs = [_band(9000, 1), _band(3000, 15), _strip(2000, 3), _wheel(500), _band(2, 1)]
    for light in ("0", str(1 << 19)):
        ctx = _context(GC_JP_CLASSES=classes, GC_JP_LIGHT_MIN=light)
        b = gcn.Batch(ctx, graphs=graphs)
        for heur in ("LF", "FF"):
            ref = [O.greedy_color(*g, O.ordering(heur, *g))[0] for g in graphs]
            for rounds in (0, 1):
                want = [O.culberson(*g, c, rounds) if rounds else c for g, c in zip(graphs, ref)]
                for _ in range(3):
                    counts = b.color(heur, recolor=rounds)
                    assert np.array_equal(b.colors(), np.concatenate(want)), (heur, rounds, light)
                    assert counts.tolist() == [O.validate(*g, c) for g, c in zip(graphs, want)]
        b.close()
        ctx.close()


def test_rounds_after_a_stopped_coloring_do_not_wait(gpu_ctx):
    """The rounds queued behind a coloring that stops have no colors to work on; their waits must not run to the limit
    (seconds)."""
    import time
    graphs = [_band(20000, 2), _wheel(3000), _strip(3000, 3)]
    ref = [O.greedy_color(*g, O.ordering("LF", *g))[0] for g in graphs]
    want = np.concatenate([O.culberson(*g, c, 2) for g, c in zip(graphs, ref)])
    for classes in ("1", "0"):  # class by class, by tickets
        ctx = _context(GC_JP_CLASSES=classes)
        b = gcn.Batch(ctx, graphs=graphs)
        b.color("FF")  # (kernels are loaded)
        t = time.perf_counter()
        b.color("LF", recolor=2)
        assert time.perf_counter() - t < 0.5
        assert np.array_equal(b.colors(), want)
        b.close()
        ctx.close()
