"""A dataflow coloring that stops before it is complete: the ticket kernels color the graph, and colors, counts and
rounds are the oracle's.  The stop is made by a wait limit of 0 (the kernel returns; nothing faults)."""
import ctypes as C
import os

import numpy as np
import pytest

import gnn_coloring as gcn
from oracle import restatement as O

pytestmark = pytest.mark.gpu


def _context(**env):
    env = dict(GC_JP_SMALL="0", **env)
    os.environ.update(env)
    try:
        return gcn.Context(int(os.environ.get("GC_DEVICE", "0")))
    finally:
        for k in env:
            del os.environ[k]


def _kernels(ctx, call):
    """The names of the kernel groups that `call` ran, and its result."""
    gcn.lib.gc_prof_read.argtypes = [C.c_void_p, C.c_void_p, C.c_void_p, C.c_void_p, C.c_int]
    names, total, launches = (C.c_char_p * 64)(), (C.c_double * 64)(), (C.c_uint64 * 64)()
    ctx.check(gcn.lib.gc_prof_enable(ctx.h, 1))
    result = call()
    n = gcn.lib.gc_prof_read(ctx.h, names, total, launches, 64)
    ctx.check(gcn.lib.gc_prof_enable(ctx.h, 0))
    return {names[i].decode() for i in range(n)}, result


def _path(n):
    i = np.arange(n - 1, dtype=np.uint32)
    return gcn.csr_from_pairs(n, i, i + 1)


GRAPHS = {
    "path": lambda: _path(5000),
    "stencil": lambda: gcn.gen_stencil27(20, 21, 22),
    "degree60": lambda: gcn.gen_er(4001, 4001 * 18, 2),
    "degree100": lambda: gcn.gen_er(3001, 3001 * 40, 3),
}


@pytest.mark.parametrize("classes", ["0", "1"])
@pytest.mark.parametrize("name", list(GRAPHS))
def test_stopped_dataflow_is_colored_by_tickets(name, classes):
    N, V, E = GRAPHS[name]()
    assert np.diff(V.astype(np.int64)).max() < 128
    ctx = _context(GC_JP_FLOW_LIMIT="0", GC_JP_CLASSES=classes)
    g = gcn.Graph(ctx, N, V, E)
    for heur in ("FF", "LF"):
        g.priority(heur)
        p = g.priorities()
        ref, _ = O.greedy_color(N, V, E, p)
        for rounds in (0, 2):
            want = O.culberson(N, V, E, ref, rounds) if rounds else ref
            for count in (True, False):
                g.priority(heur)
                names, got = _kernels(ctx, lambda: g.color(rounds, count=count))
                assert {"jp_flow", "jp_color"} <= names, "the dataflow kernel has to stop and the tickets to run"
                assert np.array_equal(g.colors(), want), (name, heur, rounds, count)
                assert got == (O.validate(N, V, E, want) if count else 0)
        assert g.recolor(1) == O.validate(N, V, E, O.culberson(N, V, E, want, 1))
        assert np.array_equal(g.colors(), O.culberson(N, V, E, want, 1))
    g.close()
    ctx.close()


def test_failed_coloring_leaves_no_colors(monkeypatch):
    """Dataflow and tickets both give up (wait limit 0): the colors written so far are not a coloring."""
    monkeypatch.setenv("GC_SPIN_LIMIT", "0")
    ctx = _context()
    N, V, E = _path(200000)
    g = gcn.Graph(ctx, N, V, E)
    g.priority("FF")
    with pytest.raises(gcn.GCError) as e:
        g.color()
    assert e.value.name == "GC_ERR_DEVICE"
    with pytest.raises(gcn.GCError) as e:
        g.colors()
    assert e.value.name == "GC_ERR_STATE"
    g.close()
    ctx.close()
