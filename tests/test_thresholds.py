"""Degree thresholds: chosen by the graph's size until somebody sets them, then taken as they are -- also values that
equal the defaults of large graphs."""
import ctypes as C
import os

import numpy as np
import pytest

import gnn_coloring as gcn
from oracle import restatement as O

pytestmark = pytest.mark.gpu


def _kernels(ctx, call):
    """The names of the kernel groups that `call` ran."""
    gcn.lib.gc_prof_read.argtypes = [C.c_void_p, C.c_void_p, C.c_void_p, C.c_void_p, C.c_int]
    names, total, launches = (C.c_char_p * 64)(), (C.c_double * 64)(), (C.c_uint64 * 64)()
    ctx.check(gcn.lib.gc_prof_enable(ctx.h, 1))
    call()
    n = gcn.lib.gc_prof_read(ctx.h, names, total, launches, 64)
    ctx.check(gcn.lib.gc_prof_enable(ctx.h, 0))
    return {names[i].decode() for i in range(n)}


def _graph():
    """A vertex of 3,000 neighbours among others of about eight."""
    N, V, E = gcn.gen_er(20000, 80000, 3)
    src = np.repeat(np.arange(N, dtype=np.uint32), np.diff(V.astype(np.int64)))
    up = src < E
    i, j = np.concatenate([src[up], np.full(3000, 7, np.uint32)]), np.concatenate([E[up], np.arange(9, 3009, dtype=np.uint32)])
    return gcn.csr_from_pairs(N, i, j)


HUB = "gnn_hub_input"


@pytest.mark.parametrize("value,hubs", [(None, True), ("2048", True), ("16384", False)])
def test_hub_degree_of_a_context(value, hubs):
    N, V, E = _graph()
    params, md = gcn.synthetic_model(2, 1002)
    if value:
        os.environ["GC_HUB_DEGREE"] = value
    ctx = gcn.Context(int(os.environ.get("GC_DEVICE", "0")))
    os.environ.pop("GC_HUB_DEGREE", None)
    g, m = gcn.Graph(ctx, N, V, E), gcn.Model(ctx, params, md)
    names = _kernels(ctx, lambda: g.priority("GNN", m))
    assert (HUB in names) == hubs, names
    assert np.array_equal(g.priorities(), O.ordering("GNN", N, V, E, params, md))
    g.close()
    m.close()
    ctx.close()


def test_thresholds_of_a_batch(gpu_ctx):
    graph = _graph()
    params, md = gcn.synthetic_model(2, 1002)
    m = gcn.Model(gpu_ctx, params, md)
    ref = O.ordering("GNN", *graph, params, md)
    b = gcn.Batch(gpu_ctx, graphs=[graph])

    def run(hubs, hub_degree, warp_degree):
        b.color("GNN", m)
        names = _kernels(gpu_ctx, lambda: gcn.lib.gc_batch_color_once(gpu_ctx.h, b.h, gcn.HEURISTICS["GNN"], m.h, 0, None))
        assert (HUB in names) == hubs, names
        assert np.array_equal(b.priorities(), ref)
        assert (b.tuning.hub_degree, b.tuning.gnn_warp_degree) == (hub_degree, warp_degree)

    run(True, 2048, 512)  # by size
    t = b.tuning
    b.tuning = t  # the same values, now set
    run(True, 2048, 512)
    t = gcn.default_tuning()
    assert (t.hub_degree, t.gnn_warp_degree) == (16384, 4096)
    b.tuning = t
    run(False, 16384, 4096)
    best, _ = b.autotune("GNN", m, effort=2)
    assert b.tuning.as_dict() == best.as_dict()
    assert best.hub_degree >= 4096
    t.hub_degree = 0
    with pytest.raises(gcn.GCError):
        b.tuning = t
    b.close()
    b = gcn.Batch(gpu_ctx, graphs=[graph])
    best, _ = b.autotune("GNN", m, effort=1)
    assert b.tuning.as_dict() == best.as_dict() and best.hub_degree == 2048
    b.close()
    m.close()
