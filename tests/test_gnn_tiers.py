"""The GNN's degree tiers against the oracle, bit for bit: at the edges of the 32-vertex groups' degrees (16, and
the input layer's chunks of 16), of the warp tier (512) and of the hubs (2,048), below and above the number of
vertices from which the groups are used, in graphs that use them throughout, in batches and after a re-upload."""
import os

import numpy as np
import pytest

import gnn_coloring as gcn
from oracle import restatement as O

pytestmark = pytest.mark.gpu


def _bicliques(degrees, a, isolated, extra, seed):
    """K(a, d) for each degree d, some vertices without neighbours, and an Erdos-Renyi part; ids shuffled."""
    rng = np.random.default_rng(seed)
    i, j, at = [], [], isolated
    for d in degrees:
        i.append(np.repeat(np.arange(at, at + a), d))
        j.append(np.tile(np.arange(at + a, at + a + d), a))
        at += a + d
    n = at + extra
    if extra:
        i.append(rng.integers(at, n, 4 * extra))
        j.append(rng.integers(at, n, 4 * extra))
    p = rng.permutation(n).astype(np.uint32)
    return gcn.csr_from_pairs(n, p[np.concatenate(i)], p[np.concatenate(j)])


SMALL = [1, 2, 7, 8, 9, 15, 16, 17, 31, 32, 33, 63, 64, 65, 127, 128]
GRAPHS = {
    "one_edge": lambda: _bicliques([1], 1, 0, 0, 0),
    "groups31": lambda: _bicliques([15], 16, 0, 0, 1),
    "groups33": lambda: _bicliques([16], 16, 1, 0, 2),
    "upto128": lambda: _bicliques(SMALL, 5, 37, 1000, 3),
    "upto129": lambda: _bicliques(SMALL + [129], 5, 37, 1000, 4),
    "wide": lambda: _bicliques(SMALL + [511, 512, 513, 600], 5, 3, 100, 5),
    "hubs": lambda: _bicliques(SMALL + [513, 2047, 2048, 2049, 5000], 5, 3, 100, 6),
    "many_upto128": lambda: _bicliques(SMALL, 5, 37, 155000, 7),
    "many_hubs": lambda: _bicliques(SMALL + [513, 2048, 2049, 9000], 5, 3000, 160000, 8),
}


@pytest.mark.parametrize("name", list(GRAPHS))
def test_tiers_match_oracle(gpu_ctx, name):
    N, V, E = GRAPHS[name]()
    for layers in (2, 3):
        params, md = gcn.synthetic_model(layers, 40 + layers)
        ref = O.ordering("GNN", N, V, E, params, md)
        for thin in (None, "0", "8", "16", "64", "200"):
            if thin is not None:
                os.environ["GC_GNN_THIN_DEGREE"] = thin
            ctx = gcn.Context(0) if thin is not None else gpu_ctx
            os.environ.pop("GC_GNN_THIN_DEGREE", None)
            g, m = gcn.Graph(ctx, N, V, E), gcn.Model(ctx, params, md)
            for _ in range(2):
                g.priority("GNN", m)
            assert np.array_equal(g.priorities(), ref), thin
            g.close()
            m.close()
            if thin is not None:
                ctx.close()


def test_tiers_in_a_batch(gpu_ctx):
    graphs = [GRAPHS[k]() for k in ("one_edge", "groups33", "upto129", "wide", "hubs", "many_hubs")]
    params, md = gcn.synthetic_model(3, 43)
    m = gcn.Model(gpu_ctx, params, md)
    b = gcn.Batch(gpu_ctx, graphs=graphs)
    ref = np.concatenate([O.ordering("GNN", N, V, E, params, md) for N, V, E in graphs])
    for _ in range(3):  # direct, then captured
        b.color("GNN", m)
        assert np.array_equal(b.priorities(), ref)
    b.close()


def test_tiers_after_reupload(gpu_ctx):
    params, md = gcn.synthetic_model(2, 42)
    m = gcn.Model(gpu_ctx, params, md)
    g = gcn.Graph(gpu_ctx, *GRAPHS["many_hubs"]())
    for k in ("many_hubs", "hubs", "upto128", "wide", "many_upto128", "hubs", "many_hubs"):
        N, V, E = GRAPHS[k]()
        gpu_ctx.check(gcn.lib.gc_graph_reupload(gpu_ctx.h, g.h, N, gcn._ptr(V, gcn.u32p), gcn._ptr(E, gcn.u32p)), k)
        g.N = N
        g.priority("GNN", m)
        assert np.array_equal(g.priorities(), O.ordering("GNN", N, V, E, params, md)), k
    g.close()
