"""GNN groups of vertices with one to four neighbours against the oracle, bit for bit: alone, beside larger degrees in
the same kernel, in the tiers of small graphs (a warp per item and no more), and where skewed graphs are not taken
throughout by the 32-vertex groups."""
import os

import numpy as np
import pytest

import gnn_coloring as gcn
from oracle import restatement as O

pytestmark = pytest.mark.gpu


def _pairs(n, i, j):
    return gcn.csr_from_pairs(n, np.asarray(i, np.uint32), np.asarray(j, np.uint32))


def _tree(n, d):
    j = np.arange(1, n)
    return _pairs(n, (j - 1) // d, j)


def _grid(a, b):
    x = np.arange(a * b).reshape(a, b)
    return _pairs(a * b, np.concatenate([x[:-1].ravel(), x[:, :-1].ravel()]), np.concatenate([x[1:].ravel(), x[:, 1:].ravel()]))


def _cliques(sizes):
    i, j, n = [], [], 0
    for s in sizes:
        a, b = np.triu_indices(s, 1)
        i.append(a + n)
        j.append(b + n)
        n += s
    return _pairs(n, np.concatenate(i), np.concatenate(j))


GRAPHS = {
    "two": lambda: _pairs(2, [0], [1]),
    **{f"path{n}": (lambda n=n: _pairs(n, np.arange(n - 1), np.arange(1, n))) for n in (7, 8, 9, 63, 64, 65, 257)},
    "tree2": lambda: _tree(1000, 2),
    "tree3": lambda: _tree(1000, 3),
    "tree40": lambda: _tree(2000, 40),
    "grid": lambda: _grid(33, 31),
    "cliques_2_to_5": lambda: _cliques([2] * 50 + [3] * 33 + [4] * 17 + [5] * 40),
    "cliques_5_to_7": lambda: _cliques([5] * 100 + [6] * 3 + [7] * 2),
    "sparse": lambda: gcn.gen_er(3000, 3300, 1),
    "many": lambda: _tree(200001, 3),
    "many_skewed": lambda: _tree(200001, 90),
}


@pytest.mark.parametrize("thin", [None, "3", "4", "5", "16", "200"])
@pytest.mark.parametrize("name", list(GRAPHS))
def test_tiny_groups_match_oracle(name, thin):
    N, V, E = GRAPHS[name]()
    if thin:
        os.environ["GC_GNN_THIN_DEGREE"] = thin
    ctx = gcn.Context(int(os.environ.get("GC_DEVICE", "0")))
    os.environ.pop("GC_GNN_THIN_DEGREE", None)
    for layers in (2, 3):
        params, md = gcn.synthetic_model(layers, 60 + layers)
        m, g = gcn.Model(ctx, params, md), gcn.Graph(ctx, N, V, E)
        ref = O.ordering("GNN", N, V, E, params, md)
        for _ in range(2):
            g.priority("GNN", m)
        assert np.array_equal(g.priorities(), ref), (name, thin, layers)
        g.close()
        b = gcn.Batch(ctx, graphs=[(N, V, E), (N, V, E)])
        b.color("GNN", m)
        assert np.array_equal(b.priorities(), np.concatenate([ref, ref])), (name, thin, layers, "batch")
        b.close()
        m.close()
    ctx.close()
