"""The dataflow coloring of graphs whose longest lists are far above the mean: leaves stay out of the queues.  Trees,
caterpillars, stars whose center comes first or last (a leaf of many neighbours), isolated vertices."""
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


def _caterpillar(n, leaves):
    sp = np.arange(n - 1)
    return _pairs(n * (1 + leaves), np.concatenate([sp, np.repeat(np.arange(n), leaves)]),
                  np.concatenate([sp + 1, n + np.arange(n * leaves)]))


def _star_last(n, spare):
    """The center has the largest id; `spare` vertices have no neighbours."""
    return _pairs(n + spare, np.arange(n - 1), np.full(n - 1, n + spare - 1))


def _hubs(n, hubs, d, seed):
    rng = np.random.default_rng(seed)
    i = np.concatenate([rng.integers(0, n, 2 * n), np.repeat(rng.choice(n, hubs, False), d)])
    return _pairs(n, i, rng.integers(0, n, len(i)))


def _bicliques(k, d):
    """Each of 60 vertices joined to the same d, k times; and a path that lowers the mean degree, to 4 at least.
    The first side, with the larger ids, are leaves of d neighbours in first fit."""
    base = (np.arange(k) * (d + 60))[:, None]
    a, b = np.repeat(np.arange(60), d) + d, np.tile(np.arange(d), 60)
    n = k * (d + 60)
    m = k * 60 * d // 8
    p = n + np.arange(m - 1)
    return _pairs(n + m, np.concatenate([(base + a).ravel(), p]), np.concatenate([(base + b).ravel(), p + 1]))


GRAPHS = {
    "tree30": lambda: _tree(20000, 30),
    "tree31": lambda: _tree(1 + 31 + 31 * 31, 31),
    "tree60": lambda: _tree(100001, 60),
    "caterpillar": lambda: _caterpillar(300, 61),
    **{f"star_last{d}": (lambda d=d: _star_last(d + 1, 40)) for d in (31, 32, 61)},
    "hubs60": lambda: _hubs(50021, 200, 40, 1),
    "hubs100": lambda: _hubs(50021, 30, 80, 2),
    **{f"bicliques{d}": (lambda d=d: _bicliques(40, d)) for d in (63, 64, 96, 127)},
}


@pytest.mark.parametrize("name", list(GRAPHS))
def test_leaves_apart_match_oracle(name):
    N, V, E = GRAPHS[name]()
    deg = np.diff(V.astype(np.int64))
    assert 4 * len(E) < deg.max() * N and deg.max() < 128
    os.environ["GC_JP_SMALL"] = "0"
    ctx = gcn.Context(int(os.environ.get("GC_DEVICE", "0")))
    del os.environ["GC_JP_SMALL"]
    g = gcn.Graph(ctx, N, V, E)
    rng = np.random.default_rng(0)
    for heur in ("FF", "LF", "SL", None, None):
        if heur:
            g.priority(heur)
        else:
            g.set_priority(rng.permutation(N).astype(np.float64))
        p = g.priorities()
        ref, _ = O.greedy_color(N, V, E, p)
        assert g.color() == O.validate(N, V, E, ref)
        assert np.array_equal(g.colors(), ref), (name, heur)
        g.recolor(1)
        assert np.array_equal(g.colors(), O.culberson(N, V, E, ref, 1)), (name, heur)
    g.close()
    ctx.close()
