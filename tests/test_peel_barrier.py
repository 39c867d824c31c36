"""Peeling where every round's counts come through the grid barrier: graphs with more vertices than the threads keep
(rounds over lists, long and short), and several contexts that peel at the same time."""
import threading

import numpy as np
import pytest

import gnn_coloring as gcn
from oracle import restatement as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["er", "rmat", "stencil"])
def test_peeling_lists_match_oracle(gpu_ctx, name):
    N, V, E = {"er": lambda: gcn.gen_er(700001, 2800000, 1), "rmat": lambda: gcn.gen_rmat(1 << 20, 4, 2),
               "stencil": lambda: gcn.gen_stencil27(90, 91, 92)}[name]()
    assert N > 148 * 1024 * 4
    g = gcn.Graph(gpu_ctx, N, V, E)
    for heur in ("SL", "SLL"):
        want = O.ordering(heur, N, V, E)
        for _ in range(3):
            g.priority(heur)
            assert np.array_equal(g.priorities(), want), (name, heur)
    g.close()


def test_contexts_that_peel_together():
    N, V, E = gcn.gen_rmat(1 << 17, 16, 3)
    want = O.ordering("SL", N, V, E)
    results = {}

    def work(k):
        ctx = gcn.Context(0)
        g = gcn.Graph(ctx, N, V, E)
        ok = True
        for _ in range(20):
            g.priority("SL")
            ok = ok and np.array_equal(g.priorities(), want)
        results[k] = ok
        g.close()
        ctx.close()

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert results == {k: True for k in range(4)}


@pytest.mark.parametrize("name", ["dense", "dense_many", "mixed", "cliques"])
def test_rounds_that_take_most_vertices(gpu_ctx, name):
    """SLL thresholds above nearly all degrees: the first round takes (almost) everything, kept or on lists."""
    N, V, E = {"dense": lambda: gcn.gen_er(20000, 1000000, 1), "dense_many": lambda: gcn.gen_er(620003, 12000000, 2),
               "mixed": lambda: gcn.gen_rmat(1 << 15, 32, 3),
               "cliques": lambda: gcn.csr_from_pairs(3000, *[np.asarray(x, np.uint32) for x in (
                   np.concatenate([np.triu_indices(30, 1)[0] + 30 * k for k in range(100)]),
                   np.concatenate([np.triu_indices(30, 1)[1] + 30 * k for k in range(100)]))])}[name]()
    g = gcn.Graph(gpu_ctx, N, V, E)
    for heur in ("SLL", "SL"):
        want = O.ordering(heur, N, V, E)
        for _ in range(2):
            g.priority(heur)
            assert np.array_equal(g.priorities(), want), (name, heur)
    g.close()
