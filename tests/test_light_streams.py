"""Batches with and without a light ticket stream against the oracle: either side of the batch size from which
there is one, with all, some and none of the tickets light."""
import os

import numpy as np
import pytest

import gnn_coloring as gcn
from oracle import restatement as O

pytestmark = pytest.mark.gpu


def _graphs():
    n = 200
    clique = gcn.csr_from_pairs(n, *(np.asarray(x, np.uint32) for x in np.triu_indices(n, 1)))
    edge = gcn.csr_from_pairs(2, np.array([0], np.uint32), np.array([1], np.uint32))
    return [gcn.gen_rmat(1 << 13, 16, 3), gcn.gen_er(5001, 30000, 4), clique, edge, gcn.gen_rmat(20003, 8, 5)]


@pytest.mark.parametrize("pick", [(0, 1, 2, 3, 4), (1, 3), (2, 2), (0, 4)])
def test_streams_match_oracle(pick):
    graphs = [_graphs()[i] for i in pick]
    total = sum(N for N, _, _ in graphs)
    for least in (0, total - 1, total):
        os.environ["GC_JP_LIGHT_MIN"] = str(least)
        ctx = gcn.Context(0)
        os.environ.pop("GC_JP_LIGHT_MIN")
        b = gcn.Batch(ctx, graphs=graphs)
        for heur in ("FF", "LF"):
            ref = np.concatenate([O.greedy_color(N, V, E, O.ordering(heur, N, V, E))[0] for N, V, E in graphs])
            for _ in range(2):  # direct, then captured
                b.color(heur)
                assert np.array_equal(b.colors(), ref), (heur, least)
        b.close()
        ctx.close()
