"""Captured batch passes stay valid when later passes of the same batch need more scratch (a wider sort)."""
import numpy as np
import pytest

import gnn_coloring as gcn
from oracle import restatement as O

pytestmark = pytest.mark.gpu


def test_replays_after_wider_sorts(gpu_ctx):
    graphs = [gcn.gen_er(30001, 120000, 1), gcn.gen_rmat(1 << 14, 8, 2), gcn.gen_stencil27(20, 21, 22)]
    params, md = gcn.synthetic_model(2, 1002)
    m = gcn.Model(gpu_ctx, params, md)

    def want(heur):
        return np.concatenate([O.greedy_color(*g, O.ordering(heur, *g, *((params, md) if heur == "GNN" else ())))[0]
                               for g in graphs])

    ref = {h: want(h) for h in ("FF", "LF", "GNN")}
    b = gcn.Batch(gpu_ctx, graphs=graphs)
    held = []
    for _ in range(3):
        for h in ("FF", "LF", "GNN"):  # sorts of one pass, of one or two, and of four
            b.color(h, m if h == "GNN" else None)
            assert np.array_equal(b.colors(), ref[h]), h
            other = gcn.Graph(gpu_ctx, *graphs[len(held) % 3])  # (takes what has been freed)
            other.priority("LF")
            other.color()
            held.append(other)
    for g in held:
        g.close()
    b.close()
    m.close()
