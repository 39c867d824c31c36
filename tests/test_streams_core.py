"""The ticket kernel's two streams behind a cluster core, which batches above a size have by default: every number of
core tickets from none to all, blocks, light warps and early decisions, on batches (direct and replayed) and on single
graphs with and without a clique of hubs, against the oracle."""
import os

import numpy as np
import pytest

import gnn_coloring as gcn
from oracle import restatement as O

pytestmark = pytest.mark.gpu


def _context(**env):
    env = dict(env, GC_JP_FLOW="0", GC_JP_SMALL="0", GC_JP_LIGHT_MIN="0")
    os.environ.update(env)
    try:
        return gcn.Context(int(os.environ.get("GC_DEVICE", "0")))
    finally:
        for k in env:
            del os.environ[k]


def _clique(n):
    return gcn.csr_from_pairs(n, *(np.asarray(x, np.uint32) for x in np.triu_indices(n, 1)))


BATCH = lambda: [gcn.gen_rmat(1 << 13, 16, 3), gcn.gen_er(5001, 60000, 4), _clique(200), gcn.gen_stencil27(12, 13, 14)]  # noqa: E731
PLAIN = {"rmat": lambda: gcn.gen_rmat(1 << 14, 16, 2), "er": lambda: gcn.gen_er(20000, 200000, 8),
         "dense": lambda: gcn.gen_er(3000, 150000, 9), "stencil": lambda: gcn.gen_stencil27(20, 21, 22)}
SETTINGS = [("0", "2", "16", "1"), ("64", "2", "1", "1"), ("777", "2", "3", "0"), ("5000", "6", "7", "1"),
            ("4097", "4", "64", "1"), ("32768", "4", "16", "1"), ("32768", "7", "1", "1"), ("32768", "1", "16", "0"), ("auto", "4", "16", "1")]


def _settings(core, light, block, decide):
    env = dict(GC_JP_LIGHT_WARPS=light, GC_JP_CORE_BLOCK=block, GC_JP_CORE_DECIDE=decide)
    return env if core == "auto" else dict(env, GC_JP_CORE=core)


@pytest.mark.parametrize("core,light,block,decide", SETTINGS)
def test_batches(core, light, block, decide):
    ctx = _context(**_settings(core, light, block, decide))
    params, md = gcn.synthetic_model(2, 1002)
    m = gcn.Model(ctx, params, md)
    graphs = BATCH()
    b = gcn.Batch(ctx, graphs=graphs)
    for heur in ("FF", "LF", "GNN"):
        ref = [O.greedy_color(*g, O.ordering(heur, *g, *((params, md) if heur == "GNN" else ())))[0] for g in graphs]
        for rounds in (0, 2):
            want = np.concatenate([O.culberson(*g, c, rounds) if rounds else c for g, c in zip(graphs, ref)])
            for _ in range(2):  # direct, then captured
                b.color(heur, m if heur == "GNN" else None, rounds)
                assert np.array_equal(b.colors(), want), (heur, rounds)
    b.close()
    m.close()
    ctx.close()


@pytest.mark.parametrize("core,light,block,decide", SETTINGS)
@pytest.mark.parametrize("name", list(PLAIN))
def test_single_graphs(name, core, light, block, decide):
    ctx = _context(**_settings(core, light, block, decide))
    N, V, E = PLAIN[name]()
    g = gcn.Graph(ctx, N, V, E)
    rng = np.random.default_rng(2)
    for heur in ("FF", "LF", None):
        if heur:
            g.priority(heur)
        else:
            g.set_priority(rng.permutation(N).astype(np.float64))
        ref, _ = O.greedy_color(N, V, E, g.priorities())
        assert g.color() == O.validate(N, V, E, ref)
        assert np.array_equal(g.colors(), ref), (name, heur)
        assert g.recolor(2) == O.validate(N, V, E, O.culberson(N, V, E, ref, 2))
        assert np.array_equal(g.colors(), O.culberson(N, V, E, ref, 2))
    g.close()
    ctx.close()
