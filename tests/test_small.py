"""Small graphs colored in one CTA against the oracle: at the edges of the level queue's light and heavy ends (96/97
neighbours), of the 32-color windows (cliques), of a level's 32 vertices, on paths (one vertex a level), with
rounds, from caller priorities and colors, and either side of the sizes that go there."""
import os

import numpy as np
import pytest

import gnn_coloring as gcn
from oracle import restatement as O

pytestmark = pytest.mark.gpu


def _pairs(n, i, j):
    return gcn.csr_from_pairs(n, np.asarray(i, np.uint32), np.asarray(j, np.uint32))


GRAPHS = {
    "vertex": lambda: _pairs(1, [], []),
    "edgeless": lambda: _pairs(77, [], []),
    "edge": lambda: _pairs(2, [0], [1]),
    "path": lambda: _pairs(3000, np.arange(2999), np.arange(1, 3000)),
    **{f"clique{n}": (lambda n=n: _pairs(n, *np.triu_indices(n, 1))) for n in (32, 33, 34, 65, 66, 97, 98, 99, 310)},
    **{f"star{n}": (lambda n=n: _pairs(n, np.zeros(n - 1), np.arange(1, n))) for n in (66, 97, 98, 3072, 3073)},
    **{f"bipartite{n}": (lambda n=n: _pairs(2 * n, np.repeat(np.arange(n), n), n + np.tile(np.arange(n), n)))
       for n in (31, 32, 33, 97)},
    "er_odd": lambda: gcn.gen_er(3071, 30011, 1),
    "er_above": lambda: gcn.gen_er(3073, 30011, 1),
    "er_rounds": lambda: gcn.gen_er(6144, 20000, 2),
    "rmat": lambda: gcn.gen_rmat(1001, 8, 3),
    "rmat_wide": lambda: gcn.gen_rmat(2047, 16, 4),
    "stencil": lambda: gcn.gen_stencil27(11, 13, 17),
}


# by rule; all here; none here, by the other kernels: as they come, all by tickets, tickets without a core
@pytest.mark.parametrize("env", ["", "SMALL=65535", "SMALL=0", "SMALL=0 FLOW=0", "SMALL=0 FLOW=0 CORE=0 CLASSES=0"])
@pytest.mark.parametrize("name", list(GRAPHS))
def test_small_matches_oracle(name, env):
    env = {"GC_JP_" + kv.split("=")[0]: kv.split("=")[1] for kv in env.split()}
    os.environ.update(env)
    ctx = gcn.Context(0)
    for k in env:
        del os.environ[k]
    N, V, E = GRAPHS[name]()
    rng = np.random.default_rng(N)
    for heur in ("FF", "LF", "SLL", "user"):
        g = gcn.Graph(ctx, N, V, E)
        if heur == "user":
            g.set_priority(rng.integers(0, 5, N).astype(np.float64))
        else:
            g.priority(heur)
        p = g.priorities()
        ref = O.greedy_color(N, V, E, p)[0]
        count = g.color()
        assert np.array_equal(g.colors(), ref)
        assert count == ref.max()
        assert np.array_equal(g.priorities(), p)
        want, used = O.culberson(N, V, E, ref, 2), g.color(2)
        assert np.array_equal(g.colors(), want) and used == want.max()
        assert np.array_equal(g.priorities(), O.culberson(N, V, E, ref, 1).astype(np.float64))
        g.close()
    wide = rng.permutation(N).astype(np.int32) + 1  # caller colors: proper, up to N
    g = gcn.Graph(ctx, N, V, E)
    g.set_colors(wide)
    assert g.recolor(1) == O.culberson(N, V, E, wide, 1).max()
    assert np.array_equal(g.colors(), O.culberson(N, V, E, wide, 1))
    g.set_colors(wide)
    g.recolor(3)
    assert np.array_equal(g.colors(), O.culberson(N, V, E, wide, 3))
    g.close()
    ctx.close()
