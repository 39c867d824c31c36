"""Small graphs whose levels hold a vertex or two, now and then or throughout: the one-CTA kernel colors them to the end
or gives them to the tickets' cluster.  Paths, bands, cliques past the 32- and 96-neighbour edges, and graphs whose
levels are wide and narrow in turn."""
import os

import numpy as np
import pytest

import gnn_coloring as gcn
from oracle import restatement as O

pytestmark = pytest.mark.gpu


def _pairs(n, i, j):
    return gcn.csr_from_pairs(n, np.asarray(i, np.uint32), np.asarray(j, np.uint32))


def _band(n, w):
    i = np.concatenate([np.arange(n - d) for d in range(1, w + 1)])
    return _pairs(n, i, np.concatenate([np.arange(n - d) + d for d in range(1, w + 1)]))


def _beads(k, wide, chain, seed):
    """A path of `chain` vertices, then `wide` vertices behind one, again and again; and a clique of 100 in the middle."""
    rng, i, j, n = np.random.default_rng(seed), [], [], 0
    for b in range(k):
        a = np.arange(n, n + chain)
        i.append(a[:-1])
        j.append(a[1:])
        w = np.arange(n + chain, n + chain + wide)
        i.append(np.full(wide, a[-1]))
        j.append(w)
        i.append(w)
        j.append(np.full(wide, n + chain + wide))  # (the next path's first vertex)
        i.append(rng.choice(w, wide))
        j.append(rng.choice(w, wide))
        if b == k // 2:
            c = np.concatenate([[a[0]], np.arange(n + chain + wide + 1, n + chain + wide + 100)])
            x, y = np.triu_indices(100, 1)
            i.append(c[x])
            j.append(c[y])
            n += 100
        n += chain + wide
    return _pairs(n + 1, np.concatenate(i), np.concatenate(j))


GRAPHS = {
    "path2": lambda: _band(2, 1),
    "path3072": lambda: _band(3072, 1),
    **{f"path{n}": (lambda n=n: _band(n, 1)) for n in (128, 129, 257, 258, 259, 260, 300)},
    "band2": lambda: _band(2000, 2),
    "band3": lambda: _band(2000, 3),
    "band15": lambda: _band(2900, 15),
    "band31": lambda: _band(600, 31),
    "band33": lambda: _band(300, 33),
    "cycle": lambda: _pairs(999, np.arange(999), (np.arange(999) + 1) % 999),
    **{f"clique{n}": (lambda n=n: _pairs(n, *np.triu_indices(n, 1))) for n in (31, 64, 96, 97, 98, 100, 101, 129, 140)},
    **{f"beads{w}": (lambda w=w: _beads(10, w, 20, w)) for w in (1, 2, 3, 4, 5, 6, 31, 33, 60)},
    "strip": lambda: _pairs(3000, np.concatenate([np.arange(2996), np.arange(0, 3000, 2)]),
                            np.concatenate([np.arange(2996) + 4, np.arange(0, 3000, 2) + 1])),
}


@pytest.mark.parametrize("small", [None, "65535"])
@pytest.mark.parametrize("name", list(GRAPHS))
def test_narrow_levels_match_oracle(name, small):
    N, V, E = GRAPHS[name]()
    if small:
        os.environ["GC_JP_SMALL"] = small
    ctx = gcn.Context(int(os.environ.get("GC_DEVICE", "0")))
    os.environ.pop("GC_JP_SMALL", None)
    g = gcn.Graph(ctx, N, V, E)
    rng = np.random.default_rng(1)
    for heur in ("FF", "LF", "SL", None):
        if heur:
            g.priority(heur)
        else:
            g.set_priority(rng.integers(0, 3, N).astype(np.float64))
        p = g.priorities()
        ref, _ = O.greedy_color(N, V, E, p)
        for rounds in (0, 1, 3):
            want = O.culberson(N, V, E, ref, rounds) if rounds else ref
            if heur:
                g.priority(heur)
            else:
                g.set_priority(p)
            assert g.color(rounds) == O.validate(N, V, E, want)
            assert np.array_equal(g.colors(), want), (name, heur, rounds)
            if heur == "LF":
                assert g.recolor(2) == O.validate(N, V, E, O.culberson(N, V, E, want, 2))
    g.close()
    ctx.close()
