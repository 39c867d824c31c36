"""CSRs that are not symmetric, against the library's contract: where a call succeeds all the same, each vertex has the
smallest color that no neighbour of its own list that precedes it has, whichever kernel colored it."""
import os

import numpy as np
import pytest

import gnn_coloring as gcn

pytestmark = pytest.mark.gpu


def _csr(lists):
    V = np.concatenate([[0], np.cumsum([len(x) for x in lists])]).astype(np.uint32)
    return len(lists), V, np.concatenate([np.sort(np.asarray(x, np.uint32)) for x in lists]).astype(np.uint32)


def _colors_by_own_lists(N, V, E, p):
    color = np.zeros(N, np.int64)
    for u in np.lexsort((np.arange(N), -p)):
        v = E[V[u]:V[u + 1]].astype(np.int64)
        before = v[(p[v] > p[u]) | ((p[v] == p[u]) & (v < u))]
        taken = set(color[before].tolist())
        color[u] = next(c for c in range(1, N + 2) if c not in taken)
    return color


def _lists(N, V, E):
    return [E[V[u]:V[u + 1]].tolist() for u in range(N)]


def test_a_vertex_named_by_one_that_it_does_not_name():
    """Vertex 41 ends a path and waits for it; vertex 42 names 41 and precedes it, one-sidedly."""
    lists = [[v for v in (u - 1, u + 1) if 0 <= v < 42] for u in range(42)] + [[41]] + [[] for _ in range(21)]
    N, V, E = _csr(lists)
    p = np.arange(N, 0, -1).astype(np.float64)
    p[42] = 100.0
    want = _colors_by_own_lists(N, V, E, p)
    ctx = gcn.Context(int(os.environ.get("GC_DEVICE", "0")))
    g = gcn.Graph(ctx, N, V, E)
    for _ in range(3):
        g.set_priority(p)
        g.color(count=False)
        assert np.array_equal(g.colors(), want)
    g.close()
    ctx.close()


@pytest.mark.parametrize("seed", range(6))
def test_entries_added_on_one_side(seed):
    """Extra entries from vertices to later ones: nobody's own predecessors change."""
    N, V, E = gcn.gen_er(900, 900 * (2 + seed), 10 + seed)
    lists, rng = _lists(N, V, E), np.random.default_rng(seed)
    for u, v in rng.integers(0, N, (1 << seed, 2)):
        u, v = min(u, v), max(u, v)
        if u != v and int(v) not in lists[u]:
            lists[u].append(int(v))
    N, V, E = _csr(lists)
    p = np.arange(N, 0, -1).astype(np.float64)  # first fit: smaller ids precede
    want = _colors_by_own_lists(N, V, E, p)
    ctx = gcn.Context(int(os.environ.get("GC_DEVICE", "0")))
    g = gcn.Graph(ctx, N, V, E)
    for _ in range(2):
        g.priority("FF")
        g.color(count=False)
        assert np.array_equal(g.colors(), want)
    g.close()
    ctx.close()


def test_a_vertex_named_by_more_than_its_counter_holds():
    """70,000 vertices name vertex 0, which names one of them; the end of a path makes the last vertex of 0's queue
    array ready once everything else is done."""
    n, chain = 70000, 3000
    lists = [[0] for _ in range(n)]
    a = n - 1
    lists[0] = [a]
    ids = [u for u in range(1, n - 1) if u % 37][:chain]  # the path, outside 0's array
    w, z = 37 * ((n - 200) // 37), n - 3
    on = next(u for u in range(w - 1, 0, -1) if u % 37)
    for k, u in enumerate(ids):
        lists[u] = ids[max(0, k - 1):k] + ids[k + 1:k + 2]
    lists[ids[-1]] += [on, w]
    lists[on], lists[w], lists[z] = [ids[-1]], [ids[-1], z], []
    N, V, E = _csr(lists)
    p = np.full(N, 2.0)
    p[ids] = np.arange(chain, 0, -1) + 10.0
    p[[0, on, w, z]] = 1.0, 1.5, 1.5, 1.0
    want = _colors_by_own_lists(N, V, E, p)
    ctx = gcn.Context(int(os.environ.get("GC_DEVICE", "0")))
    g = gcn.Graph(ctx, N, V, E)
    g.set_priority(p)
    g.color(count=False)
    assert np.array_equal(g.colors(), want)
    g.close()
    ctx.close()


@pytest.mark.parametrize("core", ["8", "64", "32768"])
def test_core_ticket_that_waits_for_a_leaf(core):
    """Vertex 1 of a path names vertex 50, which precedes it but names only vertex 60: a leaf, without a ticket.  The
    coloring fails with a status, and the context stays usable."""
    lists = [[v for v in (u - 1, u + 1) if 0 <= v < 40] for u in range(40)] + [[] for _ in range(60)]
    lists[1].append(50)
    lists[50], lists[60] = [60], [50]
    N, V, E = _csr(lists)
    p = np.arange(N, 0, -1).astype(np.float64)
    p[60], p[50] = 300.0, 200.0
    env = dict(GC_JP_SMALL="0", GC_JP_FLOW="0", GC_JP_CORE=core, GC_SPIN_LIMIT="1000")
    os.environ.update(env)
    ctx = gcn.Context(int(os.environ.get("GC_DEVICE", "0")))
    for k in env:
        del os.environ[k]
    g = gcn.Graph(ctx, N, V, E)
    g.set_priority(p)
    with pytest.raises(gcn.GCError) as e:
        g.color()
    assert e.value.name == "GC_ERR_DEVICE"
    g.close()
    N, V, E = gcn.gen_er(500, 2000, 1)
    g = gcn.Graph(ctx, N, V, E)
    g.priority("LF")
    g.color()
    assert np.array_equal(g.colors(), _colors_by_own_lists(N, V, E, g.priorities()))
    g.close()
    ctx.close()
