"""Culberson rounds class by class against the oracle: at the edges of the degree tiers (64/65 and
1,024/1,025 neighbours), at color 65 of the light tier's 64-bit mask, beyond the pending lists of the
middle and top tiers (large cliques), on skewed graphs, from caller colors, and inside batches."""
import os

import numpy as np
import pytest

import gnn_coloring as gcn
from oracle import restatement as O

pytestmark = pytest.mark.gpu


def _pairs(n, i, j):
    return gcn.csr_from_pairs(n, np.asarray(i, np.uint32), np.asarray(j, np.uint32))


def _clique(n):
    return _pairs(n, *np.triu_indices(n, 1))


def _star(n):
    return _pairs(n, np.zeros(n - 1), np.arange(1, n))


def _hubs(n, k, seed):
    """k vertices joined to each other and to a random half of the others, over a sparse graph."""
    rng = np.random.default_rng(seed)
    i, j = np.triu_indices(k, 1)
    hub = np.repeat(np.arange(k), n - k)
    leaf = np.tile(np.arange(k, n), k)
    keep = rng.random(len(hub)) < 0.5
    a, b = rng.integers(0, n, 3 * n), rng.integers(0, n, 3 * n)
    return _pairs(n, np.concatenate([i, hub[keep], a]), np.concatenate([j, leaf[keep], b]))


GRAPHS = {
    "edgeless": lambda: _pairs(100, [], []),
    "one_edge": lambda: _pairs(2, [0], [1]),
    **{f"clique{n}": (lambda n=n: _clique(n)) for n in (64, 65, 66, 67, 300, 1025, 1026, 2300)},
    **{f"star{n}": (lambda n=n: _star(n)) for n in (65, 66, 1025, 1026, 5000)},
    "hubs": lambda: _hubs(6000, 40, 1),
    "rmat": lambda: gcn.gen_rmat(1 << 15, 16, 7),
    "rmat_odd": lambda: gcn.gen_rmat(100003, 8, 8),
    "er_deg60": lambda: gcn.gen_er(20011, 600000, 9),
    "stencil": lambda: gcn.gen_stencil27(31, 33, 35),
    "er_large": lambda: gcn.gen_er((1 << 19) + 5, 3000000, 10),  # whole-warp grabs
}


@pytest.fixture(scope="module")
def gpu_ctx():
    """A context in which small graphs have no kernel of their own."""
    os.environ["GC_JP_SMALL"] = "0"
    try:
        ctx = gcn.Context(int(os.environ.get("GC_DEVICE", "0")))
    finally:
        del os.environ["GC_JP_SMALL"]
    yield ctx
    ctx.close()


@pytest.mark.parametrize("name", list(GRAPHS))
def test_rounds_match_oracle(gpu_ctx, name):
    N, V, E = GRAPHS[name]()
    for heur in ("FF", "SLL"):
        g = gcn.Graph(gpu_ctx, N, V, E)
        g.priority(heur)
        g.color()
        ref = g.colors()
        assert np.array_equal(ref, O.greedy_color(N, V, E, g.priorities())[0])
        last = None
        for r in (1, 2, 1):
            last = O.culberson(N, V, E, ref, r - 1) if r > 1 else ref
            ref = O.culberson(N, V, E, ref, r)
            count = g.recolor(r)
            assert np.array_equal(g.colors(), ref), (name, heur, r)
            assert count == O.validate(N, V, E, ref)
            assert np.array_equal(g.priorities(), last.astype(np.float64)), "keys are the colors before"
        g.priority(heur)
        assert g.color(recolor=4) == count
        assert np.array_equal(g.colors(), ref)
        g.close()


def test_rounds_from_caller_colors(gpu_ctx):
    """The first round follows the caller's colors (any values), the next ones the library's."""
    N, V, E = gcn.gen_rmat(1 << 14, 8, 5)
    rng = np.random.default_rng(3)
    c = rng.permutation(N).astype(np.int32) + 70000
    g = gcn.Graph(gpu_ctx, N, V, E)
    g.set_colors(c)
    g.recolor(3)
    assert np.array_equal(g.colors(), O.culberson(N, V, E, c, 3))
    g.close()


def test_rounds_in_a_replayed_batch(gpu_ctx):
    graphs = [GRAPHS[k]() for k in ("rmat", "clique67", "edgeless", "hubs", "stencil", "star1026")]
    b = gcn.Batch(gpu_ctx, graphs=graphs)
    for _ in range(3):
        counts = b.color("LF", recolor=3)
        allc = b.colors()
        for i, (N, V, E) in enumerate(graphs):
            p = np.diff(V.astype(np.int64)).astype(np.float64)
            ref = O.culberson(N, V, E, O.greedy_color(N, V, E, p)[0], 3)
            assert np.array_equal(b.graph_colors(i, allc), ref), i
            assert counts[i] == O.validate(N, V, E, ref)
    b.close()


def test_round_waits_are_bounded():
    """A wait limit of 0: a round whose vertices must wait ends with GC_ERR_DEVICE, and the context stays
    usable."""
    N, V, E = _clique(300)
    ok = gcn.Context(int(os.environ.get("GC_DEVICE", "0")))
    g = gcn.Graph(ok, N, V, E)
    g.priority("FF")
    g.color()
    colors = g.colors()
    g.close()
    ok.close()
    os.environ["GC_SPIN_LIMIT"] = "0"
    try:
        ctx = gcn.Context(int(os.environ.get("GC_DEVICE", "0")))
    finally:
        del os.environ["GC_SPIN_LIMIT"]
    g = gcn.Graph(ctx, N, V, E)
    g.set_colors(colors)
    with pytest.raises(gcn.GCError) as e:
        g.recolor(2)
    assert e.value.name == "GC_ERR_DEVICE"
    N2, V2, E2 = _pairs(10, [], [])
    g2 = gcn.Graph(ctx, N2, V2, E2)
    g2.priority("LF")
    assert g2.color(recolor=1) == 1
    for x in (g, g2):
        x.close()
    ctx.close()
