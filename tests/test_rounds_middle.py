"""Culberson rounds on graphs whose vertices are mostly or all of the middle tier (65 to 1,024 neighbours), few and more
than the warps that begin with it."""
import numpy as np
import pytest

import gnn_coloring as gcn
from oracle import restatement as O

pytestmark = pytest.mark.gpu


def _bicliques(k, d, light):
    """k complete bipartite graphs with d on either side, and a path of `light` vertices."""
    base = (np.arange(k) * 2 * d)[:, None]
    a, b = np.repeat(np.arange(d), d), d + np.tile(np.arange(d), d)
    p = 2 * d * k + np.arange(max(light - 1, 0))
    i, j = np.concatenate([(base + a).ravel(), p]), np.concatenate([(base + b).ravel(), p + 1])
    return gcn.csr_from_pairs(2 * d * k + light, i.astype(np.uint32), j.astype(np.uint32))


@pytest.mark.parametrize("k,d,light", [(300, 65, 0), (300, 65, 5000), (260, 70, 1), (100, 65, 0), (3, 1000, 10)])
def test_rounds_of_the_middle_tier(gpu_ctx, k, d, light):
    N, V, E = _bicliques(k, d, light)
    g = gcn.Graph(gpu_ctx, N, V, E)
    rng = np.random.default_rng(k)
    g.set_priority(rng.permutation(N).astype(np.float64))
    ref, _ = O.greedy_color(N, V, E, g.priorities())
    g.color()
    assert np.array_equal(g.colors(), ref)
    for rounds in (1, 2):
        ref = O.culberson(N, V, E, ref, rounds)
        assert g.recolor(rounds) == O.validate(N, V, E, ref)
        assert np.array_equal(g.colors(), ref), rounds
    g.close()
    wide = rng.permutation(N).astype(np.int32) + 1  # caller colors, then a round on the library's own
    g = gcn.Graph(gpu_ctx, N, V, E)
    g.set_colors(wide)
    g.recolor(2)
    assert np.array_equal(g.colors(), O.culberson(N, V, E, wide, 2))
    g.close()
