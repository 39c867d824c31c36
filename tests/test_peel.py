"""SL and SLL peeling in one kernel against the oracle: thresholds that jump (cliques, stars), lists split
between lane groups and whole CTAs (64/65, 128/129 and 512/513 neighbours and far more), graphs that need
fewer CTAs than the GPU has, and hundreds of rounds."""
import numpy as np
import pytest

import gnn_coloring as gcn
from oracle import restatement as O

pytestmark = pytest.mark.gpu


def _pairs(n, i, j):
    return gcn.csr_from_pairs(n, np.asarray(i, np.uint32), np.asarray(j, np.uint32))


def _cliques(sizes, extra):
    """Disjoint cliques (their thresholds jump) and one vertex joined to `extra` others."""
    i, j, base = [], [], 0
    for n in sizes:
        a, b = np.triu_indices(n, 1)
        i.append(a + base)
        j.append(b + base)
        base += n
    i.append(np.full(extra, base))
    j.append(np.arange(extra))
    return _pairs(base + 1, np.concatenate(i), np.concatenate(j))


GRAPHS = {
    "one": lambda: _pairs(1, [], []),
    "edgeless": lambda: _pairs(1000, [], []),
    **{f"star{n}": (lambda n=n: _pairs(n, np.zeros(n - 1), np.arange(1, n))) for n in (65, 66, 129, 130, 513, 514, 40000)},
    "cliques": lambda: _cliques((3, 66, 67, 130, 131, 514, 515), 1000),
    "er_small": lambda: gcn.gen_er(300, 2000, 1),
    "er": lambda: gcn.gen_er(50021, 700000, 2),
    "rmat": lambda: gcn.gen_rmat(1 << 16, 16, 3),
    "rmat_odd": lambda: gcn.gen_rmat(200003, 8, 4),
    "stencil": lambda: gcn.gen_stencil27(30, 31, 32),
}


@pytest.mark.parametrize("name", list(GRAPHS))
def test_peeling_matches_oracle(gpu_ctx, name):
    N, V, E = GRAPHS[name]()
    g = gcn.Graph(gpu_ctx, N, V, E)
    for heur in ("SL", "SLL", "SL"):
        g.priority(heur)
        assert np.array_equal(g.priorities(), O.ordering(heur, N, V, E)), (name, heur)
    g.close()
