"""The color count sees an improper edge at any place of a list that a warp checks alone, at the edges of its steps."""
import numpy as np
import pytest

import gnn_coloring as gcn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [257, 511, 512, 513, 1023, 1025, 1537, 2000, 2047])
def test_improper_edges_of_a_long_list(gpu_ctx, d):
    center = d // 3  # (the list holds smaller and larger ids)
    others = np.array([v for v in range(d + 1) if v != center], np.uint32)
    N, V, E = gcn.csr_from_pairs(d + 1, np.full(d, center, np.uint32), others)
    g = gcn.Graph(gpu_ctx, N, V, E)
    color = np.full(N, 2, np.int32)
    color[center] = 1
    g.set_colors(color)
    assert g.validate() == 2
    for at in {0, 1, 31, 32, 127, 128, 255, 511, 512, d // 2, d - 33, d - 32, d - 2, d - 1} & set(range(d)):
        bad = color.copy()
        bad[others[at]] = 1
        g.set_colors(bad)
        assert g.validate() == 0, at
    g.close()
