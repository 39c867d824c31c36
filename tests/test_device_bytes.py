"""The admission figure covers what a graph holds whose dataflow coloring stops and goes on by tickets."""
import os

import numpy as np
import pytest
import torch

import gnn_coloring as gcn

pytestmark = pytest.mark.gpu


def test_charge_covers_a_stopped_dataflow_coloring():
    n, chain = 12_000_000, 1000
    i = np.arange(chain, dtype=np.uint32)
    N, V, E = gcn.csr_from_pairs(n, i, i + 1)
    os.environ.update(GC_JP_FLOW_LIMIT="0", GC_JP_CORE="0")
    ctx = gcn.Context(int(os.environ.get("GC_DEVICE", "0")))
    del os.environ["GC_JP_FLOW_LIMIT"], os.environ["GC_JP_CORE"]
    small = gcn.Graph(ctx, *gcn.gen_er(100, 300, 1))  # (modules and the context's own buffers are there)
    small.priority("LF")
    small.color()
    free0 = torch.cuda.mem_get_info()[0]
    g = gcn.Graph(ctx, N, V, E)
    g.priority("FF")
    assert g.color() == 2
    held = free0 - torch.cuda.mem_get_info()[0]
    assert held <= gcn.batch_device_bytes(1, N, len(E), "FF"), held
    g.close()
    small.close()
    ctx.close()
