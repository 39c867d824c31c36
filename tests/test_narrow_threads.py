"""A wide coloring beside the work of other threads: the GPU's time is shared, so everything takes longer, and it must
not be found narrow for that."""
import threading

import numpy as np
import pytest

import gnn_coloring as gcn

pytestmark = pytest.mark.gpu

THREADS, CALLS = 16, 40


def test_mesh_beside_other_streams():
    graphs = [gcn.gen_stencil27(60, 60, 60), gcn.gen_rmat(1 << 18, 16, 1), gcn.gen_rmat(1 << 20, 16, 1)]
    small = [gcn.gen_er(int(n), 8 * int(n), i) for i, n in enumerate(np.random.default_rng(1).integers(1000, 50000, 40))]
    launches, errors, lock = [], [], threading.Lock()
    start = threading.Barrier(THREADS, timeout=60)

    def work(k):
        try:
            ctx = gcn.Context(0)
            mesh, *others = (gcn.Graph(ctx, *g) for g in graphs)
            batch = gcn.Batch(ctx, graphs=small)
            for g in (mesh, *others):
                g.priority("LF")
                g.color()
            want, mine, rng = mesh.color(), [], np.random.default_rng(k)
            start.wait()
            for _ in range(CALLS):
                before = ctx.launches
                assert mesh.color() == want
                mine.append(ctx.launches - before)
                for _ in range(rng.integers(3)):
                    if rng.integers(3) == 0:
                        batch.color("LF")
                    else:
                        (mesh, *others)[rng.integers(3)].color()
            with lock:
                launches.extend(mine)
            for o in (batch, mesh, *others, ctx):
                o.close()
        except Exception as e:  # (raised below, by the test's own thread)
            errors.append(e)
            start.abort()

    threads = [threading.Thread(target=work, args=(k,)) for k in range(THREADS)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    # A coloring that is found narrow is colored again by other kernels, with several times the launches: by the clock
    # 11 to 13 of these 640, by looks at most one in four runs.
    assert sum(n > min(launches) for n in launches) <= 2, sorted(launches)[-20:]
