"""Two contexts on two host threads: their one-kernel setups and cluster solves share the device and give the bits
that each gives alone."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def lattice(n, seed):
    rng = np.random.default_rng(seed)
    idx = np.arange(n ** 3).reshape(n, n, n)
    o = np.concatenate([np.take(idx, range(n - 1), a).reshape(-1) for a in range(3)])
    q = np.concatenate([np.take(idx, range(1, n), a).reshape(-1) for a in range(3)])
    c = rng.uniform(0.5, 2.0, o.size)
    d = np.bincount(o, c, n ** 3) + np.bincount(q, c, n ** 3) + 0.05
    rows = np.concatenate([idx.reshape(-1), o, q]).astype(np.int32)
    cols = np.concatenate([idx.reshape(-1), q, o]).astype(np.int32)
    return rows, cols, np.concatenate([d, -c, -c]), rng.uniform(-1.0, 1.0, n ** 3)


@pytest.mark.parametrize("sizes", [(12, 12), (32, 40), (12, 48)])
def test_both_at_once(sizes):
    import semo_mesh_gb300 as semo
    systems = [lattice(n, 3 + k) for k, n in enumerate(sizes)]
    alone = []
    for s in systems:
        ctx = semo.Context()
        alone.append(ctx.solve_amgcl("pressure", 1, *s).x)
        ctx.close()
    start, failed = threading.Barrier(2), []

    def work(k):
        try:
            ctx = semo.Context()
            start.wait(60)
            for _ in range(20):
                if not np.array_equal(ctx.solve_amgcl("pressure", 1, *systems[k]).x, alone[k]):
                    failed.append("thread %d: other bits" % k)
            ctx.close()
        except Exception as e:   # reported by the test's own thread
            failed.append(repr(e))

    threads = [threading.Thread(target=work, args=(k,)) for k in (0, 1)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed
