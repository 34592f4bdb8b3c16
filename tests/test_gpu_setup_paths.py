"""Which path a caller's symmetric system takes, on both sides of each limit, and the way back from the one-kernel setup.

The stage timers tell the setups apart: a level built by the level-by-level
kernels is timed as setup_aggregate, the one-kernel setup never.  The launch
counter tells the CG apart: the cluster kernel is one launch whatever the
number of iterations.  A sparse random graph has more products than the
one-kernel setup's room, so that it gives up after it has begun; the solution's
residual, formed here in FP64, is then the solver's own.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def semo():
    import semo_mesh_gb300 as S
    S.load_library()
    return S


def graph_system(o, q, n, seed):
    rng = np.random.default_rng(seed)
    c = rng.uniform(0.8, 1.2, o.size)
    d = np.bincount(o, c, n) + np.bincount(q, c, n) + 0.01
    rows = np.concatenate([np.arange(n), o, q]).astype(np.int32)
    cols = np.concatenate([np.arange(n), q, o]).astype(np.int32)
    return rows, cols, np.concatenate([d, -c, -c]), rng.uniform(-1.0, 1.0, n)


def lattice(shape, seed=3):
    n = int(np.prod(shape))
    idx = np.arange(n).reshape(shape)
    o = np.concatenate([np.take(idx, range(shape[a] - 1), a).reshape(-1) for a in range(3)])
    q = np.concatenate([np.take(idx, range(1, shape[a]), a).reshape(-1) for a in range(3)])
    return graph_system(o, q, n, seed)


def random_graph(n, degree, seed=3):
    rng = np.random.default_rng(seed)
    o, q = np.repeat(np.arange(n), degree), rng.integers(0, n, n * degree)
    key = np.unique(np.minimum(o, q) * n + np.maximum(o, q))
    o, q = key // n, key % n
    keep = o != q
    return graph_system(o[keep], q[keep], n, seed)


def solve(semo, system, precision="mixed", tol=1e-9):
    rows, cols, vals, b = system
    ctx = semo.Context(precision=precision, tol=tol)
    ctx.set_profiling(True)
    before = ctx.kernel_launches()
    r = ctx.solve_amgcl("pressure", 1, rows, cols, vals, b)
    launches = ctx.kernel_launches() - before
    levels, steps = len(ctx.hierarchy_levels()), ctx.stage_times()["setup_aggregate"][1]
    ctx.close()
    res = np.linalg.norm(b - np.bincount(rows, vals * r.x[cols], b.size))
    slack = 64 * 2.0 ** -53 * np.abs(vals).max() * np.linalg.norm(r.x)
    assert res <= tol * np.linalg.norm(b) + slack
    return levels, steps, launches


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("shape, above", [((64, 64, 64), 0), ((64, 64, 65), 1)])   # 262,144 rows and above
def test_one_kernel_setup(semo, precision, shape, above):
    levels, steps, _ = solve(semo, lattice(shape), precision)
    assert levels >= 3 and steps == above


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_no_room(semo, precision):
    system = random_graph(20000, 10)
    assert system[0].size < 2_000_000
    levels, steps, _ = solve(semo, system, precision)
    # every level that is aggregated was built by the level-by-level kernels
    assert levels >= 2 and steps == levels - 1


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("shape, cluster", [((12, 12, 12), True), ((14, 14, 14), True), ((32, 32, 32), False)])
def test_cluster_cg(semo, precision, shape, cluster):
    system = lattice(shape)
    few, many = (solve(semo, system, precision, tol)[2] for tol in (1e-2, 1e-9))
    assert (few == many) == cluster
