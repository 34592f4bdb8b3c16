"""The AMG setup of small levels in one kernel, at the sizes where it can go wrong.

Symmetric positive definite lattice systems (a 7-point stencil with seeded
coefficients) through solveAMGCL: a hierarchy that is one level, that stops at
max_levels, whose coarsest level is inverted in the kernel (64 rows) or after
it, levels of one block and of many, rows longer than a warp's table.
Reference: numpy's dense solve.  Tolerance: the solve stops at 1e-11 relative
residual, so the relative error is at most the condition number times that
(and the reference's own, the condition number times some 1e-14).  Two solves
give the same bits.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def semo():
    import semo_mesh_gb300 as S
    S.load_library()
    return S


def lattice(shape, seed, hub=0):
    """COO triple of a lattice Laplacian with a reaction term; hub: that many extra strong entries in row 0."""
    rng = np.random.default_rng(seed)
    N = int(np.prod(shape))
    idx = np.arange(N).reshape(shape)
    o, q = [], []
    for a in range(3):
        o.append(np.take(idx, range(shape[a] - 1), a).reshape(-1))
        q.append(np.take(idx, range(1, shape[a]), a).reshape(-1))
    o, q = np.concatenate(o), np.concatenate(q)
    if hub:
        far = rng.choice(np.arange(2, N), size=min(hub, N - 2), replace=False)
        o, q = np.concatenate([o, np.zeros(far.size, int)]), np.concatenate([q, far])
    c = rng.uniform(0.5, 2.0, o.size)
    d = np.bincount(o, c, N) + np.bincount(q, c, N) + 0.01
    rows = np.concatenate([np.arange(N), o, q]).astype(np.int32)
    cols = np.concatenate([np.arange(N), q, o]).astype(np.int32)
    vals = np.concatenate([d, -c, -c])
    A = np.zeros((N, N))
    np.add.at(A, (rows, cols), vals)
    return rows, cols, vals, A, rng.uniform(-1.0, 1.0, N)


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("shape, coarse, levels, hub", [
    ((1, 1, 1), 64, 24, 0), ((2, 1, 1), 1, 24, 0), ((4, 4, 4), 64, 24, 0), ((5, 13, 1), 64, 24, 0),
    ((5, 13, 1), 8, 24, 0), ((9, 9, 9), 64, 24, 0), ((9, 9, 9), 200, 24, 0), ((9, 9, 9), 64, 2, 0),
    ((11, 12, 13), 4, 24, 0), ((11, 12, 13), 4, 24, 1200), ((16, 16, 8), 64, 24, 300)])
def test_sizes(semo, precision, shape, coarse, levels, hub):
    rows, cols, vals, A, b = lattice(shape, 7, hub)
    bar = np.linalg.cond(A) * 1.01e-11
    ctx = semo.Context(precision=precision, tol=1e-11, coarse_enough=coarse, max_levels=levels)
    x = ctx.solve_amgcl("pressure", 1, rows, cols, vals, b)
    ref = np.linalg.solve(A, b)
    assert np.linalg.norm(x.x - ref) <= bar * np.linalg.norm(ref)
    lev = ctx.hierarchy_levels()
    assert lev[0]["rows"] == b.size and len(lev) <= levels
    again = ctx.solve_amgcl("pressure", 1, rows, cols, vals, b)
    assert np.array_equal(x.x, again.x) and x.info["iterations"] == again.info["iterations"]
    ctx.close()


def test_levels_of_both_setups_agree(semo):
    """A context whose setup runs beside the momentum pass and one whose does not take a 48^3 level differently; the
    aggregation is the same, so the levels are."""
    from semo_mesh_gb300.cases import vof_case
    case = vof_case(48)
    rows = []
    for overlap in (True, False):
        ctx = semo.Context(overlap_setup=overlap, reuse_hierarchy=False)
        ctx.set_case(case)
        ctx.outer_iteration()
        rows.append([(v["rows"], v["nnz_A"], v["nnz_P"]) for v in ctx.hierarchy_levels()])
        ctx.close()
    assert rows[0] == rows[1]
