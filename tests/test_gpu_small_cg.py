"""CG of small systems in one cluster kernel, and the V-cycle's smallest levels in one block.

Lattice systems whose sizes meet the edges: one row, fewer rows than blocks,
runs of rows that are no multiple of four, the largest that still fits and the
first that does not; one level, two and more; a zero right-hand side, a guess
that is the solution, an indefinite matrix, the iteration cap.  Reference:
numpy's dense solve where it is affordable, else the residual in FP64.
Tolerance: the solve stops at 1e-10 relative residual, so the relative error is
at most the condition number times that, and the residual that numpy forms of
the returned solution differs from the tolerance by rounding (n 2^-53 |A||x|).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
TOL = 1e-10


@pytest.fixture(scope="module")
def semo():
    import semo_mesh_gb300 as S
    S.load_library()
    return S


def lattice(shape, seed, shift=0.05):
    rng = np.random.default_rng(seed)
    N = int(np.prod(shape))
    idx = np.arange(N).reshape(shape)
    o = np.concatenate([np.take(idx, range(shape[a] - 1), a).reshape(-1) for a in range(3)])
    q = np.concatenate([np.take(idx, range(1, shape[a]), a).reshape(-1) for a in range(3)])
    c = rng.uniform(0.5, 2.0, o.size)
    d = np.bincount(o, c, N) + np.bincount(q, c, N) + shift
    rows = np.concatenate([np.arange(N), o, q]).astype(np.int32)
    cols = np.concatenate([np.arange(N), q, o]).astype(np.int32)
    return rows, cols, np.concatenate([d, -c, -c]), rng.uniform(-1.0, 1.0, N)


def matvec(rows, cols, vals, x):
    return np.bincount(rows, vals * x[cols], x.size)


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("shape", [(1, 1, 1), (3, 1, 1), (7, 3, 1), (9, 7, 1), (13, 5, 1), (9, 11, 7), (14, 14, 14),
                                   (13, 17, 23), (16, 20, 25), (20, 20, 20), (20, 21, 20), (22, 22, 22)])
def test_sizes(semo, precision, shape):
    rows, cols, vals, b = lattice(shape, 5)
    ctx = semo.Context(precision=precision, tol=TOL)
    res = ctx.solve_amgcl("pressure", 1, rows, cols, vals, b)
    r = np.linalg.norm(b - matvec(rows, cols, vals, res.x))
    slack = b.size * 2.0 ** -53 * np.abs(vals).max() * np.linalg.norm(res.x)
    assert r <= TOL * np.linalg.norm(b) + slack and res.info["rel_residual"] <= TOL
    assert abs(res.info["rel_residual"] * np.linalg.norm(b) - r) <= slack
    if b.size <= 1200:
        A = np.zeros((b.size, b.size))
        np.add.at(A, (rows, cols), vals)
        ref = np.linalg.solve(A, b)
        assert np.linalg.norm(res.x - ref) <= 1.01 * np.linalg.cond(A) * TOL * np.linalg.norm(ref)
    again = ctx.solve_amgcl("pressure", 1, rows, cols, vals, b)
    assert np.array_equal(again.x, res.x)
    # from a guess near the solution: fewer iterations; from the solution itself: none or one
    near = ctx.solve_amgcl("pressure", 1, rows, cols, vals, b, res.x * (1.0 + 1e-6))
    assert near.info["iterations"] <= res.info["iterations"] and near.info["rel_residual"] <= TOL
    assert ctx.solve_amgcl("pressure", 1, rows, cols, vals, b, res.x).info["iterations"] <= 1
    ctx.close()


def test_outcomes(semo):
    rows, cols, vals, b = lattice((9, 11, 7), 5)
    ctx = semo.Context(tol=TOL)
    zero = ctx.solve_amgcl("pressure", 1, rows, cols, vals, 0.0 * b)
    assert zero.info["iterations"] == 0 and not zero.x.any() and zero.info["rel_residual"] == 0.0
    n = b.size
    bad = vals.copy()
    bad[:n] *= -1.0   # negative diagonal: p.Ap <= 0
    with pytest.raises(semo.SemoError) as e:
        ctx.solve_amgcl("pressure", 1, rows, cols, bad, b)
    assert e.value.status in (5, 6, 7)
    assert ctx.solve_amgcl("pressure", 1, rows, cols, vals, b).info["rel_residual"] <= TOL   # usable after it
    ctx.close()
    ctx = semo.Context(tol=TOL, max_iter=2)
    with pytest.raises(semo.SemoError) as e:
        ctx.solve_amgcl("pressure", 1, rows, cols, vals, b)
    assert e.value.status == 5
    ctx.close()
