"""The coarsest level's inverse and its product, as the whole solver of a small dense system.

Symmetric positive definite matrices B B^T + I of 1 to 64 rows: Gauss-Jordan then
takes pivots off the diagonal.  Above 64 rows the other inverse is used.  The solve
stops at 1e-11 relative residual, so the error is at most the condition number
times that (and numpy's, the condition number times some 1e-14).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("n", [1, 2, 15, 16, 17, 31, 33, 48, 63, 64, 65, 97])
def test_dense(precision, n):
    import semo_mesh_gb300 as semo
    rng = np.random.default_rng(n)
    B = rng.uniform(-1.0, 1.0, (n, n))
    A = B @ B.T + np.eye(n)
    r, c = (a.reshape(-1).astype(np.int32) for a in np.indices((n, n)))
    b = rng.uniform(-1.0, 1.0, n)
    ctx = semo.Context(precision=precision, tol=1e-11, coarse_enough=100)
    x = ctx.solve_amgcl("pressure", 1, r, c, A.reshape(-1), b)
    ref = np.linalg.solve(A, b)
    assert np.linalg.norm(x.x - ref) <= 1.01e-11 * np.linalg.cond(A) * np.linalg.norm(ref)
    assert x.info["iterations"] <= (1 if precision == "fp64" else 4)
    ctx.close()
