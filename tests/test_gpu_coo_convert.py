"""Caller-supplied COO systems whose entries come in any order (semo_solve_coo, semo_solve_coo_multi).

The conversion to CSR runs on the device, 8 lanes a row, up to 512 entries a
row and on the host above that.  Systems with one row of the lengths at which
those can go wrong, entries shuffled, duplicates among them, against numpy's
dense solve.  Tolerance: the solves stop at 1e-12 relative residual and the
matrices' condition numbers are below 1e3 (checked), so 1e-9.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def semo():
    import semo_mesh_gb300 as S
    S.load_library()
    return S


def system(n, row_len, symmetric, seed):
    """A diagonally dominant tridiagonal-plus-one-long-row system as a shuffled COO triple."""
    rng = np.random.default_rng(seed)
    r, c, v = [], [], []
    for i in range(n - 1):
        r += [i, i + 1]; c += [i + 1, i]; v += [-0.2, -0.2 if symmetric else -0.1]
    long = n // 2
    k = max(row_len - 3, 0)   # the row's diagonal and two neighbours are there already
    others = rng.choice([j for j in range(n) if abs(j - long) > 1], size=min(k, n - 3), replace=False)
    for j in others:
        r.append(long); c.append(j); v.append(-0.5 / max(k, 1))
        if symmetric:
            r.append(j); c.append(long); v.append(-0.5 / max(k, 1))
    r += [3, 3]; c += [4, 2]; v += [-0.05, -0.05]   # duplicates add up
    if symmetric:
        r += [4, 2]; c += [3, 3]; v += [-0.05, -0.05]
    order = rng.permutation(len(r))
    rows = np.concatenate([np.arange(n), np.array(r)[order]]).astype(np.int32)
    cols = np.concatenate([np.arange(n), np.array(c)[order]]).astype(np.int32)
    vals = np.concatenate([np.full(n, 2.0), np.array(v)[order]])
    A = np.zeros((n, n))
    np.add.at(A, (rows, cols), vals)
    assert np.linalg.cond(A) < 1e3
    return rows, cols, vals, A, rng.uniform(-1.0, 1.0, size=(3, n))


@pytest.mark.parametrize("row_len", [3, 8, 9, 33, 511, 512, 513])
def test_long_rows(semo, row_len):
    n = 700
    ctx = semo.Context(precision="fp64", tol=1e-12, mom_tol=1e-12)
    rows, cols, vals, A, B = system(n, row_len, True, row_len)
    x = ctx.solve_amgcl("pressure", 1, rows, cols, vals, B[0]).x
    ref = np.linalg.solve(A, B[0])
    assert np.linalg.norm(x - ref) < 1e-9 * np.linalg.norm(ref)
    rows, cols, vals, A, B = system(n, row_len, False, row_len)
    for j, r in enumerate(ctx.solve_amgcl("momentum", 1, rows, cols, vals, *B)):
        ref = np.linalg.solve(A, B[j])
        assert np.linalg.norm(r.x - ref) < 1e-9 * np.linalg.norm(ref)
    ctx.close()


def test_first_error_is_reported(semo):
    ctx = semo.Context()
    n = 40
    i = np.arange(n, dtype=np.int32)
    one = np.ones(n)
    for bad, status, word in ((("v", 7, np.nan), 6, "matrix value"), (("r", 9, n), 1, "out of range"),
                              (("c", 9, -1), 1, "out of range"), (("d", 5, 0.0), 1, "row 5 has a zero diagonal"),
                              (("b", 3, np.inf), 6, "rhs")):
        r, c, v, b = i.copy(), i.copy(), one.copy(), one.copy()
        {"v": v, "r": r, "c": c, "d": v, "b": b}[bad[0]][bad[1]] = bad[2]
        with pytest.raises(semo.SemoError) as e:
            ctx.solve_amgcl("volume_fraction", 1, r, c, v, b)
        assert e.value.status == status and word in str(e.value)
    # entry 4 is not finite, entry 6 out of range: the first one counts
    r, v = i.copy(), one.copy()
    v[4], r[6] = np.inf, -3
    with pytest.raises(semo.SemoError) as e:
        ctx.solve_amgcl("volume_fraction", 1, r, i, v, one)
    assert e.value.status == 6
    ctx.close()
