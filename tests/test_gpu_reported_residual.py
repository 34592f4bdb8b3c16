"""The batched BiCGStab's info.rel_residual is |b - A x| / |b| of the returned x and the caller's A, in FP64.

On a diagonal matrix every row of b - A x is one product and one subtraction,
whose roundings numpy repeats exactly, so the reported value is numpy's up to
the order of the sum of squares (n 2^-53 relative).  On general rows (a
dominant and a nearly singular diagonal) it is within the rounding of the
product, (w + 1) 2^-53 (|A||x| + |b|) a row, of the extended-precision one.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -53


@pytest.fixture(scope="module")
def semo():
    import semo_mesh_gb300 as S
    S.load_library()
    return S


@pytest.mark.parametrize("n", [1, 33, 5000])
@pytest.mark.parametrize("guess", [False, True])
def test_diagonal(semo, n, guess):
    rng = np.random.default_rng(n)
    i = np.arange(n, dtype=np.int32)
    d = rng.uniform(0.5, 3.0, n)
    b = rng.uniform(-1.0, 1.0, (3, n))
    x0 = [rng.uniform(-1.0, 1.0, n) for _ in range(3)] if guess else []
    ctx = semo.Context(mom_tol=1e-12)
    out = list(ctx.solve_amgcl("momentum", 1, i, i, d, *b, *x0))
    out.append(ctx.solve_amgcl("volume_fraction", 1, i, i, d, b[0], *x0[:1]))
    ctx.close()
    for j, r in enumerate(out):
        assert r.info["rel_residual"] <= 1e-12
        if guess:
            continue   # the residual is of the correction's system
        bj = b[j % 3]
        ref = np.linalg.norm(bj - d * r.x) / np.linalg.norm(bj)
        assert abs(r.info["rel_residual"] - ref) <= 2 * n * EPS * ref


@pytest.mark.parametrize("n", [5, 1000, 40000])
@pytest.mark.parametrize("width, shift", [(4, 1.5), (6, 1.5), (9, 1.5), (6, 0.6)])
def test_general_rows(semo, n, width, shift):
    rng = np.random.default_rng(n + width)
    w = min(width, n - 1)
    i = np.repeat(np.arange(n), w)
    j = (i + 1 + np.tile(np.arange(w), n) * max(1, (n - 1) // w)) % n
    keep = i != j
    i, j = i[keep], j[keep]
    v = rng.uniform(-1.0, 1.0, i.size)
    d = shift * np.bincount(i, np.abs(v), n) + 0.1
    rows = np.concatenate([i, np.arange(n)]).astype(np.int32)
    cols = np.concatenate([j, np.arange(n)]).astype(np.int32)
    vals = np.concatenate([v, d])
    b = rng.uniform(-1.0, 1.0, (3, n))
    ctx = semo.Context(mom_tol=1e-11, mom_max_iter=2000)
    out = ctx.solve_amgcl("momentum", 1, rows, cols, vals, *b)
    ctx.close()
    L = np.longdouble
    for k, r in enumerate(out):
        ax, mag = np.zeros(n, L), np.zeros(n, L)
        prod = vals.astype(L) * r.x.astype(L)[cols]
        np.add.at(ax, rows, prod)
        np.add.at(mag, rows, np.abs(prod))
        exact = float(np.sqrt(np.sum((b[k] - ax) ** 2)))
        slack = (w + 2) * EPS * float(np.sqrt(np.sum((mag + np.abs(b[k])) ** 2))) + 2 * n * EPS * exact
        assert abs(r.info["rel_residual"] * np.linalg.norm(b[k]) - exact) <= slack
