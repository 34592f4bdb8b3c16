"""Pressure systems whose finest level is laid out in slices of equal width, and those next to them.

Widths 5, 6 and 7 (lattices of 4, 5 and 6 neighbours) take the layout; width 4
and 8, a row far longer than the others, and columns more than 32,767 from
their row don't.  Sizes about a multiple of 32 rows, above the largest system
that one cluster kernel solves.  The reported residual is compared with numpy's
(they differ by the rounding of a row's products and sum, w + 2 roundings of
|A||x| + |b|), and a right-hand side scaled by a power of two has to scale the
solution exactly: every step of the solve does, conversions included.
"""
import numpy as np
import pytest

from test_gpu_small_cg import lattice, matvec

pytestmark = pytest.mark.gpu
TOL = 1e-10


@pytest.fixture(scope="module")
def semo():
    import semo_mesh_gb300 as S
    S.load_library()
    return S


def add_links(sys, o, q, c=0.7):
    rows, cols, vals, b = sys
    n = b.size
    vals = np.concatenate([vals, np.full(2 * len(o), -c)])
    vals[:n] += c * (np.bincount(o, minlength=n) + np.bincount(q, minlength=n))
    return (np.concatenate([rows, o, q]).astype(np.int32), np.concatenate([cols, q, o]).astype(np.int32), vals, b)


def system(kind):
    if kind == "line":        # width 3
        return lattice((9000, 1, 1), 3)
    if kind == "hex wide":    # width 8: a link across each even row
        s = lattice((21, 22, 23), 3)
        i = np.arange(0, s[3].size // 2 - 1)
        return add_links(s, i, s[3].size - 1 - i)
    if kind == "long row":
        s = lattice((21, 22, 23), 3)
        return add_links(s, np.zeros(300, int), np.arange(5000, 8000, 10))
    if kind == "far":
        rows, cols, vals, b = lattice((41, 42, 41), 3)
        p = np.random.default_rng(1).permutation(b.size).astype(np.int32)
        return p[rows], p[cols], vals, b
    return lattice(kind, 3)


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("kind", [(96, 97, 1), (97, 97, 1), (65, 66, 2), (21, 21, 21), (20, 24, 20), (21, 23, 21), (31, 31, 31),
                                  "line", "hex wide", "long row", "far"])
def test_residual_and_scaling(semo, precision, kind):
    rows, cols, vals, b = system(kind)
    ctx = semo.Context(precision=precision, tol=TOL)
    res = ctx.solve_amgcl("pressure", 1, rows, cols, vals, b)
    r = np.linalg.norm(b - matvec(rows, cols, vals, res.x))
    width = np.bincount(rows).max()
    slack = 2 * (width + 2) * 2.0 ** -53 * np.linalg.norm(matvec(rows, cols, np.abs(vals), np.abs(res.x)) + np.abs(b))
    assert r <= TOL * np.linalg.norm(b) + slack and res.info["rel_residual"] <= TOL
    assert abs(res.info["rel_residual"] * np.linalg.norm(b) - r) <= slack
    for k in (-40, 40):
        scaled = ctx.solve_amgcl("pressure", 1, rows, cols, vals, np.ldexp(b, k))
        assert scaled.info["iterations"] == res.info["iterations"]
        assert np.array_equal(scaled.x, np.ldexp(res.x, k))
    ctx.close()
