"""The batched BiCGStab's off-diagonal layouts through the caller's COO systems.

Rows of equal width (4, 5 or 6 off-diagonal entries: equally wide slices known
to the compiler) and ragged ones (slice pointers), at sizes around a slice, a
block and more than one sweep of the fixed grid, with the diagonal in any place
of a row, repeated diagonals and rows without off-diagonals.  The bar is the
solver's own contract, checked in extended precision: |b - A x| <= tol |b| plus
the rounding of the product, 16 eps (|A| |x| + |b|) in every row.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
TOL = 1e-11


def system(n, width, ragged, seed):
    """Strictly diagonally dominant, columns spread over the whole matrix, entries of a row in random order."""
    rng = np.random.default_rng(seed)
    w = min(width, n - 1)
    rows, cols, vals = [], [], []
    count = rng.integers(0, w + 1, n) if ragged else np.full(n, w)
    total = np.zeros(n)
    for j in range(w):
        i = np.nonzero(count > j)[0]
        c = (i + 1 + j * max((n - 1) // max(w, 1), 1) % max(n - 1, 1)) % n
        c = np.where(c == i, (i + 1) % n, c)
        v = rng.uniform(-1.0, 1.0, i.size)
        rows.append(i); cols.append(c); vals.append(v)
        np.add.at(total, i, np.abs(v))
    d = 1.5 * total + rng.uniform(0.1, 2.0, n)
    i = np.arange(n)
    if ragged:   # the diagonal in two parts, the first the larger
        rows += [i, i]; cols += [i, i]; vals += [0.9 * d, 0.1 * d]
    else:
        rows.append(i); cols.append(i); vals.append(d * rng.choice([-1.0, 1.0], n))
    r, c, v = (np.concatenate(a) for a in (rows, cols, vals))
    if not ragged:
        o = rng.permutation(r.size)
        r, c, v = r[o], c[o], v[o]
    return r.astype(np.int32), c.astype(np.int32), v


@pytest.mark.parametrize("n", [1, 5, 31, 33, 128, 4865, 78001, 160000])
@pytest.mark.parametrize("width,ragged", [(3, False), (4, False), (5, False), (6, False), (7, False), (6, True)])
def test_layouts(n, width, ragged):
    import semo_mesh_gb300 as semo
    r, c, v = system(n, width, ragged, 100 * n + width)
    b = np.random.default_rng(n).uniform(-1.0, 1.0, (3, n))
    ctx = semo.Context(precision="fp64", mom_tol=TOL)
    out = list(ctx.solve_amgcl("momentum", 1, r, c, v, *b)) + [ctx.solve_amgcl("volume_fraction", 1, r, c, v, b[0])]
    ctx.close()
    for j, res in enumerate(out):
        bj = b[j % 3].astype(np.longdouble)
        prod = v.astype(np.longdouble) * res.x.astype(np.longdouble)[c]
        ax, mag = np.zeros(n, np.longdouble), np.zeros(n, np.longdouble)
        np.add.at(ax, r, prod)
        np.add.at(mag, r, np.abs(prod))
        rounding = 16 * np.finfo(np.float64).eps * np.linalg.norm((mag + np.abs(bj)).astype(np.float64))
        got = np.linalg.norm((bj - ax).astype(np.float64))
        assert got <= TOL * np.linalg.norm(b[j % 3]) + rounding, (j, res.info)
