"""Gradients keep FP64's accuracy where a cell's weights or values are of very different sizes.

Lattices of 8^3 cells: cells stretched up to 2^10 : 1 with a field 2^20 times
larger along the long side, a cell beside one whose value is 2^20 times the
others' in the plane where its weight is zero, fields far below 1, sign
patterns.  Reference: the least-squares sums in longdouble, with the library's
own cell centres and inverse of the normal matrix.  Tolerance, per component c of an
interior cell with entries k: with a = sum w d phi, every product's and
addition's rounding is at most (n + 3) 2^-53 of the sum of |w d phi| (n = 26,
the term phi_i sum w d included), which the inverse's row carries on:
sum_b |minv_cb| (n + 6) 2^-53 sum_k |w d_b| (|phi_k| + |phi_i|).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
N = 8
EPS = 2.0 ** -53


@pytest.fixture(scope="module")
def semo():
    import semo_mesh_gb300 as S
    S.load_library()
    return S


def field(kind, n):
    """(z, y, x) values."""
    rng = np.random.default_rng(5)
    f = rng.uniform(0.5, 1.0, (n, n, n))
    x = np.arange(n)
    if kind == "columns":      # large along x, and the same for every y and z of a column but for the noise
        return f * np.where(x % 4 == 3, 2.0 ** 20, 1.0)[None, None, :]
    if kind == "one":
        f[4, 4, 4] = 2.0 ** 20
        return f
    if kind == "plane":
        f[:, 4, :] *= 2.0 ** 30
        return f
    if kind == "negative":
        return -f
    if kind == "small":
        return f * 2.0 ** -970
    return f * rng.choice([-1.0, 1.0], f.shape)


@pytest.mark.parametrize("stretch", [(0, 0, 0), (0, 0, 10), (10, 0, 0), (0, 5, 10)])
@pytest.mark.parametrize("kind", ["columns", "one", "plane", "negative", "small", "signs"])
def test_stretched_lattice(semo, stretch, kind):
    from dataclasses import replace
    from semo_mesh_gb300.cases import Case
    from semo_mesh_gb300.meshgen import hex_box
    scale = np.array([2.0 ** -s for s in stretch])
    mesh = hex_box(N)
    mesh = replace(mesh, points=mesh.points * scale)
    f = field(kind, N)
    flat = f.reshape(-1)
    npatch = len(mesh.patch_names)
    case = Case(name="t", mesh=mesh, P=flat, U=flat, V=-flat, W=flat, VF=np.ones(N ** 3),
                bc_type=np.zeros((npatch, 3), np.int32), bc_value=np.zeros((npatch, 5)))
    ctx = semo.Context(precision="fp64")
    ctx.set_case(case)
    ctx.assemble()
    got = {k: ctx.get_array("grad_" + k, 3 * N ** 3).reshape(N, N, N, 3) for k in ("P", "U", "V", "W")}
    cc = ctx.get_array("geometry:cell_c", 3 * N ** 3).reshape(N, N, N, 3).astype(np.longdouble)
    m = ctx.get_array("geometry:lsq_minv", 6 * N ** 3).reshape(N, N, N, 6)
    ctx.close()
    L = np.longdouble
    inner = (slice(1, -1),) * 3
    a, b = np.zeros((3, N - 2, N - 2, N - 2), L), np.zeros((3, N - 2, N - 2, N - 2), L)
    c = f.astype(L)[inner]
    for off in np.ndindex(3, 3, 3):
        o = np.array(off) - 1
        if not o.any():
            continue
        there = tuple(slice(s, s + N - 2) for s in off)
        d = cc[there] - cc[inner]
        w = L(1) / (d * d).sum(axis=-1)
        q = f.astype(L)[there]
        for k in range(3):
            a[k] += w * d[..., k] * (q - c)
            b[k] += np.abs(w * d[..., k]) * (np.abs(q) + np.abs(c))
    at = [[0, 1, 2], [1, 3, 4], [2, 4, 5]]
    for k in range(3):
        minv = [m[inner][..., at[k][j]].astype(L) for j in range(3)]
        ref = sum(minv[j] * a[j] for j in range(3))
        bar = 32 * EPS * sum(np.abs(minv[j]) * b[j] for j in range(3))
        for name, sign in (("P", 1), ("U", 1), ("V", -1), ("W", 1)):
            err = np.abs(sign * got[name][inner][..., k].astype(L) - ref)
            assert (err <= bar).all(), (name, k, float((err / bar).max()))
