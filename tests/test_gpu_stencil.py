"""The fixed-point stencil pass: gradients and limits against FP64 in numpy.

Meshes where it can go wrong: one cell (no stencil), small lattices, an odd
jittered box, jittered tetrahedra (stencils of more than 64 entries, where the
sums are carried); fields of one value, of values 2^60 apart in one stencil, all
zero, near the bottom of the range, with a large common part.  Reference: the LSQ sums in numpy's
longdouble from the library's own cell centres' geometry, computed here from the
mesh (plain lattice) -- or, on jittered meshes, exactness for linear fields.
Tolerance: the fixed-point sum of n entries is within n 2^-53 of the largest
product |g||phi| (derivation in the kernel's header), and the weights' rounding
adds as much: 4 n 2^-53 max|g| max|phi|.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def semo():
    import semo_mesh_gb300 as S
    S.load_library()
    return S


def context(semo, mesh, U, V, W, P):
    from semo_mesh_gb300.cases import Case
    npatch = len(mesh.patch_names)
    case = Case(name="t", mesh=mesh, P=P, U=U, V=V, W=W, VF=np.ones(mesh.n_cells),
                bc_type=np.zeros((npatch, 3), np.int32), bc_value=np.zeros((npatch, 5)))
    ctx = semo.Context(precision="fp64")
    ctx.set_case(case)
    ctx.assemble()
    return ctx


def lattice_gradient(f, n):
    """LSQ over the 26 neighbours and the boundary faces (zero gradient there) of the n^3 unit box, in longdouble."""
    h = np.longdouble(1.0) / n
    f = f.astype(np.longdouble).reshape(n, n, n)
    pad, live = np.zeros((n + 2,) * 3, np.longdouble), np.zeros((n + 2,) * 3, np.longdouble)
    pad[1:-1, 1:-1, 1:-1], live[1:-1, 1:-1, 1:-1] = f, 1
    M, r = np.zeros((3, 3, n, n, n), np.longdouble), np.zeros((3, n, n, n), np.longdouble)
    big = np.zeros((n, n, n), np.longdouble)
    for off in np.ndindex(3, 3, 3):
        d = (np.array(off) - 1) * h
        if not d.any():
            continue
        at = tuple(slice(o, o + n) for o in off)
        w = live[at] / (d @ d)
        big = np.maximum(big, np.abs(pad[at]) * live[at])
        for a in range(3):
            r[a] += w * d[a] * (pad[at] - f)
            for b in range(3):
                M[a, b] += w * d[a] * d[b]
    for a in range(3):
        for end in (0, n - 1):
            at = [slice(None)] * 3
            at[a] = end
            M[a, a][tuple(at)] += 1
    # M is diagonal on the lattice but at the corners and edges: invert by cofactors
    g = np.empty_like(r)
    det = (M[0, 0] * (M[1, 1] * M[2, 2] - M[1, 2] ** 2) - M[0, 1] * (M[0, 1] * M[2, 2] - M[1, 2] * M[0, 2])
           + M[0, 2] * (M[0, 1] * M[1, 2] - M[1, 1] * M[0, 2]))
    inv = [[M[1, 1] * M[2, 2] - M[1, 2] ** 2, M[0, 2] * M[1, 2] - M[0, 1] * M[2, 2], M[0, 1] * M[1, 2] - M[0, 2] * M[1, 1]],
           [None, M[0, 0] * M[2, 2] - M[0, 2] ** 2, M[0, 1] * M[0, 2] - M[0, 0] * M[1, 2]],
           [None, None, M[0, 0] * M[1, 1] - M[0, 1] ** 2]]
    for a in range(3):
        g[a] = sum(inv[min(a, b)][max(a, b)] * r[b] for b in range(3)) / det
    return g.reshape(3, -1), np.maximum(big, np.abs(f)).reshape(-1)


@pytest.mark.parametrize("n", [2, 4, 8])   # powers of two: the lattice's centres are exact
@pytest.mark.parametrize("kind", ["uniform", "offset", "spread", "constant", "zero", "tiny"])
def test_lattice(semo, n, kind):
    from semo_mesh_gb300.meshgen import hex_box
    mesh = hex_box(n)
    rng = np.random.default_rng(n)
    nc = mesh.n_cells
    f = {"uniform": rng.uniform(-1, 1, nc), "offset": 1e5 + rng.uniform(-1, 1, nc),
         "spread": rng.uniform(-1, 1, nc) * 2.0 ** rng.integers(-60, 1, nc), "constant": np.full(nc, -3.7),
         "zero": np.zeros(nc), "tiny": rng.uniform(-1, 1, nc) * 1e-280}[kind]
    ctx = context(semo, mesh, f, -f, np.zeros(nc), np.zeros(nc))
    ref, big = lattice_gradient(f, n)
    ref = ref[::-1]   # (z, y, x) -> x, y, z
    # |g| <= |M^-1| |w d| <= n_scale / h: the largest weight of a two-cell side is below 2 / h
    bar = 4 * 26 * 2.0 ** -53 * (2.0 * n) * big.astype(float)
    for name, sign in (("grad_U", 1.0), ("grad_V", -1.0)):
        g = ctx.get_array(name, 3 * nc).reshape(nc, 3)
        for a in range(3):
            assert (np.abs(sign * g[:, a] - ref[a].astype(float)) <= bar).all(), (name, a)
    assert not ctx.get_array("grad_W", 3 * nc).any()
    mm = ctx.get_array("minmax_uvw", 6 * nc).reshape(nc, 6)
    pad = np.pad(f.reshape(n, n, n), 1, mode="edge")
    win = [pad[tuple(slice(o, o + n) for o in off)].reshape(-1) for off in np.ndindex(3, 3, 3)]
    assert np.array_equal(mm[:, 0], np.max(win, axis=0)) and np.array_equal(mm[:, 1], np.min(win, axis=0))
    ctx.close()


@pytest.mark.parametrize("tets", [False, True])
def test_linear_fields_on_jittered_meshes(semo, tets):
    """Away from the boundary (whose faces hold the cell's value) LSQ is exact for linear fields."""
    from semo_mesh_gb300.meshgen import hex_box, tet_box
    mesh = tet_box(6, jitter=0.15, seed=3) if tets else hex_box(9, jitter=0.25, seed=3)
    nc = mesh.n_cells
    ctx0 = context(semo, mesh, np.zeros(nc), np.zeros(nc), np.zeros(nc), np.zeros(nc))
    cc = ctx0.get_array("geometry:cell_c", 3 * nc).reshape(nc, 3)
    f = 2.0 + cc @ np.array([0.3, -1.1, 0.7])
    ctx = context(semo, mesh, f, np.zeros(nc), np.zeros(nc), f)
    inner = np.ones(nc, bool)
    inner[mesh.owner[mesh.n_internal:]] = False
    h = 1.0 / (6 if tets else 9)
    # 4 n 2^-53 max|g| max|phi| with n <= 200 entries, |g| <= 40 / h on these meshes, |phi| <= 5
    bar = 4 * 200 * 2.0 ** -53 * (40.0 / h) * 5.0
    for name in ("grad_U", "grad_P"):
        g = ctx.get_array(name, 3 * nc).reshape(nc, 3)[inner]
        assert np.abs(g - np.array([0.3, -1.1, 0.7])).max() <= bar
    ctx.close()
