"""An adjoint whose hierarchy belongs to another matrix than the assembled one is refused.

semo_vjp_fields and semo_vjp_source reuse the hierarchy and the FP64 operator
of the last solve.  After an assembly with another time step, or after a
caller's system, these are not the assembled matrix's: the call ends in an
error and not in a gradient, on meshes of one cell type (equally wide slices),
on tetrahedra, and on systems that one cluster kernel solves.  A new assembly
of the same matrix, and a new solve, give the first gradient again.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
NOT_CONVERGED, STATE = 5, 8


@pytest.fixture(scope="module")
def semo():
    import semo_mesh_gb300 as S
    S.load_library()
    return S


def case_of(n, tets):
    from semo_mesh_gb300.cases import Case, vof_case, with_fields
    if not tets:
        return with_fields(vof_case(n), seed=3, p_scale=10.0)
    from semo_mesh_gb300.meshgen import tet_box
    mesh = tet_box(n, jitter=0.1, seed=2)
    rng = np.random.default_rng(4)
    bt = np.zeros((len(mesh.patch_names), 3), np.int32)
    bt[mesh.patch_names.index("zmax"), 0] = 1
    u = rng.uniform(-1.0, 1.0, (4, mesh.n_cells))
    return Case(name="tets", mesh=mesh, P=u[0], U=u[1], V=u[2], W=u[3], VF=np.ones(mesh.n_cells), bc_type=bt,
                bc_value=np.zeros((len(mesh.patch_names), 5)), dt=1e-3)


def laplacian(n):
    """A caller's chain system of n rows."""
    i = np.arange(n)
    rows = np.concatenate([i, i[:-1], i[1:]]).astype(np.int32)
    cols = np.concatenate([i, i[1:], i[:-1]]).astype(np.int32)
    return rows, cols, np.concatenate([np.full(n, 2.1), np.full(2 * (n - 1), -1.0)]), np.sin(i * 0.1)


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("n, tets", [(14, False), (24, False), (6, True), (13, True)])
def test_assembled_anew(semo, n, tets, precision):
    case = case_of(n, tets)
    ctx = semo.Context(precision=precision, tol=1e-9)
    ctx.set_case(case)
    ctx.assemble()
    ctx.solve()
    g = np.random.default_rng(1).uniform(-1.0, 1.0, ctx.n_cells)
    first, grad, _ = ctx.vjp_fields(g)
    dt = case.dt
    case.dt = 3.0 * dt
    ctx.set_physics(case)
    ctx.assemble()
    for call in (ctx.vjp_fields, ctx.vjp_source):
        with pytest.raises(semo.SemoError) as e:
            call(g)
        assert e.value.status in (STATE, NOT_CONVERGED)
    # the same matrix assembled once more is the hierarchy's again
    case.dt = dt
    ctx.set_physics(case)
    ctx.assemble()
    _, _, info = ctx.vjp_fields(g)
    assert info["rel_residual"] <= 1e-9   # of the assembled matrix
    ctx.solve()
    fresh, grad2, _ = ctx.vjp_fields(g)
    assert np.array_equal(fresh, first) and all(np.array_equal(grad[k], grad2[k]) for k in grad)
    ctx.close()


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("rows", [0, 1, 4096])   # as many as the mesh has cells, one more, far more
def test_after_a_callers_system(semo, rows, precision):
    case = case_of(24, False)
    ctx = semo.Context(precision=precision, tol=1e-9)
    ctx.set_case(case)
    ctx.assemble()
    ctx.solve()
    g = np.random.default_rng(1).uniform(-1.0, 1.0, ctx.n_cells)
    first, _, _ = ctx.vjp_fields(g)
    ctx.solve_amgcl("pressure", 1, *laplacian(ctx.n_cells + rows))
    for call in (ctx.vjp_fields, ctx.vjp_source):
        with pytest.raises(semo.SemoError) as e:
            call(g)
        assert e.value.status in (STATE, NOT_CONVERGED)
    ctx.solve()
    again, _, _ = ctx.vjp_fields(g)
    assert np.array_equal(again, first)
    ctx.close()
