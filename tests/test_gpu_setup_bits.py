"""The pressure hierarchy does not depend on where it is built: beside the momentum pass (overlap_setup), alone, or
kept from an earlier call (reuse_hierarchy) give the same bits, at sizes where the one-kernel setup's limits lie."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def semo():
    import semo_mesh_gb300 as S
    S.load_library()
    return S


def case_of(n):
    from semo_mesh_gb300.cases import vof_case, with_fields, with_history
    return with_history(with_fields(vof_case(n), seed=31, p_scale=50.0), seed=32)


def equal(a, b):
    return all(np.array_equal(a[k], b[k]) for k in ("P", "U", "V", "W"))


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("n", [40, 41, 48, 61])
def test_beside_alone_and_kept(semo, n, precision):
    case = case_of(n)
    runs = []
    for overlap, reuse in ((True, False), (False, False), (True, True), (False, True)):
        ctx = semo.Context(precision=precision, overlap_setup=overlap, reuse_hierarchy=reuse)
        ctx.set_case(case)
        norms, info = ctx.outer_iteration()
        f1 = ctx.fields()
        # a further correction: the hierarchy is rebuilt alone, or the one of the call above
        n2, info2 = ctx.calc_pressure_eq()
        runs.append((norms, info[3]["iterations"], n2, info2["iterations"], f1, ctx.fields()))
        ctx.close()
    for r in runs[1:]:
        assert r[:4] == runs[0][:4]
        assert equal(r[4], runs[0][4]) and equal(r[5], runs[0][5])
