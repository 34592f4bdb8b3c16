"""Device memory that a pressure hierarchy keeps: what its levels hold, not the scratch of their construction."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def used_bytes():
    """Bytes in use in the device's stream-ordered pool."""
    import glob
    lib = None
    for name in ["libcudart.so.13", "libcudart.so"] + glob.glob("/usr/local/cuda/lib64/libcudart.so*"):
        try:
            lib = ctypes.CDLL(name)
            break
        except OSError:
            continue
    if lib is None:
        pytest.skip("no libcudart")
    pool, value = ctypes.c_void_p(), ctypes.c_uint64()
    assert lib.cudaDeviceSynchronize() == 0
    assert lib.cudaDeviceGetDefaultMemPool(ctypes.byref(pool), 0) == 0
    assert lib.cudaMemPoolGetAttribute(pool, 7, ctypes.byref(value)) == 0   # cudaMemPoolAttrUsedMemCurrent
    return value.value


@pytest.mark.parametrize("precision, size", [("mixed", 4), ("fp64", 8)])
def test_levels_only(precision, size):
    import semo_mesh_gb300 as semo
    n = 40
    idx = np.arange(n ** 3).reshape(n, n, n)
    o = np.concatenate([np.take(idx, range(n - 1), a).reshape(-1) for a in range(3)])
    q = np.concatenate([np.take(idx, range(1, n), a).reshape(-1) for a in range(3)])
    diag = (np.bincount(o, minlength=n ** 3) + np.bincount(q, minlength=n ** 3) + 0.01)
    rows = np.concatenate([idx.reshape(-1), o, q]).astype(np.int32)
    cols = np.concatenate([idx.reshape(-1), q, o]).astype(np.int32)
    vals = np.concatenate([diag, np.full(2 * o.size, -1.0)])
    ctx = semo.Context(precision=precision)
    before = used_bytes()
    ctx.solve_amgcl("pressure", 1, rows, cols, vals, np.sin(np.arange(n ** 3)))
    kept = used_bytes() - before
    lev = ctx.hierarchy_levels()
    entries = sum(v["nnz_A"] + v["nnz_P"] + v["nnz_R"] for v in lev)
    nrows = sum(v["rows"] for v in lev)
    ctx.close()
    # an entry of A, P, R in CSR and in a sliced copy with up to an eighth of padding, the FP64 operator's sliced copy;
    # a level's vectors (5), pointers (5) and the Krylov vectors (4 of FP64) a row; the coarsest inverse, reductions
    # and the pool's rounding in the last term
    bound = entries * (4 + size) * 2.125 + 10 * 1.125 * rows.size + nrows * (5 * size + 20 + 32) + (4 << 20)
    assert kept <= bound, (kept, bound)
