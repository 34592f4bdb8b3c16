"""Places and sizes near the ends of 32 bits: the rule for equally wide slices, and a thread's row.

The systems that reach them have hundreds of millions of rows, so the helpers
(index.h) are compiled for the host and compared with Python's integers.
"""
import ctypes
import os
import subprocess

import pytest

from semo_mesh_gb300.build import CSRC

INT_MAX = 2 ** 31 - 1
SRC = r'''
#include "index.h"
extern "C" long long even(int w, int lo, int hi, long long nslices, long long slots) {
    return semo::even_slots(w, lo, hi, nslices, slots);
}
extern "C" long long row(unsigned b, unsigned t, unsigned i, int lanes) { return semo::row_of(b, t, i, lanes); }
'''


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("index")
    src, out = os.path.join(d, "index.cpp"), os.path.join(d, "libindex.so")
    with open(src, "w") as f:
        f.write(SRC)
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, src, "-o", out], check=True)
    L = ctypes.CDLL(out)
    L.even.argtypes, L.even.restype = [ctypes.c_int] * 3 + [ctypes.c_longlong] * 2, ctypes.c_longlong
    L.row.argtypes, L.row.restype = [ctypes.c_uint] * 3 + [ctypes.c_int], ctypes.c_longlong
    return L


@pytest.mark.parametrize("width", [3, 4, 5, 6, 7, 8])
def test_even_slots(lib, width):
    for nslices in (1, 2, 1000, 9_000_000, 9_586_980, 9_586_981, 9_590_000, 11_184_810, 11_184_811, 60_000_000):
        full = 32 * width * nslices
        for slots in (full, full - full // 9, full - full // 9 - 32, full // 2, min(full, 1_950_000_000), INT_MAX):
            got = lib.even(width, 5, 7, nslices, slots)
            take = 5 <= width <= 7 and full <= slots + slots // 8 and full < INT_MAX
            assert got == (full if take else 0), (nslices, slots)
            assert got < INT_MAX


def test_row_of(lib):
    for lanes in (1, 8, 32):
        for n in (1, 255, 256, 2 ** 28 - 1, 2 ** 28, 2 ** 28 + 5, 300_000_000, INT_MAX):
            blocks = (n * lanes + 255) // 256
            for b in (0, blocks // 2, blocks - 1):
                for t in (0, 7, 8, 255):
                    assert lib.row(b, 256, t, lanes) == (b * 256 + t) // lanes
            assert lib.row(blocks - 1, 256, (n * lanes - 1) % 256, lanes) == n - 1
