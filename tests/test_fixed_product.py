"""The setup's FP64 fixed-point product, round(a b 2^sc) to the nearest integer with ties to even, against exact
rational arithmetic: the header's function compiled for the host."""
import ctypes
import os
import random
import subprocess
from fractions import Fraction

import pytest

from semo_mesh_gb300.build import CSRC, nvcc

SRC = r'''
#include "amg_rows.cuh"
extern "C" long long fixed(double a, double b, int sc) { return semo::amg::fixed_product(a, b, sc); }
'''


@pytest.fixture(scope="module")
def fixed(tmp_path_factory):
    d = tmp_path_factory.mktemp("fixed")
    src, lib = os.path.join(d, "fixed.cu"), os.path.join(d, "libfixed.so")
    with open(src, "w") as f:
        f.write(SRC)
    subprocess.run([nvcc(), "-gencode", "arch=compute_103a,code=sm_103a", "-std=c++17", "-Xcompiler", "-fPIC", "-shared", "-I", CSRC, src, "-o",
                    lib], check=True)
    f = ctypes.CDLL(lib).fixed
    f.argtypes, f.restype = [ctypes.c_double, ctypes.c_double, ctypes.c_int], ctypes.c_longlong
    return f


def cases():
    rng = random.Random(5)
    for _ in range(4000):
        a = rng.uniform(-1.0, 1.0) * 2.0 ** rng.randint(-60, 60)
        b = rng.uniform(-1.0, 1.0) * 2.0 ** rng.randint(-60, 60)
        p = abs(Fraction(a) * Fraction(b))
        top = 0
        while p * Fraction(2) ** top >= Fraction(2) ** 62:
            top -= 1
        while p and p * Fraction(2) ** (top + 1) < Fraction(2) ** 62:
            top += 1
        for sc in (top, top - 1, top - rng.randint(2, 61), top - 62, top - 63, top - 64, top - 130):
            yield a, b, sc
    for a in (0.0, -0.0, 5e-324, 2.0 ** -1022, 1.0, 3.0, -3.0, 2.0 ** 31 - 1):   # subnormals, exact ties, small integers
        for b in (0.0, 5e-324, 1.0, 0.5, -0.5, 1.5, 2.0 ** 29):
            for sc in (-3, -1, 0, 1, 2):
                yield a, b, sc


def test_rounding(fixed):
    n = 0
    for a, b, sc in cases():
        exact = Fraction(a) * Fraction(b) * Fraction(2) ** sc
        assert abs(exact) < 2 ** 62
        assert fixed(a, b, sc) == round(exact), (a, b, sc)   # Fraction rounds ties to even
        n += 1
    assert n > 20000
