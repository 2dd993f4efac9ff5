"""Host (CPU) test of the twiddles' source (simple3.0_b200/csrc/unit_root.h, built here with g++): every root
of unity within half a unit in the last place of its value (and a thousandth for the extended precision it is
evaluated in), the quarter turns exact."""
import ctypes as C
import math
import os
import subprocess
from decimal import Decimal, getcontext

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "simple3.0_b200", "csrc")
PI = Decimal("3.14159265358979323846264338327950288419716939937510582097494459")


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("roots") / "libunit_root_host.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, "-o", out,
                    os.path.join(HERE, "unit_root_host.cpp")], check=True)
    return C.CDLL(out)


def exact(e, n):
    """cos and sin of 2 pi e / n by their series, 50 digits"""
    getcontext().prec = 60
    a = 2 * PI * e / n
    c = s = Decimal(0)
    term = Decimal(1)
    for k in range(120):
        if k % 2 == 0:
            c += term if k % 4 == 0 else -term
        else:
            s += term if k % 4 == 1 else -term
        term = term * a / (k + 1)
    return c, s


@pytest.mark.parametrize("n", [4, 34, 100, 128, 360, 600])
def test_rounded_once(lib, n):
    cs = np.zeros((2 * n, 2))
    lib.unit_roots(C.c_longlong(-n), 2 * n, C.c_longlong(n), cs.ctypes.data_as(C.c_void_p))
    assert np.array_equal(cs[:n], cs[n:])            # negative exponents
    for e in range(n):
        for got, want in zip(cs[n + e], exact(e, n)):
            if abs(want) < Decimal("1e-40"):
                assert got == 0.0
            else:
                assert abs(Decimal(float(got)) - want) <= Decimal(math.ulp(float(got))) * Decimal("0.501")
