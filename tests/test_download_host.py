"""Host (CPU) tests of a large result's way to the caller (simple3.0_b200/csrc/download.h, built here with
g++ over a device whose copies land when they are waited for): page-locked memory takes one direct copy,
a large result into pageable memory pieces through two pinned buffers, the plain copy serves where there are none, and a
failed copy's status is returned."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "simple3.0_b200", "csrc")
PIECE, LARGE = 4 << 20, 32 << 20


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("download") / "libdownload_host.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-pthread", "-I", CSRC, "-o", out,
                    os.path.join(HERE, "download_host.cpp")], check=True)
    L = C.CDLL(out)

    def call(nbytes, page_locked=False, pieces=2, fail=-1):
        src = np.random.default_rng(nbytes).integers(0, 256, nbytes, dtype=np.uint8)
        dst = np.zeros(nbytes, np.uint8)
        copies, direct = C.c_int(), C.c_int()
        st = L.download_run(src.ctypes.data_as(C.c_void_p), dst.ctypes.data_as(C.c_void_p), C.c_size_t(nbytes),
                            int(page_locked), pieces, fail, C.byref(copies), C.byref(direct))
        return st, copies.value, direct.value, np.array_equal(src, dst)

    return call


@pytest.mark.parametrize("nbytes", [1, 2 * PIECE, LARGE - 1, LARGE, LARGE + 1, LARGE + PIECE + 4097])
def test_route_and_contents(run, nbytes):
    n = -(-nbytes // PIECE)
    large = nbytes >= LARGE
    assert run(nbytes) == (0, n if large else 1, 0 if large else 1, True)
    assert run(nbytes, page_locked=True) == (0, 1, 1, True)
    for pieces in (0, 1):
        assert run(nbytes, pieces=pieces) == (0, 1, 1, True)


@pytest.mark.parametrize("fail", [0, 1, 2])
def test_failed_copy(run, fail):
    st, copies, _, _ = run(LARGE, fail=fail)
    assert st == 7 and copies == fail + 1
