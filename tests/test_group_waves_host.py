"""Host (CPU) tests of the grouped search's launches (simple3.0_b200/csrc/group_waves.h, built here with
g++): the waves of a batch cover every (row, column) of their groups once and keep the budgets, and no
two waves of one launch share a column -- stage 2's blocks each merge into their column's top 8 without
any order between them, so a group cut by rows must be searched in successive launches."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "simple3.0_b200", "csrc")
GIB = 1 << 30


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("waves") / "libgroup_waves_host.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, "-o", out,
                    os.path.join(HERE, "group_waves_host.cpp")], check=True)
    L = C.CDLL(out)

    def call(P, ns, groups, z_wave=GIB, z_max=2 * GIB, d_max=GIB):
        dlen = {64: 64, 180: 200, 300: 300}[P]
        geom = np.array([P, ns, dlen, P // 2 + 1, 64, 128], np.int32)
        g = np.ascontiguousarray(groups, np.int32)
        waves, sets, sums = np.zeros((4096, 8), np.int32), np.zeros(4096, np.int32), np.zeros((4096, 3), np.uint64)
        p = lambda a: a.ctypes.data_as(C.c_void_p)
        n = L.group_waves_run(p(geom), len(g), p(g), C.c_size_t(z_wave), C.c_size_t(z_max), C.c_size_t(d_max), 4096,
                              p(waves), p(sets), p(sums))
        assert n > 0
        return waves[:n], sets[:n], sums[:sets[n - 1] + 1]

    return call


@pytest.mark.parametrize("P,ns,groups,cut", [
    (64, 81, [(0, 200 * 81, 0, 256)], True),                                       # 8192 rows a wave, then 8008
    (300, 1, [(0, 300, 0, 1500)], True),                                           # 256 rows, then 44: 1.2 GiB together
    (300, 1, [(0, 57, 0, 865), (57, 207, 865, 1315), (207, 308, 1315, 2565)], False),
    (180, 3, [(0, 33, 0, 75), (33, 54, 75, 105), (54, 93, 105, 170)], False),       # tiles shared, columns not
    (64, 81, [(0, 405, 0, 40), (405, 30000, 40, 900), (30000, 30081, 900, 1000)], True),
    (180, 1, [(5, 3000, 0, 3000), (3000, 6007, 3000, 8192)], True),
])
def test_waves_and_their_launches(run, P, ns, groups, cut):
    waves, sets, sums = run(P, ns, groups)
    assert (len(waves) > len(groups)) == cut
    at = 0
    for r_lo, r_end, c_lo, c_hi in groups:      # the rows of a group one after another, once
        r = r_lo
        while r < r_end:
            w = waves[at]
            assert w[0] == r and tuple(w[4:6]) == (c_lo, c_hi)
            assert w[2] % 64 == 0 and w[3] % 64 == 0 and w[2] <= w[0] < w[1] <= w[3]
            assert w[6] * 128 <= c_lo and c_hi <= w[7] * 128
            z = P * (w[3] - w[2]) * (w[7] - w[6]) * 128 * 8
            assert z <= GIB or w[3] - w[2] == 64
            r, at = w[1], at + 1
        assert r == r_end
    assert at == len(waves)
    assert np.all(np.diff(sets) >= 0) and np.all(np.diff(sets) <= 1)
    for s in range(sets[-1] + 1):
        mine = waves[sets == s]
        held = np.zeros(mine[:, 5].max(), int)
        for w in mine:
            held[w[4]:w[5]] += 1
        assert held.max() == 1, "two waves of one launch share a column"
        z = sum(P * int(w[3] - w[2]) * int(w[7] - w[6]) * 128 * 8 for w in mine)
        assert z == sums[s][0] and (z <= 2 * GIB or len(mine) == 1)
        assert sums[s][1] <= GIB or len(mine) == 1
    if not cut:
        assert sets[-1] == 0                     # groups that fit share their launch
