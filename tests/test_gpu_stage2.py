"""GPU tests of the search's second stage at the edges of its row pairs, row groups (64 rows) and column
sets, for each transform length: the top-1 search against the written-out correlations of the same
kernel (the same values, the lowest rotation among equals), the re-scored search, and groups whose
first row is odd.

The re-scored best may differ from the screening's best only where the screening's FP32 values at the
two poses differ by less than the sum of both roundings: each correlation is a transform of P
FP32 sums over the shells, a few 2^-24 relative to its norm (<= 1), so 2e-6 covers both."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def build(pkg, name, nrefs, nptcls, eo=None):
    w = getattr(pkg.synth, name)(nrefs=nrefs, nptcls=nptcls)
    refs, R = pkg.synth.make_refs(w)
    parts = pkg.synth.make_particles(w, R)
    pc = pkg.polarft_corrcalc()
    pc.new(nrefs, (1, nptcls), box=w.box, nrots=w.nrots, kfromto=(w.kfrom, w.kto), ctf=True, ctf_frame="ptcl", eoarr=eo)
    pc.set_refs(1, refs.numpy(), True)
    pc.set_refs(1, refs.numpy() * np.complex64(0.8 + 0.2j), False)
    pc.polarize_ptcls(0, parts.cmat.numpy())
    pc.create_polar_absctfmats(pkg.ctfparams_array(nptcls, smpd=w.smpd, kv=w.kv, cs=w.cs, fraca=w.fraca,
                                                   dfx=parts.dfx, dfy=parts.dfy, angast=parts.angast))
    return w, pc


@pytest.mark.parametrize("name", ["config0", "config1", "geometry_c"])
@pytest.mark.parametrize("precision", ["fp32", "bf16x3"])
@pytest.mark.parametrize("nrefs,ns", [(1, 1), (2, 1), (31, 1), (32, 2), (43, 3), (65, 1)])
def test_rows(pkg, name, precision, nrefs, ns):
    w, pc = build(pkg, name, nrefs, 4)
    shifts = np.array([[0.0, 0.0], [1.0, -0.5], [-0.5, 0.5]], np.float32)[:ns]
    cc = pc.corr_all_prec(shifts, precision).reshape(4, -1)
    top = pc.search_best(shifts, precision, ntop=0)
    idx = cc.argmax(1)
    assert np.array_equal(top["corr"], cc.max(1))
    assert np.array_equal((top["iref"] - 1) * ns * w.nrots + top["ishift"] * w.nrots + top["irot"] - 1, idx)
    for ntop in (1, 8):
        best = pc.search_best(shifts, precision, ntop=ntop)
        at = (best["iref"] - 1) * ns * w.nrots + best["ishift"] * w.nrots + best["irot"] - 1
        tol = 2e-6 if precision == "fp32" else 2e-5     # the screening's BF16 split: 5.8e-6 a value
        assert np.all(cc.max(1) - cc[np.arange(4), at] <= tol)
    pc.kill()


@pytest.mark.parametrize("name", ["config0", "config1", "geometry_c"])
def test_groups_from_odd_rows(pkg, name):
    """rows of a group that start and end inside a row pair, columns of both parities"""
    groups = [(1, 3, 1, 5), (4, 5, 6, 4), (9, 1, 10, 3)]
    w, pc = build(pkg, name, 9, 12, eo=[i % 2 for i in range(12)])
    shifts = np.array([[0.0, 0.0], [1.0, -0.5], [-0.5, 0.5]], np.float32)
    cc = pc.corr_all_prec(shifts, "fp32")
    for ntop in (0, 8):
        got = pc.search_groups(groups, shifts, "fp32", ntop=ntop)
        for r0, nr, s0, n in groups:
            for i in range(s0 - 1, s0 - 1 + n):
                b = got[i]
                assert r0 <= b["iref"] < r0 + nr
                mine = cc[i, r0 - 1:r0 - 1 + nr]
                assert mine.max() - cc[i, b["iref"] - 1, b["ishift"], b["irot"] - 1] <= 2e-6
                assert abs(b["corr"] - mine.max()) <= 2e-6
    pc.kill()
