"""GPU tests of the exact correlations by transforms (the lengths 64, 180 and 300): every correlation
against the FP64 oracle at the edges of the kernel's shell pairs, item chunks and modes, and the same
bits for a request alone, in a batch and in a search.

Tolerance without a CTF: the operands are the reference times the shift phase in FP32 -- the phase's
rounding and the complex product's, at most 4 half-ulps (2^-24) of each sample's modulus -- so by
Cauchy-Schwarz a correlation of unit vectors moves by at most 4 * 2^-24 = 2.4e-7; the FP32 square sum
of the particle (a few 1e-8 relative) and the result's rounding (6e-8) leave 4e-7."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
TOL = 4e-7


def build(pkg, name, nrefs, nptcls, frame, kstop=None, ctf=False, kto=None):
    w = getattr(pkg.synth, name)(nrefs=nrefs, nptcls=nptcls)
    if kto:
        w.kto = kto
    refs, R = pkg.synth.make_refs(w)
    parts = pkg.synth.make_particles(w, R)
    pc = pkg.polarft_corrcalc()
    pc.new(nrefs, (1, nptcls), box=w.box, nrots=w.nrots, kfromto=(w.kfrom, w.kto), kstop=kstop, ctf=ctf, ctf_frame=frame,
           eoarr=[0] * nptcls)
    pc.set_refs(1, refs.numpy(), True)
    pc.polarize_ptcls(0, parts.cmat.numpy())
    if ctf:
        pc.create_polar_absctfmats(pkg.ctfparams_array(nptcls, smpd=w.smpd, kv=w.kv, cs=w.cs, fraca=w.fraca,
                                                       dfx=parts.dfx, dfy=parts.dfy, angast=parts.angast))
    return w, pc, refs.numpy()


@pytest.mark.parametrize("frame", ["ref", "ptcl"])
@pytest.mark.parametrize("name,kstop", [("config0", 20), ("config0", 2), ("config0", 9), ("config1", 40), ("config1", 37),
                                        ("geometry_c", 60), ("geometry_c", 55)])
def test_every_correlation(pkg, O, name, kstop, frame):
    """odd and even shell counts, one shell, shells beyond kstop; 5 references = a chunk and a remainder"""
    w, pc, refs = build(pkg, name, 5, 3, frame, kstop=kstop)
    g = O.geom(w.nrots, w.kfrom, w.kto, w.box, kstop=kstop)
    ptcls = np.stack([pc.get_ptcl_pft(i + 1) for i in range(3)])
    for shifts in (None, np.array([[0.0, 0.0], [1.5, -0.75], [-2.0, 2.0]], np.float32)):
        want = O.allcorrs64(g, O.tables(g), refs, ptcls, None, shifts, frame)
        assert np.max(np.abs(pc.corr_all(shifts) - want)) < TOL
    pc.kill()


@pytest.mark.parametrize("frame", ["ref", "ptcl"])
@pytest.mark.parametrize("name,kstop", [("config0", 20), ("config0", 9), ("config1", 37), ("geometry_c", 60), ("geometry_c", 55)])
def test_every_correlation_with_a_ctf(pkg, O, name, kstop, frame):
    """the third channel with a CTF that varies over samples and shells.  The stored |CTF| are FP32 of FP32
    arguments: chi, some 30 here, is off by up to 2^-24 chi and a few of its terms' roundings, 4e-6, at each sample
    on its own, and a correlation of unit vectors moves by the root mean square of that over |CTF|: 1e-5"""
    w, pc, refs = build(pkg, name, 5, 3, frame, kstop=kstop, ctf=True)
    parts = pkg.synth.make_particles(w, pkg.synth.make_refs(w)[1])
    g = O.geom(w.nrots, w.kfrom, w.kto, w.box, kstop=kstop)
    t = O.tables(g)
    ptcls = np.stack([pc.get_ptcl_pft(i + 1) for i in range(3)])
    ctfs = np.stack([O.ctfmat(g, t, O.make_ctf(w.smpd, w.kv, w.cs, w.fraca, float(parts.dfx[i]), float(parts.dfy[i]),
                                               float(parts.angast[i]))) for i in range(3)])
    for shifts in (None, np.array([[0.0, 0.0], [1.5, -0.75], [-2.0, 2.0]], np.float32)):
        want = O.allcorrs64(g, t, refs, ptcls, ctfs, shifts, frame)
        assert np.max(np.abs(pc.corr_all(shifts) - want)) < 1e-5
    pc.kill()


@pytest.mark.parametrize("name", ["config0", "config1", "geometry_c"])
@pytest.mark.parametrize("frame", ["ref", "ptcl"])
@pytest.mark.parametrize("nrefs,nptcls,ns", [(1, 3, 0), (2, 3, 1), (3, 2, 1), (4, 2, 2), (9, 2, 1), (21, 1, 2), (7, 40, 1)])
def test_batch_and_search_equal_single_calls(pkg, name, frame, nrefs, nptcls, ns):
    """1 to 42 items a particle: a single item, chunks, a particle's items shared between blocks"""
    if name != "config0" and nptcls > 10:
        nptcls = 12
    w, pc, refs = build(pkg, name, nrefs, nptcls, frame, ctf=True, kto=11)
    shifts = None if ns == 0 else np.array([[0.5, -1.0], [-1.0, 0.25]], np.float32)[:ns]
    cc = pc.corr_all(shifts)
    for i in (0, nptcls - 1):
        for r in (0, nrefs - 1):
            for s in range(max(1, ns)):
                assert np.array_equal(cc[i, r, s], pc.gencorrs(r + 1, i + 1, None if ns == 0 else shifts[s]))
    best = pc.search_best(shifts, "exact")
    flat = cc.reshape(nptcls, -1).argmax(1)
    assert np.array_equal(best["corr"], cc.reshape(nptcls, -1).max(1))
    assert np.array_equal(best["iref"] - 1, flat // (max(1, ns) * w.nrots))
    assert np.array_equal(best["irot"] - 1, flat % w.nrots)
    pc.kill()


def test_zero_reference_is_never_the_best(pkg):
    """0 / 0 is not a number and takes no part in a maximum, as with the direct sums"""
    w, pc, refs = build(pkg, "config0", 3, 2, "ptcl", ctf=True)
    zero = refs.copy()
    zero[1] = 0
    pc.set_refs(1, zero, True)
    cc = pc.corr_all(None)
    assert np.all(np.isnan(cc[:, 1])) and np.all(np.isfinite(cc[:, [0, 2]]))
    assert np.all(pc.search_best(None, "exact")["iref"] != 2)
    pc.set_refs(1, np.zeros_like(refs), True)
    best = pc.search_best(None, "exact")
    assert np.all(best["iref"] == 0) and np.all(best["irot"] == 0) and np.all(np.isneginf(best["corr"]))
    pc.kill()


def test_weak_ctf(pkg, O):
    """|CTF| of 4e-9 at most (defocus 1e-10 um, no spherical aberration or amplitude contrast): the correlations
    are those of any multiple of it.  It is stored in FP32, off by a few 2^-24 a sample: 1e-6"""
    w = pkg.synth.config0(nrefs=5, nptcls=3)
    refs, R = pkg.synth.make_refs(w)
    parts = pkg.synth.make_particles(w, R)
    pc = pkg.polarft_corrcalc()
    pc.new(5, (1, 3), box=w.box, nrots=w.nrots, kfromto=(w.kfrom, w.kto), ctf=True, ctf_frame="ptcl", eoarr=[0] * 3)
    pc.set_refs(1, refs.numpy(), True)
    pc.polarize_ptcls(0, parts.cmat.numpy())
    df = np.full(3, 1e-10, np.float32)
    pc.create_polar_absctfmats(pkg.ctfparams_array(3, smpd=w.smpd, kv=w.kv, cs=0.0, fraca=0.0, dfx=df, dfy=df))
    g = O.geom(w.nrots, w.kfrom, w.kto, w.box)
    t = O.tables(g)
    ctf = O.ctfmat(g, t, O.make_ctf(w.smpd, w.kv, 0.0, 0.0, 1e-10, 1e-10, 0.0))
    assert 0 < ctf.max() < 1e-8
    ptcls = np.stack([pc.get_ptcl_pft(i + 1) for i in range(3)])
    want = O.allcorrs64(g, t, refs.numpy(), ptcls, np.stack([ctf] * 3) / ctf.max(), None, "ptcl")
    assert np.max(np.abs(pc.corr_all(None) - want)) < 1e-6
    assert np.max(np.abs(pc.search_best(None, "exact")["corr"] - want.reshape(3, -1).max(1))) < 1e-6
    pc.kill()


@pytest.mark.parametrize("name", ["config0", "config1", "geometry_c"])
def test_reference_where_the_ctf_almost_vanishes(pkg, O, name):
    """a reference on one shell, the defocus such that |CTF| is near 2e-6 there (and not on the shells it is
    transformed with): the correlations times the particle's norm are those of a handle of that shell alone,
    up to each value's rounding, the FP32 square sums (2^-24 and some each) and what the transforms leave: 3e-7"""
    w = getattr(pkg.synth, name)(nrefs=1, nptcls=2)
    refs, R = pkg.synth.make_refs(w)
    parts = pkg.synth.make_particles(w, R)
    k = w.kfrom + 6
    g = O.geom(w.nrots, w.kfrom, w.kto, w.box)
    t = O.tables(g)

    def shell(df):
        return np.median(O.ctfmat(g, t, O.make_ctf(w.smpd, w.kv, w.cs, w.fraca, float(df), float(df), 0.0))[k - w.kfrom])

    dfs = np.arange(0.2, 12.0, 0.002)     # towards a zero of the shell's CTF, then to where FP32 defocus values give 2e-6
    df = dfs[np.argmin([shell(x) for x in dfs])]
    for step in (1e-4, 1e-5, 1e-6):
        near = df + step * np.arange(-30, 31)
        df = near[np.argmin([abs(shell(x) - 2e-6) for x in near])]
    df = np.full(2, df, np.float32)
    assert shell(df[0]) < 1e-5
    one = np.zeros_like(refs.numpy())
    one[:, k - w.kfrom] = refs.numpy()[:, k - w.kfrom]
    got = []
    ptcls = None
    for lo, hi in ((w.kfrom, w.kto), (k, k)):
        pc = pkg.polarft_corrcalc()
        pc.new(1, (1, 2), box=w.box, nrots=w.nrots, kfromto=(lo, hi), ctf=True, ctf_frame="ptcl", eoarr=[0] * 2)
        pc.set_refs(1, one[:, lo - w.kfrom:hi + 1 - w.kfrom], True)
        if ptcls is None:
            pc.polarize_ptcls(0, parts.cmat.numpy())
            ptcls = np.stack([pc.get_ptcl_pft(i + 1) for i in range(2)])
        else:
            pc.set_ptcls(0, ptcls[:, k - w.kfrom:k + 1 - w.kfrom])
        pc.create_polar_absctfmats(pkg.ctfparams_array(2, smpd=w.smpd, kv=w.kv, cs=w.cs, fraca=w.fraca, dfx=df, dfy=df))
        norm = np.sqrt([np.float64(pc.get_sqsum_ptcl(i + 1)) for i in range(2)])
        got.append(pc.corr_all(None).astype(np.float64)[:, 0, 0] * norm[:, None])
        pc.kill()
    assert np.all(np.isfinite(got[0]))
    scale = np.abs(got[1]).max(1, keepdims=True)
    assert np.max(np.abs(got[0] - got[1]) / scale) < 3e-7


def test_large_result_into_page_locked_memory(pkg):
    """36 MB of correlations, past the 32 MiB that go in pieces: page-locked and pageable destinations hold the same"""
    import ctypes as C

    import torch
    w, pc, refs = build(pkg, "config0", 64, 1100, "ref")
    want = pc.corr_all(None)
    got = torch.zeros(want.shape, dtype=torch.float32).pin_memory()
    pc._check(pc._L.pftcc_corr_all(pc._h, 0, None, C.cast(got.data_ptr(), C.POINTER(C.c_float))))
    assert np.array_equal(got.numpy(), want)
    pc.kill()
