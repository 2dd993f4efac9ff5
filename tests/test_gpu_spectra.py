"""GPU tests of the search's spectra, normaliser, FP32 contraction and re-score at the edges of their
shell batches (8 shells, two to a transform), column groups (8) and candidate counts, against the FP64
oracle; and of the gridding and CTF kernels' image groups and the adjoint's shell segments against the
same work done one piece at a time.

Tolerances.  FP32 m-domain correlations: |cc| <= 1, each a transform of FP32 sums over at most 2 P Ks
products, 1e-5 as the search tests hold them to.  The adjoint's values are FP64 sums of at most 1e4 terms
in another order: 1e-12 of their scale.  Pieces: the same operations on each image, so the same bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def build(pkg, name, nrefs, nptcls, kstop=None, frame="ptcl", ctf=True, nrots=None):
    kw = {} if nrots is None else {"nrots": nrots}
    w = getattr(pkg.synth, name)(nrefs=nrefs, nptcls=nptcls, **kw)
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
    return w, pc, refs.numpy(), parts


@pytest.mark.parametrize("name,ks", [("config0", k) for k in (1, 2, 7, 8, 9, 16, 17)] +
                         [("config1", k) for k in (8, 33, 38)] + [("geometry_c", k) for k in (17, 58)])
def test_shell_batches(pkg, O, name, ks):
    w, pc, refs, parts = build(pkg, name, 3, 9, kstop=1 + ks)
    g = O.geom(w.nrots, w.kfrom, w.kto, w.box, kstop=1 + ks)
    t = O.tables(g)
    ptcls = np.stack([pc.get_ptcl_pft(i + 1) for i in range(9)])
    ctfs = np.stack([O.ctfmat(g, t, O.make_ctf(w.smpd, w.kv, w.cs, w.fraca, float(parts.dfx[i]), float(parts.dfy[i]),
                                               float(parts.angast[i]))) for i in range(9)])
    for shifts in (None, np.array([[0.0, 0.0], [1.5, -0.75]], np.float32)):
        want = O.allcorrs64(g, t, refs, ptcls, ctfs, shifts, "ptcl")
        assert np.max(np.abs(pc.corr_all_prec(shifts, "fp32") - want)) < 1e-5
        assert np.max(np.abs(pc.corr_all_prec(shifts, "bf16x3") - want)) < 1e-4
        best = want.reshape(9, -1).max(1)
        for ntop in (1, 2, 7, 8):      # 3 or 6 candidates: some of the 8 are empty
            assert np.max(np.abs(pc.search_best(shifts, "fp32", ntop=ntop)["corr"] - best)) < 1e-5
    pc.kill()


@pytest.mark.parametrize("n", [1, 17, 595, 1187, 1601])
def test_image_groups(pkg, n):
    """gridding takes up to four images a block, the CTF one, four or sixteen; box 48 with kto at its limit"""
    w = pkg.synth.config0(nrefs=1, nptcls=n)
    w.box, w.kto = 48, 22
    rng = np.random.default_rng(n)
    img = (rng.standard_normal((n, 48, 25)) + 1j * rng.standard_normal((n, 48, 25))).astype(np.complex64)
    ref = (rng.standard_normal((1, 21, 64)) + 1j * rng.standard_normal((1, 21, 64))).astype(np.complex64)
    df, ast = rng.uniform(1, 3, n).astype(np.float32), rng.uniform(0, 180, n).astype(np.float32)

    def handle(sel):
        pc = pkg.polarft_corrcalc()
        pc.new(1, (1, len(sel)), box=48, nrots=128, kfromto=(2, 22), ctf=True, ctf_frame="ref")
        pc.set_refs(1, ref, True)
        pc.polarize_ptcls(0, img[sel])
        pc.create_polar_absctfmats(pkg.ctfparams_array(len(sel), dfx=df[sel], dfy=df[sel] - 0.05, angast=ast[sel]))
        return pc

    every = handle(np.arange(n))
    for i in sorted({0, n // 2, n - 2 if n > 1 else 0, n - 1}):
        one = handle(np.array([i]))
        assert np.array_equal(every.get_ptcl_pft(i + 1), one.get_ptcl_pft(1))
        assert every.get_sqsum_ptcl(i + 1) == one.get_sqsum_ptcl(1)
        assert np.array_equal(every.gencorrs(1, i + 1), one.gencorrs(1, 1))
        one.kill()
    every.kill()


@pytest.mark.parametrize("box,kto,nrots,n", [(64, 20, 128, 1187), (128, 40, 360, 593), (128, 40, 360, 889),
                                              (128, 40, 360, 890), (200, 60, 600, 593), (200, 60, 600, 889),
                                              (200, 60, 600, 891), (240, 118, 360, 3)])
def test_image_groups_against_the_oracle(pkg, O, box, kto, nrots, n):
    """gridding with one to four images a block (from 592, 888 and 1184 images on; box 200's window leaves room
    for three, box 240's largest for one), remainders of each, against the oracle's polarize: nine products
    summed in FP32, at most 2^-24 (9 + 1) of the taps' moduli, and the weights' rounding: 2e-6 of the largest
    sample.  The square sums: the FP32 sum of 2 K P squares in a tree after a thread's share, 1e-5 relative"""
    rng = np.random.default_rng(n)
    kfrom = kto - 5
    img = (rng.standard_normal((n, box, box // 2 + 1)) + 1j * rng.standard_normal((n, box, box // 2 + 1))).astype(np.complex64)
    pc = pkg.polarft_corrcalc()
    pc.new(1, (1, n), box=box, nrots=nrots, kfromto=(kfrom, kto))
    pc.polarize_ptcls(0, img)
    g = O.geom(nrots, kfrom, kto, box)
    t = O.tables(g)
    for i in sorted({0, 1, 2, 3, n // 2, n - 4, n - 3, n - 2, n - 1} & set(range(n))):
        want = O.polarize(g, t, img[i])
        got = pc.get_ptcl_pft(i + 1)
        assert np.max(np.abs(got - want)) < 2e-6 * np.max(np.abs(want))
        assert abs(pc.get_sqsum_ptcl(i + 1) / np.sum(np.abs(want) ** 2) - 1) < 1e-5
    pc.kill()


@pytest.mark.parametrize("box,kto", [(242, 40), (258, 127)])
def test_boxes_past_the_gridding_are_refused(pkg, box, kto):
    """box 258's window would not be addressed by 16-bit offsets either"""
    pc = pkg.polarft_corrcalc()
    pc.new(1, (1, 1), box=box, nrots=128, kfromto=(2, kto))
    img = np.zeros((1, box, box // 2 + 1), np.complex64)
    for _ in range(2):
        with pytest.raises(pkg.PftccError):
            pc.polarize_ptcls(0, img)
    pc.kill()


@pytest.mark.parametrize("nrots,kstop", [(128, 20), (128, 2), (128, 5), (100, 20), (34, 20), (360, 40), (600, 60)])
def test_adjoint_segments(pkg, nrots, kstop):
    """without a CTF the adjoint is the drop-in gradient (which keeps one segment)"""
    name = {360: "config1", 600: "geometry_c"}.get(nrots, "config0")
    w, pc, refs, _ = build(pkg, name, 3, 4, kstop=kstop, frame="ref", ctf=False, nrots=nrots)
    rng = np.random.default_rng(nrots)
    n = 9
    iref, ip, rot = rng.integers(1, 4, n), rng.integers(1, 5, n), rng.integers(1, nrots + 1, n)
    sh = rng.uniform(-2, 2, (n, 2))
    f, g = pc.grad_batch(iref, ip, rot, sh[:, 0], sh[:, 1], 0.0)
    for i in range(n):
        f1, g1 = pc.gencorr_grad_for_rot_8(int(iref[i]), int(ip[i]), sh[i], int(rot[i]))
        assert abs(f[i] - f1) < 1e-12 and np.max(np.abs(g[i, :2] - g1)) < 1e-12 and g[i, 2] == 0.0
    pc.kill()
