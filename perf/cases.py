"""What the library's speed is measured on: calls a 2D classification or 3D refinement makes through
``polarft_corrcalc``, over the three geometries of the package's workloads (box 64 / 128 rotations /
shells 2..20, box 128 / 360 / 2..40, box 200 / 600 / 2..60).

``listed()`` are the cases, ``draw(rng)`` gives more of the same ranges, ``prepare`` makes a case's
handle and inputs from a seed, ``run`` is one pass, ``work`` the bytes and operations a pass cannot do
without, ``tolerance`` how far two correct implementations may differ, and ``exact`` the same outputs in
64 bits by plain torch.  Data: a volume of Gaussian blobs, references its central sections (the odd
half's carry noise of their own), particles the even sections rotated, shifted, times |CTF|, with white
noise at signal-to-noise 0.1."""
import importlib.util
import math
import os
import sys

import numpy as np
import torch

GEOMETRIES = {64: (128, 2, 20), 128: (360, 2, 40), 200: (600, 2, 60)}   # box: rotations, first and last shell
DEV = "cuda"


def _package():
    if "simple3_0_b200" not in sys.modules:
        where = os.path.join(os.getcwd(), "simple3.0_b200")
        spec = importlib.util.spec_from_file_location("simple3_0_b200", os.path.join(where, "__init__.py"),
                                                      submodule_search_locations=[where])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["simple3_0_b200"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["simple3_0_b200"]


def _case(kind, box, nrefs, nptcls, **more):
    nrots, kfrom, kto = GEOMETRIES[box]
    c = {"kind": kind, "box": box, "nrots": nrots, "kfrom": kfrom, "kto": kto, "nrefs": nrefs, "nptcls": nptcls,
         "grid": 0, "frame": "ref", "precision": "exact", "euclid": False, "pairs": 0, "groups": ""}
    c.update(more)
    return c


def listed():
    named = {
        # one drop-in gencorrs(iref, iptcl, shvec) call, as the host strategies make them one by one
        "gencorrs_box64": _case("gencorrs", 64, 20, 50),
        # a host strategy's batch of such pairs into its own device buffer, the largest box
        "pairs_box200": _case("pairs", 200, 60, 500, pairs=500),
        # every correlation of a small 2D classification, returned to the host
        "corr_all_box64": _case("corr_all", 64, 100, 1000),
        # the greedy search of the same classification, the tensor-core path
        "search_box64": _case("search", 64, 100, 1000, frame="ptcl", precision="bf16x3"),
        # the headline step: new particles gridded, their CTF made, the exhaustive search on a 9 x 9 shift grid
        "step_box128": _case("step", 128, 500, 20000, grid=9, frame="ptcl", precision="bf16x3"),
        # the plain FP32 path on the same grid
        "search_fp32_box128": _case("search", 128, 100, 1000, grid=9, frame="ptcl", precision="fp32"),
        # the tensor-core search with the reference's own CTF frame: its candidates re-scored exactly
        "search_ref_box128": _case("search", 128, 100, 1000, grid=9, precision="bf16x3"),
        # chunks of a streaming classification in one handle, each against its own references
        "groups_box200": _case("groups", 200, 308, 5130, frame="ptcl", precision="bf16x3",
                               groups="57x1730 150x900 101x2500"),
        # the noise-weighted Euclidean objective, odd sizes
        "euclid_box128": _case("search", 128, 61, 777, grid=5, frame="ptcl", precision="bf16x3", euclid=True),
        # the adjoint of a continuous refinement: value and shift / defocus gradients, 11 rotations a particle
        "grad_box128": _case("grad", 128, 100, 2000, pairs=22000),
        # a 3D refinement round: both half-volumes projected into the references, then the greedy search
        "project_box128": _case("project", 128, 500, 2000, frame="ptcl", precision="bf16x3"),
    }
    return [dict(c, name=n) for n, c in named.items()]


def draw(rng):
    def logint(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    box = rng.choice([64, 128, 200])
    kind = rng.choice(["gencorrs", "pairs", "corr_all", "search", "search", "search", "step", "groups", "grad", "project"])
    if kind == "project":
        box = rng.choice([64, 128])
    if kind == "gencorrs":
        c = _case(kind, box, rng.randint(5, 60), rng.randint(10, 200))
    elif kind == "pairs":
        c = _case(kind, box, rng.randint(10, 100), rng.randint(50, 600), pairs=logint(20, 3000))
    elif kind == "corr_all":
        c = _case(kind, box, logint(10, 100), logint(20, 1000 if box == 64 else 200))
    elif kind == "search":
        grid = rng.choice([0, 0, 3, 5, 9])
        precision = rng.choice(["bf16x3", "bf16x3", "fp32", "exact"])
        frame = rng.choice(["ptcl", "ptcl", "ref"])
        euclid = frame == "ptcl" and precision != "exact" and rng.random() < 0.25
        small = precision == "exact"
        c = _case(kind, box, logint(10, 40 if small else 300), logint(30, 100 if small else 3000),
                  grid=min(grid, 3) if small else grid, frame=frame, precision=precision, euclid=euclid)
    elif kind == "step":
        c = _case(kind, box, logint(50, 300), logint(500, 4000), grid=rng.choice([0, 3, 5, 9]), frame="ptcl",
                  precision="bf16x3")
    elif kind == "groups":
        sizes = [(rng.randint(50, 300), logint(300, 3000)) for _ in range(rng.randint(2, 4))]
        c = _case(kind, box, sum(r for r, _ in sizes), sum(p for _, p in sizes), frame="ptcl", precision="bf16x3",
                  groups=" ".join("%dx%d" % s for s in sizes))
    elif kind == "grad":
        c = _case(kind, box, rng.randint(10, 200), logint(100, 2000), pairs=logint(50, 22000))
    else:
        c = _case(kind, box, logint(50, 500), logint(300, 3000), frame="ptcl", precision="bf16x3")
    c["kto"] -= rng.randint(0, 5)     # the resolution limit moves as a run goes on
    return c


# ---- inputs ------------------------------------------------------------------------------
def _shifts(case):
    n = case["grid"]
    if not n:
        return None
    s = (np.arange(n) - (n - 1) / 2) * 0.5
    return np.stack(np.meshgrid(s, s, indexing="ij"), -1).reshape(-1, 2).astype(np.float32)


def _grid(case):
    """the polar coordinates (single precision, as the reference's tables), FP64 tensors (K, P)"""
    n, ang = case["nrots"], np.float32(2 * math.pi) / np.float32(case["nrots"])
    a = (np.arange(n // 2, dtype=np.float32) * ang).astype(np.float32)
    k = np.arange(case["kfrom"], case["kto"] + 1, dtype=np.float32)[:, None]
    sin, cos = (f(a.astype(np.float64)).astype(np.float32)[None] for f in (np.sin, np.cos))
    x, y = (sin * k).astype(np.float32), (-cos * k).astype(np.float32)
    return tuple(torch.as_tensor(v, dtype=torch.float64, device=DEV) for v in (x, y))


def _abs_ctf(case, p, ddf=0.0, sel=None):
    """|CTF| on the polar grid in 64 bits, (n, K, P), and its derivative by the defocus in microns"""
    x, y = _grid(case)
    s2, ang = (x * x + y * y) / case["box"] ** 2, torch.atan2(y, x)
    kv = 3.0e5
    wl = 12.26 / math.sqrt(kv + 0.9784 * kv * kv / 1.0e6) / p["smpd"]
    cs, sc = p["cs"] * 1.0e7 / p["smpd"], 1.0e4 / p["smpd"]
    dfx, dfy, ast = (torch.as_tensor(p[k], dtype=torch.float64, device=DEV)[:, None, None] for k in ("dfx", "dfy", "ast"))
    if sel is not None:
        dfx, dfy, ast = dfx[sel], dfy[sel], ast[sel]
    ast = ast * math.pi / 180.0
    df = 0.5 * (dfx + dfy + 2 * ddf + torch.cos(2 * (ang - ast)) * (dfx - dfy)) * sc
    chi = math.pi * wl * s2 * (df - 0.5 * wl * wl * s2 * cs) + math.atan(p["fraca"] / math.sqrt(1 - p["fraca"] ** 2))
    s = torch.sin(chi)
    return s.abs(), torch.where(s >= 0, 1.0, -1.0) * torch.cos(chi) * math.pi * wl * s2 * sc


def _ext(a):
    """samples continued over the full circle by conjugate symmetry, (..., K, 2P)"""
    return torch.cat([a, a.conj()], -1)


def _phase(case, shifts):
    """the shift phases, (n, K, P)"""
    x, y = _grid(case)
    s = torch.as_tensor(np.asarray(shifts), dtype=torch.float64, device=DEV)
    a = math.pi / (case["box"] // 2) * (s[:, 0, None, None] * x + s[:, 1, None, None] * y)
    return torch.polar(torch.ones_like(a), a)


def _euler(e):
    """rotation matrices R3 R2 R1 of Spider Euler triplets in degrees, (n, 3, 3)"""
    t = torch.deg2rad(torch.as_tensor(e, dtype=torch.float64, device=DEV))
    c, s, z, o = torch.cos(t), torch.sin(t), torch.zeros_like(t[:, 0]), torch.ones_like(t[:, 0])

    def rz(i):
        return torch.stack([c[:, i], s[:, i], z, -s[:, i], c[:, i], z, z, z, o], -1).reshape(-1, 3, 3)

    ry = torch.stack([c[:, 1], z, -s[:, 1], z, o, z, s[:, 1], z, c[:, 1]], -1).reshape(-1, 3, 3)
    return rz(2) @ ry @ rz(0)


def _inputs(case, seed):
    S = _package().synth
    make = {64: S.config0, 128: S.config1, 200: S.geometry_c}[case["box"]]
    w = make(nrefs=case["nrefs"], nptcls=case["nptcls"], kto=case["kto"], seed_base=100 * seed + 7)
    K, P, N, n = w.K, w.pftsz, w.nrots, case["nptcls"]
    g = torch.Generator(device=DEV).manual_seed(seed)
    r = np.random.default_rng(seed)
    d = {"w": w}
    if case["kind"] == "project":
        blobs = S.make_blobs(w)
        d["euls"] = np.stack([r.uniform(0, 360, w.nrefs), np.degrees(np.arccos(r.uniform(-1, 1, w.nrefs))),
                              r.uniform(0, 360, w.nrefs)], -1).astype(np.float32)
        x, y = _grid(case)
        loc = (x[..., None] * _euler(d["euls"])[:, None, None, 0] + y[..., None] * _euler(d["euls"])[:, None, None, 1]) / w.box
        d["even"] = S._blob_ft(blobs, loc[..., 0], loc[..., 1], loc[..., 2], DEV, torch.float64).to(torch.complex64)
        f = torch.fft.fftfreq(w.box, device=DEV)
        m, k, h = torch.meshgrid(f, f, f[: w.box // 2 + 1].abs(), indexing="ij")
        vol = S._blob_ft(blobs, h, k, m, DEV, torch.float32)
        noise = torch.randn(vol.shape, generator=g, device=DEV, dtype=torch.complex64) * vol.abs().mean()
        d["volumes"] = [(vol + s * 0.1 * noise).cpu().numpy() for s in (1, -1)]
    else:
        refs, R = S.make_refs(w, device=DEV)
        d["even"] = refs
    even = d["even"]
    spread = even.abs().square().mean(-1, keepdim=True).sqrt()
    d["odd"] = even + 0.05 * spread * torch.randn(even.shape, generator=g, device=DEV, dtype=torch.complex64)
    d["ctf"] = {k: float(np.float32(getattr(w, k))) for k in ("smpd", "cs", "fraca")}      # the records are single precision
    d["ctf"]["dfx"], d["ctf"]["dfy"], d["ctf"]["ast"] = S.ctf_params(w, n)
    d["eo"] = r.integers(0, 2, n).astype(np.int32)
    truth = r.integers(0, w.nrefs, n)
    for i, (first, nref, slot, count) in enumerate(_groups(case)):
        truth[slot - 1:slot - 1 + count] = first - 1 + r.integers(0, nref, count)
    d["truth"], d["rot"] = truth, r.integers(0, N, n)
    half = max(0.5, 0.25 * (case["grid"] - 1)) if case["grid"] else 0.5
    d["shift"] = r.uniform(-half, half, (n, 2)).astype(np.float32)
    shells = torch.arange(w.kfrom, w.kto + 1, device=DEV, dtype=torch.float32)
    if case["kind"] in ("step", "groups"):      # Cartesian half-plane transforms, to be gridded
        parts = S.make_particles(w, R, device=DEV, chunk=1024, noise=False)
        c = parts.cmat
        d["ctf"].update(dfx=parts.dfx, dfy=parts.dfy, ast=parts.angast)
        for i in range(0, n, 2048):
            v = c[i:i + 2048]
            level = (10.0 * v.abs().square().mean((1, 2), keepdim=True)).sqrt()
            v += level * torch.randn(v.shape, generator=g, device=DEV, dtype=torch.complex64)
        d["cmats"] = c
    else:
        ptcls = torch.empty((n, K, P), dtype=torch.complex64, device=DEV)
        for i in range(0, n, 1024):
            sl = slice(i, min(n, i + 1024))
            at = (torch.arange(P, device=DEV) - torch.as_tensor(d["rot"][sl], device=DEV)[:, None]) % N
            src = _ext(even[torch.as_tensor(truth[sl], device=DEV)])
            v = torch.gather(src, 2, at[:, None].expand(-1, K, -1)).to(torch.complex128)
            v = v * _phase(case, d["shift"][sl]) * _abs_ctf(case, d["ctf"], sel=sl)[0]
            power = (v.abs().square().mean(-1) * shells).sum(-1) * 2 * math.pi / case["box"] ** 2   # mean over the plane
            noise = torch.randn(v.shape, generator=g, device=DEV, dtype=torch.complex64)
            ptcls[sl] = (v + (10.0 * power).sqrt()[:, None, None] * noise).to(torch.complex64)
        d["ptcls"] = ptcls
        if case["euclid"]:
            level = ptcls.abs().square().mean((1, 2)).cpu().numpy()[:, None]
            d["sigma2"] = (level * r.uniform(0.5, 2.0, (n, K))).astype(np.float32)
    m = case["pairs"] or 1
    d["iref"], d["iptcl"] = r.integers(1, w.nrefs + 1, m).astype(np.int32), r.integers(1, n + 1, m).astype(np.int32)
    if case["kind"] == "grad":      # every particle against its own reference near its pose
        d["iptcl"] = (np.arange(m) % n + 1).astype(np.int32)
        d["iref"] = (truth[d["iptcl"] - 1] + 1).astype(np.int32)
        d["irot"] = ((d["rot"][d["iptcl"] - 1] + np.arange(m) // n - 5) % N + 1).astype(np.int32)
        d["ddf"] = r.uniform(-0.1, 0.1, m)
    d["pair_shift"] = r.uniform(-2, 2, (m, 2)).astype(np.float32)
    return d


def _groups(case):
    """(first reference, references, first slot, slots) of each group, counted from 1"""
    out, ref, slot = [], 1, 1
    for part in case["groups"].split():
        a, b = (int(v) for v in part.split("x"))
        out.append((ref, a, slot, b))
        ref, slot = ref + a, slot + b
    return out


def prepare(case, seed):
    pkg, d = _package(), _inputs(case, seed)
    w, p = d["w"], d["ctf"]
    pc = pkg.polarft_corrcalc()
    pc.new(w.nrefs, (1, w.nptcls), box=w.box, nrots=w.nrots, kfromto=(w.kfrom, w.kto), ctf=True,
           ctf_frame=case["frame"], eoarr=d["eo"])
    ctfp = pkg.ctfparams_array(w.nptcls, smpd=w.smpd, kv=w.kv, cs=w.cs, fraca=w.fraca, dfx=p["dfx"], dfy=p["dfy"],
                               angast=p["ast"])
    s = {"case": case, "pc": pc, "ctfp": ctfp, "shifts": _shifts(case), "groups": _groups(case)}
    if case["kind"] == "project":
        s["volumes"], s["euls"] = d["volumes"], d["euls"]
    else:
        pc.set_refs(1, d["even"].cpu().numpy(), True)
        pc.set_refs(1, d["odd"].cpu().numpy(), False)
    if "cmats" in d:
        s["cmats"] = d["cmats"]
    else:
        pc.set_ptcls(0, d["ptcls"].cpu().numpy())
        pc.create_polar_absctfmats(ctfp)
    if case["euclid"]:
        pc.set_objfun(1)
        pc.assign_sigma2_noise(d["sigma2"])
    s.update(iref=d["iref"], iptcl=d["iptcl"], pair_shift=d["pair_shift"])
    if case["kind"] == "pairs":
        s["out"] = torch.empty((case["pairs"], w.nrots), dtype=torch.float32, device=DEV)
    if case["kind"] == "grad":
        s.update(irot=d["irot"], ddf=d["ddf"])
    torch.cuda.synchronize()      # the library works on its own stream
    return s


def run(s):
    case, pc, kind = s["case"], s["pc"], s["case"]["kind"]
    if kind == "gencorrs":
        return pc.gencorrs(int(s["iref"][0]), int(s["iptcl"][0]), s["pair_shift"][0])
    if kind == "pairs":
        pc.gencorrs_noalloc(s["iref"], s["iptcl"], s["pair_shift"], s["out"].data_ptr())
        return s["out"]
    if kind == "corr_all":
        return pc.corr_all(None)
    if kind == "grad":
        sx, sy = s["pair_shift"][:, 0], s["pair_shift"][:, 1]
        f, g = pc.grad_batch(s["iref"], s["iptcl"], s["irot"], sx, sy, s["ddf"])
        return {"f": f, "grad": g}
    if kind == "project":
        for vol, iseven in zip(s["volumes"], (True, False)):
            pc.set_volume_ft(vol)
            pc.fproject_polar(1, s["euls"], iseven=iseven)
    if kind in ("step", "groups"):
        pc.polarize_ptcls_dev(0, case["nptcls"], s["cmats"].data_ptr())
        pc.create_polar_absctfmats(s["ctfp"])
    if kind == "groups":
        b = pc.search_groups(s["groups"], s["shifts"], case["precision"], ntop=8)
    else:
        b = pc.search_best(s["shifts"], case["precision"], ntop=0 if case["precision"] == "exact" else 8)
    return {"iref": b["iref"].copy(), "irot": b["irot"].copy(), "ishift": b["ishift"].copy(), "corr": b["corr"].copy()}


def work(case):
    K, N = case["kto"] - case["kfrom"] + 1, case["nrots"]
    P, ns = N // 2, max(1, case["grid"] ** 2)
    pft, image = 8 * K * P, 8 * case["box"] * (case["box"] // 2 + 1)
    nr, n, m = case["nrefs"], case["nptcls"], max(1, case["pairs"])
    fft = 5 * N * math.log2(N)
    held = 2 * nr * pft + n * 1.5 * pft                      # both reference sets, particles and |CTF|
    if case["kind"] == "grad":
        return {"bytes": min(nr, m) * 2 * pft + min(n, m) * pft + m * (40 + 32), "flops": m * K * P * 60.0}
    if case["kind"] in ("gencorrs", "pairs"):      # one transform of the prepared reference and particle shells each
        return {"bytes": min(2 * nr, m) * pft + min(n, m) * 1.5 * pft + m * 4 * N,
                "flops": m * (K * (fft + 3 * P * 8) + fft / 2)}
    pairs = sum(a * b for _, a, _, b in _groups(case)) or nr * n
    spectra = (nr * ns + n) * K * fft / 2
    flops = spectra + pairs * ns * (8.0 * K * (P + 1) + fft / 2)      # the contraction over the shells, one transform a triple
    if case["kind"] == "corr_all":
        return {"bytes": held + 4 * pairs * ns * N, "flops": flops}
    extra = {"step": n * image, "groups": n * image, "project": 2 * 8 * case["box"] ** 2 * (case["box"] // 2 + 1)}
    return {"bytes": held + extra.get(case["kind"], 0) + 16 * n, "flops": flops}


def tolerance(case):
    """Measured against ``exact`` (the largest of the listed and drawn cases' errors, times about four)."""
    if case["kind"] == "grad":      # FP64 sums, cancelling in the gradients
        return {"rel": 1e-11, "max": 1e-8}
    if case["kind"] in ("gencorrs", "pairs", "corr_all"):      # FP32 operands, one rounding of each value
        return {"rel": 5e-7, "max": 4e-5}
    return {"rel": 5e-7, "max": 4e-5, "differ": 0.005}


# ---- the same outputs in 64 bits -----------------------------------------------------------
def _gridded(case, cmats):
    """polarize in 64 bits: the 3 x 3 Kaiser-Bessel window around the nearest pixel, its weights normalised"""
    x, y = _grid(case)
    box = case["box"]

    def window(v):
        w0 = torch.sign(v) * torch.floor(v.abs() + 0.5) - 1
        at = w0[..., None] + torch.arange(3, device=DEV)
        return at.long(), torch.special.i0(7.4 * (1 - (2 / 3 * (at - v[..., None])) ** 2).clamp(min=0).sqrt())

    hx, wx = window(x)
    ky, wy = window(y)
    h, k = torch.broadcast_tensors(hx[..., None, :], ky[..., :, None])
    wt = wx[..., None, :] * wy[..., :, None]
    wt = wt / wt.sum((-1, -2), keepdim=True)
    conj = h < 0
    at = torch.where(conj, -k, k) % box * (box // 2 + 1) + h.abs()
    out = torch.empty((cmats.shape[0],) + x.shape, dtype=torch.complex128, device=DEV)
    for i in range(0, cmats.shape[0], 64):
        v = cmats[i:i + 64].reshape(-1, box * (box // 2 + 1))[:, at.reshape(-1)].reshape((-1,) + at.shape).to(torch.complex128)
        out[i:i + 64] = (torch.where(conj, v.conj(), v) * wt).sum((-1, -2))
    return out


def _projected(case, vol, euls):
    """fproject_polar in 64 bits: the 3 x 3 x 3 window of the volume's transform, normalised"""
    x, y = _grid(case)
    box, v = case["box"], torch.as_tensor(vol, device=DEV).to(torch.complex128)
    R, out = _euler(euls), []
    for i in range(0, len(euls), 16):
        loc = x[..., None] * R[i:i + 16, None, None, 0] + y[..., None] * R[i:i + 16, None, None, 1]
        w0 = torch.sign(loc) * torch.floor(loc.abs() + 0.5) - 1
        at = w0[..., None] + torch.arange(3, device=DEV)
        wt = torch.special.i0(7.4 * (1 - (2 / 3 * (at - loc[..., None])) ** 2).clamp(min=0).sqrt())
        at = at.long()
        h, k, m = torch.broadcast_tensors(at[..., 0, None, None, :], at[..., 1, None, :, None], at[..., 2, :, None, None])
        w = wt[..., 0, None, None, :] * wt[..., 1, None, :, None] * wt[..., 2, :, None, None]
        neg = h < 0
        val = v[torch.where(neg, -m, m) % box, torch.where(neg, -k, k) % box, h.abs()]
        val = torch.where(neg, val.conj(), val)
        out.append((val * w).sum((-1, -2, -3)) / w.sum((-1, -2, -3)))
    return torch.cat(out)


def _spectra(a):
    return torch.fft.fft(_ext(a), dim=-1)[..., : a.shape[-1] + 1]


def _pair_corrs(case, refs, ptcls, ctf, phase):
    """every rotation's correlation in the reference frame, pair by pair, (m, N)"""
    a = refs * ctf * (1.0 if phase is None else phase)
    c = torch.fft.irfft((_spectra(a).conj() * _spectra(ptcls)).sum(-2), n=case["nrots"], dim=-1) / 2
    return c / torch.sqrt(a.abs().square().sum((-1, -2)) * ptcls.abs().square().sum((-1, -2)))[:, None]


def _pxls(case):
    k = np.arange(1, case["kto"] + 1)
    sh = np.floor(np.hypot(k[:, None], k[None]) + 0.5)
    return np.array([(sh == s).sum() for s in range(case["kfrom"], case["kto"] + 1)], np.float64)


def _search64(case, d, refs, ptcls, cols, out):
    """the best correlation of the particles `cols` over the references (set, shift, rotation) in 64 bits"""
    N, P = case["nrots"], case["nrots"] // 2
    sh = _shifts(case)
    ns = 1 if sh is None else len(sh)
    phase = None if sh is None else _phase(case, sh)
    wk = None
    if case["euclid"]:
        wk = torch.as_tensor(_pxls(case) / P / d["sigma2"][cols].astype(np.float64), device=DEV)
    UA = torch.cat([_spectra(r[None] if phase is None else r[None] * phase) for r in refs.to(torch.complex128)])   # (rows, K, M)
    UA = UA.permute(2, 0, 1).contiguous()
    RU = torch.fft.rfft(refs.to(torch.complex128).abs().square(), dim=-1)          # (refs, K, J)
    step = max(1, int(3e8 / (len(UA[0]) * N)))
    for i in range(0, len(cols), step):
        c = cols[i:i + step]
        q = ptcls[c].to(torch.complex128)
        ctf = _abs_ctf(case, d["ctf"], sel=c)[0]
        B, C = _spectra(q * ctf), torch.fft.rfft(ctf.square(), dim=-1)
        energy = q.abs().square().sum(-1)
        if wk is not None:
            B, C, energy = B * wk[i:i + step, :, None], C * wk[i:i + step, :, None], energy * wk[i:i + step]
        energy = energy.sum(-1)
        X = torch.matmul(UA.conj(), B.permute(2, 1, 0))                              # (M, rows, cols)
        cc = torch.fft.irfft(X, n=N, dim=0).reshape(N, -1, ns, len(c)) / 2
        D = torch.fft.irfft(torch.einsum("rkj,ckj->jrc", RU.conj(), C), n=P, dim=0)
        D = torch.cat([D, D])[:, :, None]
        cc = cc - (D + energy) / 2 if wk is not None else cc / torch.sqrt(D * energy)
        if case["frame"] == "ptcl":
            out[c] = cc.amax((0, 1, 2))
            continue
        top = cc.amax(0).reshape(-1, len(c)).topk(8, 0).indices                       # the candidates, then their own frame
        best = torch.full((len(c),), -2.0, dtype=torch.float64, device=DEV)
        for t in top:
            ph = None if phase is None else phase[t % ns]
            best = torch.maximum(best, _pair_corrs(case, refs[t // ns].to(torch.complex128), q, ctf, ph).amax(-1))
        out[c] = best


def exact(case, seed):
    K, P, kind = case["kto"] - case["kfrom"] + 1, case["nrots"] // 2, case["kind"]
    triples = case["nrefs"] * case["nptcls"] * max(1, case["grid"] ** 2)
    if kind == "step" or (kind in ("search", "groups", "project") and triples * K * P > 8e10):
        return None
    d = _inputs(case, seed)
    sets = [d["even"], d["odd"]]
    if kind in ("gencorrs", "pairs", "corr_all") or (kind == "search" and case["precision"] == "exact" and case["frame"] == "ref"):
        listed_pairs = kind in ("gencorrs", "pairs")
        ir = d["iref"] - 1 if listed_pairs else np.tile(np.arange(case["nrefs"]), case["nptcls"])
        ip = d["iptcl"] - 1 if listed_pairs else np.repeat(np.arange(case["nptcls"]), case["nrefs"])
        sh = d["pair_shift"] if listed_pairs else None
        grid = _shifts(case)
        got = []
        for i in range(0, len(ir), 1000):
            a, p = ir[i:i + 1000], ip[i:i + 1000]
            both = torch.stack(sets)[torch.as_tensor(d["eo"][p], device=DEV).long(), torch.as_tensor(a, device=DEV)]
            both, q, ctf = both.to(torch.complex128), d["ptcls"][p].to(torch.complex128), _abs_ctf(case, d["ctf"], sel=p)[0]
            if grid is not None:
                got.append(torch.stack([_pair_corrs(case, both, q, ctf, _phase(case, g[None])).amax(-1) for g in grid]).amax(0))
            else:
                c = _pair_corrs(case, both, q, ctf, None if sh is None else _phase(case, sh[i:i + 1000]))
                got.append(c.cpu() if kind != "search" else c.amax(-1))
        got = torch.cat(got)
        if kind == "gencorrs":
            return got[0]
        if kind == "pairs":
            return got
        if kind == "corr_all":
            return got.reshape(case["nptcls"], case["nrefs"], 1, case["nrots"])
        return {"iref": None, "irot": None, "ishift": None, "corr": got.reshape(case["nptcls"], -1).amax(-1)}
    if kind == "grad":
        x, y = _grid(case)
        A = math.pi / (case["box"] // 2)
        wt = torch.arange(case["kfrom"], case["kto"] + 1, device=DEV, dtype=torch.float64)[:, None]
        fs, gs = [], []
        for i in range(0, case["pairs"], 1000):
            p = d["iptcl"][i:i + 1000] - 1
            r = torch.stack(sets)[torch.as_tensor(d["eo"][p], device=DEV).long(), torch.as_tensor(d["iref"][i:i + 1000] - 1, device=DEV).long()]
            ctf, dctf = _abs_ctf(case, d["ctf"], torch.as_tensor(d["ddf"][i:i + 1000], device=DEV)[:, None, None], p)
            ph = _phase(case, d["pair_shift"][i:i + 1000])
            at = (torch.arange(P, device=DEV) + torch.as_tensor(d["irot"][i:i + 1000] - 1, device=DEV)[:, None]) % (2 * P)
            q = torch.gather(_ext(d["ptcls"][p].to(torch.complex128)), 2, at[:, None].expand(-1, K, -1))
            a, b = r * ph * ctf, r * ph * dctf

            def dot(u, v):
                return (wt * (u * v.conj()).real).sum((-1, -2))

            sa = dot(a, a)
            den = torch.sqrt(sa * dot(q, q))
            f = dot(a, q) / den
            fs.append(f)
            gs.append(torch.stack([dot(1j * A * x * a, q) / den, dot(1j * A * y * a, q) / den,
                                   dot(b, q) / den - f * dot(a, b) / sa], -1))
        return {"f": torch.cat(fs), "grad": torch.cat(gs)}
    ptcls = _gridded(case, d["cmats"]) if "cmats" in d else d["ptcls"]
    if kind == "project":
        sets = [_projected(case, v, d["euls"]) for v in d["volumes"]]
    out = torch.zeros(case["nptcls"], dtype=torch.float64, device=DEV)
    for first, nref, slot, count in _groups(case) or [(1, case["nrefs"], 1, case["nptcls"])]:
        for eo in (0, 1):
            cols = np.flatnonzero(d["eo"][slot - 1:slot - 1 + count] == eo) + slot - 1
            if len(cols):
                _search64(case, d, sets[eo][first - 1:first - 1 + nref], ptcls, cols, out)
    return {"iref": None, "irot": None, "ishift": None, "corr": out}
