"""Timed cases of the reconstruction path through its public entry points.

Four kinds of work, each called as a user's program calls it:

* ``chain``: a block of a parallel-beam scan, uint16 counts on the device to the reconstructed
  volume (pipeline.ParallelChain.run_device: FullLogNorm, optional spot and ring cleaning,
  ProjectionFilterSingle, MultiProjectionBPparallel);
* ``fdk``: a cone-beam scan, uint16 counts to the volume (pipeline.FdkPipeline.run_device), with
  FP32, BF16 or FP16 filtered projections, optionally with the uint16 slices that are written out;
* ``clean``: one projection cleaner on a block (FullLogNorm of the counts into the block, then the
  cleaner in place), as ReconEngine runs a configured preprocessing module;
* ``pair``: one gradient of a differentiable reconstruction (joseph.project with the projector
  pair matched to the backprojector): projections, and gradients in the volume, the centre of
  rotation and the tilt.

``exact`` evaluates the chains without cleaners, the cone-beam scans and the projector pair in
64 bits with plain torch. The cleaners have no such value here: their results are selected or
replaced pixels and a wavelet band filter with the reference's own border rules.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from imagingsuite_b200 import joseph as J
from imagingsuite_b200 import modules as M
from imagingsuite_b200 import phantom, pipeline

DEV = "cuda"
I0 = 3.0e4
NFLAT = NDARK = 5
GRAY = (0.0, 1.0e-2)  # gray interval of the stored slices


def listed():
    return [
        # a few slices of a small detector: the preview a user repeats while looking for the
        # centre of rotation (launches and host time count)
        chain("preview", 180, 8, 128),
        # the benchmark's C1 block: 360 projections of 256 x 64
        chain("parallel_c1", 360, 64, 256),
        # an ordinary scan on an odd detector, dose correction from an open-beam region, tilted
        # axis of rotation
        chain("parallel_tilt", 625, 60, 1001, tilt=0.3, dose=True),
        # slices of the production scan (2048 columns, 1125 projections) with spots and ring
        # artefacts, both cleaners on
        chain("production", 1125, 64, 2048, spot="both", ring="daub15"),
        # the benchmark's C2 cone-beam scan in FP32, with the uint16 slices that are stored
        fdk("fdk_c2", 720, 512, 512, u16=True),
        # a wide cone-beam scan with 16-bit filtered projections
        fdk("fdk_bf16", 600, 512, 768, precision="bf16"),
        # a quick cone-beam scan on a cropped, odd-sized detector
        fdk("fdk_odd", 200, 203, 301),
        # spot cleaning as the module is configured by default: peaks, 4 neighbours
        clean("spot_peaks", 64, 700, 1000, "spot", mode="peaks"),
        # wavelet ring cleaning alone, ragged sinograms, a shorter wavelet and one level more
        clean("ring_wavelet", 401, 50, 750, "ring", wname="daub5", decnum=3),
        # the median-based ring cleaner
        clean("ring_medianmix", 180, 500, 750, "medianmix"),
        # the alternative spot cleaner with its default ring detection
        clean("spot2_ring", 180, 500, 750, "spot2"),
        # one gradient step of the reconstruction with centre and tilt as unknowns
        pair("gradient", 256, 64, 180, tilt=0.4),
    ]


def chain(name, nproj, nv, nu, spot="", ring="", tilt=0.0, dose=False):
    return {"name": name, "kind": "chain", "nproj": nproj, "nv": nv, "nu": nu, "spot": spot, "ring": ring,
            "tilt": tilt, "dose": dose}


def fdk(name, nproj, nv, nu, precision="fp32", u16=False):
    return {"name": name, "kind": "fdk", "nproj": nproj, "nv": nv, "nu": nu, "precision": precision, "u16": u16}


def clean(name, nproj, nv, nu, module, mode="", wname="", decnum=0):
    return {"name": name, "kind": "clean", "nproj": nproj, "nv": nv, "nu": nu, "module": module, "mode": mode,
            "wname": wname, "decnum": decnum}


def pair(name, n, nz, nproj, tilt=0.0):
    return {"name": name, "kind": "pair", "n": n, "nz": nz, "nproj": nproj, "tilt": tilt}


# --------------------------------------------------------------------------------- drawn cases

MOST_CHAIN = 2.4e11   # voxel updates of a drawn chain (the production case has 2.8e11)
MOST_FDK = 9.0e10     # voxel updates of a drawn cone-beam scan (the 512^3 case has 9.7e10)
MOST_PIXELS = 6.0e7   # pixels of a block that is cleaned
MOST_PAIR = 7.0e8     # voxel updates of a gradient


def _between(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("chain", "chain", "fdk", "fdk", "clean", "clean", "pair"))
    if kind == "chain":
        nproj, nv, nu = _between(rng, 120, 1200), _between(rng, 8, 128), _between(rng, 96, 2048)
        clean_it = rng.random() < 0.4
        while nproj * nv * float(nu) * nu > MOST_CHAIN:
            nv = max(8, nv // 2)
            nproj = max(120, nproj * 3 // 4)
        c = chain("", nproj, nv, nu, spot=rng.choice(("holes", "peaks", "both")) if clean_it else "",
                  ring=rng.choice(("daub5", "daub10", "daub15")) if clean_it else "",
                  tilt=rng.choice((0.0, 0.0, round(rng.uniform(-0.6, 0.6), 2))), dose=rng.random() < 0.5)
    elif kind == "fdk":
        nproj, nv, nu = _between(rng, 90, 1000), _between(rng, 48, 768), _between(rng, 64, 1024)
        while nproj * nv * float(nu) * nu > MOST_FDK:
            nproj, nv, nu = max(90, nproj * 3 // 4), max(48, nv * 3 // 4), max(64, nu * 7 // 8)
        c = fdk("", nproj, nv, nu, precision=rng.choice(("fp32", "fp32", "bf16", "fp16")), u16=rng.random() < 0.5)
    elif kind == "clean":
        module = rng.choice(("spot", "ring", "medianmix", "spot2"))
        nproj, nv, nu = _between(rng, 140, 800), _between(rng, 16, 512), _between(rng, 160, 2048)
        while nproj * nv * float(nu) > MOST_PIXELS:
            nproj, nv = max(140, nproj * 3 // 4), max(16, nv * 3 // 4)
        c = clean("", nproj, nv, nu, module, mode=rng.choice(("holes", "peaks", "both")) if module == "spot" else "",
                  wname=rng.choice(("daub5", "daub10", "daub15")) if module == "ring" else "",
                  decnum=rng.choice((1, 2, 3)) if module == "ring" else 0)
    else:
        n, nz, nproj = _between(rng, 64, 512), 4 * _between(rng, 2, 32), _between(rng, 60, 360)
        while nproj * nz * float(n) * n > MOST_PAIR:
            nproj, nz = max(60, nproj * 3 // 4), max(8, nz // 8 * 4)
            n = max(64, n * 7 // 8)
        c = pair("", n, nz, nproj, tilt=rng.choice((0.0, round(rng.uniform(-0.6, 0.6), 2))))
    del c["name"]
    return c


# -------------------------------------------------------------------------------------- inputs


def _weights(nproj, arc):
    return np.full(nproj, np.float32(math.radians(arc) / nproj))


def _counts(integrals, seed, defects):
    """uint16 projections, flats and darks (Poisson counts plus a dark level of 100 +- 3); with
    `defects`, 0.05 % white or tripled pixels and 1 % of the columns with a gain error in the
    projections only."""
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    shape = integrals.shape[1:]

    def u16(t):
        return torch.clamp(torch.round(t), 0, 65535).to(torch.int32).to(torch.uint16)

    def dark(n):
        return torch.randn((n, *shape), generator=g, device=DEV) * 3.0 + 100.0

    darks = dark(NDARK)
    flats = torch.poisson(torch.full((NFLAT, *shape), I0, device=DEV), generator=g) + dark(NFLAT)
    proj = torch.poisson(I0 * torch.exp(-integrals), generator=g)
    proj += dark(integrals.shape[0])
    if defects:
        cols = torch.randperm(shape[1], generator=g, device=DEV)[:max(1, shape[1] // 100)]
        proj[:, :, cols] *= 1.005 + 0.025 * torch.rand(cols.numel(), generator=g, device=DEV)
        n = max(1, proj.numel() // 4000)
        at = torch.randint(proj.numel(), (2, n), generator=g, device=DEV)
        flat = proj.view(-1)
        flat[at[0]] = 65535.0
        flat[at[1]] *= 3.0
    return u16(proj), u16(flats), u16(darks)


def _config(case):
    nu, nv, nproj = case["nu"], case["nv"], case["nproj"]
    cfg = M.ReconConfig()
    pi = cfg.ProjectionInfo
    pi.roi = pi.projection_roi = (0, 0, nu, nv)
    pi.nDims = (nu, nv, nproj)
    pi.nOBCount, pi.nDCCount = NFLAT, NDARK
    if case["kind"] == "fdk":
        # the detector's field of view in voxels of the reconstruction: magnification 2, piercing
        # point and centre off the pixel grid as on a real scanner
        pi.fSOD, pi.fSDD, pi.fResolution = 300.0, 600.0, (0.2, 0.2)
        cfg.MatrixInfo.fVoxelSize = (0.1, 0.1, 0.1)
        pi.fpPoint = ((nu - 1) / 2 + 0.13, (nv - 1) / 2 - 0.21)
        pi.fCenter = (nu - 1) / 2 + 0.07
    else:
        pi.fCenter = (nu - 1) / 2
        if case.get("dose"):
            pi.dose_roi = (2, 1, 2 + max(4, nu // 16), nv - 1)
        if case.get("tilt"):
            pi.bCorrectTilt, pi.fTiltAngle, pi.fTiltPivotPosition = True, case["tilt"], (nv - 1) / 2
    return cfg


def _norm(cfg, case, darks, flats):
    norm = M.FullLogNorm()
    norm.Configure(cfg, {"usenormregion": "true" if case.get("dose") else "false", "uselut": "false",
                         "referenceaverage": "ImageAverage"})
    norm.SetReferenceImages(darks, flats)
    return norm


def _spot(cfg, mode):
    m = M.MorphSpotCleanModule()
    m.Configure(cfg, {"connectivity": "conn4" if mode == "peaks" else "conn8", "cleanmethod": "morphcleanreplace",
                      "detectionmethod": "morphdetect" + mode, "threshold": "0.1 0.1", "sigma": "0.01 0.01",
                      "edgesmooth": "5", "maxarea": "30", "removeinfnan": "false", "clampdata": "false",
                      "minlevel": "-0.1", "maxlevel": "12", "threading": "false"})
    return m


def _ring(cfg, wname, decnum=2):
    m = M.WaveletRingClean()
    m.Configure(cfg, {"wname": wname, "sigma": "0.05", "decnum": str(decnum), "parallel": "false",
                      "method": "verticalfft"})
    return m


def _cleaner(cfg, case):
    if case["module"] == "spot":
        return _spot(cfg, case["mode"])
    if case["module"] == "ring":
        return _ring(cfg, case["wname"], case["decnum"])
    if case["module"] == "medianmix":
        m = M.MedianMixRingClean()
        m.Configure(cfg, {"threshold": "0.025", "width": "0.0025"})
        return m
    m = M.SpotClean2()
    m.Configure(cfg, {"gamma": "0.1", "sigma": "0.001", "iterations": "1", "maxlevel": "5", "minlevel": "-0.1",
                      "maxarea": "20", "detectionmethod": "ring"})
    return m


def _parallel_inputs(case, seed):
    ells = phantom.ellipsoids(seed, 5)
    nproj, nv, nu = case["nproj"], case["nv"], case["nu"]
    line = phantom.parallel_integrals_torch(ells, nproj, nu, nv, DEV, v0=(nu - nv) // 2, chunk=32)
    defects = case["kind"] == "clean" or bool(case["spot"] or case["ring"])
    return _counts(line, seed, defects)


def _fdk_inputs(case, seed):
    nproj, nv, nu = case["nproj"], case["nv"], case["nu"]
    ells = phantom.ellipsoids(seed, 5)
    line = phantom.cone_integrals_torch(ells, nproj, nu, nv, 300.0, 600.0, 0.2, 0.1 * nu, DEV, chunk=16)
    return _counts(line, seed, False)


def _pair_inputs(case, seed):
    n, nz = case["n"], case["nz"]
    truth = phantom.voxelize_torch(phantom.ellipsoids(seed, 5), n, nz, DEV, fov_margin=4)
    truth = truth.permute(1, 2, 0).contiguous()
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    vol = truth * 0.8 + 0.02 / n * torch.randn(truth.shape, generator=g, device=DEV)
    # measured projections with a residual slope of the beam profile, in both directions
    slope = torch.arange(n, device=DEV) / n * (0.5 + torch.arange(nz, device=DEV) / nz)[:, None]
    measured = slope + 0.1 * torch.randn((case["nproj"], nz, n), generator=g, device=DEV)
    return vol, measured


def _angles(case):
    arc = 360.0 if case["kind"] == "fdk" else 180.0
    return (np.arange(case["nproj"]) * arc / case["nproj"]).astype(np.float32), arc


def prepare(case, seed):
    s = {"case": case}
    angles, arc = _angles(case)
    if case["kind"] == "pair":
        s["vol"], s["measured"] = _pair_inputs(case, seed)
        s["op"] = J.MatchedOperator(case["n"], case["nz"], angles)
        s["centre"] = torch.tensor(case["n"] / 2 + 1.75, requires_grad=True)
        s["tilt"] = torch.tensor(float(case["tilt"]), requires_grad=True)
        s["vol"].requires_grad_(True)
        return s
    cfg = _config(case)
    weights = _weights(case["nproj"], arc)
    if case["kind"] == "fdk":
        counts, flats, darks = _fdk_inputs(case, seed)
        s["pipe"] = pipeline.FdkPipeline(cfg, angles, weights, darks, flats, precision=case["precision"])
        s["counts"] = counts
        return s
    counts, flats, darks = _parallel_inputs(case, seed)
    s["counts"] = counts
    norm = _norm(cfg, case, darks, flats)
    if case["kind"] == "clean":
        s["norm"], s["module"] = norm, _cleaner(cfg, case)
        s["block"] = torch.empty(counts.shape, dtype=torch.float32, device=DEV)
        return s
    filt = M.ProjectionFilterSingle()
    filt.Configure(cfg, {"filtertype": "hanning", "cutoff": "0.5", "order": "1", "usebias": "true",
                         "biasweight": "0.1", "paddingdoubler": "2"})
    bp = M.MultiProjectionBPparallel()
    bp.Configure(cfg, {"ProjectionBufferSize": "16", "SliceBlock": "32", "SubVolume": "1 1", "precision": "fp32",
                       "referencecompat": "true"})
    bp.SetROI((0, 0, case["nu"], case["nv"]))
    s["chain"] = pipeline.ParallelChain(norm, filt, bp, angles, weights,
                                        spot=_spot(cfg, case["spot"]) if case["spot"] else None,
                                        ring=_ring(cfg, case["ring"]) if case["ring"] else None)
    return s


def run(s):
    case = s["case"]
    if case["kind"] == "chain":
        return s["chain"].run_device(s["counts"])
    if case["kind"] == "fdk":
        vol = s["pipe"].run_device(s["counts"])
        if not case["u16"]:
            return vol
        slices = M.slices_u16(vol, "MatrixXYZ", GRAY)
        return {"volume": vol, "slices": slices.view(torch.int16)}
    if case["kind"] == "clean":
        block = s["norm"].ProcessCore(s["counts"], {}, out=s["block"])
        return s["module"].ProcessCore(block, {})
    proj = J.project(s["vol"], s["centre"], s["tilt"], s["op"])
    gvol, gcentre, gtilt = torch.autograd.grad(proj, (s["vol"], s["centre"], s["tilt"]), proj - s["measured"])
    return {"projections": proj, "volume": gvol, "centre": gcentre, "tilt": gtilt}


# ------------------------------------------------------------------------------------ the work


def _inside(n):
    return math.pi / 4 * n * n


def work(case):
    """Each input and output once; per voxel update inside the reconstructed circle a multiply and
    an add for every sample that enters it, and the row filter's transforms."""
    if case["kind"] == "pair":
        n, nz, nproj = case["n"], case["nz"], case["nproj"]
        vol, proj = n * n * nz, nproj * n * nz
        # projections: two samples per update, and two more for the derivative; gradient: two
        return {"bytes": 4.0 * (2 * vol + 3 * proj), "flops": 12.0 * _inside(n) * nz * nproj}
    nproj, nv, nu = case["nproj"], case["nv"], case["nu"]
    px = float(nproj) * nv * nu
    if case["kind"] == "clean":
        return {"bytes": 6.0 * px, "flops": 8.0 * px}
    length = 2.0 ** math.ceil(math.log2(2 * nu))
    fft = nproj * nv * 5.0 * length * math.log2(length)
    per = 2.0 if case["kind"] == "fdk" else 4.0
    used = nproj if case["kind"] == "fdk" else nproj - nproj // 16
    vol = float(nu) * nu * nv
    out = vol * (6.0 if case.get("u16") else 4.0)
    return {"bytes": 2.0 * px + out, "flops": fft + per * _inside(nu) * nv * used}


# ------------------------------------------------------------------- values in 64 bits (torch)


def _median_of_row_means(frames, roi):
    x0, y0, x1, y1 = roi
    means = frames[:, y0:y1, x0:x1].double().mean(dim=2).sort(dim=1).values
    h = means.shape[1]
    return means[:, h // 2] if h % 2 else 0.5 * (means[:, h // 2 - 1] + means[:, h // 2])


def _lognorm64(counts, flats, darks, roi, chunk=64):
    dark, flat = darks.double().mean(dim=0), flats.double().mean(dim=0)
    open_beam = flat - dark
    if roi is None:
        dose = torch.zeros(counts.shape[0], dtype=torch.float64, device=DEV)
    else:
        darkdose = _median_of_row_means(darks.float(), roi).mean()
        open_beam = open_beam / (_median_of_row_means(flats.float(), roi) - darkdose).mean()
        dose = torch.log(torch.clamp(_median_of_row_means(counts.float(), roi) - darkdose, min=1.0))
    logflat = torch.where(open_beam > 0, torch.log(open_beam), torch.zeros_like(open_beam))
    out = torch.empty(counts.shape, dtype=torch.float64, device=DEV)
    for a in range(0, counts.shape[0], chunk):
        v = counts[a:a + chunk].float().double() - dark
        out[a:a + chunk] = torch.where(v > 0, logflat - torch.log(v.clamp_min(1e-300)) + dose[a:a + chunk, None, None],
                                       torch.zeros_like(v))
    return out


def _hann64(proj, nu, cutoff=0.5, bias=0.1, doubler=2, chunk=8):
    """ProjectionFilterSingle with its sigmoid tapers (the right one shifted by 16 samples), Hann
    window and unfiltered Nyquist bin."""
    n = 2 ** (math.ceil(math.log2(nu)) + doubler)
    half, ins = n // 2, n // 2 - nu // 2
    k = torch.arange(half, dtype=torch.float64, device=DEV)
    cut = int(2 * cutoff * half)
    resp = k / (half - 1) * (0.5 + 0.5 * torch.cos(k / (cut - 1) * math.pi * cutoff))
    resp[cut:] = 0
    resp[0] = bias * resp[1]
    resp = torch.cat([resp, torch.ones(1, dtype=torch.float64, device=DEV)])
    x = torch.arange(ins, dtype=torch.float64, device=DEV) / ins - 0.5
    taper = 1 / (1 + torch.exp(-x / 0.07))
    out = torch.empty_like(proj)
    for a in range(0, proj.shape[0], chunk):
        p = proj[a:a + chunk]
        line = torch.zeros((*p.shape[:2], n + 16), dtype=torch.float64, device=DEV)
        line[..., ins:ins + nu] = p
        line[..., :ins] = p[..., :1] * taper
        line[..., n + 16 - ins:] = p[..., -1:] * taper.flip(0)
        spec = torch.fft.rfft(line[..., :n]) * resp
        out[a:a + chunk] = torch.fft.irfft(spec, n=n)[..., ins:ins + nu] * (n * math.pi / (4 * half))
    return out


def _circle(n, tilt=0.0, slices=0):
    """First and last column of each row (half-open on the left) of the reconstructed circle."""
    c = n // 2
    r = c - 1 - (math.floor(math.tan(math.radians(abs(tilt))) * slices) if tilt else 0)
    rows = []
    for i in range(n):
        left = r * r - (i - c) ** 2
        if left < 0:
            rows.append((0, 0))
        else:
            rows.append((math.ceil(c - math.sqrt(left)), min(n - 1, math.floor(c + math.sqrt(left)))))
    return torch.tensor(rows, device=DEV)


def _parallel64(case, seed):
    counts, flats, darks = _parallel_inputs(case, seed)
    cfg = _config(case)
    pi = cfg.ProjectionInfo
    nproj, nv, nu = case["nproj"], case["nv"], case["nu"]
    proj = _hann64(_lognorm64(counts, flats, darks, pi.dose_roi if case["dose"] else None), nu)
    angles, arc = _angles(case)
    proj *= float(np.float32(math.radians(arc) / nproj))
    mask = _circle(nu, case["tilt"], nv)
    one = torch.arange(1, nu + 1, device=DEV)
    x, y = one.double()[None, :], one.double()[:, None]
    inside = (one[None, :] > mask[:, :1]) & (one[None, :] <= mask[:, 1:])
    groups = nv // 4
    inc = 4 * math.tan(math.radians(case["tilt"]))
    off = -pi.fTiltPivotPosition * math.tan(math.radians(case["tilt"])) if case["tilt"] else 0.0
    shift = 2 * inc * torch.arange(groups, dtype=torch.float64, device=DEV).repeat_interleave(4)
    vol = torch.zeros((nu * nu, nv), dtype=torch.float64, device=DEV)
    part = vol[:, :4 * groups]
    for k in range(nproj):
        if k % 16 == 15:  # a full buffer of 16 is flushed without its last projection
            continue
        a = -math.radians(float(angles[k]))
        s, c = math.sin(a), math.cos(a)
        pos = (nu // 2) * (s - c) + pi.fCenter + c * y - off - s * x
        n = pos.trunc()
        ok = (inside & (n >= 0) & (n <= nu - 2)).reshape(-1, 1)
        frac, n = (pos - n).reshape(-1, 1), n.clamp(0, nu - 2).long().reshape(-1)
        wb = (frac - shift).abs() if case["tilt"] else frac.abs()
        p = proj[k, :4 * groups].t().contiguous()
        term = torch.addcmul(p[n] * (1 - wb), p[n + 1], wb)
        part += torch.where(ok, term, torch.zeros_like(term))
    return vol.view(nu, nu, nv)


def _ramp64(proj, nu, nv, chunk=8):
    """FDKbp_single's ramp filter: 5 edge rows replaced by the sixth, twice the padded width."""
    n = 2 * 2 ** math.ceil(math.log2(nu))
    k = torch.arange(n, dtype=torch.float64, device=DEV)
    ramp = torch.minimum(k, n - k) * (0.54 + 0.46 * (torch.cos(2 * math.pi * k / n) + 1)) / (n / 2)
    left = (n - nu) // 2
    out = torch.empty_like(proj)
    for a in range(0, proj.shape[0], chunk):
        p = proj[a:a + chunk].clone()
        p[:, :5] = p[:, 5:6]
        p[:, nv - 5:] = p[:, nv - 6:nv - 5]
        line = torch.zeros((*p.shape[:2], n), dtype=torch.float64, device=DEV)
        line[..., left:left + nu] = p
        out[a:a + chunk] = torch.fft.irfft(torch.fft.rfft(line) * ramp[:n // 2 + 1], n=n)[..., left:left + nu]
    return out


def _fdk64(case, seed):
    counts, flats, darks = _fdk_inputs(case, seed)
    cfg = _config(case)
    pi = cfg.ProjectionInfo
    nproj, nv, nu = case["nproj"], case["nv"], case["nu"]
    f = lambda v: float(np.float32(v))  # noqa: E731  (the configuration's values are 32-bit)
    sod, sdd, pix, vox = f(pi.fSOD), f(pi.fSDD), f(pi.fResolution[0]), f(cfg.MatrixInfo.fVoxelSize[0])
    pu, pv, centre = f(pi.fpPoint[0]), f(pi.fpPoint[1]), f(pi.fCenter)
    angles, arc = _angles(case)
    proj = _ramp64(_lognorm64(counts, flats, darks, None), nu, nv)
    proj *= f(math.radians(arc) / nproj) * (sod / sdd) ** 3
    # detector rows the geometry reaches: the image centre counts from the first of them
    radius = nu * vox / 2
    first = pv - (pv * vox * sdd / (sod - radius)) / pix
    first = 0 if first <= 0 else int(first) - 8
    ic = (pu, pv - first)
    o = (-(nu - centre) * vox - vox / 2, -(nu - centre) * vox - vox / 2, -(nv - pv) * vox - vox / 2)
    ax = torch.arange(nu, dtype=torch.float64, device=DEV) * vox
    x, y = (o[0] + ax)[None, :], (o[1] + ax)[:, None]
    z = (o[2] + torch.arange(nv, dtype=torch.float64, device=DEV) * vox)[:, None, None]
    mask = _circle(nu)
    col = torch.arange(nu, device=DEV)[None, :]
    inside = (col > mask[:, :1]) & (col <= mask[:, 1:])
    offcentre = (pu - centre) * vox
    vol = torch.zeros((nv, nu, nu), dtype=torch.float64, device=DEV)
    for k in range(nproj):
        a = -math.radians(float(angles[k]))
        ca, sa = math.cos(a), math.sin(a)
        # camera at sod (ca, sa, 0): depth along the axis, offset across it, height
        w = (-ca * x - sa * y + sod) / sdd
        u = (-sa * x + ca * y - offcentre) / pix
        c = torch.floor((u + ic[0] * w) / w + 0.5)
        ok2 = inside & (c >= 0) & (c < nu)
        r = torch.floor((ic[1] * w - z / pix) / w + 0.5)
        at = r.clamp(0, nv - 1).mul_(nu).add_(c.clamp(0, nu - 1)).long()
        val = proj[k].reshape(-1)[at]
        vol += torch.where(ok2 & (r >= 0) & (r < nv), val / (w * w), torch.zeros_like(val))
    vol = vol.flip(0, 2)
    return {"volume": vol, "slices": None} if case["u16"] else vol


def _pair64(case, seed):
    vol, measured = _pair_inputs(case, seed)
    n, nz, nproj = case["n"], case["nz"], case["nproj"]
    vol, measured = vol.double(), measured.double()
    angles, _ = _angles(case)
    mask = _circle(n)
    one = torch.arange(1, n + 1, device=DEV)
    inside = (one[None, :] > mask[:, :1]) & (one[None, :] <= mask[:, 1:])
    at = inside.nonzero()
    y, x = at[:, 0].double() + 1, at[:, 1].double() + 1
    zc = torch.arange(nz, dtype=torch.float64, device=DEV) - (nz - 1) / 2
    tilt = float(np.float32(case["tilt"]))
    centre = n / 2 + 1.75 + math.tan(math.radians(tilt)) * zc
    v = vol[at[:, 0], at[:, 1]]
    zi = torch.arange(nz, device=DEV)[None, :]
    proj = torch.zeros((nproj, nz * n), dtype=torch.float64, device=DEV)
    gvol, gcentre, gtilt = torch.zeros_like(v), 0.0, 0.0
    dtan = math.radians(1.0) / math.cos(math.radians(tilt)) ** 2
    for k in range(nproj):
        a = -math.radians(float(angles[k]))
        s, c = math.sin(a), math.cos(a)
        pos = ((n // 2) * (s - c) + c * y - s * x)[:, None] + centre
        m = pos.trunc()
        ok = (m >= 0) & (m <= n - 2)
        wb = (pos - m).abs()
        m = (m.clamp(0, n - 2).long() + zi * n).reshape(-1)
        zero = torch.zeros_like(v)
        va, vb, vv = (torch.where(ok, t, zero).reshape(-1) for t in (v * (1 - wb), v * wb, v))
        d = torch.zeros(nz * n, dtype=torch.float64, device=DEV)
        proj[k].index_add_(0, m, va).index_add_(0, m + 1, vb)
        d.index_add_(0, m, -vv).index_add_(0, m + 1, vv)
        g = proj[k] - measured[k].reshape(-1)
        gvol += torch.where(ok, g[m].view_as(v) * (1 - wb) + g[m + 1].view_as(v) * wb, zero)
        per = (d * g).view(nz, n).sum(1)
        gcentre, gtilt = gcentre + per.sum(), gtilt + (per * zc).sum() * dtan
    out = torch.zeros_like(vol)
    out[at[:, 0], at[:, 1]] = gvol
    return {"projections": proj.view(nproj, nz, n), "volume": out, "centre": gcentre.cpu(), "tilt": gtilt.cpu()}


def exact(case, seed):
    if case["kind"] == "chain":
        return None if case["spot"] or case["ring"] else _parallel64(case, seed)
    if case["kind"] == "fdk":
        return _fdk64(case, seed)
    return _pair64(case, seed) if case["kind"] == "pair" else None
