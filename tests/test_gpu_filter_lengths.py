"""Row filters at every transform length of their kernels and at the widths around its steps: against the
FP64 oracle within the FFT tolerance (1e-5 relative RMS, float transforms of up to 2^14 points), odd row
counts (a lone last row) and rows that do not depend on their neighbours' pairing partner's size."""
import numpy as np
import pytest
import torch

import oracle as O
from imagingsuite_b200 import modules as M

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return float(np.linalg.norm(a.astype(np.float64) - b) / np.linalg.norm(b))


@pytest.mark.parametrize("nu", [2, 31, 64, 65, 128, 129, 256, 257, 511, 513, 1024, 1025, 2048, 2049, 4096])
@pytest.mark.parametrize("rows", [(1, 1), (3, 5)])
def test_projection_filter(cuda, nu, rows):
    rng = np.random.default_rng(nu)
    p = rng.standard_normal((*rows, nu)).astype(np.float32)
    cfg = M.ReconConfig()
    cfg.ProjectionInfo.roi = (0, 0, nu, rows[1])
    f = M.ProjectionFilterSingle()
    f.Configure(cfg, {"filtertype": "hanning", "cutoff": "0.5", "order": "1", "usebias": "true", "biasweight": "0.1",
                      "paddingdoubler": "2"})
    t = torch.from_numpy(p).to(cuda)
    w = torch.linspace(0.5, 1.5, rows[0], device=cuda)
    f.ProcessCore(t, {}, weights=w)
    exp = O.projfilter(p, O.projfilter_plan(nu)) * w.cpu().numpy()[:, None, None]
    assert _rel(t.cpu().numpy(), exp) < 1e-5


@pytest.mark.parametrize("nu", [12, 64, 65, 129, 257, 513, 1025, 2049, 4097, 8192])
def test_fdk_filter_and_its_scales(cuda, nu):
    """The FDK ramp filter, and the 16-bit form's scales from the largest |value| that the filter collects:
    they equal those of the filtered projections quantised apart."""
    rng = np.random.default_rng(nu)
    nproj, nv = 2, 13
    p = rng.standard_normal((nproj, nv, nu)).astype(np.float32)
    w = np.array([0.7, 1.3], np.float32)
    cfg = M.ReconConfig()
    pi = cfg.ProjectionInfo
    pi.fSOD, pi.fSDD, pi.fResolution = 300.0, 600.0, (0.2, 0.2)
    pi.fpPoint, pi.fCenter = ((nu - 1) / 2, (nv - 1) / 2), (nu - 1) / 2
    cfg.MatrixInfo.fVoxelSize = (0.1, 0.1, 0.1)
    og = O.fdk_geom(300.0, 600.0, pi.fpPoint, pi.fCenter, (0.2, 0.2), (0.1, 0.1, 0.1), 0, False, 0.0, 0.0)
    t = torch.from_numpy(p).to(cuda)
    res = {}
    for prec in ("fp32", "bf16", "fp16"):
        f = M.FDKbp_single()
        f.Configure(cfg, {"ProjectionBufferSize": "16", "SliceBlock": "32", "SubVolume": "1 1", "precision": prec})
        f.SizeU, f.SizeV = nu, nv
        g = (torch.from_numpy(w).to(cuda), None, None, None, np.float32(0.25), np.float32(0.5), 1, (0, 0), None)
        res[prec] = f.ramp_filter(t, g)
    exp = O.fdk_prepare(p, w, og)
    assert _rel(res["fp32"][0].cpu().numpy(), exp) < 1e-5
    for prec in ("bf16", "fp16"):
        bits, scale = M.quantize(res["fp32"][0], prec)
        assert torch.equal(scale, res[prec][1]) and torch.equal(bits.view(torch.int16), res[prec][0].view(torch.int16))


@pytest.mark.parametrize("nu", [12, 33, 99, 130, 301])
def test_scales_from_a_maximum_in_any_column(cuda, nu):
    """Each projection's largest |value| in another column, so in another lane of the kernel's warps: the
    scales equal those of the filtered projections quantised apart."""
    nv = 13
    g = torch.Generator(device=cuda).manual_seed(nu)
    p = 0.01 * torch.randn((nu, nv, nu), device=cuda, generator=g)
    c = torch.arange(nu, device=cuda)
    p[c, 6, c] = 10.0 * 1.37 ** (c % 17).float()
    geo = (torch.ones(nu, device=cuda), None, None, None, np.float32(0.25), np.float32(0.5), 1, (0, 0), None)
    res = {}
    for prec in ("fp32", "bf16", "fp16"):
        f = M.FDKbp_single()
        f.Configure(M.ReconConfig(), {"ProjectionBufferSize": "16", "SliceBlock": "32", "SubVolume": "1 1", "precision": prec})
        f.SizeU, f.SizeV = nu, nv
        res[prec] = f.ramp_filter(p, geo)
    for prec in ("bf16", "fp16"):
        bits, scale = M.quantize(res["fp32"][0], prec)
        assert torch.equal(scale, res[prec][1]) and torch.equal(bits.view(torch.int16), res[prec][0].view(torch.int16))
