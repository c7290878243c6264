"""FDK backprojection on detectors whose rows TMA cannot address (and 16-bit rows on such detectors): the
re-pitched staged path gives the direct-load kernel's volume bit for bit (the same float operations on
the same samples), for whole volumes, slice ranges and continued sums."""
import numpy as np
import pytest
import torch

import oracle as O
from imagingsuite_b200 import modules as M

pytestmark = pytest.mark.gpu


def _fdk(nu, nv, precision):
    cfg = M.ReconConfig()
    pi = cfg.ProjectionInfo
    pi.roi = pi.projection_roi = (0, 0, nu, nv)
    pi.fSOD, pi.fSDD, pi.fResolution = 300.0, 600.0, (0.2, 0.2)
    cfg.MatrixInfo.fVoxelSize = (0.1, 0.1, 0.1)
    pi.fpPoint, pi.fCenter = ((nu - 1) / 2 + 0.13, (nv - 1) / 2 - 0.21), (nu - 1) / 2 + 0.07
    f = M.FDKbp_single()
    f.Configure(cfg, {"ProjectionBufferSize": "16", "SliceBlock": "32", "SubVolume": "1 1", "precision": precision})
    f.SetROI((0, 0, nu, nv))
    return f


@pytest.mark.parametrize("nu,nv", [(65, 33), (66, 32), (67, 64), (97, 31), (100, 47), (130, 40)])
@pytest.mark.parametrize("precision", ["fp32", "bf16", "fp16"])
def test_widths_equal_direct_loads(cuda, nu, nv, precision):
    g = torch.Generator(device=cuda).manual_seed(nu)
    nproj = 29
    proj = torch.randn((nproj, nv, nu), device=cuda, generator=g)
    ang = (np.arange(nproj) * 360.0 / nproj).astype(np.float32)
    f = _fdk(nu, nv, precision)
    geo = f.prepare(ang, np.ones(nproj, np.float32), proj.device)
    assert nu % 8 == 0 or geo[8] is None and geo[7][0] > 0
    filt, scale = f.ramp_filter(proj, geo)
    vols = {}
    for staging in (True, False):
        f.staging = staging
        f.backproject(filt, scale, geo, accumulate=False)
        vols[staging, "whole"] = f.volume.clone()
        f.backproject(filt, scale, geo, accumulate=True)  # the sums continued
        f.backproject(filt, scale, geo, k_range=(5, min(nv, 38)), accumulate=True)
        vols[staging, "more"] = f.volume.clone()
    for k in ("whole", "more"):
        assert torch.equal(vols[True, k], vols[False, k])


@pytest.mark.parametrize("nu", [66, 99])
def test_odd_width_equals_oracle(cuda, nu):
    rng = np.random.default_rng(nu)
    nproj, nv = 24, 36
    filt = rng.standard_normal((nproj, nv, nu)).astype(np.float32)
    ang = (np.arange(nproj) * 15.0).astype(np.float32)
    f = _fdk(nu, nv, "fp32")
    geo = f.prepare(ang, np.ones(nproj, np.float32), torch.device("cuda", 0))
    f.backproject(torch.from_numpy(filt).to(cuda), None, geo, accumulate=False)
    pi, mi = f.mConfig.ProjectionInfo, f.mConfig.MatrixInfo
    og = O.fdk_geom(pi.fSOD, pi.fSDD, pi.fpPoint, pi.fCenter, pi.fResolution, mi.fVoxelSize, pi.eDirection, False, 0.0, 0.0)
    assert np.array_equal(f.volume.cpu().numpy(), O.fdk_bp(filt, ang, og))
