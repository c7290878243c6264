"""FDK staging: the largest boxes that two CTAs' shared memory holds, and geometries whose source plane
passes through a tile."""
import ctypes

import numpy as np
import pytest
import torch

from imagingsuite_b200 import _lib as L
from imagingsuite_b200 import modules as M

pytestmark = pytest.mark.gpu


def _module(nu, nv, sod, sdd, res, vox):
    cfg = M.ReconConfig()
    pi = cfg.ProjectionInfo
    pi.fSOD, pi.fSDD, pi.fResolution = sod, sdd, (res, res)
    pi.fpPoint = ((nu - 1) / 2.0 + 0.13, (nv - 1) / 2.0 - 0.21)
    pi.fCenter = (nu - 1) / 2.0 + 0.07
    pi.nDims = (nu, nv, 0)
    cfg.MatrixInfo.fVoxelSize = (vox, vox, vox)
    m = M.FDKbp_single()
    m.Configure(cfg, {"ProjectionBufferSize": "16", "SliceBlock": "32", "SubVolume": "1 1"})
    m.SetROI((0, 0, nu, nv))
    return m


def _backproject(cuda, m, filt, ang, box):
    nproj, nv, nu = filt.shape
    xip, yip, zip_, *_, uni = m.partials(ang)
    X, Y, Z = (torch.from_numpy(a).to(cuda) for a in (xip, yip, zip_))
    vol = torch.full((nv, nu, nu), 7.0, device=cuda)
    L.check(L.lib().mr_fdk_backproject(filt.data_ptr(), L.MR_F32, None, nu, nv, nproj, X.data_ptr(), Y.data_ptr(),
                                       Z.data_ptr(), uni, m._mask.data_ptr(), *box, 0, vol.data_ptr(),
                                       torch.cuda.current_stream().cuda_stream))
    return vol


def _word():
    st = ctypes.c_int(-1)
    L.check(L.lib().mr_device_status(ctypes.byref(st)))
    return st.value


# up to 12544 bytes a box (batches of four projections), on widths whose geometry is copied 16 and 4
# bytes at a time
@pytest.mark.parametrize("nu,nv", [(96, 64), (98, 35)])
@pytest.mark.parametrize("box", [(40, 33), (40, 41), (48, 64), (56, 54), (56, 55), (56, 56)])
def test_box_is_staged(cuda, nu, nv, box):
    rng = np.random.default_rng(box[1])
    filt = torch.from_numpy(rng.standard_normal((21, nv, nu)).astype(np.float32)).to(cuda)
    ang = (np.arange(21) * 17.0).astype(np.float32)
    m = _module(nu, nv, 300.0, 600.0, 0.2, 0.12)
    assert _word() == 0
    L.check(L.lib().mr_set_wait_limit(0))  # only the staged kernel waits
    try:
        _backproject(cuda, m, filt, ang, box)
        assert _word() == 1
    finally:
        L.check(L.lib().mr_set_wait_limit(-1))
    got, direct = _backproject(cuda, m, filt, ang, box), _backproject(cuda, m, filt, ang, (0, 0))
    assert _word() == 0
    assert torch.equal(got, direct)


# the source inside the volume, detector pixels of a third to all of the source's distance: tiles with
# corners on both sides of the source plane whose footprints would fit the box
@pytest.mark.parametrize("sod,sdd,res", [(2.0, 4.0, 2.0), (1.0, 3.0, 1.0), (1.5, 2.0, 2.0), (0.8, 4.0, 1.5)])
def test_source_plane_inside_a_tile(cuda, sod, sdd, res):
    nu, nv, box = 64, 64, (56, 56)
    ang = np.array([0.0, 30.0, 90.0, 135.0, 180.0, 200.0, 270.0, 301.0], np.float32)
    m = _module(nu, nv, sod, sdd, res, 0.1)
    xip, yip, zip_, *_, uni = m.partials(ang)
    assert uni
    fits = 0  # such tiles
    for p in range(ang.size):
        for j0 in range(0, nu, 8):
            for i0 in range(0, nu, 32):
                i, j = np.array([i0, i0 + 31])[:, None], np.array([j0, j0 + 7])[None]
                X, Y = xip[p, i], yip[p, j]
                d = zip_[p, 0, 2] + Y[..., 2] + X[..., 2]
                if d.min() < 0 < d.max():
                    c = (zip_[p, 0, 0] + Y[..., 0] + X[..., 0]) / d + 0.5
                    r = np.stack([(zip_[p, k, 1] + Y[..., 1] + X[..., 1]) / d + 0.5 for k in (0, 31)])
                    fits += np.ptp(c) < 50 and np.ptp(r) < 50 and c.max() > -1 and c.min() < nu and r.max() > -1 and r.min() < nv
    assert fits > 0
    rng = np.random.default_rng(3)
    filt = torch.from_numpy(rng.standard_normal((ang.size, nv, nu)).astype(np.float32)).to(cuda)
    got, direct = _backproject(cuda, m, filt, ang, box), _backproject(cuda, m, filt, ang, (0, 0))
    assert torch.equal(got, direct)
