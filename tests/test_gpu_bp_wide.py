"""Parallel-beam backprojection on very wide detectors, where one step of the detector position is a
noticeable part of a column and the positions of neighbouring rows can round to columns two apart:
every float operation restated with numpy, bit for bit."""
import numpy as np
import pytest
import torch

from imagingsuite_b200 import _lib as L

pytestmark = pytest.mark.gpu


def _geometry(ang, nu, centre):
    s, c, su = (np.empty_like(ang) for _ in range(3))
    L.check(L.lib().mr_bp_parallel_geometry(ang.ctypes.data_as(L.P_float), ang.size, nu, centre, 0,
                                            *(v.ctypes.data_as(L.P_float) for v in (s, c, su))))
    return s, c, su


# (columns, angle, 1-based row): a voxel of this row and the one below it read columns two apart
@pytest.mark.parametrize("nu,angle,row", [(20000, 2.834629774093628, 16741), (20000, 2.848041296005249, 16639)])
def test_neighbouring_rows_two_columns_apart(cuda, nu, angle, row):
    nv, rows = 4, 8
    rng = np.random.default_rng(row)
    ang = np.array([angle, 0.0, 2.5, 177.2, 91.0], np.float32)
    proj = rng.standard_normal((ang.size, nv, nu)).astype(np.float32)
    sn, cs, su = _geometry(ang, nu, (nu - 1) / 2)
    x, y = np.arange(1, nu + 1, dtype=np.float32)[None], np.arange(row, row + rows, dtype=np.float32)[:, None]
    exp = np.zeros((rows, nu, nv), np.float32)
    apart = 0
    for i in range(ang.size):
        u = (su[i] + cs[i] * y) - sn[i] * x
        n = u.astype(np.int64)
        ok = (n >= 0) & (n <= nu - 2)
        apart = max(apart, int(np.abs(np.diff(n, axis=0))[ok[1:] & ok[:-1]].max()))
        f = np.abs(u - n.astype(np.float32))
        n = np.where(ok, n, 0)
        for z in range(nv):
            t = proj[i, z][n] * (np.float32(1) - f) + proj[i, z][n + 1] * f
            exp[:, :, z] = np.where(ok, exp[:, :, z] + t, exp[:, :, z])
    assert apart == 2
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(cuda)  # noqa: E731
    mask = dev(np.tile(np.array([0, nu], np.int32), nu))
    p, s, c, u0 = dev(proj), dev(sn), dev(cs), dev(su)
    vol = torch.zeros((nu, nu, nv), device=cuda)
    L.check(L.lib().mr_bp_parallel_rows(p.data_ptr(), ang.size, L.MR_F32, None, None, None, s.data_ptr(), c.data_ptr(),
                                        u0.data_ptr(), ang.size, nu, nv, mask.data_ptr(), 0, 0.0, 0.0, row - 1,
                                        row - 1 + rows, vol.data_ptr(), torch.cuda.current_stream().cuda_stream))
    assert np.array_equal(vol[row - 1:row - 1 + rows].cpu().numpy(), exp)
