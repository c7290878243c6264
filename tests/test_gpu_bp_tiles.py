"""Tiles and projection layouts of the staged parallel-beam backprojector: every tile height with its
remainders, rows whose pitch or base the TMA unit cannot address, weights, positions off the detector
and cos = +-1, against the oracle bit for bit (every float operation is the reference's)."""
import numpy as np
import pytest
import torch

import oracle as O
from imagingsuite_b200 import _lib as L
from imagingsuite_b200 import modules as M

pytestmark = pytest.mark.gpu


def _text(a):
    return " ".join("%.9g" % v for v in a)


def _module(cls, nu, nv, centre, tilt, params):
    cfg = M.ReconConfig()
    pi = cfg.ProjectionInfo
    pi.fCenter, pi.bCorrectTilt, pi.fTiltAngle, pi.fTiltPivotPosition = centre, tilt != 0, tilt, nv / 2
    pi.roi = (0, 0, nu, nv)
    pi.nDims = (nu, nv, 0)
    bp = cls()
    bp.Configure(cfg, {"ProjectionBufferSize": "16", "SliceBlock": "32", "SubVolume": "1 1", **params})
    bp.SetROI((0, 0, nu, nv))
    return bp


# (nv, nu): 8-slice tiles (few tiles or short remainders), 16-slice, 32-slice; widths that are and are
# not multiples of 4; the last voxel column and row alone in their tile; partial last tiles
@pytest.mark.parametrize("nv,nu", [(4, 48), (8, 49), (11, 65), (16, 129), (20, 130), (28, 225), (36, 161), (40, 226),
                                   (64, 161), (96, 163)])
@pytest.mark.parametrize("tilt", [0.0, -0.7])
@pytest.mark.parametrize("shift", [0.0, 21.3])
def test_tiles_bit_exact(cuda, nv, nu, tilt, shift):
    rng = np.random.default_rng(nv * nu)
    nproj = 37
    proj = rng.standard_normal((nproj, nv, nu)).astype(np.float32)
    ang = np.concatenate([[0.0, 90.0, 180.0, 270.0], rng.uniform(-200, 400, nproj - 4)]).astype(np.float32)
    w = rng.uniform(0.5, 1.5, nproj).astype(np.float32)
    centre = (nu - 1) / 2.0 + shift
    bp = _module(M.MultiProjectionBPparallel, nu, nv, centre, tilt, {})
    bp.Process(torch.from_numpy(proj).to(cuda), {"angles": _text(ang), "weights": _text(w)})
    exp = O.bp_parallel(proj, ang, w, centre, buffersize=16, correcttilt=tilt != 0, tiltangle=tilt, tiltpivot=nv / 2,
                        nslices=nv)
    assert np.array_equal(bp.GetVolume().cpu().numpy(), exp)


@pytest.mark.parametrize("nv,nu,offset", [(24, 100, 1), (24, 101, 0), (24, 102, 3)])
def test_projection_base_off_16_bytes(cuda, nv, nu, offset):
    """Contiguous projections that start `offset` floats into an allocation, prefiltered weights."""
    g = torch.Generator(device=cuda).manual_seed(3)
    nproj = 50
    flat = torch.randn(nproj * nv * nu + offset, device=cuda, generator=g)
    view = flat[offset:].view(nproj, nv, nu)
    ang = (np.arange(nproj) * 180.0 / nproj).astype(np.float32)
    params = {"angles": _text(ang), "weights": _text(np.ones(nproj))}
    bp = _module(M.MultiProjectionBPparallel, nu, nv, nu / 2, 0.0, {})
    bp.Process(view, params, prefiltered_weights=True)
    exp = O.bp_parallel(view.cpu().numpy(), ang, np.ones(nproj, np.float32), nu / 2, buffersize=16)
    assert np.array_equal(bp.GetVolume().cpu().numpy(), exp)


def test_repitched_runs_continue_the_sums(cuda):
    """More projections than one scratch run holds: the volume carries the sums between the runs, as in
    the direct-load kernel."""
    nproj, nv, nu = 1400, 4000, 49
    g = torch.Generator(device=cuda).manual_seed(4)
    proj = torch.randn((nproj, nv, nu), device=cuda, generator=g)
    ang = (np.arange(nproj) * 180.0 / nproj).astype(np.float32)
    w = np.linspace(0.5, 1.5, nproj).astype(np.float32)
    vols = []
    for staging in (True, False):
        bp = _module(M.MultiProjectionBPparallel, nu, nv, (nu - 1) / 2, 0.0, {})
        bp.staging = staging
        bp.Process(proj, {"angles": _text(ang), "weights": _text(w)})
        vols.append(bp.GetVolume())
    assert torch.equal(vols[0], vols[1])


@pytest.mark.parametrize("nu", [96, 97])
def test_values_that_are_not_finite(cuda, nu):
    """Infinities and NaN reach the voxels they reach in the direct-load kernel, and no others."""
    g = torch.Generator(device=cuda).manual_seed(5)
    nproj, nv = 40, 32
    proj = torch.randn((nproj, nv, nu), device=cuda, generator=g)
    proj[3, 5, nu // 2] = float("inf")
    proj[20, 9, nu // 3] = float("nan")
    ang = (np.arange(nproj) * 180.0 / nproj).astype(np.float32)
    vols = []
    for staging in (True, False):
        bp = _module(M.MultiProjectionBPparallel, nu, nv, (nu - 1) / 2, 0.0, {})
        bp.staging = staging
        bp.Process(proj, {"angles": _text(ang), "weights": _text(np.ones(nproj))}, prefiltered_weights=True)
        vols.append(bp.GetVolume().cpu().numpy())
    assert np.isnan(vols[1]).any() and np.array_equal(vols[0], vols[1], equal_nan=True)


@pytest.mark.parametrize("nu", [64, 66])
def test_slab_count_below_the_list(cuda, nu):
    """Without an index list fewer slabs than projections are refused, with tilt correction they never were."""
    nv, nproj = 8, 20
    g = torch.Generator(device=cuda).manual_seed(nu)
    p = torch.randn((nproj, nv, nu), device=cuda, generator=g)
    sn, cs, su = (torch.rand(nproj, device=cuda, generator=g) * s + o for s, o in ((0.7, 0.0), (0.3, 0.7), (2.0, 0.0)))
    mask = torch.tensor([0, nu], dtype=torch.int32, device=cuda).repeat(nu)
    vols = {}
    for tilt, nslabs in ((1, nproj), (1, nproj - 1), (1, 0), (0, nproj - 1)):
        vol = torch.zeros((nu, nu, nv), device=cuda)
        st = L.lib().mr_bp_parallel_staged(p.data_ptr(), nslabs, L.MR_F32, None, None, None, sn.data_ptr(), cs.data_ptr(),
                                           su.data_ptr(), nproj, nu, nv, mask.data_ptr(), tilt, 0.3, 0.01, vol.data_ptr(),
                                           torch.cuda.current_stream().cuda_stream)
        assert st == (L.MR_OK if tilt else L.MR_ERR_ARGUMENT)
        vols[tilt, nslabs] = vol
    assert torch.equal(vols[1, nproj], vols[1, nproj - 1]) and torch.equal(vols[1, nproj], vols[1, 0])
    assert not bool(vols[0, nproj - 1].any())
