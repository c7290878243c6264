"""Thin tiles of the staged parallel-beam backprojector: 4-slice tiles (fewer than 74 16-slice tiles), 8- and
16-slice ones beyond, with their remainders, in every mode, with footprints that lie partly and wholly outside
the detector on either side and projection counts around a batch of 16 and 32, against the oracle bit for bit
(every float operation is the reference's)."""
import numpy as np
import pytest
import torch

import oracle as O
from imagingsuite_b200 import modules as M

pytestmark = pytest.mark.gpu


def _text(a):
    return " ".join("%.9g" % v for v in a)


@pytest.mark.parametrize("variant", ["parallel", "serial", "nn"])
@pytest.mark.parametrize("tilt", [0.0, 0.6])
@pytest.mark.parametrize("nproj,nv,nu,shift", [(32, 4, 48, -19.7), (33, 5, 64, 0.3), (16, 13, 65, 40.4), (65, 8, 131, -0.5),
                                               (17, 20, 96, 70.0), (31, 9, 161, 12.6), (33, 17, 162, -30.2),
                                               (20, 48, 100, 25.0)])
def test_thin_tiles_bit_exact(cuda, variant, tilt, nproj, nv, nu, shift):
    rng = np.random.default_rng(nproj * nv + nu)
    proj = rng.standard_normal((nproj, nv, nu)).astype(np.float32)
    ang = np.concatenate([[0.0, 90.0, 180.0, 270.0], rng.uniform(-200, 400, nproj - 4)]).astype(np.float32)
    w = rng.uniform(0.5, 1.5, nproj).astype(np.float32)
    centre = (nu - 1) / 2.0 + shift
    cfg = M.ReconConfig()
    pi = cfg.ProjectionInfo
    pi.fCenter, pi.bCorrectTilt, pi.fTiltAngle, pi.fTiltPivotPosition = centre, tilt != 0, tilt, nv / 2
    pi.roi = (0, 0, nu, nv)
    pi.nDims = (nu, nv, 0)
    bp = {"parallel": M.MultiProjectionBPparallel, "serial": M.MultiProjectionBP, "nn": M.NearestNeighborBP}[variant]()
    bp.Configure(cfg, {"ProjectionBufferSize": "16", "SliceBlock": "32", "SubVolume": "1 1"})
    bp.SetROI((0, 0, nu, nv))
    bp.Process(torch.from_numpy(proj).to(cuda), {"angles": _text(ang), "weights": _text(w)})
    exp = O.bp_parallel(proj, ang, w, centre, buffersize=16, correcttilt=tilt != 0, tiltangle=tilt, tiltpivot=nv / 2,
                        nslices=nv, serial=variant == "serial", nn=variant == "nn")
    assert np.array_equal(bp.GetVolume().cpu().numpy(), exp)
