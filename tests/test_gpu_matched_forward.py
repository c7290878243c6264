"""The matched pair's forward projection on both sides of the line between its kernels (400 bins), at odd and
small widths, partial slice groups, one and two CTAs per projection, centres that put part of the volume off the
detector, steep tilts and masks with holes, against the oracle's transpose in FP64. A bin sums at most a few
times n products of FP32 values in FP32: 1e-6 of the projections' norm, as for the pair's other tests; the
derivative is compared as there."""
import math

import numpy as np
import pytest
import torch

import oracle as O
from imagingsuite_b200 import _lib as L

pytestmark = pytest.mark.gpu

ANGLES = np.array([0.0, 1.0, 44.9, 45.0, 60.3, 90.0, 117.7, 135.0, 179.2, 200.0, 270.0, 315.0, 333.3], np.float32)


def _forward(x, ang, centre, tan, pivot, mask, derivative):
    n, _, nz = x.shape
    sc, su = O.mbp_geometry(ang, n, nz, centre, tan, pivot, 0)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    xt, sct, sut, mt = dev(x), dev(sc), dev(su), dev(mask.view(np.int32))
    proj = torch.full((ang.size, nz, n), np.nan, device="cuda")
    d = torch.full_like(proj, np.nan) if derivative else None
    L.check(L.lib().mr_mbp_forward(xt.data_ptr(), n, nz, sct.data_ptr(), sut.data_ptr(), ang.size, mt.data_ptr(),
                                   proj.data_ptr(), None if d is None else d.data_ptr(),
                                   torch.cuda.current_stream().cuda_stream))
    return proj.cpu().numpy(), None if d is None else d.cpu().numpy()


@pytest.mark.parametrize("n,nz", [(2, 4), (5, 1), (31, 33), (101, 8), (400, 4), (401, 4), (407, 36), (523, 3)])
@pytest.mark.parametrize("tilt,shift,holes", [(0.4, 0.2, False), (-0.9, 17.3, True), (30.0, -5.0, True)])
def test_forward(cuda, n, nz, tilt, shift, holes):
    rng = np.random.default_rng(n * 100 + nz)
    x = rng.standard_normal((n, n, nz)).astype(np.float32)
    centre, tan, pivot = n / 2 + shift, math.tan(math.radians(tilt)), (nz - 1) / 2
    mask = O.circle_mask(n, n).reshape(-1, 2).astype(np.uint32)
    inside = x.copy()
    if holes:  # rows cut short at random: columns with gaps
        mask[:, 0] += (rng.random(n) * (mask[:, 1] - mask[:, 0]) / 2).astype(np.uint32)
        mask[rng.random(n) < 0.1] = 0
        for y, (a, b) in enumerate(mask):
            inside[y, :a] = 0.0
            inside[y, b:] = 0.0
    exp, dexp = O.mbp_forward64(inside, ANGLES, centre, tan, pivot, derivative=True)
    for derivative in (False, True):
        got, d = _forward(x, ANGLES, centre, tan, pivot, np.ascontiguousarray(mask), derivative)
        assert np.sqrt(np.sum((got - exp) ** 2)) <= 1e-6 * np.sqrt(np.sum(exp ** 2))
        if derivative:
            assert np.abs(d - dexp).max() <= 1e-3 * np.abs(dexp).max()


def test_forward_two_ctas(cuda):
    """More than 74 and fewer than 148 (projection, slice group) pairs take one CTA each, 60 take two."""
    rng = np.random.default_rng(3)
    x = rng.standard_normal((65, 65, 4)).astype(np.float32)
    mask = O.circle_mask(65, 65).astype(np.uint32)
    for nproj in (60, 100):
        ang = (np.arange(nproj) * 3.1).astype(np.float32)
        exp = O.mbp_forward64(x, ang, 32.9, 0.01, 1.5)
        got, _ = _forward(x, ang, 32.9, 0.01, 1.5, mask, False)
        assert np.sqrt(np.sum((got - exp) ** 2)) <= 1e-6 * np.sqrt(np.sum(exp ** 2))


# more pairs than the GPU has SMs: half as many threads up to 48 bins, whole ones beyond, two CTAs each where the
# lines are long enough for the number of waves (130 bins, 160 pairs) and one where not
@pytest.mark.parametrize("n,nz,nproj", [(3, 33, 80), (16, 4, 150), (48, 34, 100), (49, 4, 160), (130, 4, 160), (130, 34, 160)])
def test_forward_several_waves(cuda, n, nz, nproj):
    rng = np.random.default_rng(n)
    x = rng.standard_normal((n, n, nz)).astype(np.float32)
    mask = O.circle_mask(n, n).astype(np.uint32)
    ang = (np.arange(nproj) * 2.3).astype(np.float32)
    exp, dexp = O.mbp_forward64(x, ang, n / 2 + 0.2, 0.01, nz / 2, derivative=True)
    for derivative in (False, True):
        got, d = _forward(x, ang, n / 2 + 0.2, 0.01, nz / 2, mask, derivative)
        assert np.sqrt(np.sum((got - exp) ** 2)) <= 1e-6 * np.sqrt(np.sum(exp ** 2))
        if derivative:
            assert np.abs(d - dexp).max() <= 1e-3 * np.abs(dexp).max()
