"""The matched pair's adjoint with tilt, staged by TMA: widths that are not a multiple of 4 or narrower than
the staged box, partial slice tiles, steep tilts whose footprints leave the box, centres that put part of the
volume off the detector, and runs of padded copies, bit for bit against the oracle (the same float operations
in the same order)."""
import math

import numpy as np
import pytest
import torch

import oracle as O
from imagingsuite_b200 import _lib as L
from imagingsuite_b200 import joseph as J

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nz", [(17, 4), (31, 36), (47, 32), (48, 8), (50, 40), (63, 68), (64, 33), (97, 32), (190, 36)])
@pytest.mark.parametrize("tilt,shift", [(0.4, 0.2), (-0.9, 17.3), (35.0, 0.0)])
def test_adjoint_bit_exact(cuda, n, nz, tilt, shift):
    rng = np.random.default_rng(n * nz)
    ang = np.concatenate([[0.0, 90.0, 180.0], rng.uniform(0, 360, 34)]).astype(np.float32)
    nproj = ang.size
    p = rng.standard_normal((nproj, nz, n)).astype(np.float32)
    centre, pivot, tan = n / 2 + shift, (nz - 1) / 2, math.tan(math.radians(tilt))
    sc, su = O.mbp_geometry(ang, n, nz, centre, tan, pivot, 0)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(cuda)  # noqa: E731
    mask = dev(O.circle_mask(n, n).view(np.int32))
    pt, sct, sut = dev(p), dev(sc), dev(su)
    vol = torch.full((n, n, nz), 7.0, device=cuda)
    st = torch.cuda.current_stream().cuda_stream
    L.check(L.lib().mr_mbp_adjoint(pt.data_ptr(), n, nz, sct.data_ptr(), sut.data_ptr(), nproj, mask.data_ptr(), 0,
                                   vol.data_ptr(), st))
    exp = O.mbp_adjoint(p[:, :, :], ang, centre, tan, pivot, 0)
    assert np.array_equal(vol.cpu().numpy(), exp)
    # continued sums leave everything outside the circle alone
    vol += 1.0
    before = vol.cpu().numpy()
    L.check(L.lib().mr_mbp_adjoint(pt.data_ptr(), n, nz, sct.data_ptr(), sut.data_ptr(), 0, mask.data_ptr(), 1,
                                   vol.data_ptr(), st))
    assert np.array_equal(vol.cpu().numpy(), before)


def test_padded_runs_continue_the_sums(cuda):
    """More projections than one run of padded copies: equal to two accumulating calls."""
    n, nz, nproj = 45, 2048, 400  # 48 * 2048 floats each, 170 a run
    g = torch.Generator(device=cuda).manual_seed(2)
    p = torch.randn((nproj, nz, n), device=cuda, generator=g)
    ang = (np.arange(nproj) * 0.45).astype(np.float32)
    whole = J.MatchedOperator(n, nz, ang).adjoint(p, n / 2, 0.3)
    out = torch.zeros_like(whole)
    for a, b in ((0, 100), (100, 230), (230, 400)):
        J.MatchedOperator(n, nz, ang[a:b]).adjoint(p[a:b].contiguous(), n / 2, 0.3, out=out, accumulate=True)
    assert torch.equal(whole, out)


@pytest.mark.parametrize("n,tilt", [(31, 0.4), (65, -0.9)])
def test_adjoint_without_scratch(cuda, n, tilt):
    """No room for the padded copies: the same values by guarded loads."""
    nz, ang = 8, (np.arange(40) * 4.5).astype(np.float32)
    g = torch.Generator(device=cuda).manual_seed(n)
    p = torch.randn((40, nz, n), device=cuda, generator=g)
    op = J.MatchedOperator(n, nz, ang)
    exp = op.adjoint(p, n / 2 + 1.3, tilt)
    L.check(L.lib().mr_debug_fail_allocation(0))
    try:
        got = op.adjoint(p, n / 2 + 1.3, tilt)
    finally:
        L.check(L.lib().mr_debug_fail_allocation(-1))
    assert torch.equal(got, exp)


@pytest.mark.parametrize("n,nz", [(64, 32), (61, 12), (192, 64)])
def test_accumulate_keeps_what_is_outside_the_circle(cuda, n, nz):
    """A volume of nonzero values: untouched outside the circle; inside, one call continues it as two do."""
    g = torch.Generator(device=cuda).manual_seed(1)
    p = torch.randn((40, nz, n), device=cuda, generator=g)
    op = J.MatchedOperator(n, nz, (np.arange(40) * 4.5).astype(np.float32))
    preset = torch.rand((n, n, nz), device=cuda, generator=g) + 1.0
    one, two = preset.clone(), preset.clone()
    op.adjoint(p, n / 2 + 0.3, 0.4, out=one, accumulate=True)
    for a, b in ((0, 17), (17, 40)):
        J.MatchedOperator(n, nz, op.angles[a:b]).adjoint(p[a:b].contiguous(), n / 2 + 0.3, 0.4, out=two, accumulate=True)
    m = op._mask.cpu().numpy().view(np.uint32).reshape(-1, 2)
    x = np.arange(1, n + 1)
    inside = torch.from_numpy((x > m[:, :1]) & (x <= m[:, 1:])).to(cuda)
    assert torch.equal(one[~inside], preset[~inside])
    assert torch.equal(one, two)
    assert bool((one[inside] != preset[inside]).any(dim=1).all())
