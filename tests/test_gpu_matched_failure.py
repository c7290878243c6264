"""Bounded waits of the matched adjoint without a fault: with the wait limit at 0 every tile gives up, the
device word is set, its voxels are NaN (a gradient that passes for a value would be worse), copies in
flight are waited for, and with the limit restored the result is exact; cgls and fbp raise."""
import ctypes

import numpy as np
import pytest
import torch

from imagingsuite_b200 import _lib as L
from imagingsuite_b200 import joseph as J

pytestmark = pytest.mark.gpu


def _word():
    st = ctypes.c_int(-1)
    L.check(L.lib().mr_device_status(ctypes.byref(st)))
    return st.value


@pytest.fixture
def zero_wait_limit():
    assert _word() == 0
    L.check(L.lib().mr_set_wait_limit(0))
    try:
        yield
    finally:
        L.check(L.lib().mr_set_wait_limit(-1))
        _word()


def _operator(cuda, n, nz, nproj):
    g = torch.Generator(device=cuda).manual_seed(n)
    ang = (np.arange(nproj) * 180.0 / nproj).astype(np.float32)
    return J.MatchedOperator(n, nz, ang), torch.randn((nproj, nz, n), device=cuda, generator=g)


# one batch of projections, several, rows copied to a padded pitch, the two tile heights
@pytest.mark.parametrize("n,nz,nproj", [(64, 8, 3), (64, 32, 40), (61, 8, 20), (192, 64, 40)])
def test_expiry_is_loud_and_recovered(cuda, n, nz, nproj):
    op, p = _operator(cuda, n, nz, nproj)
    exp = op.adjoint(p, n / 2 + 0.3, 0.4)
    assert _word() == 0
    L.check(L.lib().mr_set_wait_limit(0))
    try:
        got = op.adjoint(p, n / 2 + 0.3, 0.4)
        assert _word() == 1
    finally:
        L.check(L.lib().mr_set_wait_limit(-1))
    assert _word() == 0  # reading cleared it
    inside = exp[:, :, 0] != 0
    assert bool(torch.isnan(got[inside]).all()) and bool((got[~inside] == 0).all())
    assert torch.equal(op.adjoint(p, n / 2 + 0.3, 0.4), exp)


@pytest.mark.parametrize("tilt", [0.0, 0.4])
def test_cgls_and_fbp_raise(cuda, zero_wait_limit, tilt):
    op, p = _operator(cuda, 64, 8, 20)
    for call in (lambda: J.cgls(op, p, torch.zeros((64, 64, 8), device=cuda), 32.0, tilt, iterations=2),
                 lambda: J.fbp(op, p, 32.0, tilt)):
        with pytest.raises(L.MrError) as e:
            call()
        assert e.value.status == L.MR_ERR_DEVICE
        assert _word() == 0
