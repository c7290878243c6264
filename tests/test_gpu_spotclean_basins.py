"""MorphSpotClean's two reconstructions: merged basins (few images) and row sweeps with a worklist (many
images) against the oracle bit for bit (thresholds only, no sigmoid), at sizes around the strips the
passes work on, on noise, plateaus, ramps, terraces and spirals, and at image counts on both sides of the
rule that chooses between them. Reconstructions are minima and maxima of pixel values, so there is no
tolerance."""
import ctypes

import numpy as np
import pytest
import torch

import oracle as O
from imagingsuite_b200 import _lib as L
from imagingsuite_b200 import modules as M

pytestmark = pytest.mark.gpu
DET = {"holes": 0, "peaks": 1, "both": 2}


def _clean(stack, detect, conn8, th=(0.3, 0.25)):
    t = torch.from_numpy(np.ascontiguousarray(stack, np.float32)).cuda()
    M.morph_spot_clean(t, DET[detect], conn8, th, (0.0, 0.0))
    st = ctypes.c_int(-1)
    L.check(L.lib().mr_device_status(ctypes.byref(st)))
    assert st.value == 0
    return t.cpu().numpy()


def _image(kind, h, w, rng):
    y, x = np.mgrid[0:h, 0:w].astype(np.float32)
    if kind == "noise":
        return rng.standard_normal((h, w))
    if kind == "plateau":
        return np.round(rng.standard_normal((h, w)))
    if kind == "ramp":  # one long descent, with spots
        return 0.01 * (x + 3 * y) + 2.0 * (rng.random((h, w)) < 0.01)
    if kind == "terraces":
        return np.floor((x + y) / 7) * 0.5 - 3.0 * (rng.random((h, w)) < 0.02)
    r = np.hypot(x - w / 2, y - h / 2)  # a spiral wall: long winding paths to the border
    return 2.0 * (np.sin(r / 2.5 + np.arctan2(y - h / 2, x - w / 2)) > 0) + 0.1 * rng.standard_normal((h, w))


@pytest.mark.parametrize("kind", ["noise", "plateau", "ramp", "terraces", "spiral"])
@pytest.mark.parametrize("h,w", [(5, 1), (6, 7), (22, 20), (23, 51), (54, 50), (55, 81), (118, 111)])
def test_basins_equal_oracle(cuda, kind, h, w):
    rng = np.random.default_rng(h * w)
    stack = np.stack([_image(kind, h, w, rng) for _ in range(3)]).astype(np.float32)
    for detect in DET:
        for conn8 in (True, False):
            exp = O.morphspotclean(stack, detect, conn8, (0.3, 0.25), (0.0, 0.0))
            assert np.array_equal(_clean(stack, detect, conn8), exp), (detect, conn8)


@pytest.mark.parametrize("detect", ["holes", "peaks", "both"])
@pytest.mark.parametrize("conn8", [True, False])
def test_many_images_equal_few(cuda, detect, conn8):
    """700 small images go through the sweeps; each alone through the basins."""
    rng = np.random.default_rng(11)
    stack = rng.standard_normal((700, 13, 40)).astype(np.float32)
    stack[::7] = np.round(stack[::7])
    got = _clean(stack, detect, conn8)
    parts = np.concatenate([_clean(stack[a:a + 250], detect, conn8) for a in range(0, 700, 250)])
    assert np.array_equal(got, parts)
    exp = O.morphspotclean(stack[:20], detect, conn8, (0.3, 0.25), (0.0, 0.0))
    assert np.array_equal(got[:20], exp)


@pytest.mark.parametrize("h,w,n", [(6400, 12, 1), (6400, 6, 600)])
def test_tall_images_replay_the_band_in_global_memory(cuda, h, w, n):
    """Border columns beyond a CTA's shared memory (peaks), on both reconstructions."""
    rng = np.random.default_rng(12)
    stack = np.repeat(rng.standard_normal((1, h, w)).astype(np.float32), n, axis=0)
    got = _clean(stack, "peaks", True)
    exp = O.morphspotclean(stack[:1], "peaks", True, (0.3, 0.25), (0.0, 0.0))
    assert np.array_equal(got[0], exp[0]) and np.array_equal(got[-1], exp[0])


def test_infinities_and_nan(cuda):
    """Infinities are heights like others; a NaN pixel stays NaN and lets paths through."""
    rng = np.random.default_rng(13)
    img = rng.standard_normal((1, 60, 70)).astype(np.float32)
    img[0, 20, 20], img[0, 30, 40] = np.inf, -np.inf
    for detect in DET:
        assert np.array_equal(_clean(img, detect, True), O.morphspotclean(img, detect, True, (0.3, 0.25), (0.0, 0.0)))
    img[0, 10, 10] = np.nan
    low = img.copy()
    low[0, 10, 10] = -np.inf  # the height a NaN has for holes
    got, exp = _clean(img, "holes", True), _clean(low, "holes", True)
    same = np.ones(img.shape, bool)
    same[0, 10, 10] = False
    assert np.isnan(got[0, 10, 10]) and np.array_equal(got[same], exp[same])
