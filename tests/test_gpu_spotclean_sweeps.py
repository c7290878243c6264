"""MorphSpotClean's row sweeps and worklist (many images) against the oracle bit for bit: every chunk
length of the sweep kernel (rows of up to 374, 630, 1142, 2166 and 4214 pixels), images whose paths wind
through noise so that the worklist overflows into dense passes and finishes them, and the same in the
bounds-checked build."""
import ctypes

import numpy as np
import pytest
import torch

import oracle as O
from imagingsuite_b200 import _lib as L
from imagingsuite_b200 import modules as M

pytestmark = pytest.mark.gpu
DET = {"holes": 0, "peaks": 1, "both": 2}
MANY = 600  # images from which every mode and width takes the sweeps


def _clean(stack, detect, conn8, th, edge):
    t = torch.from_numpy(np.ascontiguousarray(stack, np.float32)).cuda()
    M.morph_spot_clean(t, DET[detect], conn8, th, (0.0, 0.0), edge)
    st = ctypes.c_int(-1)
    L.check(L.lib().mr_device_status(ctypes.byref(st)))
    assert st.value == 0
    return t


def _check(img, detect, conn8, th, edge=5):
    """All repetitions of the images equal the oracle's."""
    exp = torch.from_numpy(O.morphspotclean(img, detect, conn8, th, (0.0, 0.0), edge=edge)).cuda()
    k = img.shape[0]
    n = -(-MANY // k) * k
    got = _clean(np.tile(img, (n // k, 1, 1)), detect, conn8, th, edge)
    assert torch.equal(got.view(n // k, *img.shape), exp.expand(n // k, *img.shape))


def _noisy_profile(h, w, n, seed):
    rng = np.random.default_rng(seed)
    yy, xx = np.mgrid[:h, :w]
    base = 1.5 * np.exp(-((xx - w / 2) / (0.3 * w)) ** 2 - ((yy - h / 2) / (0.6 * h)) ** 2)
    img = (base + rng.normal(0, 0.03, (n, h, w))).astype(np.float32)
    img[0, h // 3, w // 7] += 1.0
    img[-1, h // 2, w // 2] -= 1.0
    return img


@pytest.mark.parametrize("detect", ["holes", "peaks", "both"])
@pytest.mark.parametrize("conn8", [True, False])
@pytest.mark.parametrize("h,w", [(9, 374), (12, 375), (7, 630), (14, 1000), (6, 1142), (11, 2048), (8, 2166), (6, 3000),
                                 (5, 4214)])
def test_chunk_lengths(cuda, detect, conn8, h, w):
    rng = np.random.default_rng(h * w)
    img = rng.standard_normal((3, h, w)).astype(np.float32)
    img[1] = np.round(img[1])
    img[2] = np.cumsum(img[2], axis=1) * np.float32(0.05)
    _check(img, detect, conn8, (0.3, 0.25))


@pytest.mark.parametrize("detect", ["holes", "peaks", "both"])
@pytest.mark.parametrize("conn8", [True, False])
@pytest.mark.parametrize("h,w", [(96, 700), (40, 300), (30, 1500)])
def test_worklist_completion(cuda, detect, conn8, h, w):
    _check(_noisy_profile(h, w, 2, h + w), detect, conn8, (0.1, 0.1))


# stacks beyond the number up to which basins are merged at their width and neighbourhood (230, 139 and
# 118 reconstructions; with 'both', two per image) equal their parts below it
@pytest.mark.parametrize("detect,conn8,w,n,part", [("holes", True, 990, 240, 80), ("both", True, 990, 117, 39),
                                                   ("peaks", False, 990, 150, 50), ("holes", False, 1270, 120, 40)])
def test_line_between_the_reconstructions(cuda, detect, conn8, w, n, part):
    img = _noisy_profile(12, w, n, w + n)
    got = _clean(img, detect, conn8, (0.1, 0.1), 5)
    parts = torch.cat([_clean(img[a:a + part], detect, conn8, (0.1, 0.1), 5) for a in range(0, n, part)])
    assert torch.equal(got, parts)
    exp = O.morphspotclean(img[:3], detect, conn8, (0.1, 0.1), (0.0, 0.0), edge=5)
    assert np.array_equal(got[:3].cpu().numpy(), exp)


@pytest.mark.parametrize("detect", ["holes", "peaks", "both"])
def test_checked_build(cuda, detect, monkeypatch):
    img = np.tile(_noisy_profile(40, 300, 2, 9), (MANY // 2, 1, 1))
    product = _clean(img, detect, False, (0.1, 0.1), 5)
    checked = L.load(L.CHECKED_LIB_PATH)
    monkeypatch.setattr(L, "_lib", checked)
    word = ctypes.c_ulonglong(1)
    L.check(checked.mr_bounds_status(ctypes.byref(word)))  # clear
    got = _clean(img, detect, False, (0.1, 0.1), 5)
    L.check(checked.mr_bounds_status(ctypes.byref(word)))
    assert word.value == 0
    assert torch.equal(got, product)
