"""MorphSpotClean on images with NaN (removeinfnan off), in both reconstructions (merged basins for few
images, row sweeps for many). The reference's comparisons are false for a NaN: such a pixel keeps its
NaN, paths do not lead through it, and none starts at it when it lies on the padded border. Bit for bit
against the oracle; edge lengths above 1 only between the two reconstructions, because a median of
samples with NaN depends on how it is formed."""
import numpy as np
import pytest
import torch

import oracle as O
from imagingsuite_b200 import modules as M

pytestmark = pytest.mark.gpu
DET = {"holes": 0, "peaks": 1, "both": 2}
MANY = 600  # images from which every mode takes the sweeps


def _clean(stack, detect, conn8, edge):
    t = torch.from_numpy(np.array(stack, np.float32)).cuda()
    M.morph_spot_clean(t, DET[detect], conn8, (0.3, 0.25), (0.0, 0.0), edge)
    return t.cpu().numpy()


def _images(h, w):
    """NaN in the rows that become the padded border (4 and h - 5), in the corners, in the middle, as a
    closed wall around a region, as a line from edge to edge, and in half of the pixels."""
    rng = np.random.default_rng(h * w)
    x = rng.standard_normal((9, h, w)).astype(np.float32)
    x[0, 4, 3] = np.nan
    x[1, h - 5, [2, w - 3]] = np.nan
    x[2, 4, :] = np.nan
    x[2, h - 5, ::2] = np.nan
    x[3, [0, 0, -1, -1], [0, -1, 0, -1]] = np.nan
    x[4, h // 2, w // 2] = np.nan
    x[5, 6:13, 6] = x[5, 6:13, 14] = x[5, 6, 6:15] = x[5, 12, 6:15] = np.nan
    x[5, 9, 9] = 9.0  # the image's maximum inside the wall
    x[6, h // 2, :] = np.nan
    x[7][rng.random((h, w)) < 0.5] = np.nan
    x[8] = np.round(x[8])
    x[8][rng.random((h, w)) < 0.05] = np.nan
    x[8][rng.random((h, w)) < 0.05] = np.inf
    x[8][rng.random((h, w)) < 0.05] = -np.inf
    return x


@pytest.mark.parametrize("detect", ["holes", "peaks", "both"])
@pytest.mark.parametrize("conn8", [True, False])
@pytest.mark.parametrize("h,w", [(21, 23), (60, 70)])
@pytest.mark.parametrize("many", [False, True])
def test_equal_oracle(cuda, detect, conn8, h, w, many):
    img = _images(h, w)
    exp = O.morphspotclean(img, detect, conn8, (0.3, 0.25), (0.0, 0.0), edge=1)
    got = _clean(np.resize(img, (MANY + 3, h, w)) if many else img, detect, conn8, 1)
    assert np.array_equal(got, np.resize(exp, got.shape), equal_nan=True)


@pytest.mark.parametrize("detect", ["holes", "peaks", "both"])
@pytest.mark.parametrize("edge", [5, 9])
def test_few_equal_many(cuda, detect, edge):
    img = _images(40, 52)
    few = _clean(img, detect, True, edge)
    many = _clean(np.resize(img, (MANY, 40, 52)), detect, True, edge)
    assert np.array_equal(many, np.resize(few, many.shape), equal_nan=True)


@pytest.mark.parametrize("many", [False, True])
def test_nan_bits_stay(cuda, many):
    bits = np.array([0x7FC00001, 0xFFC12345, 0x7F800001, 0xFFFFFFFF, 0x7FFFFFFF], np.uint32)
    img = np.random.default_rng(4).standard_normal((1, 20, 30)).astype(np.float32)
    img.view(np.uint32)[0, 7, 3:28:5] = bits
    got = _clean(np.repeat(img, MANY if many else 1, axis=0), "both", True, 5)
    assert np.array_equal(got[-1].view(np.uint32)[7, 3:28:5], bits)
