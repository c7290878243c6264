"""MorphSpotClean's merging of basins when it takes more rounds than are launched one by one: a chain of
minima between walls whose heights are the trailing zeros of their number, where every component's lowest
edge leads to its twin, so that a round halves the components and does no more (2^k minima take k + 1
rounds; noise needs a third of that). Bit for bit against the oracle."""
import ctypes

import numpy as np
import pytest
import torch

import oracle as O
from imagingsuite_b200 import _lib as L
from imagingsuite_b200 import modules as M

pytestmark = pytest.mark.gpu
DET = {"holes": 0, "peaks": 1, "both": 2}


def _chain(log2):
    """2^log2 minima down the middle column, the outer columns and ends above every wall."""
    k = np.arange(1, 1 << log2)
    col = np.full(2 * k.size + 1, -1.0, np.float32)
    col[1::2] = np.log2(k & -k)
    img = np.full((col.size + 16, 3), 40.0, np.float32)
    img[8:-8, 1] = col
    return img[None]


@pytest.mark.parametrize("detect,sign", [("holes", 1), ("peaks", -1), ("both", 1), ("both", -1)])
@pytest.mark.parametrize("conn8", [True, False])
@pytest.mark.parametrize("log2", [10, 12, 14])  # 11, 13 and 15 rounds
def test_halving_rounds(cuda, detect, sign, conn8, log2):
    img = sign * _chain(log2)
    t = torch.from_numpy(img.copy()).cuda()
    M.morph_spot_clean(t, DET[detect], conn8, (0.5, 0.5), (0.0, 0.0), 1)
    st = ctypes.c_int(-1)
    L.check(L.lib().mr_device_status(ctypes.byref(st)))
    assert st.value == 0
    exp = O.morphspotclean(img, detect, conn8, (0.5, 0.5), (0.0, 0.0), edge=1)
    assert np.array_equal(t.cpu().numpy(), exp)
    inner = exp[0, 8:-8, 1]
    assert float(np.abs(inner - img[0, 8:-8, 1]).max()) > log2  # filled to the outer walls


