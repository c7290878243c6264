"""The 5x5 median's tiled kernel against the oracle, bit for bit: images at the smallest size it takes, widths and
heights on both sides of its tiles (2 columns x 16 rows per thread, 64 columns x 64 rows per CTA), one image and
several, and values with ties, zeros of both signs, NaN and infinities."""
import numpy as np
import pytest
import torch

import oracle as O
from imagingsuite_b200 import modules as M

pytestmark = pytest.mark.gpu


def _special(rng, shape):
    img = rng.integers(-3, 4, shape).astype(np.float32)
    img[(img == 0) & (rng.random(shape) < 0.5)] = -0.0
    for v in (np.nan, np.inf, -np.inf, np.finfo(np.float32).max, np.finfo(np.float32).min):
        img[rng.random(shape) < 0.01] = v
    return img


@pytest.mark.parametrize("h,w", [(5, 6), (6, 5), (6, 6), (6, 7), (7, 6), (7, 9), (19, 67), (20, 68), (21, 69), (22, 70),
                                 (36, 131), (37, 132), (67, 64), (68, 65), (69, 66), (133, 200)])
@pytest.mark.parametrize("nimg", [1, 3])
def test_median55(cuda, h, w, nimg):
    rng = np.random.default_rng(h * 1000 + w)
    stack = rng.standard_normal((nimg, h, w)).astype(np.float32)
    if nimg > 1:
        stack[1] = _special(rng, (h, w))
        stack[2] = rng.integers(0, 3, (h, w))
    got = M.median_filter(torch.from_numpy(stack).cuda(), 5, 5).cpu().numpy()
    for i in range(nimg):
        assert np.array_equal(got[i].view(np.uint32), O.median_filter(stack[i], 5, 5).view(np.uint32)), i
