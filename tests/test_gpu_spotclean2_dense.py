"""SpotClean2's ring detection and component areas where nearly every weight is nonzero (one component
holds most of an image) and where none is, at sizes around the kernels' tiles, bit for bit against the
oracle."""
import numpy as np
import pytest
import torch

import oracle as O
from imagingsuite_b200 import modules as M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h,w", [(16, 31), (17, 32), (63, 33), (64, 64), (65, 130), (130, 257)])
@pytest.mark.parametrize("gamma", [-0.2, 0.05, 10.0])
@pytest.mark.parametrize("maxarea", [0, 7])
def test_dense_weights(cuda, h, w, gamma, maxarea):
    rng = np.random.default_rng(h * w)
    p = (0.3 + rng.normal(0, 0.05, (3, h, w))).astype(np.float32)
    p[1, h // 2:] = 0.25  # a flat half
    p[2][rng.random((h, w)) < 0.02] += 1.5
    mod = M.SpotClean2()
    mod.Configure(M.ReconConfig(), {"gamma": str(gamma), "sigma": "0.02", "iterations": "1", "maxlevel": "5",
                                    "minlevel": "-0.1", "maxarea": str(maxarea), "detectionmethod": "ring"})
    t = torch.from_numpy(p).to(cuda)
    mod.Process(t)
    exp = O.spotclean2(p, "ring", gamma, 0.02, 1, -0.1, 5.0, maxarea)
    assert np.array_equal(t.cpu().numpy().view(np.uint32), np.ascontiguousarray(exp, np.float32).view(np.uint32))
