"""MorphSpotClean on a large image with little device memory left: what the merging of basins needs is not
there, and the row sweeps, which need a third of it, give the same image."""
import pytest
import torch
from cuda.bindings import runtime as rt

from imagingsuite_b200 import modules as M

pytestmark = pytest.mark.gpu


def test_large_image_with_little_memory(cuda):
    g = torch.Generator(device=cuda).manual_seed(1)
    img = torch.randn((1, 7000, 4000), device=cuda, generator=g)  # 1.1 GB of basins, 0.4 of sweeps
    exp = img.clone()
    M.morph_spot_clean(exp, 2, False, (0.5, 0.5), (0.0, 0.0), 5)
    torch.cuda.synchronize()
    # return what the library's stream-ordered pool and torch hold, then leave 0.7 GB
    err, pool = rt.cudaDeviceGetDefaultMemPool(0)
    assert int(err) == 0 and int(rt.cudaMemPoolTrimTo(pool, 0)[0]) == 0
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    hold = torch.empty(free - (700 << 20), dtype=torch.uint8, device=cuda)
    try:
        M.morph_spot_clean(img, 2, False, (0.5, 0.5), (0.0, 0.0), 5)
        torch.cuda.synchronize()
    finally:
        del hold
        torch.cuda.empty_cache()
    assert torch.equal(img, exp)
