"""The list of a mask's set pixels: masks of less than a tile, of exactly one, of
one pixel more, of as many tiles as a block adds up by itself and of one more.
A PatchMatch call without sweeps evaluates one candidate per listed pixel: as
many as the mask has, a match for each of them and none elsewhere."""
import numpy as np
import pytest

from nli_gb300 import _abi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(8, 4), (33, 31), (32, 32), (41, 25), (2048, 1024), (2049, 1024), (2047, 1027)])
@pytest.mark.parametrize("density", [0.0005, 0.3, 1.0])
def test_every_set_pixel_is_listed_once(gpu_ctx, w, h, density):
    rng = np.random.default_rng(w + h)
    tgt = (rng.random((h, w)) < density).astype(np.uint8) * 255
    tgt[-1, -1] = 1
    img = rng.uniform(0, 255, (h, w, 1)).astype(np.float32)
    src = np.ones((h, w), np.uint8)
    d = _abi.DistanceParams(_abi.NLI_DIST_L2_NORM, 1, 1, 10000.0, 0.3, 0.6)
    before = gpu_ctx.counters()["candidates"]
    nnf, _, _ = gpu_ctx.patchmatch(d, _abi.PatchMatchParams(0, 30, -1), img, src, img, tgt)
    assert gpu_ctx.counters()["candidates"] - before == np.count_nonzero(tgt)
    nnf = nnf.cpu().numpy().reshape(h, w, 2)
    assert np.array_equal(nnf[..., 0] >= 0, tgt != 0)
