"""PatchMatch targets with sides above 65535, which the entry point takes (only
source sides are limited): every target point's distance must be that of its own
patch and its match's, and the default kernels (grouped, four and two warps per
point) must find the one-point kernels' field, on both sides of the 16-bit line."""
import numpy as np
import pytest

from nli_gb300 import _abi

pytestmark = pytest.mark.gpu

SW, SH = 60, 50


# 24 rows or columns hold 16 points across: 912 of them are the last that four warps
# share on 152 SMs, 1824 of two, beyond 7296 a warp takes three
@pytest.mark.parametrize("along", [30, 100, 600, 0])
@pytest.mark.parametrize("shape", [(65536, 24), (65537, 24), (70000, 24), (24, 70000)])
def test_wide_target(gpu_ctx, shape, along):
    W, H = shape
    rng = np.random.default_rng(W + along)
    src = rng.uniform(0, 255, (SH, SW, 3)).astype(np.float32)
    tgt = rng.uniform(0, 255, (H, W, 3)).astype(np.float32)
    smask = np.zeros((SH, SW), np.uint8)
    smask[4:-4, 4:-4] = 1
    tmask = np.zeros((H, W), np.uint8)
    inside = tmask[4:-4, 4:-4] if W > H else tmask[4:-4, 4:-4].T
    n = inside.shape[1]
    line = 65536 - 4
    # points on both sides of the line (as far as there are any), and the last ones
    inside[:, min(line - along // 2, n - along) if along else 0:line + along // 2 if along else n] = 1
    inside[:, -3:] = 1
    d = _abi.DistanceParams(_abi.NLI_DIST_L2_COMBINED, 9, 9, 10000.0, 0.3, 0.0)
    pm = _abi.PatchMatchParams(3, 30, -1)
    out = []
    for variant in (0, 2):
        gpu_ctx.set_tuning(gpu_ctx.TUNE_PM_VARIANT, variant)
        try:
            gpu_ctx.set_seed(21)
            nnf, dist, _ = gpu_ctx.patchmatch(d, pm, src, smask, tgt, tmask)
        finally:
            gpu_ctx.set_tuning(gpu_ctx.TUNE_PM_VARIANT, 0)
        out.append((nnf.cpu().numpy().reshape(H, W, 2), dist.cpu().numpy().reshape(H, W)))
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
    nnf, dist = out[0]
    ty, tx = np.nonzero(tmask)
    assert (nnf[ty, tx] >= 0).all()
    pairs = np.stack([nnf[ty, tx, 0], nnf[ty, tx, 1], tx, ty], 1).astype(np.int32)
    want = gpu_ctx.distance_pairs(d, src, tgt, pairs).cpu().numpy()
    # 31 * 81 operations on floats of one sign: relative error below 2600 * 2^-24
    assert np.allclose(dist[ty, tx], want, rtol=2e-4, atol=1e-6)
