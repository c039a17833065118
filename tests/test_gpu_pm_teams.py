"""PatchMatch calls of few points, where four or two warps share a point: the
matches must be those of the same points in a large call.  The small call's
points lie further from the large call's other points than any step of
propagation reaches, and the source mask, the random streams and the images
are shared, so the comparison is bit for bit after several sweeps."""
import numpy as np
import pytest

from nli_gb300 import _abi

pytestmark = pytest.mark.gpu

W, H = 170, 140
JUMP = 16  # the longest step, of the first sweep


# on 152 SMs: the last count that four warps share, the first of two, their
# last, and the first of none
@pytest.mark.parametrize("points", [1, 2, 911, 912, 913, 1824, 1825])
@pytest.mark.parametrize("kind,C,P,window,shots", [
    (_abi.NLI_DIST_L2_COMBINED, 3, 9, -1, 30), (_abi.NLI_DIST_L2_COMBINED, 3, 9, 1, 3),
    (_abi.NLI_DIST_L2_COMBINED, 1, 5, 100000, 1), (_abi.NLI_DIST_L2_RGBD, 4, 9, -1, 30),
    (_abi.NLI_DIST_L2_NORM, 3, 7, 2000, 30), (_abi.NLI_DIST_L1_NORM, 2, 3, -1, 30),
    (_abi.NLI_DIST_L1_NORM, 3, 15, -1, 30)])
def test_matches_do_not_depend_on_teams(gpu_ctx, kind, C, P, window, shots, points):
    from nli_gb300 import workloads as wl
    rng = np.random.default_rng(50 + C)
    img, _ = wl.voronoi_texture(W, H, 14, rng)
    if C == 4:
        img = np.concatenate([img, rng.uniform(0.5, 5, (H, W, 1)).astype(np.float32)], -1)
    img = np.ascontiguousarray(img[..., :C])
    r = P // 2
    inside = np.zeros((H, W), np.uint8)
    inside[r:H - r, r:W - r] = 1
    src = inside.copy()
    src[60:120, 20:120] = 0  # some draws are refused
    few = np.zeros_like(inside)
    top = max(r - 1, 0)  # a row whose patches leave the image, then rows with some that do
    few[top:top + 13].ravel()[:points] = 1
    many = few.copy()
    many[top + 13 + JUMP:] = inside[top + 13 + JUMP:]
    assert many.sum() >= 3 * 16 * 152
    d = _abi.DistanceParams(kind, P, P, 10000.0, 0.3, 0.6)
    out = []
    for tgt in (many, few):
        gpu_ctx.set_seed(9)
        nnf, dist, _ = gpu_ctx.patchmatch(d, _abi.PatchMatchParams(3, shots, window), img, src, img, tgt)
        out.append((nnf.cpu().numpy().reshape(H, W, 2), dist.cpu().numpy().reshape(H, W)))
    on = few != 0
    assert np.array_equal(out[0][0][on], out[1][0][on])
    assert np.array_equal(out[0][1][on], out[1][1][on])
    assert (out[1][0][~on] == -1).all()
    assert points < 911 or (out[1][0][on] >= 0).any()
