"""The slope stage of PatchMatch's lower bound, which calls of 48 points per SM
and more use: fields, distances and energy bit for bit those of evaluating every
candidate, on fields that have converged over several sweeps and a warm start
(where the bound is tight), for the L2 kinds on one to four channels, flat and
narrow weights, and square, even and non-square patches."""
import numpy as np
import pytest

from nli_gb300 import _abi
from test_gpu_pm_bound import both, npy

pytestmark = pytest.mark.gpu

W, H = 150, 120


def scene(C, noise):
    from nli_gb300 import workloads as wl
    rng = np.random.default_rng(60 + C)
    img, _ = wl.voronoi_texture(W, H, 12, rng)
    if C == 4:
        img = np.concatenate([img, rng.uniform(0.5, 5, (H, W, 1)).astype(np.float32)], -1)
    img = np.ascontiguousarray(img[..., :C])
    return (img + rng.normal(0, noise, img.shape)).astype(np.float32) if noise else img


@pytest.mark.parametrize("noise", [0.0, 3.0])
@pytest.mark.parametrize("sigma", [10000.0, 2.5])
@pytest.mark.parametrize("kind,C,px,py", [
    (_abi.NLI_DIST_L2_COMBINED, 3, 9, 9), (_abi.NLI_DIST_L2_COMBINED, 1, 9, 9), (_abi.NLI_DIST_L2_COMBINED, 2, 7, 7),
    (_abi.NLI_DIST_L2_COMBINED, 4, 5, 5), (_abi.NLI_DIST_L2_COMBINED, 3, 8, 8), (_abi.NLI_DIST_L2_COMBINED, 3, 11, 4),
    (_abi.NLI_DIST_L2_COMBINED, 3, 1, 7), (_abi.NLI_DIST_L2_RGBD, 4, 9, 9), (_abi.NLI_DIST_L2_RGBD, 4, 6, 13),
    (_abi.NLI_DIST_L2_NORM, 3, 9, 9), (_abi.NLI_DIST_L2_NORM, 1, 4, 4), (_abi.NLI_DIST_L2_NORM, 2, 15, 15),
    (_abi.NLI_DIST_L2_NORM, 4, 3, 10)])
def test_fields_are_those_of_every_candidate(gpu_ctx, kind, C, px, py, sigma, noise):
    img = scene(C, noise)
    rx, ry = px // 2, py // 2
    inside = np.zeros((H, W), np.uint8)
    inside[ry:H - ry, rx:W - rx] = 1
    src = inside.copy()
    src[40:75, 50:100] = 0  # targets in here cannot match themselves
    assert inside.sum() >= 48 * 152
    d = _abi.DistanceParams(kind, px, py, sigma, 0.3, 0.6)
    # the source is another image, so that no distance is 0
    other = np.ascontiguousarray(img[::-1, ::-1])

    def run():
        gpu_ctx.set_seed(31)
        nnf, dist, e = gpu_ctx.patchmatch(d, _abi.PatchMatchParams(6, 30, -1), other, src, img, inside)
        gpu_ctx.set_seed(32)
        warm = gpu_ctx.patchmatch(d, _abi.PatchMatchParams(3, 30, -1), other, src, img, inside, init=nnf)
        return [npy(nnf), npy(dist), e, npy(warm[0]), npy(warm[1]), warm[2]]

    (off, n_off), (on, n_on), (dev, n_dev) = both(gpu_ctx, run)
    for a, b, c in zip(off, on, dev):
        assert np.array_equal(np.asarray(a), np.asarray(b))
        assert np.array_equal(np.asarray(a), np.asarray(c))
    assert (off[0].reshape(H, W, 2)[inside != 0] >= 0).all()
    assert n_dev <= n_on < n_off
