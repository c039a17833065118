"""Groups of target points in the PatchMatch kernels: how many points a warp
takes at a time follows from the call's size and search window, and the
lower bound's slopes from its size, but a point's match must not.  A call on
all target points (groups of three, two or one) and one on a part of them
(one point per group) are compared after a sweep on the points whose
neighbours are the same in both: bit for bit, with the source mask, the
random streams and the images shared."""
import numpy as np
import pytest

from nli_gb300 import _abi

pytestmark = pytest.mark.gpu

W, H = 170, 140
JUMP = 16  # of the first sweep


def scene(C):
    from nli_gb300 import workloads as wl
    rng = np.random.default_rng(40 + C)
    img, _ = wl.voronoi_texture(W, H, 14, rng)
    if C == 4:
        img = np.concatenate([img, rng.uniform(0.5, 5, (H, W, 1)).astype(np.float32)], -1)
    return np.ascontiguousarray(img[..., :C])


def masks(P):
    r = P // 2
    inside = np.zeros((H, W), np.uint8)
    inside[r:H - r, r:W - r] = 1
    src = inside.copy()
    src[H // 3:H // 3 + 30, W // 3:W // 3 + 40] = 0  # some draws are refused
    part = np.zeros_like(inside)
    part[20:101, 30:111] = inside[20:101, 30:111]
    # points whose neighbours at distance 1 and JUMP are all in the part
    same = np.zeros_like(inside)
    same[20 + JUMP:101 - JUMP, 30 + JUMP:111 - JUMP] = 1
    return src, inside, part, same != 0


# window 2000: 11 search windows (two points per group at most); 100000: 17 (one)
@pytest.mark.parametrize("kind,C,P,window", [
    (_abi.NLI_DIST_L2_COMBINED, 3, 9, -1), (_abi.NLI_DIST_L2_COMBINED, 3, 9, 2000),
    (_abi.NLI_DIST_L2_COMBINED, 3, 9, 100000), (_abi.NLI_DIST_L2_COMBINED, 1, 7, -1),
    (_abi.NLI_DIST_L2_COMBINED, 2, 5, -1), (_abi.NLI_DIST_L2_RGBD, 4, 9, -1), (_abi.NLI_DIST_L2_RGBD, 4, 11, -1),
    (_abi.NLI_DIST_L2_NORM, 3, 7, -1), (_abi.NLI_DIST_L2_NORM, 4, 15, 2000), (_abi.NLI_DIST_L1_NORM, 3, 5, -1),
    (_abi.NLI_DIST_L1_NORM, 3, 3, -1)])
def test_matches_do_not_depend_on_grouping(gpu_ctx, kind, C, P, window):
    img = scene(C)
    src, full, part, same = masks(P)
    assert full.sum() >= 3 * 16 * 152 > part.sum()  # grouped, one by one
    d = _abi.DistanceParams(kind, P, P, 10000.0, 0.3, 0.6)
    for sweeps in (0, 1):
        pm = _abi.PatchMatchParams(sweeps, 30, window)
        out = []
        for tgt in (full, part):
            gpu_ctx.set_seed(7)
            nnf, dist, _ = gpu_ctx.patchmatch(d, pm, img, src, img, tgt)
            out.append((nnf.cpu().numpy().reshape(H, W, 2), dist.cpu().numpy().reshape(H, W)))
        where = part != 0 if sweeps == 0 else same
        assert np.array_equal(out[0][0][where], out[1][0][where])
        assert np.array_equal(out[0][1][where], out[1][1][where])
        assert (out[0][0][where] >= 0).any()


@pytest.mark.parametrize("points", [1, 2, 3, 4, 7295, 7296, 7297])
def test_every_point_is_visited_once(gpu_ctx, points):
    """Target counts around a group and around the line between one and
    three points per group: every target point gets a match whose distance
    is that of the two patches, no other pixel is touched."""
    img = scene(3)
    src, full, _, _ = masks(9)
    ys, xs = np.nonzero(full)
    tgt = np.zeros_like(full)
    tgt[ys[:points], xs[:points]] = 1
    d = _abi.DistanceParams(_abi.NLI_DIST_L2_COMBINED, 9, 9, 10000.0, 0.3, 0.6)
    gpu_ctx.set_seed(11)
    nnf, dist, _ = gpu_ctx.patchmatch(d, _abi.PatchMatchParams(2, 30, -1), img, src, img, tgt)
    nnf, dist = nnf.cpu().numpy().reshape(H, W, 2), dist.cpu().numpy().reshape(H, W)
    on = tgt != 0
    assert (nnf[~on] == -1).all() and (dist[~on] == np.finfo(np.float32).max).all()
    assert (nnf[on] >= 0).all()
    ty, tx = np.nonzero(on)
    pairs = np.stack([nnf[on][:, 0], nnf[on][:, 1], tx, ty], 1).astype(np.int32)
    want = gpu_ctx.distance_pairs(d, img, img, pairs).cpu().numpy()
    # 31 * 81 operations on floats of one sign: relative error below 2600 * 2^-24
    assert np.allclose(dist[on], want, rtol=2e-4, atol=1e-6)
