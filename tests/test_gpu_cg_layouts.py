"""The CG's CTA layouts at the sizes where they change: systems of one unknown,
around the one-CTA limit, around the unknowns per thread that the kernels are
compiled for, several CTAs per pixel row (a neighbour's range is then not the
next one), ranges that end in the middle of a row, and the first sizes past a
cluster.  Plain and preconditioned solves against an exact FP64 solve."""
import numpy as np
import pytest
import torch

import update64

pytestmark = pytest.mark.gpu

# image size and the hole's rectangle (x, y, w, h)
CASES = [
    ((40, 40), (20, 20, 1, 1)),        # one unknown
    ((40, 40), (18, 20, 2, 1)),
    ((64, 64), (16, 16, 32, 32)),      # 1024: one CTA
    ((64, 64), (16, 16, 33, 32)),      # 1056: two CTAs
    ((64, 96), (12, 20, 41, 51)),      # 2091: three CTAs of 697
    ((900, 40), (20, 18, 850, 3)),     # ranges of 850: a neighbour per unknown and side in the next CTA
    ((3100, 30), (30, 14, 3000, 2)),   # ranges of 1000: the row below is three CTAs away
    ((160, 160), (13, 15, 131, 127)),  # 16637: 16 CTAs of 1040
    ((240, 240), (20, 20, 201, 201)),  # 40401: 5 per thread
    ((280, 280), (12, 12, 255, 256)),  # 65280: 8 per thread
    ((290, 290), (12, 12, 257, 256)),  # 65792: past a cluster
]


@pytest.mark.parametrize("pre", [0, 1])
@pytest.mark.parametrize("size,rect", CASES)
def test_layouts_against_fp64(gpu_ctx, size, rect, pre):
    from nli_gb300 import workloads as wl
    W, H = size
    x, y, w, h = rect
    rng = np.random.default_rng(W + w)
    img, _ = wl.voronoi_texture(W, H, 12, rng)
    img = np.ascontiguousarray(img[..., :1])
    mask = np.zeros((H, W), np.uint8)
    mask[y:y + h, x:x + w] = 1
    p = wl.params("nlpoisson", scales=1, cg_tol=1e-12, cg_iters=2000)
    ext = gpu_ctx.extended_domain(mask, 9, 9)
    # any field will do: every pixel of the domain copies from a random place
    nnf = np.stack([rng.integers(0, W, (H, W)), rng.integers(0, H, (H, W))], -1).astype(np.int32)
    conf = gpu_ctx.confidence_mask(mask, 5.0, 0.1)
    gpu_ctx.set_tuning(gpu_ctx.TUNE_CG_PRECOND, pre)
    try:
        out, total = gpu_ctx.update(p.update, img, img, mask, ext, nnf, conf)
    finally:
        gpu_ctx.set_tuning(gpu_ctx.TUNE_CG_PRECOND, 0)
    out = out.cpu().numpy().reshape(H, W, 1)
    plan = update64.Plan(nnf, mask != 0, ext.cpu().numpy(), conf.double().cpu().numpy())
    want = update64.poisson_fast(img.astype(np.float64), float(p.update.lambda_), float(p.update.sigma), plan)
    hole = mask != 0
    assert np.array_equal(out[~hole], img[~hole])
    d, dw = out[hole].astype(np.float64) - img[hole], want[hole] - img[hole]
    # |r| < 1e-6 |r0| and a condition number of at most (0.05 + 8 * 0.95) / 0.05
    assert np.linalg.norm(d - dw) <= 2e-4 * np.linalg.norm(dw)
    assert abs(total - (d * d).sum()) <= 1e-5 * (d * d).sum()
