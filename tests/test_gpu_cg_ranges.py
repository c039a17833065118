"""Systems beyond a cluster whose sums leave the range of single floats: images
scaled by up to 2^60 and down to 2^-100 against an exact FP64 solve, and the
adjoint of scaled gradients against that of the unscaled ones, plain and
preconditioned, one channel and three side by side."""
import numpy as np
import pytest

import update64

pytestmark = pytest.mark.gpu


def field(rng, W, H):
    return np.stack([rng.integers(0, W, (H, W)), rng.integers(0, H, (H, W))], -1).astype(np.int32)


def params(method, sigma, **kw):
    from nli_gb300 import workloads as wl
    return wl.params(method, scales=1, psigma=sigma, cg_tol=1e-12, cg_iters=2000, **kw).update


def large_case(C):
    """65792 unknowns a channel, past what a cluster takes."""
    from nli_gb300 import workloads as wl
    n = 290
    rng = np.random.default_rng(7)
    img, _ = wl.voronoi_texture(n, n, 12, rng)
    img = np.ascontiguousarray(img[..., :C])
    mask = np.zeros((n, n), np.uint8)
    mask[12:12 + 256, 12:12 + 257] = 1
    return img, mask, field(rng, n, n)


@pytest.mark.parametrize("pre", [0, 1])
@pytest.mark.parametrize("scale", [2.0 ** 60, 2.0 ** 30, 1.0, 2.0 ** -40, 2.0 ** -70, 2.0 ** -100])
def test_large_solve_scaled(gpu_ctx, scale, pre):
    img, mask, nnf = large_case(1)
    ext = gpu_ctx.extended_domain(mask, 9, 9)
    conf = gpu_ctx.confidence_mask(mask, 5.0, 0.1)
    p = params("nlpoisson", 10000.0)
    scaled = img * np.float32(scale)
    gpu_ctx.set_tuning(gpu_ctx.TUNE_CG_PRECOND, pre)
    try:
        out, _ = gpu_ctx.update(p, scaled, scaled, mask, ext, nnf, conf)
    finally:
        gpu_ctx.set_tuning(gpu_ctx.TUNE_CG_PRECOND, 0)
    out = out.cpu().numpy().reshape(img.shape).astype(np.float64) / scale
    plan = update64.Plan(nnf, mask != 0, ext.cpu().numpy(), conf.double().cpu().numpy())
    want = update64.poisson_fast(img.astype(np.float64), float(p.lambda_), float(p.sigma), plan)
    hole = mask != 0
    d, dw = out[hole] - img[hole], want[hole] - img[hole]
    # |r| < 1e-6 |r0| and a condition number of at most (0.05 + 8 * 0.95) / 0.05
    assert np.linalg.norm(d - dw) <= 2e-4 * np.linalg.norm(dw)


@pytest.mark.parametrize("scale", [2.0 ** 70, 2.0 ** -70])
def test_large_adjoint_is_linear(gpu_ctx, scale):
    img, mask, nnf = large_case(3)
    ext = gpu_ctx.extended_domain(mask, 9, 9)
    conf = gpu_ctx.confidence_mask(mask, 5.0, 0.1)
    p = params("nlpoisson", 10000.0)
    rng = np.random.default_rng(8)
    g = (rng.standard_normal(img.shape) * (mask != 0)[..., None]).astype(np.float32)
    out, _ = gpu_ctx.update(p, img, img, mask, ext, nnf, conf)
    res = []
    for s in (1.0, scale):
        gi, gl, _, gs = gpu_ctx.update_backward(p, img, out, mask, ext, nnf, conf, g * np.float32(s))
        res.append((gi.double().cpu().numpy() / s, gl / s, gs / s))
    (a, la, sa), (b, lb, sb) = res
    # two solves, each off by at most 1.5e-4 of z; the gathers' transpose takes that to
    # the image within a factor of 30
    assert np.linalg.norm(a - b) <= 1e-2 * np.linalg.norm(a)
    assert abs(la - lb) <= 1e-2 * abs(la) and abs(sa - sb) <= 1e-2 * abs(sa)
