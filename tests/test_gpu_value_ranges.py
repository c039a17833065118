"""The adjoints where weights and values lie far from one, against FP64: weight
sums below the smallest normal float, patch sigmas whose derivative lies below
it, and images and confidences scaled up and down."""
import numpy as np
import pytest
import torch

import update64

pytestmark = pytest.mark.gpu

W, H = 37, 29


def field(rng, W=W, H=H):
    return np.stack([rng.integers(0, W, (H, W)), rng.integers(0, H, (H, W))], -1).astype(np.int32)


def params(method, sigma, **kw):
    from nli_gb300 import workloads as wl
    return wl.params(method, scales=1, psigma=sigma, cg_tol=1e-12, cg_iters=2000, **kw).update


def means64(img, sigma, nnf, dom, conf, g):
    u = torch.tensor(img, dtype=torch.float64, requires_grad=True)
    s = torch.tensor(sigma, dtype=torch.float64, requires_grad=True)
    (update64.means(u, s, nnf, dom != 0, conf) * torch.tensor(g, dtype=torch.float64)).sum().backward()
    return u.grad.numpy(), s.grad.item()


def means_ours(ctx, img, sigma, nnf, dom, conf, g):
    gi, _, _, ds = ctx.update_backward(params("nlmeans", sigma), img, img, dom, dom, nnf, conf, g)
    return gi.cpu().numpy().reshape(img.shape).astype(np.float64), ds


# taps that have a match, as offsets from the hole pixel; at sigma 0.42 a corner's
# weight is 3e-40, its neighbour's 1e-31
@pytest.mark.parametrize("taps", [[(-4, -4)], [(-4, -4), (4, 4)], [(-4, -4), (-4, -3)], [(-4, -3), (4, 3)]])
@pytest.mark.parametrize("C", [1, 3])
def test_means_adjoint_subnormal_weights(gpu_ctx, taps, C):
    rng = np.random.default_rng(3)
    img = rng.uniform(0, 255, (H, W, C)).astype(np.float32)
    dom = np.zeros((H, W), np.uint8)
    dom[14, 18] = 1
    nnf = np.full((H, W, 2), -1, np.int32)
    for dx, dy in taps:
        nnf[14 + dy, 18 + dx] = (12 + dx, 10 + dy + 2 * dx)
    g = rng.standard_normal((H, W, C)).astype(np.float32)
    want, ds_want = means64(img, 0.42, nnf, dom, None, g)
    got, ds = means_ours(gpu_ctx, img, 0.42, nnf, dom, None, g)
    # a weight of 3e-40 is a multiple of 1.4e-45
    eps = 1e-5
    assert (np.abs(got - want) <= eps * (1.0 + np.abs(want))).all()
    r2 = 32
    assert abs(ds - ds_want) <= eps * np.abs(g[14, 18]).sum() * 255 * r2 / 0.42 ** 3


def test_means_adjoint_subnormal_confidence(gpu_ctx):
    rng = np.random.default_rng(4)
    img = rng.uniform(0, 255, (H, W, 3)).astype(np.float32)
    dom = np.zeros((H, W), np.uint8)
    dom[8:20, 9:25] = 1
    nnf = field(rng)
    conf = np.full((H, W), 2.0 ** -126, np.float32)
    nnf[dom == 0] = -1
    g = rng.standard_normal((H, W, 3)).astype(np.float32)
    want, ds_want = means64(img, 3.0, nnf, dom, conf.astype(np.float64), g)
    got, ds = means_ours(gpu_ctx, img, 3.0, nnf, dom, conf, g)
    # weights of 2^-131.4 (the middle) to 2^-134 (a corner) on a grid of 2^-149, each half a
    # step off, and the patch weights' own 2^-22
    eps = 2.0 ** -150 / 2.0 ** -134 + 2.0 ** -22
    assert (np.abs(got - want) <= eps * 2 * np.abs(g).max() * 40).all()
    assert abs(ds - ds_want) <= eps * np.abs(g[dom != 0]).sum() * 255 * 32 / 27


@pytest.mark.parametrize("sigma", [1e13, 1e6, 3.0])
@pytest.mark.parametrize("scale", [2.0 ** 119.5, 1.0, 2.0 ** -100])
def test_means_adjoint_scaled(gpu_ctx, sigma, scale):
    rng = np.random.default_rng(5)
    img = (rng.uniform(-255, 255, (H, W, 2)) * scale).astype(np.float32)
    assert np.isfinite(img).all()
    dom = np.zeros((H, W), np.uint8)
    dom[rng.random((H, W)) < 0.3] = 1
    nnf = field(rng)
    g = rng.standard_normal((H, W, 2)).astype(np.float32)
    want, ds_want = means64(img, sigma, nnf, dom, None, g)
    got, ds = means_ours(gpu_ctx, img, sigma, nnf, dom, None, g)
    eps = 16 * 2.0 ** -24  # of the float weights, on the sum of the terms' sizes
    assert (np.abs(got - want) <= eps * 40).all()
    assert abs(ds - ds_want) <= eps * np.abs(g[dom != 0]).astype(np.float64).sum() * 510 * scale * 32 / sigma ** 3


@pytest.mark.parametrize("sigma", [1e13, 3.0])
@pytest.mark.parametrize("scale,conf", [(1.0, 1.0), (2.0 ** 100, 1.0), (2.0 ** -100, 1.0), (1.0, 2.0 ** -70),
                                        (1.0, 2.0 ** 60)])
def test_poisson_adjoint_scaled(gpu_ctx, sigma, scale, conf):
    """dL/du does not depend on the image's scale (the step is linear in it) nor
    on the confidence's (it cancels), dL/dsigma follows the image's."""
    rng = np.random.default_rng(6)
    img = (rng.uniform(0, 255, (H, W, 2)) * scale).astype(np.float32)
    dom = np.zeros((H, W), np.uint8)
    dom[6:18, 5:20] = 1
    ext = gpu_ctx.extended_domain(dom, 9, 9).cpu().numpy()
    nnf = field(rng)
    cf = (rng.uniform(0.1, 1, (H, W)) * conf).astype(np.float32)
    g = (rng.standard_normal((H, W, 2)) * (dom != 0)[..., None]).astype(np.float32)
    u = torch.tensor(img / scale, dtype=torch.float64, requires_grad=True)
    s = torch.tensor(sigma, dtype=torch.float64, requires_grad=True)
    out = update64.poisson(u, 0.05, s, nnf, dom != 0, ext, cf.astype(np.float64) / conf)
    (out * torch.tensor(g, dtype=torch.float64)).sum().backward()
    p = params("nlpoisson", sigma, lam=0.05)
    o32 = (out.detach().numpy() * scale).astype(np.float32)
    gi, _, _, ds = gpu_ctx.update_backward(p, img, o32, dom, ext, nnf, cf, g)
    gi = gi.cpu().numpy().reshape(H, W, 2).astype(np.float64)
    want = u.grad.numpy()
    # the solve's |r| < 1e-6 |r0| with a condition number of 153, as tests of the adjoint allow
    assert np.linalg.norm(gi - want) <= 1e-4 * np.linalg.norm(want)
    assert abs(ds / scale - s.grad.item()) <= 1e-3 * abs(s.grad.item())
