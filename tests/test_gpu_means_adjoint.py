"""The NL-means adjoint's warp per pixel at its edges: one to four channels,
patches of fewer and of more taps than a warp has lanes, windows clipped at
the corners, pixels without any valid candidate and single-pixel holes,
against FP64 autograd of the FP64 step."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

W, H = 37, 29


@pytest.mark.parametrize("C", [1, 2, 3, 4])
@pytest.mark.parametrize("px,py", [(1, 1), (5, 5), (5, 7), (9, 9), (11, 3)])
@pytest.mark.parametrize("hole", ["pixel", "corner", "spread"])
def test_against_fp64_autograd(gpu_ctx, C, px, py, hole):
    import torch
    import update64
    from nli_gb300 import workloads as wl
    rng = np.random.default_rng(100 * C + px)
    img = rng.uniform(0, 255, (H, W, C)).astype(np.float32)
    dom = np.zeros((H, W), np.uint8)
    if hole == "pixel":
        dom[14, 18] = 1
    elif hole == "corner":
        dom[:6, :7] = 1
    else:
        dom[rng.random((H, W)) < 0.3] = 1
    nnf = np.stack([rng.integers(0, W, (H, W)), rng.integers(0, H, (H, W))], -1).astype(np.int32)
    nnf[rng.random((H, W)) < 0.2] = -1
    conf = rng.uniform(0.1, 1, (H, W)).astype(np.float32)
    sigma = 3.0
    p = wl.params("nlmeans", patch=9, psigma=sigma).update
    p.patch_x, p.patch_y = px, py
    g = rng.standard_normal((H, W, C)).astype(np.float32)
    out = img.copy()
    gi, _, _, ds = gpu_ctx.update_backward(p, img, out, dom, dom, nnf, conf, g)
    u = torch.tensor(img, dtype=torch.float64, requires_grad=True)
    s = torch.tensor(sigma, dtype=torch.float64, requires_grad=True)
    (update64.means(u, s, nnf, dom != 0, conf, px, py) * torch.tensor(g, dtype=torch.float64)).sum().backward()
    want, got = u.grad.numpy(), gi.cpu().numpy().reshape(H, W, C).astype(np.float64)
    # the float weights: argument, exponential, division and confidence give 6 * 2^-24
    # each, the ratio to their sum twice that, the result's rounding one more,
    # on the sum of the terms' sizes
    eps = 16 * 2.0 ** -24
    a = torch.tensor(img, dtype=torch.float64, requires_grad=True)
    (update64.means(a, sigma, nnf, dom != 0, conf, px, py) * torch.tensor(np.abs(g), dtype=torch.float64)).sum().backward()
    assert (np.abs(got - want) <= eps * a.grad.numpy() + 1e-12).all()
    # per pixel and channel at most |g| |rho - m| |u - out|
    r2 = (px // 2) ** 2 + (py // 2) ** 2
    scale = np.abs(g[dom != 0]).sum() * r2 / sigma ** 3 * 255
    assert abs(ds - (s.grad.item() if s.grad is not None else 0.0)) <= eps * scale + 1e-12
