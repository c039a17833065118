"""NL-medians at the candidate counts where its kernel changes: windows of one
block of 32 candidates and its neighbours, of three blocks (the most of the
smaller kernel) and more, many equal values, and signed zeros, against a
plain restatement (values sorted with ties in candidate order, the weights
subtracted one after the other in float): the same values, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

W, H = 45, 40


def weighted_medians(img, mask, nnf, conf, weights, px, py):
    out = img.copy()
    hx, hy = px // 2, py // 2
    for y, x in zip(*np.nonzero(mask)):
        xa, xb, ya, yb = max(x - hx, 0), min(x + hx, W - 1), max(y - hy, 0), min(y + hy, H - 1)
        vals, ws = [], []
        for i in range(xa, xb + 1):
            for j in range(ya, yb + 1):
                if nnf[j, i, 0] == -1:
                    continue
                qx, qy = nnf[j, i, 0] + x - i, nnf[j, i, 1] + y - j
                if 0 <= qx < W and 0 <= qy < H:
                    w = weights[j - ya, i - xa]
                    vals.append(img[qy, qx])
                    ws.append(np.float32(w * conf[j, i]) if mask[j, i] else w)
        if not vals:
            continue
        vals, ws = np.array(vals, np.float32), np.array(ws, np.float32)
        tw = np.float32(0)
        for w in ws:
            tw = np.float32(tw + w)
        for c in range(img.shape[2]):
            t, half, out[y, x, c] = tw, np.float32(tw / np.float32(2)), 0
            for k in np.argsort(vals[:, c], kind="stable"):
                t = np.float32(t - ws[k])
                if t < half:
                    out[y, x, c] = vals[k, c]
                    break
    return out


# 25, 27, 35, 63, 81, 99, 121 and 225 candidates
@pytest.mark.parametrize("px,py", [(5, 5), (3, 9), (5, 7), (7, 9), (9, 9), (9, 11), (11, 11), (15, 15)])
@pytest.mark.parametrize("values", ["noise", "few", "zeros"])
def test_blocks_against_restatement(gpu_ctx, px, py, values):
    from nli_gb300 import workloads as wl
    rng = np.random.default_rng(px * 16 + py)
    img = rng.uniform(0, 255, (H, W, 3)).astype(np.float32)
    if values == "few":
        img = np.floor(img / 64) * 64
    if values == "zeros":
        img = np.where(img < 128, np.float32(-0.0), np.float32(0.0)) + (img > 200) * np.float32(3.0)
    img = np.ascontiguousarray(img, np.float32)
    mask = np.zeros((H, W), np.uint8)
    mask[16:22, 18:26] = 1
    mask[0:6, 0:5] = 1  # windows clipped at the corner
    p = wl.params("nlmedians", patch=9, psigma=3.0)
    p.update.patch_x, p.update.patch_y = px, py
    ext = gpu_ctx.extended_domain(mask, px, py).cpu().numpy()
    nnf = np.stack([rng.integers(0, W, (H, W)), rng.integers(0, H, (H, W))], -1).astype(np.int32)
    nnf[rng.uniform(size=(H, W)) < 0.05] = -1
    conf = gpu_ctx.confidence_mask(mask, 5.0, 0.1).cpu().numpy()
    out, _ = gpu_ctx.update(p.update, img, img, mask, ext, nnf, conf)
    want = weighted_medians(img, mask, nnf, conf, gpu_ctx.gaussian_weights(px, py, 3.0, 3.0), px, py)
    assert np.array_equal(out.cpu().numpy().reshape(H, W, 3), want)
