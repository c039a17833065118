"""The NL-Poisson solvers of the largest systems: the grid kernel with its vectors
in memory and its bounded grid barrier (images wider than 65535 pixels, and more
unknowns than the SMs hold) against an exact FP64 solve, through a barrier that
times out, and in the captured loop and a batch; and systems whose channels are
solved by several launches (ranges of up to 4096 unknowns on 152 SMs hold three
channels of 204800 at once, two of 311296), or by the launch with double sums for
some of the channels, against the same channels one by one."""
import numpy as np
import pytest

import update64
from test_gpu_graph_loop import same

pytestmark = pytest.mark.gpu

WIDE, H, CROP = 65600, 16, 720


def wide_case(C, seed=1):
    """An image of 65600 x 16 whose hole (6000 pixels) and matches lie in its
    last 720 columns, and the same case cropped to these."""
    rng = np.random.default_rng(seed)
    img = rng.uniform(0, 255, (H, CROP, C)).astype(np.float32)
    mask = np.zeros((H, CROP), np.uint8)
    mask[3:13, 60:660] = 1
    ext = np.zeros_like(mask)
    ext[:, 56:664] = 1
    nnf = np.stack([rng.integers(20, CROP, (H, CROP)), rng.integers(0, H, (H, CROP))], -1).astype(np.int32)
    conf = rng.uniform(0.2, 1, (H, CROP)).astype(np.float32)
    off = WIDE - CROP

    def put(a, fill=0):
        out = np.full((H, WIDE) + a.shape[2:], fill, a.dtype)
        out[:, off:] = a
        return out

    shifted = nnf + np.array([off, 0], np.int32)
    return (img, mask, ext, nnf, conf), (put(img), put(mask), put(ext), put(shifted, -1), put(conf))


def params(**kw):
    from nli_gb300 import workloads as wl
    return wl.params("nlpoisson", scales=1, cg_tol=1e-12, cg_iters=2000, **kw)


@pytest.mark.parametrize("pre", [0, 1])
@pytest.mark.parametrize("C", [1, 3])
def test_grid_kernel_against_fp64(gpu_ctx, C, pre):
    (img, mask, ext, nnf, conf), wide = wide_case(C)
    p = params().update
    gpu_ctx.set_tuning(gpu_ctx.TUNE_CG_PRECOND, pre)
    gpu_ctx.set_tuning(gpu_ctx.TUNE_CG_UNKNOWNS_PER_CTA, 1 << 30)
    try:
        out, total = gpu_ctx.update(p, wide[0], wide[0], *wide[1:])
    finally:
        gpu_ctx.set_tuning(gpu_ctx.TUNE_CG_UNKNOWNS_PER_CTA, 1024)
        gpu_ctx.set_tuning(gpu_ctx.TUNE_CG_PRECOND, 0)
    out = out.cpu().numpy().reshape(H, WIDE, C)
    assert np.array_equal(out[wide[1] == 0], wide[0][wide[1] == 0])
    out = out[:, WIDE - CROP:]
    plan = update64.Plan(nnf, mask != 0, ext, conf.astype(np.float64))
    want = update64.poisson_fast(img.astype(np.float64), float(p.lambda_), float(p.sigma), plan)
    hole = mask != 0
    d, dw = out[hole].astype(np.float64) - img[hole], want[hole] - img[hole]
    # |r| < 1e-6 |r0| and a condition number of at most (0.05 + 8 * 0.95) / 0.05 times the
    # coefficients' spread, which random confidences of 81 taps keep below 3
    assert np.linalg.norm(d - dw) <= 6e-4 * np.linalg.norm(dw)
    assert abs(total - (d * d).sum()) <= 1e-5 * (d * d).sum()


def test_grid_kernel_timeout_and_recovery(gpu_ctx):
    from nli_gb300 import NliError
    ctx = gpu_ctx
    _, wide = wide_case(1)
    p = params().update
    ctx.set_tuning(ctx.TUNE_CG_UNKNOWNS_PER_CTA, 1 << 30)
    try:
        clean, t_clean = ctx.update(p, wide[0], wide[0], *wide[1:])
        ctx.grid_wait_limit(1)
        with pytest.raises(NliError) as e:
            ctx.update(p, wide[0], wide[0], *wide[1:])
        assert e.value.status == -7 and "timed out" in str(e.value)  # NLI_E_TIMEOUT
        ctx.grid_wait_limit(0)
        again, t_again = ctx.update(p, wide[0], wide[0], *wide[1:])
    finally:
        ctx.grid_wait_limit(0)
        ctx.set_tuning(ctx.TUNE_CG_UNKNOWNS_PER_CTA, 1024)
    assert np.array_equal(again.cpu().numpy(), clean.cpu().numpy())
    assert t_again == t_clean


@pytest.mark.parametrize("pre", [0, 1])
def test_grid_kernel_in_graph_and_batch(gpu_ctx, pre):
    """630 000 unknowns a channel, beyond what 152 SMs hold, in whole runs."""
    from nli_gb300 import workloads as wl
    rng = np.random.default_rng(2)
    img, _ = wl.voronoi_texture(960, 760, 20, rng)
    img = np.ascontiguousarray(img[..., :1])
    mask = np.zeros((760, 960), np.uint8)
    mask[30:730, 30:930] = 1
    assert mask.sum() > 152 * 4096
    p = wl.params("nlpoisson", scales=1, iters=3, tol=0.0, cg_tol=1e-12, cg_iters=4, pm_iters=1, init="avg")

    def run(graph):
        gpu_ctx.set_tuning(gpu_ctx.TUNE_GRAPH_LOOP, graph)
        gpu_ctx.set_seed(gpu_ctx.batch_seed(5, 0))
        n = gpu_ctx.launch_count()
        out, st = gpu_ctx.process(img, mask, p)
        return out, st, gpu_ctx.launch_count() - n

    gpu_ctx.set_tuning(gpu_ctx.TUNE_CG_PRECOND, pre)
    try:
        captured, host = run(1), run(0)
        gpu_ctx.set_tuning(gpu_ctx.TUNE_GRAPH_LOOP, 1)
        gpu_ctx.set_seed(5)
        batch, _ = gpu_ctx.process_batch([(img, mask)], [p])
    finally:
        gpu_ctx.set_tuning(gpu_ctx.TUNE_GRAPH_LOOP, 1)
        gpu_ctx.set_tuning(gpu_ctx.TUNE_CG_PRECOND, 0)
    same(captured, host)
    assert np.array_equal(batch[0], host[0])
    assert not np.array_equal(host[0], img)


@pytest.mark.parametrize("pre", [0, 1])
@pytest.mark.parametrize("n,C,scales", [
    (460, 3, (1, 1, 1)),                      # 211600: two channels, then one
    (460, 4, (1, 1, 1, 1)),                   # two and two
    (559, 3, (1, 1, 1)),                      # 312481: one after the other
    (460, 3, (2.0 ** -70, 1, 2.0 ** 60)),     # doubles for the first and the last
    (300, 3, (1, 2.0 ** -70, 0)),             # side by side; nothing to solve in the last
])
def test_channels_as_one_by_one(gpu_ctx, n, C, scales, pre):
    size = n + 24
    rng = np.random.default_rng(n + C)
    img = rng.uniform(0, 255, (size, size, C)).astype(np.float32) * np.array(scales, np.float32)
    mask = np.zeros((size, size), np.uint8)
    mask[12:12 + n, 12:12 + n] = 1
    ext = gpu_ctx.extended_domain(mask, 9, 9)
    nnf = np.stack([rng.integers(0, size, (size, size)), rng.integers(0, size, (size, size))], -1).astype(np.int32)
    conf = gpu_ctx.confidence_mask(mask, 5.0, 0.1)
    p = params().update
    gpu_ctx.set_tuning(gpu_ctx.TUNE_CG_PRECOND, pre)
    try:
        out = gpu_ctx.update(p, img, img, mask, ext, nnf, conf)[0].cpu().numpy().reshape(img.shape)
        one = [gpu_ctx.update(p, c, c, mask, ext, nnf, conf)[0].cpu().numpy().reshape(c.shape)
               for c in (np.ascontiguousarray(img[..., k:k + 1]) for k in range(C))]
    finally:
        gpu_ctx.set_tuning(gpu_ctx.TUNE_CG_PRECOND, 0)
    hole = mask != 0
    assert np.array_equal(out[~hole], img[~hole])
    for k in range(C):
        a = out[hole][:, k].astype(np.float64) - img[hole][:, k]
        b = one[k][hole][:, 0].astype(np.float64) - img[hole][:, k]
        if scales[k] == 0:
            assert (a == 0).all()
            continue
        # each |r| < 1e-6 |r0| with a condition number of at most 153
        assert np.linalg.norm(a - b) <= 4e-4 * np.linalg.norm(b) and np.linalg.norm(b) > 0
