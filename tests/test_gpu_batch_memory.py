"""A lockstep batch holds the tables of PatchMatch's lower bound that its calls
read: one float4 per pixel (means) for the L1 distance, three with the slopes, six
with the deviations (NLI_TUNE_PM_BOUND 2)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIDE = 1000


@pytest.mark.parametrize("method,bound,tables", [("nlmedians", 0, 0), ("nlmedians", 1, 1), ("nlpoisson", 1, 3),
                                                 ("nlpoisson", 2, 6)])
def test_tables_held(gpu_ctx, method, bound, tables):
    import torch
    import __graft_entry__ as ge
    from nli_gb300 import workloads as wl
    pkg = ge.package()
    rng = np.random.default_rng(1)
    img = rng.uniform(0, 255, (SIDE, SIDE, 3)).astype(np.float32)
    mask = np.zeros((SIDE, SIDE), np.uint8)
    mask[400:410, 400:410] = 1
    p = wl.params(method, scales=1, iters=1, pm_iters=1, init="avg")
    used = []
    for b in (0, bound):
        ctx = pkg.Context(0)
        try:
            ctx.set_tuning(ctx.TUNE_PM_BOUND, b)
            torch.cuda.synchronize()
            free = torch.cuda.mem_get_info()[0]
            ctx.process_batch([(img, mask)], [p])
            used.append(free - torch.cuda.mem_get_info()[0])
        finally:
            ctx.close()
    # a buffer is allocated an eighth larger than asked for, and rounded up to 2 MB
    assert abs((used[1] - used[0]) - tables * 16 * (SIDE + 1) ** 2 * 9 / 8) <= 8 << 20
