"""The counts of evaluated candidates and of those at their point's match by the
early-termination test say the same for the three ways the 9x9 kernels work (in
teams, one point or up to three points per warp; and the one-point variants)."""
import numpy as np
import pytest

from nli_gb300 import _abi
from test_gpu_pm_variants import npy, run_all, scene

pytestmark = pytest.mark.gpu


# 152 SMs: teams up to 1824 points, one point per group up to 4864, then two and three
@pytest.mark.parametrize("points", [300, 1500, 4000, 6000, 9000])
@pytest.mark.parametrize("kind,C", [(_abi.NLI_DIST_L2_COMBINED, 3), (_abi.NLI_DIST_L2_RGBD, 4),
                                    (_abi.NLI_DIST_L1_NORM, 1)])
@pytest.mark.parametrize("bound", [0, 1])
def test_counts_do_not_depend_on_the_variant(gpu_ctx, kind, C, points, bound):
    img, _ = scene(C, 70 + C, 130, 100, 10)
    src = np.zeros((100, 130), np.uint8)
    src[4:-4, 4:-4] = 1
    tgt = np.zeros_like(src)
    ys, xs = np.nonzero(src)
    tgt[ys[:points], xs[:points]] = 1
    d = _abi.DistanceParams(kind, 9, 9, 3.0, 0.4, 0.3)
    other = np.ascontiguousarray(img[::-1])

    def one():
        before = gpu_ctx.counters()
        gpu_ctx.set_seed(5)
        nnf, dist, _ = gpu_ctx.patchmatch(d, _abi.PatchMatchParams(4, 30, -1), other, src, img, tgt)
        after = gpu_ctx.counters()
        return npy(nnf), npy(dist), [after[k] - before[k] for k in ("candidates", "candidates_partial")]

    gpu_ctx.set_tuning(gpu_ctx.TUNE_PM_BOUND, bound)
    try:
        runs = run_all(gpu_ctx, one)
    finally:
        gpu_ctx.set_tuning(gpu_ctx.TUNE_PM_BOUND, 1)
    for nnf, dist, counts in runs:
        assert np.array_equal(nnf, runs[0][0]) and np.array_equal(dist, runs[0][1])
        assert counts == runs[0][2]
    assert 0 < runs[0][2][1] < runs[0][2][0]
