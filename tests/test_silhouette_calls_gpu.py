"""What a silhouette call leaves alone: the caller's scores when a label is out of range, host memory
that it does not need."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bad", [-2, 4000, 2**31 - 1])
@pytest.mark.parametrize("want_mean", [True, False])
def test_scores_untouched_by_a_label_out_of_range(gpu_context, bad, want_mean):
    import torch
    from cluestering_alpaka3_b200 import capi
    n = 4000
    rng = np.random.default_rng(3)
    lab = rng.integers(-1, 5, n).astype(np.int32)
    lab[n - 7] = bad
    c = torch.from_numpy(rng.normal(0, 3, size=(2, n)).astype(np.float32)).cuda()
    d = torch.from_numpy(lab).cuda()
    per = torch.full((n,), -7.0, device="cuda")
    mean = ctypes.c_float(-3.0)
    torch.cuda.synchronize()
    with pytest.raises(capi.ClueOutOfRange):
        capi.check(capi.lib.clue_silhouette(gpu_context.handle, 2, n, ctypes.c_void_p(c.data_ptr()),
                                            ctypes.c_void_p(d.data_ptr()), ctypes.c_void_p(per.data_ptr()),
                                            ctypes.byref(mean) if want_mean else None, None))
    assert bool((per == -7.0).all()) and mean.value == -3.0


def test_pinned_memory_only_for_the_mean():
    """20M points without a mean: no host memory of their size is pinned (it shows as shared memory of
    the process)."""
    import torch
    from cluestering_alpaka3_b200 import capi

    def pinned():
        for line in open("/proc/self/status"):
            if line.startswith("RssShmem"):
                return int(line.split()[1]) << 10
        return 0

    n = 20_000_000
    lab = torch.full((n,), -1, dtype=torch.int32, device="cuda")
    lab[:100] = torch.arange(100, dtype=torch.int32, device="cuda") % 2
    c = torch.rand(2, n, device="cuda")
    torch.cuda.synchronize()
    ctx = capi.Context(0)
    try:
        args = (ctx.handle, 2, n, ctypes.c_void_p(c.data_ptr()), ctypes.c_void_p(lab.data_ptr()), None)
        ctx.cluster_centroids_device(c.data_ptr(), lab.data_ptr(), 2, n, 2, torch.empty(4, device="cuda").data_ptr())
        before = pinned()
        capi.check(capi.lib.clue_silhouette(*args, None, None))
        assert pinned() - before < 5 * n // 2
        mean = ctypes.c_float(np.nan)
        capi.check(capi.lib.clue_silhouette(*args, ctypes.byref(mean), None))
        assert np.isfinite(mean.value)
    finally:
        ctx.close()
