"""Contexts kept for the next create: same results, default settings, nothing of the last owner, several
threads, bounded memory."""
import threading

import numpy as np
import pytest

from parity_util import assert_exact, gpu_args, random_blobs, run_both

pytestmark = pytest.mark.gpu


def test_next_context_is_as_new():
    from cluestering_alpaka3_b200 import capi
    rng = np.random.default_rng(1)
    c, w = random_blobs(rng, 3000, 2, nblobs=5, extent=40.0)
    defaults = None
    for k in range(6):
        ctx = capi.Context(0)
        defaults = defaults or ctx.tuning()
        assert ctx.tuning() == defaults and ctx.kernel_launches == 0
        with pytest.raises(capi.ClueError):
            ctx.read_info()  # no run of this context yet
        with pytest.raises(capi.ClueError):
            ctx.near_counts()
        with pytest.raises(capi.ClueError):
            ctx.stage_times()
        assert_exact(*run_both(ctx, c, w, dc=1.0, rhoc=2.0, dm=1.5))
        ctx.set_tuning(nh_split_lanes=k, symmetric_density=0)
        ctx.set_timing(True)
        assert_exact(*run_both(ctx, c[:, :500], w[:500], dc=1.0, rhoc=2.0, dm=1.5))
        ctx.close()


def test_threads_and_memory_bound():
    import torch
    from cluestering_alpaka3_b200 import capi
    rng = np.random.default_rng(2)
    c, w = random_blobs(rng, 4000, 2, nblobs=6, extent=40.0)
    args = gpu_args(dc=1.0, rhoc=2.0, dm=1.5)
    first = capi.Context(0)
    want = first.make_clusters_host(c, w, *args)
    first.close()
    bad = []

    def work(seed):
        try:
            for k in range(8):
                ctx = capi.Context(0)
                m = 4000 - 37 * ((seed + k) % 5)
                got = ctx.make_clusters_host(c[:, :m], w[:m], *args)
                if m == 4000 and not np.array_equal(got.cluster_index, want.cluster_index):
                    bad.append((seed, k))
                ctx.close()
        except Exception as e:  # noqa: BLE001 (a thread's failure is the test's)
            bad.append((seed, e))

    threads = [threading.Thread(target=work, args=(s,)) for s in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
    # a large context is not kept
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    big = capi.Context(0)
    big.reserve(2, 4_000_000)
    assert big.workspace_bytes > 64 << 20
    big.close()
    assert free - torch.cuda.mem_get_info()[0] < 64 << 20
