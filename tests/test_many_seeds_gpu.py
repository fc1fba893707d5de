"""Calls whose points are mostly seeds: the seeds are ranked by several blocks (by launches of their own
above 262144 points), each of which scans all seed bits."""
import numpy as np
import pytest

from parity_util import gpu_args

pytestmark = pytest.mark.gpu


def _scattered(n, events, seed):
    """Points that are nobody's neighbours; one in three too light for a seed."""
    rng = np.random.default_rng(seed)
    side = int(np.ceil(n ** 0.5))
    grid = rng.permutation(side * side)[:n]
    c = np.stack([grid % side, grid // side]).astype(np.float32)
    w = np.where(rng.random(n) < 0.67, 1.5, 0.5).astype(np.float32)
    off = np.unique(np.concatenate([[0, n], rng.integers(1, n, size=events - 1)])).astype(np.int32)
    return c, w, off


@pytest.mark.parametrize("n,events", [(n, e) for n in (31, 4095, 4096, 4097, 8193, 100_000, 262_144, 262_145)
                                      for e in (1, 30, 1000) if e == 1 or 4 * e <= n])
def test_labels(gpu_context, n, events):
    c, w, off = _scattered(n, events, n + events)
    args = gpu_args(dc=0.5, rhoc=1.0, dm=0.5)
    got, ncl = gpu_context.batch_host(c, w, off, *args)
    seed = w > 1.0
    np.testing.assert_array_equal(got.is_seed, seed.astype(np.int32))
    rank = np.cumsum(seed) - seed
    first = np.repeat(rank[off[:-1]], np.diff(off))
    np.testing.assert_array_equal(got.cluster_index, np.where(seed, rank - first, -1))
    np.testing.assert_array_equal(ncl, np.add.reduceat(seed, off[:-1]))
    assert (got.info.n_seeds, got.info.n_clusters) == (seed.sum(), seed.sum())


def test_label_stage_does_not_grow_with_the_seeds():
    """Stage time of 262144 points, 175k of them seeds: one block alone took 0.14 ms, the stage takes 0.02."""
    import torch
    from cluestering_alpaka3_b200 import capi
    n = 262_144
    c, w, _ = _scattered(n, 1, 1)
    d, dw = torch.from_numpy(c).cuda(), torch.from_numpy(w).cuda()
    lab = torch.empty(n, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    ctx = capi.Context(0)
    try:
        ctx.set_timing(True)
        ms = []
        for _ in range(10):
            ctx.make_clusters_device(d.data_ptr(), dw.data_ptr(), 2, n, {"cluster_index": lab.data_ptr()},
                                     *gpu_args(dc=0.5, rhoc=1.0, dm=0.5))
            ms.append(ctx.stage_times()[3])
        assert min(ms) < 0.07
    finally:
        ctx.close()
