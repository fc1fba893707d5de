"""The one-launch first stage (single events of up to 131072 points, small batches): sizes around its clusters, tile counts around
its radix digits, and the same bits as the separate launches that larger calls take."""
import numpy as np
import pytest

from parity_util import assert_exact, gpu_args, random_blobs, run_both

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,ppbin", [(1, 128), (2, 1), (32, 128), (33, 4), (1023, 128), (1025, 128), (2049, 7),
                                     (4097, 128), (8192, 128), (8193, 20), (30000, 60), (65537, 128), (131072, 128),
                                     (131073, 128)])
@pytest.mark.parametrize("ndim", [1, 2, 3])
def test_sizes_against_oracle(gpu_context, n, ppbin, ndim):
    rng = np.random.default_rng(n + ndim)
    c, w = random_blobs(rng, n, ndim, nblobs=min(40, n), extent=300.0, sigma=1.0)
    assert_exact(*run_both(gpu_context, c, w, dc=0.8 if ndim > 1 else 0.02, rhoc=2.0, dm=1.2 if ndim > 1 else 0.04,
                           ppbin=ppbin))


@pytest.mark.parametrize("ndim", [5, 10])
@pytest.mark.parametrize("n,ppbin", [(3000, 1), (3000, 128), (9000, 40)])
def test_many_dimensions_against_oracle(gpu_context, n, ppbin, ndim):
    rng = np.random.default_rng(n)
    c, w = random_blobs(rng, n, ndim, nblobs=6, extent=40.0, sigma=1.0)
    assert_exact(*run_both(gpu_context, c, w, dc=1.0 + 0.3 * ndim, rhoc=2.0, dm=1.0 + 0.3 * ndim, ppbin=ppbin))


@pytest.mark.parametrize("kernel,metric,wrapped", [
    (("exp", (1.0, 1.0)), ("euclidean", ()), ()),                       # symmetric density, one sort
    (("gaus", (0.0, 0.7, 1.0)), ("weighted_euclidean", (1.0, 2.0)), ()),  # one-sided spatial density
    (("exp", (1.0, 1.0)), ("periodic_euclidean", (0.0, 60.0)), (0, 1)),
    (("flat", (0.5,)), ("euclidean", ()), (1, 0)),
])
def test_same_bits_as_separate_launches(gpu_context, kernel, metric, wrapped):
    """Events alone and in a small batch (one launch) against the same events beside one that is too
    large for it (separate launches)."""
    rng = np.random.default_rng(5)
    sizes = [1, 40, 1000, 1500, 5000, 129, 20000, 32768, 66000]
    evs = [random_blobs(rng, s, 2, nblobs=min(8, s), extent=60.0) for s in sizes]
    args = gpu_args(dc=1.5, rhoc=3.0, dm=2.0, kernel=kernel, metric=metric, wrapped=wrapped)

    def batch(k):
        off = np.concatenate([[0], np.cumsum(sizes[:k])]).astype(np.int32)
        r, ncl = gpu_context.batch_host(np.ascontiguousarray(np.concatenate([e[0] for e in evs[:k]], axis=1)),
                                        np.concatenate([e[1] for e in evs[:k]]), off, *args)
        return r, ncl, off

    large, ncl_large, off = batch(len(sizes))
    small, ncl_small, _ = batch(len(sizes) - 1)
    np.testing.assert_array_equal(ncl_small, ncl_large[:-1])
    m = off[-2]
    for k in ("cluster_index", "is_seed", "nearest_higher", "rho", "delta"):
        np.testing.assert_array_equal(getattr(small, k).view(np.uint32), getattr(large, k)[:m].view(np.uint32), k)
    for e, (c, w) in enumerate(evs[:-1]):
        alone = gpu_context.make_clusters_host(c, w, *args)
        a, b = off[e], off[e + 1]
        for k in ("cluster_index", "is_seed", "rho", "delta"):
            np.testing.assert_array_equal(getattr(alone, k).view(np.uint32), getattr(large, k)[a:b].view(np.uint32),
                                          f"{k} of event {e}")
        nh = large.nearest_higher[a:b]
        np.testing.assert_array_equal(alone.nearest_higher, np.where(nh >= 0, nh - a, nh))


def test_graphs_of_alternating_cluster_sizes(gpu_context):
    """Blocking calls keep one executable graph per cluster size."""
    rng = np.random.default_rng(3)
    evs = [random_blobs(rng, n, 2, nblobs=5, extent=40.0) for n in (9000, 700, 3000, 140000, 5000, 1500, 9001, 700)]
    for _ in range(2):
        for c, w in evs:
            assert_exact(*run_both(gpu_context, c, w, dc=1.0, rhoc=2.0, dm=1.5))
