"""Where the one-launch first stage hands over to the separate launches: many events, many tiles.  The
route shows in the launches counted; the bits are the same on both sides of the line."""
import numpy as np
import pytest

from oracle import oracle as O
from parity_util import gpu_args, oracle_cfg, random_blobs

pytestmark = pytest.mark.gpu
NAMES = ("cluster_index", "is_seed", "rho", "nearest_higher", "delta")
EXP = ("exp", (1.0, 1.0))


def _launches(ctx, call):
    before = ctx.kernel_launches
    r = call()
    return r, ctx.kernel_launches - before


@pytest.mark.parametrize("kernel", [("flat", (0.5,)), EXP])
def test_tiny_events(gpu_context, kernel):
    rng = np.random.default_rng(4)
    E, m = 6001, 5
    c = rng.uniform(0, 20, size=(2, E * m)).astype(np.float32)
    w = rng.uniform(0.5, 1.5, E * m).astype(np.float32)
    args = gpu_args(dc=6.0, rhoc=1.2, dm=9.0, kernel=kernel)
    got = {}
    for k in (2282, 2283, E):
        off = (np.arange(k + 1) * m).astype(np.int32)
        (r, ncl), n = _launches(gpu_context, lambda: gpu_context.batch_host(
            np.ascontiguousarray(c[:, :k * m]), np.ascontiguousarray(w[:k * m]), off, *args))
        assert (n < 12) == (k + k * m // 512 <= 2304)
        got[k] = r, ncl
    for k in (2282, 2283):
        np.testing.assert_array_equal(got[k][1], got[E][1][:k])
        for f in NAMES:
            np.testing.assert_array_equal(getattr(got[k][0], f).view(np.uint32),
                                          getattr(got[E][0], f)[:k * m].view(np.uint32), f)
    if kernel[0] == "flat":
        ref = O.run_events(c, w, (np.arange(E + 1) * m).astype(np.int32), oracle_cfg(dc=6.0, rhoc=1.2, dm=9.0))
        for f in NAMES:
            np.testing.assert_array_equal(getattr(got[E][0], f).view(np.uint32), getattr(ref, f).view(np.uint32), f)


@pytest.mark.parametrize("n,ppbin,own", [(30000, 12, True), (11800, 1, True), (12400, 1, False)])
def test_many_tiles(gpu_context, n, ppbin, own):
    """A single event by k_build (own) or not, and in a batch that has too many tiles for it."""
    c, w = random_blobs(np.random.default_rng(n), n, 2, nblobs=n // 800, extent=40.0 * (n / 3000) ** 0.5)
    small = random_blobs(np.random.default_rng(1), 500, 2, nblobs=3, extent=30.0)
    args = gpu_args(dc=0.8, rhoc=2.0, dm=1.2, ppbin=ppbin, kernel=EXP)
    alone, k = _launches(gpu_context, lambda: gpu_context.make_clusters_host(c, w, *args))
    assert (k < 10) == own
    off = np.array([0, n, n + 500], np.int32)
    (r, _), k = _launches(gpu_context, lambda: gpu_context.batch_host(
        np.ascontiguousarray(np.concatenate([c, small[0]], axis=1)), np.concatenate([w, small[1]]), off, *args))
    assert k > 15
    for f in NAMES:
        np.testing.assert_array_equal(getattr(r, f)[:n].view(np.uint32), getattr(alone, f).view(np.uint32), f)
    flat = gpu_args(dc=0.8, rhoc=2.0, dm=1.2, ppbin=ppbin)
    _, k = _launches(gpu_context, lambda: gpu_context.make_clusters_host(c, w, *flat))
    assert k < 10  # the other sweeps' three sorts cost more
