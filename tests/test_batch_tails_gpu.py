"""Batches whose last events lie inside the last, partial block of 32 records: every event's bits are
those of the event alone.  (Few points per tile, so that such an event has several blocks and its sums
a received part.)"""
import numpy as np
import pytest

from parity_util import gpu_args, random_blobs

pytestmark = pytest.mark.gpu


# head % 32 + the tail is below 32, so the tail's events share one partial block with the head's last points
@pytest.mark.parametrize("head", [1985, 530017])  # one launch for the first stage, separate launches
@pytest.mark.parametrize("tail", [(1,), (7,), (30,), (1, 9, 18)])
@pytest.mark.parametrize("kernel", [("exp", (1.0, 1.0)), ("gaus", (0.0, 0.7, 1.0))])
def test_small_events_in_the_last_block(gpu_context, head, tail, kernel):
    rng = np.random.default_rng(head + len(tail))
    extent = 60.0 * (head / 1985) ** 0.5
    evs = [random_blobs(rng, head, 2, nblobs=max(4, head // 500), extent=extent)]
    for m in tail:  # neighbours within dc of one another
        evs.append((rng.normal(5.0, 0.4, size=(2, m)).astype(np.float32), rng.uniform(0.5, 1.5, m).astype(np.float32)))
    off = np.concatenate([[0], np.cumsum([e[1].size for e in evs])]).astype(np.int32)
    last = (off[-1] - 1) // 32 * 32
    assert off[-1] % 32 and last < off[1]
    args = gpu_args(dc=1.2, rhoc=2.0, dm=1.8, ppbin=6, kernel=kernel)
    got, ncl = gpu_context.batch_host(np.ascontiguousarray(np.concatenate([e[0] for e in evs], axis=1)),
                                      np.concatenate([e[1] for e in evs]), off, *args)
    for e, (c, w) in enumerate(evs):
        alone = gpu_context.make_clusters_host(np.ascontiguousarray(c), w, *args)
        a, b = off[e], off[e + 1]
        for k in ("rho", "delta", "is_seed", "cluster_index"):
            np.testing.assert_array_equal(getattr(got, k)[a:b].view(np.uint32), getattr(alone, k).view(np.uint32),
                                          f"{k} of event {e}")
        nh = got.nearest_higher[a:b]
        np.testing.assert_array_equal(np.where(nh >= 0, nh - a, nh), alone.nearest_higher)
        assert ncl[e] == alone.info.n_clusters
