"""Metric values below zero (a negative weight of the weighted Euclidean metric): the least one wins."""
import numpy as np
import pytest

from parity_util import gpu_args

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [40, 120, 3000])
@pytest.mark.parametrize("weights", ["ones", "random"])
def test_negative_weight(gpu_context, n, weights):
    rng = np.random.default_rng(n)
    c = rng.uniform(0, 30.0, size=(2, n)).astype(np.float32)
    w = np.ones(n, np.float32) if weights == "ones" else rng.uniform(0.5, 1.5, n).astype(np.float32)
    mw = np.array([-0.5, 1.0], np.float32)
    got = gpu_context.make_clusters_host(c, w, *gpu_args(dc=2.0, rhoc=1e9, dm=4.0,
                                                         metric=("weighted_euclidean", tuple(mw))))
    assert got.info.label_rounds == 1  # (no chain without an end)
    nh = got.nearest_higher
    i = np.nonzero(nh >= 0)[0]
    higher = (got.rho[nh[i]] > got.rho[i]) | ((got.rho[nh[i]] == got.rho[i]) & (nh[i] > i))
    assert i.size > n // 2 and higher.all()
    if n > 128:
        return
    # one tile: every denser point within dm is a candidate, the least metric value wins
    s = np.zeros((n, n), np.float32)
    for d in (1, 0):
        t = c[d][:, None] - c[d][None, :]
        s = (mw[d] * t) * t + s
    cand = (got.rho[None, :] > got.rho[:, None]) | ((got.rho[None, :] == got.rho[:, None]) &
                                                    (np.arange(n)[None, :] > np.arange(n)[:, None]))
    cand &= s <= np.float32(16.0)
    s = np.where(cand, s, np.inf)
    np.testing.assert_array_equal(nh, np.where(cand.any(1), s.argmin(1), -1))
