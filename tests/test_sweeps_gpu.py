"""Edges of the neighbour sweeps against the oracle, bit for bit (flat kernel): blocks of 32, super-blocks
of 1024 records, more than 32 tiles in a search box, boxes that wrap, and many equal distances."""
import numpy as np
import pytest

from parity_util import assert_exact, random_blobs, run_both

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ndim,n,ppbin,dc,dm", [
    (2, 1, 128, 1.0, 1.0), (2, 31, 128, 5.0, 9.0), (2, 33, 128, 5.0, 9.0), (2, 129, 128, 5.0, 9.0),
    (2, 9000, 3000, 1.5, 3.0),    # tiles of several super-blocks
    (1, 5000, 2500, 0.4, 0.9),
    (2, 3001, 8, 2.0, 60.0),      # hundreds of tiles in a box, rings beyond the neighbours
    (3, 2500, 6, 3.0, 45.0),
    (4, 3000, 16, 4.0, 30.0),     # no ring order above three dimensions
    (7, 900, 4, 6.0, 12.0),
])
@pytest.mark.parametrize("tiebreak", ["reference", "rho_index"])
def test_nearest_higher_edges(gpu_context, ndim, n, ppbin, dc, dm, tiebreak):
    rng = np.random.default_rng(n + ndim)
    c, w = random_blobs(rng, n, ndim, nblobs=min(6, n), extent=60.0, sigma=1.5)
    assert_exact(*run_both(gpu_context, c, w, dc=dc, rhoc=2.0, dm=dm, ppbin=ppbin, tiebreak=tiebreak))


@pytest.mark.parametrize("n,ppbin", [(700, 128), (4000, 1500)])
@pytest.mark.parametrize("wrapped", [(), (1, 0), (1, 1)])
def test_nearest_higher_lattice(gpu_context, n, ppbin, wrapped):
    """Integer coordinates and weights: equal distances and equal densities in every block."""
    rng = np.random.default_rng(n)
    c = rng.integers(0, 25, size=(2, n)).astype(np.float32)
    w = rng.integers(1, 4, size=n).astype(np.float32)
    for tiebreak in ("reference", "rho_index"):
        assert_exact(*run_both(gpu_context, c, w, dc=1.0, rhoc=2.0, dm=4.0, ppbin=ppbin, wrapped=wrapped,
                               tiebreak=tiebreak))


@pytest.mark.parametrize("n", [1, 4, 31, 32, 33, 63, 64, 65, 95, 96, 97, 127, 130, 1021])
@pytest.mark.parametrize("ndim,metric,wrapped", [
    (1, ("euclidean", ()), ()), (2, ("euclidean", ()), ()), (2, ("periodic_euclidean", (0.0, 40.0)), (0, 1)),
    (3, ("weighted_euclidean", (0.5, 2.0, 1.0)), ()), (4, ("chebyshev", ()), ()), (9, ("manhattan", ()), ()),
])
def test_reference_order_density_edges(gpu_context, n, ndim, metric, wrapped):
    """Sums of whole and partial buffers of 32 kept candidates; all candidates kept, few, one."""
    rng = np.random.default_rng(7 * n + ndim)
    c, w = random_blobs(rng, n, ndim, nblobs=min(3, n), extent=40.0, sigma=1.0)
    w -= np.float32(0.8)  # negative weights too
    for dc, ppbin in ((0.4, 128), (2.5, 128), (200.0, 128), (3.0, 16)):
        assert_exact(*run_both(gpu_context, c, w, dc=dc, rhoc=0.5, dm=dc, ppbin=ppbin, metric=metric, wrapped=wrapped))


@pytest.mark.parametrize("n,fall", [(33, 0), (3000, 0), (100000, 0), (100000, 97)])
@pytest.mark.parametrize("blocking", [True, False])
def test_label_chains(gpu_context, n, fall, blocking):
    """One chain through all points (each point's nearest higher is the next one), whole or cut into
    pieces of `fall` points: one label round, several enqueued rounds, rounds from the host."""
    import torch
    from cluestering_alpaka3_b200 import capi
    from oracle import oracle as O
    from parity_util import gpu_args, oracle_cfg
    c = np.arange(n, dtype=np.float32)[None]
    w = (1.0 + np.arange(n) % fall if fall else 1.0 + np.arange(n)).astype(np.float32)
    kw = dict(dc=0.5, rhoc=1.5, dm=1.5)
    ref = O.run(c, w, oracle_cfg(**kw))
    dc, dw = torch.from_numpy(c).cuda(), torch.from_numpy(w).cuda()
    out = {k: torch.empty(n, dtype=torch.int32, device="cuda") for k in ("cluster_index", "is_seed", "nearest_higher")}
    torch.cuda.synchronize()
    gpu_context.make_clusters_device(dc.data_ptr(), dw.data_ptr(), 1, n, {k: t.data_ptr() for k, t in out.items()},
                                     *gpu_args(**kw), blocking=blocking)
    info = gpu_context.read_info()
    assert isinstance(info, capi.RunInfo) and info.n_clusters == ref.stats["n_clusters"]
    for k, t in out.items():
        np.testing.assert_array_equal(t.cpu().numpy(), getattr(ref, k), err_msg=k)


@pytest.mark.parametrize("n", [1, 31, 33, 64, 127, 1025])
@pytest.mark.parametrize("ndim", [1, 2, 3, 4, 9])
@pytest.mark.parametrize("kernel,metric", [(("exp", (1.0, 1.0)), "euclidean"), (("gaus", (0.0, 0.5, 1.0)), "euclidean"),
                                           (("exp", (1.0, 1.0)), "manhattan"), (("gaus", (0.0, 0.5, 1.0)), "chebyshev"),
                                           (("gaus", (1.0, 2.0, 1.5)), "euclidean")])
def test_symmetric_density_edges(gpu_context, n, ndim, kernel, metric):
    """Whole and partial blocks against each other, every kernel form and metric of the symmetric sweep,
    by the tolerance rule (densities within 1e-5 of FP64, everything after them exact)."""
    from oracle import oracle as O
    from parity_util import check_tolerant, gpu_args, oracle_cfg
    rng = np.random.default_rng(100 * n + ndim)
    c, w = random_blobs(rng, n, ndim, nblobs=min(3, n), extent=25.0, sigma=1.0)
    for dc in (0.7, 3.0, 100.0):
        kw = dict(dc=dc, rhoc=1.0, dm=1.3 * dc, kernel=kernel, metric=(metric, ()), ppbin=100)
        got = gpu_context.make_clusters_host(c, w, *gpu_args(**kw))
        cfg = oracle_cfg(**kw)
        check_tolerant(c, w, cfg, got, ref=O.run(c, w, cfg), rtol=1e-5)
