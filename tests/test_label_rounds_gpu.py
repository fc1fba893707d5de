"""Chains that outlast the first label round, in every kind of call: a ramp of more points than the GPU
holds threads, each point's nearest higher the next one.  The first round's last running points climb
into points that no thread has moved yet, one hop at a time, and stop after 4096 of them; the labels
are completed by later rounds, and the run's status is good afterwards."""
import numpy as np
import pytest

from oracle import oracle as O
from parity_util import gpu_args, oracle_cfg

pytestmark = pytest.mark.gpu

KW = dict(dc=0.5, rhoc=1.5, dm=1.5, seed_dc=1.2)  # one seed: the last point
OUT = ("cluster_index", "is_seed", "nearest_higher")


def _ramps(sizes):
    """Coordinates, weights, offsets and the oracle's outputs of one ramp per size."""
    c = np.concatenate([np.arange(n, dtype=np.float32) for n in sizes])[None]
    w = 1.0 + c[0]
    refs = [O.run(np.arange(n, dtype=np.float32)[None], 1.0 + np.arange(n, dtype=np.float32), oracle_cfg(**KW))
            for n in sizes]
    return np.ascontiguousarray(c), w, np.concatenate([[0], np.cumsum(sizes)]).astype(np.int32), refs


def _device(c, w):
    import torch
    n = w.size
    dc, dw = torch.from_numpy(c).cuda(), torch.from_numpy(w).cuda()
    out = {k: torch.empty(n, dtype=torch.int32, device="cuda") for k in OUT}
    torch.cuda.synchronize()
    return dc, dw, out


@pytest.mark.parametrize("blocking", [True, False])
@pytest.mark.parametrize("bfs", [0, 1])
def test_one_event(blocking, bfs):
    from cluestering_alpaka3_b200 import capi
    n = 1 << 20
    c, w, _, (ref,) = _ramps([n])
    dc, dw, out = _device(c, w)
    ctx = capi.Context(0)
    try:
        ctx.set_tuning(labels_bfs=bfs)
        for _ in range(2):  # a call's status is its own
            ctx.make_clusters_device(dc.data_ptr(), dw.data_ptr(), 1, n, {k: t.data_ptr() for k, t in out.items()},
                                     *gpu_args(**KW), blocking=blocking)
            info = ctx.read_info()
            assert info.label_rounds > 1  # the first round did not do it
            assert (info.n_clusters, info.n_seeds) == (ref.stats["n_clusters"], ref.stats["n_seeds"])
            for k, t in out.items():
                np.testing.assert_array_equal(t.cpu().numpy(), getattr(ref, k), err_msg=k)
            ctx.near_counts()
    finally:
        ctx.close()


@pytest.mark.parametrize("blocking", [True, False])
def test_batch(gpu_context, blocking):
    c, w, off, refs = _ramps([1000, 700_000, 500_001])
    dc, dw, out = _device(c, w)
    gpu_context.batch_device(dc.data_ptr(), dw.data_ptr(), 1, off, {k: t.data_ptr() for k, t in out.items()},
                             *gpu_args(**KW), blocking=blocking)
    info = gpu_context.read_info()
    assert info.label_rounds > 1
    assert info.n_clusters == sum(r.stats["n_clusters"] for r in refs)
    for e, ref in enumerate(refs):
        a, b = off[e], off[e + 1]
        nh = out["nearest_higher"][a:b].cpu().numpy()
        np.testing.assert_array_equal(np.where(nh >= 0, nh - a, nh), ref.nearest_higher)
        np.testing.assert_array_equal(out["cluster_index"][a:b].cpu().numpy(), ref.cluster_index)


def test_host_memory(gpu_context):
    c, w, _, (ref,) = _ramps([600_011])
    got = gpu_context.make_clusters_host(c, w, *gpu_args(**KW))
    assert got.info.label_rounds > 1
    np.testing.assert_array_equal(got.cluster_index, ref.cluster_index)
    assert gpu_context.read_info().n_clusters == ref.stats["n_clusters"]
