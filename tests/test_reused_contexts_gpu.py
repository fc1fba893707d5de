"""Contexts made from an idle one (clue_context_destroy keeps small ones): what they hold, what they say
of themselves and what a program can rely on is as with a new one."""
import numpy as np
import pytest

from parity_util import gpu_args, random_blobs

pytestmark = pytest.mark.gpu


def _leave_idle(ndim, n):
    """Leaves two idle contexts that ran n points of ndim dimensions."""
    from cluestering_alpaka3_b200 import capi
    c, w = random_blobs(np.random.default_rng(1), n, ndim, nblobs=max(4, n // 1000), extent=30.0 * max(1, n / 4000) ** 0.5)
    ctxs = [capi.Context(0) for _ in range(2)]
    for ctx in ctxs:
        ctx.make_clusters_host(c, w, *gpu_args(dc=0.5, rhoc=2.0, dm=0.8))
    for ctx in ctxs:
        ctx.close()


def _drop_idle():
    """Takes the idle contexts and closes them too large to be kept."""
    from cluestering_alpaka3_b200 import capi
    ctxs = [capi.Context(0) for _ in range(2)]
    for ctx in ctxs:
        ctx.reserve(2, 3_000_000)
    for ctx in ctxs:
        ctx.close()


@pytest.mark.parametrize("last,own", [((10, 3000), (2, 4_000_000)), ((2, 300_000), (10, 20_000))])
@pytest.mark.parametrize("first", [0, 200])
def test_larger_allocation_ignores_the_last_owner(last, own, first):
    """An earlier owner's record words do not multiply a later one's points, nor its points their words."""
    from cluestering_alpaka3_b200 import capi
    c, w = random_blobs(np.random.default_rng(2), 200, 2, nblobs=2, extent=30.0)

    def held():
        ctx = capi.Context(0)
        if first:  # a call that fits what is there
            ctx.make_clusters_host(c, w, *gpu_args(dc=1.0, rhoc=2.0, dm=1.5))
        ctx.reserve(*own)
        b = ctx.workspace_bytes
        ctx.close()
        return b

    _drop_idle()
    new = held()
    _drop_idle()
    _leave_idle(*last)
    assert held() <= new + (12 << 20)  # (staging buffers of the last owner, 9.6 MB, are not the workspace's)
    _drop_idle()


def test_server_stays_inside_its_budget():
    """Slots hold what was reserved for them, not a larger idle context's buffers."""
    import torch
    from cluestering_alpaka3_b200 import capi
    _drop_idle()
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    _leave_idle(2, 300_000)
    budget = 24 << 20
    cfg = capi.ServerConfig(ndim=2, n_slots=2, max_batch_events=16, max_event_points=20000, device_budget_bytes=budget)
    srv = capi.Server(cfg, *gpu_args(dc=1.0, rhoc=2.0, dm=1.5))
    try:
        _drop_idle()  # those that the server did not take
        held = free - torch.cuda.mem_get_info()[0]
        assert srv.stats()["device_bytes"] <= budget
        assert held <= budget + (24 << 20)  # (allocations of the driver, 2 MB each)
    finally:
        srv.close()


def test_no_status_and_no_bytes_before_a_call():
    """The last owner's run is nobody's business, also after calls that are not runs."""
    import torch
    from cluestering_alpaka3_b200 import capi
    _leave_idle(2, 3000)
    ctx = capi.Context(0)
    try:
        assert ctx.workspace_bytes == 0
        for call in ("none", "reserve", "get_clusters"):
            if call == "reserve":
                ctx.reserve(2, 100)
                assert ctx.workspace_bytes > 0
            elif call == "get_clusters":
                lab = torch.zeros(64, dtype=torch.int32, device="cuda")
                off, pts = torch.empty(65, dtype=torch.int32, device="cuda"), torch.empty_like(lab)
                torch.cuda.synchronize()
                assert ctx.get_clusters(lab.data_ptr(), 64, off.data_ptr(), pts.data_ptr()) == (1, 64)
            with pytest.raises(capi.ClueError):
                ctx.read_info()
            with pytest.raises(capi.ClueError):
                ctx.near_counts()
        c, w = random_blobs(np.random.default_rng(2), 200, 2, nblobs=2, extent=30.0)
        got = ctx.make_clusters_host(c, w, *gpu_args(dc=1.0, rhoc=2.0, dm=1.5))
        assert ctx.read_info().n_clusters == got.info.n_clusters
    finally:
        ctx.close()
