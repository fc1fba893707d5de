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


RESET = r'''
import ctypes, sys
import numpy as np
sys.path[:0] = [ROOT, ROOT + "/tests"]
from cluestering_alpaka3_b200 import capi
from parity_util import gpu_args, random_blobs
c, w = random_blobs(np.random.default_rng(1), 3000, 2, nblobs=4, extent=30.0)
args = gpu_args(dc=1.0, rhoc=2.0, dm=1.5)
vp, n = ctypes.c_void_p, 8 << 20
first = capi.Context(0)
want = first.make_clusters_host(c, w, *args)
second = capi.Context(0)
second.make_clusters_host(c, w, *args)
first.close()
second.close()
assert ctypes.CDLL("libcuda.so.1").cuDevicePrimaryCtxReset_v2(0) == 0  # what cudaDeviceReset does
# the program's own memory, perhaps where the contexts' was
bufs, data = [], np.arange(n, dtype=np.uint8)
for _ in range(6):
    p = vp()
    capi.check(capi.lib.clue_device_alloc(0, n, ctypes.byref(p)))
    capi.check(capi.lib.clue_memcpy_htod(p, data.ctypes.data, n, None))
    bufs.append(p)
if WHAT == "failing allocation":  # gives the idle contexts back
    p = vp()
    assert capi.lib.clue_device_alloc(0, 1 << 45, ctypes.byref(p)) != 0
for _ in range(3):
    ctx = capi.Context(0)
    got = ctx.make_clusters_host(c, w, *args)
    assert np.array_equal(got.cluster_index, want.cluster_index)
    assert np.array_equal(got.rho.view(np.uint32), want.rho.view(np.uint32))
    ctx.close()
back = np.empty_like(data)
for p in bufs:
    capi.check(capi.lib.clue_memcpy_dtoh(back.ctypes.data, p, n, None))
    capi.check(capi.lib.clue_stream_synchronize(None))
    assert np.array_equal(back, data)
    capi.check(capi.lib.clue_device_free(p))
print("ok")
'''


@pytest.mark.parametrize("what", ["create", "failing allocation"])
def test_device_reset_forgets_idle_contexts(what):
    """A program that resets its device between contexts (in a child process: the reset ends all that
    the process has on the device)."""
    import os
    import subprocess
    import sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", f"ROOT = {root!r}\nWHAT = {what!r}\n" + RESET], capture_output=True,
                       text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr


def test_release_gives_the_memory_back():
    import torch
    from cluestering_alpaka3_b200 import capi
    _leave_idle(2, 3000)  # (kernels loaded, streams made)
    capi.release_idle_contexts()
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    _leave_idle(2, 300_000)
    assert free - torch.cuda.mem_get_info()[0] > 60 << 20
    capi.release_idle_contexts()
    capi.release_idle_contexts()  # nothing left
    assert free - torch.cuda.mem_get_info()[0] < 8 << 20
    ctx = capi.Context(0)
    c, w = random_blobs(np.random.default_rng(2), 200, 2, nblobs=2, extent=30.0)
    ctx.make_clusters_host(c, w, *gpu_args(dc=1.0, rhoc=2.0, dm=1.5))
    ctx.close()
