"""Long chains: ramps, each point's nearest higher the next one, of more points than the GPU holds
threads.  The first label round climbs them in passes; what it leaves, which the checked build is told to
let happen (CLUE_LABEL_HOPS jumps a round), is completed by later rounds, enqueued or from the host, and the
run's status is good afterwards."""
import os
import subprocess
import sys

import numpy as np
import pytest

from oracle import oracle as O
from parity_util import gpu_args, oracle_cfg

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CHECKED = os.path.join(ROOT, "cluestering_alpaka3_b200", "libclue_b200_checked.so")

KW = dict(dc=0.5, rhoc=1.5, dm=1.5, seed_dc=1.2)  # one seed: the last point
OUT = ("cluster_index", "is_seed", "nearest_higher")


def ramps(sizes):
    """Coordinates, weights, offsets and the oracle's outputs of one ramp per size."""
    c = np.concatenate([np.arange(n, dtype=np.float32) for n in sizes])[None]
    refs = [O.run(np.arange(n, dtype=np.float32)[None], 1.0 + np.arange(n, dtype=np.float32), oracle_cfg(**KW))
            for n in sizes]
    return np.ascontiguousarray(c), 1.0 + c[0], np.concatenate([[0], np.cumsum(sizes)]).astype(np.int32), refs


def device(c, w):
    import torch
    n = w.size
    dc, dw = torch.from_numpy(c).cuda(), torch.from_numpy(w).cuda()
    out = {k: torch.empty(n, dtype=torch.int32, device="cuda") for k in OUT}
    torch.cuda.synchronize()
    return dc, dw, out


def check_event(ctx, n, blocking, bfs, rounds):
    from cluestering_alpaka3_b200 import capi
    c, w, _, (ref,) = ramps([n])
    dc, dw, out = device(c, w)
    ctx.set_tuning(labels_bfs=bfs)
    for _ in range(2):  # a call's status is its own
        ctx.make_clusters_device(dc.data_ptr(), dw.data_ptr(), 1, n, {k: t.data_ptr() for k, t in out.items()},
                                 *gpu_args(**KW), blocking=blocking)
        if rounds is None:
            with pytest.raises(capi.ClueError, match="deeper than the enqueued label rounds"):
                ctx.read_info()
            continue
        info = ctx.read_info()
        assert rounds(info.label_rounds), info.label_rounds
        assert (info.n_clusters, info.n_seeds) == (ref.stats["n_clusters"], ref.stats["n_seeds"])
        for k, t in out.items():
            np.testing.assert_array_equal(t.cpu().numpy(), getattr(ref, k), err_msg=k)
        ctx.near_counts()
    ctx.set_tuning(labels_bfs=0)


def check_batch(ctx, sizes, blocking, rounds):
    c, w, off, refs = ramps(sizes)
    dc, dw, out = device(c, w)
    ctx.batch_device(dc.data_ptr(), dw.data_ptr(), 1, off, {k: t.data_ptr() for k, t in out.items()},
                     *gpu_args(**KW), blocking=blocking)
    info = ctx.read_info()
    assert rounds(info.label_rounds), info.label_rounds
    assert info.n_clusters == sum(r.stats["n_clusters"] for r in refs)
    for e, ref in enumerate(refs):
        a, b = off[e], off[e + 1]
        nh = out["nearest_higher"][a:b].cpu().numpy()
        np.testing.assert_array_equal(np.where(nh >= 0, nh - a, nh), ref.nearest_higher)
        np.testing.assert_array_equal(out["cluster_index"][a:b].cpu().numpy(), ref.cluster_index)


def check_host(ctx, n, rounds):
    c, w, _, (ref,) = ramps([n])
    got = ctx.make_clusters_host(c, w, *gpu_args(**KW))
    assert rounds(got.info.label_rounds), got.info.label_rounds
    np.testing.assert_array_equal(got.cluster_index, ref.cluster_index)
    assert ctx.read_info().n_clusters == ref.stats["n_clusters"]


@pytest.mark.parametrize("blocking", [True, False])
@pytest.mark.parametrize("n,bfs", [(1 << 20, 0), (1 << 20, 1), (2_200_001, 0)])  # one and four chains a thread
def test_long_chain(blocking, n, bfs):
    from cluestering_alpaka3_b200 import capi
    ctx = capi.Context(0)
    try:
        check_event(ctx, n, blocking, bfs, lambda r: r >= 1)
    finally:
        ctx.close()


@pytest.mark.parametrize("blocking", [True, False])
def test_long_chains_of_a_batch(gpu_context, blocking):
    check_batch(gpu_context, [1000, 700_000, 500_001], blocking, lambda r: r >= 1)


def test_long_chain_in_host_memory(gpu_context):
    check_host(gpu_context, 600_011, lambda r: r >= 1)


def test_label_time_of_a_long_chain():
    """1M points: 16 ms when a chain was climbed to its end at once, 0.06 in passes."""
    from cluestering_alpaka3_b200 import capi
    n = 1 << 20
    c, w = np.arange(n, dtype=np.float32)[None], 1.0 + np.arange(n, dtype=np.float32)
    dc, dw, out = device(c, w)
    ctx = capi.Context(0)
    try:
        ctx.set_timing(True)
        ms = []
        for _ in range(5):
            ctx.make_clusters_device(dc.data_ptr(), dw.data_ptr(), 1, n, {k: t.data_ptr() for k, t in out.items()},
                                     *gpu_args(**KW))
            ms.append(ctx.stage_times()[3])
        assert min(ms) < 0.4
    finally:
        ctx.close()


LATER = r'''
import sys
sys.path[:0] = [ROOT, ROOT + "/tests"]
from cluestering_alpaka3_b200 import capi
import test_label_rounds_gpu as t
ctx = capi.Context(0)
more = lambda r: r > 1
if HOPS == 2:  # the host continues; four rounds of two jumps reach 256 points at most
    for bfs in (0, 1):
        t.check_event(ctx, 20_000, True, bfs, more)
    t.check_event(ctx, 1_000_003, True, 0, more)
    t.check_event(ctx, 20_000, False, 0, None)
    t.check_batch(ctx, [1000, 20_000, 33, 9000], True, more)
    t.check_batch(ctx, [1000, 700_000, 33, 9000], True, more)
    t.check_host(ctx, 20_000, more)
else:  # four rounds of sixteen jumps reach 65536 points at least
    t.check_event(ctx, 20_000, False, 0, more)
    t.check_batch(ctx, [1000, 20_000, 33, 9000], False, more)
ctx.close()
print("ok")
'''


@pytest.mark.parametrize("hops", [2, 16])
def test_later_rounds(hops):
    env = dict(os.environ, CLUE_B200_LIB=CHECKED, CLUE_LABEL_HOPS=str(hops))
    r = subprocess.run([sys.executable, "-c", f"ROOT = {ROOT!r}\nHOPS = {hops}\n" + LATER], env=env,
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stdout + r.stderr
