"""The one-launch first stage on a device that does not give it the clusters it asks for: smaller ones,
none, a refused launch, another size than asked for.  The checked build is told to find each
(CLUE_BUILD_CLUSTERS); its outputs are the default build's, bit for bit, in every kind of call."""
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CHECKED = os.path.join(ROOT, "cluestering_alpaka3_b200", "libclue_b200_checked.so")

CASES = r'''
import sys, numpy as np
sys.path.insert(0, ROOT); sys.path.insert(0, ROOT + "/tests")
import torch
from cluestering_alpaka3_b200 import capi
from parity_util import gpu_args, random_blobs
rng = np.random.default_rng(11)
OUT_NAMES = ("cluster_index", "is_seed", "rho", "nearest_higher", "delta")
out = {}

def device(c, w):
    n = w.size
    t = {k: torch.empty(n, dtype=torch.float32 if k in ("rho", "delta") else torch.int32, device="cuda") for k in OUT_NAMES}
    d = torch.from_numpy(c).cuda(), torch.from_numpy(w).cuda()
    torch.cuda.synchronize()
    return d, t

ctx = capi.Context(0)
evs = [random_blobs(rng, n, 2, nblobs=4, extent=40.0) for n in (900, 12000, 3000, 700, 12000)]
off = np.concatenate([[0], np.cumsum([e[1].size for e in evs])]).astype(np.int32)
c = np.ascontiguousarray(np.concatenate([e[0] for e in evs], axis=1))
w = np.concatenate([e[1] for e in evs])
for name, kernel in (("flat", ("flat", (0.5,))), ("exp", ("exp", (1.0, 1.0)))):
    args = gpu_args(dc=1.0, rhoc=2.0, dm=1.5, kernel=kernel)
    for k, (ce, we) in enumerate(evs):  # graphs of several cluster sizes
        out[f"{name} blocking {k}"] = ctx.make_clusters_host(np.ascontiguousarray(ce), we, *args)
    out[f"{name} batch"], _ = ctx.batch_host(c, w, off, *args)
    (dc, dw), t = device(evs[1][0], evs[1][1])
    ctx.make_clusters_device(dc.data_ptr(), dw.data_ptr(), 2, evs[1][1].size, {k: v.data_ptr() for k, v in t.items()},
                             *args, blocking=False)
    ctx.read_info()
    out[f"{name} async"] = {k: v.cpu().numpy() for k, v in t.items()}
    (dc, dw), t = device(c, w)
    side = torch.cuda.Stream()
    g = ctx.capture_batch(dc.data_ptr(), dw.data_ptr(), 2, off, {k: v.data_ptr() for k, v in t.items()}, *args,
                          stream=side.cuda_stream)
    g.launch(side.cuda_stream)
    side.synchronize()
    out[f"{name} graph"] = {k: v.cpu().numpy() for k, v in t.items()}
get = lambda r, f: r[f] if isinstance(r, dict) else getattr(r, f)
np.savez(OUT, launches=ctx.kernel_launches, **{f"{k}.{f}": get(r, f) for k, r in out.items() for f in OUT_NAMES})
'''


def _run(path, lib=None, clusters=""):
    env = {k: v for k, v in os.environ.items() if k not in ("CLUE_B200_LIB", "CLUE_BUILD_CLUSTERS")}
    if lib:
        env.update(CLUE_B200_LIB=lib, CLUE_BUILD_CLUSTERS=clusters)
    code = f"ROOT = {ROOT!r}\nOUT = {path!r}\n" + CASES
    r = subprocess.run([sys.executable, "-c", code], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    return np.load(path)


@pytest.fixture(scope="module")
def default(tmp_path_factory):
    return _run(str(tmp_path_factory.mktemp("build") / "default.npz"))


@pytest.mark.parametrize("clusters", ["", "fit 8", "fit 3", "fit 1", "fit 0", "refuse", "half", "double"])
def test_outputs_do_not_depend_on_the_clusters(default, tmp_path, clusters):
    got = _run(str(tmp_path / "got.npz"), CHECKED, clusters)
    assert sorted(got.files) == sorted(default.files)
    separate = clusters in ("fit 0", "refuse")  # some 20 launches in place of one
    assert (int(got["launches"]) > int(default["launches"]) + 150) == separate
    for k in got.files:
        if k != "launches":
            np.testing.assert_array_equal(got[k].view(np.uint32), default[k].view(np.uint32), err_msg=k)
