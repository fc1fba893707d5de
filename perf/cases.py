"""Performance cases of the clustering library: what its users have it do, by call and by size.

Every case is a dict of plain values.  ``listed()`` gives the fixed cases, ``draw(rng)`` one more
of the same ranges, ``prepare(case, seed)`` the inputs, context and buffers that a user's program
has before the call, ``run(state)`` one pass through the public entry points, ``work(case)`` the
bytes and operations the pass cannot do without, and ``exact(case, seed)`` the computed outputs
in 64 bits (plain torch, no code of the library).

A case's ``call`` names the entry point:

  event       one event, device memory        Context.make_clusters_device (blocking)
  host        one event, host memory          Context.make_clusters_host
  python      one event, the Python class     clusterer.fit_predict
  batch       many events, device memory      Context.batch_device (blocking)
  graph       many events, captured once      Context.capture_batch, Graph.launch
  batch_host  many events, pinned host memory Context.batch_host
  serve       single events submitted         Server.submit / Server.wait
  clusters    after clustering                Context.get_clusters, Context.cluster_centroids_device
  silhouette  after clustering                Context.silhouette_device

and its ``data`` the distribution:

  blobs       isotropic Gaussian blobs (sigma 1) with 10% uniform noise
  blobs3d     anisotropic 3-D blobs (per-axis sigma U[0.2, 1]) with 15% noise, lognormal weights
  calo        2-D calorimeter-like events: 3-30 energy-weighted showers with 20% noise
  barrel      a detector barrel, eta x phi with phi periodic, showers with 15% noise
"""
import math

import numpy as np
import torch

from cluestering_alpaka3_b200 import capi

_EVENT_OUT = ("cluster_index", "is_seed", "rho", "nearest_higher", "delta")
_BATCH_OUT = ("cluster_index", "is_seed", "rho", "nearest_higher")
_FLOAT_OUT = ("rho", "delta")


def listed():
    return [
        # A script clustering a small table through the Python front end, a new object per table
        # (the reference's usual Python session).
        {"name": "python_2k", "call": "python", "data": "blobs", "dim": 2, "n": 2000, "kernel": "flat"},
        # The smallest device-resident call: one small event inside a larger GPU program.
        {"name": "event_2d_1k", "call": "event", "data": "blobs", "dim": 2, "n": 1000, "kernel": "flat"},
        # The 16k-point 2-D set of the benchmark (flat kernel, bit-exact reference order).
        {"name": "event_2d_16k", "call": "event", "data": "blobs", "dim": 2, "n": 16384, "kernel": "flat"},
        # The 1M-point 2-D set: one large plain clustering.
        {"name": "event_2d_1m", "call": "event", "data": "blobs", "dim": 2, "n": 1048576, "kernel": "flat"},
        # The 4M-point 3-D set with the Gaussian kernel: the largest single event.
        {"name": "event_3d_4m", "call": "event", "data": "blobs3d", "dim": 3, "n": 4194304, "kernel": "gaus"},
        # Five coordinates per point, odd count, the exponential kernel and the Manhattan metric.
        {"name": "event_5d_30k", "call": "event", "data": "blobs", "dim": 5, "n": 30011, "kernel": "exp",
         "metric": "manhattan"},
        # A detector barrel: one periodic coordinate, periodic metric, exponential kernel.
        {"name": "barrel_50k", "call": "event", "data": "barrel", "dim": 2, "n": 50021, "kernel": "exp",
         "metric": "periodic"},
        # The flagship: 4096 uneven calorimeter events replayed as one captured graph.
        {"name": "calo_graph_4096", "call": "graph", "data": "calo", "dim": 2, "events": 4096, "median": 2000,
         "kernel": "exp"},
        # The same work arriving in pinned host memory, labels and seed flags going back.
        {"name": "calo_host_2048", "call": "batch_host", "data": "calo", "dim": 2, "events": 2048, "median": 2000,
         "kernel": "exp"},
        # Online clustering: a burst of 4-D events submitted to the request loop.
        {"name": "serve_4d_24", "call": "serve", "data": "blobs", "dim": 4, "events": 24, "median": 2000,
         "kernel": "flat"},
        # After a large clustering: members and centroid of every cluster.
        {"name": "clusters_1m", "call": "clusters", "data": "blobs", "dim": 2, "n": 1000003},
        # Quality of a clustering: every point against every clustered point.
        {"name": "silhouette_32k", "call": "silhouette", "data": "blobs", "dim": 2, "n": 32768},
    ]


def _log_int(rng, lo, hi):
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return max(lo, min(hi, n | 1 if rng.random() < 0.7 else n))


def draw(rng):
    call = rng.choice(["event", "event", "event", "host", "python", "batch", "graph", "batch_host", "serve", "clusters",
                       "silhouette"])
    if call in ("event", "host"):
        if rng.random() < 0.2:
            return {"call": call, "data": "barrel", "dim": 2, "n": _log_int(rng, 1000, 400000),
                    "kernel": rng.choice(["flat", "exp", "gaus"]), "metric": "periodic"}
        if rng.random() < 0.15:
            return {"call": call, "data": "blobs3d", "dim": 3, "n": _log_int(rng, 2000, 3000000),
                    "kernel": rng.choice(["exp", "gaus"])}
        dim = rng.choice([1, 2, 2, 2, 3, 3, 4, 5, 6])
        return {"call": call, "data": "blobs", "dim": dim,
                "n": _log_int(rng, 500, {1: 400000, 2: 1048576, 3: 500000}.get(dim, 60000)),
                "kernel": rng.choice(["flat", "flat", "exp", "gaus"]),
                "metric": rng.choice(["euclidean", "euclidean", "euclidean", "weighted_euclidean", "manhattan",
                                      "chebyshev", "weighted_chebyshev"])}
    if call == "python":
        return {"call": call, "data": "blobs", "dim": rng.choice([2, 3]), "n": _log_int(rng, 500, 30000),
                "kernel": rng.choice(["flat", "exp", "gaus"])}
    if call in ("batch", "graph", "batch_host"):
        data, dim, kernel = rng.choice([("calo", 2, "exp"), ("calo", 2, "flat"), ("blobs", 4, "flat"),
                                        ("blobs", 3, "gaus")])
        return {"call": call, "data": data, "dim": dim, "kernel": kernel, "median": _log_int(rng, 300, 3000),
                "events": _log_int(rng, 4, 2500 if data == "calo" else 500)}
    if call == "serve":
        return {"call": call, "data": "blobs", "dim": 4, "events": rng.randint(1, 60),
                "median": _log_int(rng, 500, 4000), "kernel": "flat"}
    if call == "clusters":
        return {"call": call, "data": "blobs", "dim": rng.choice([2, 3, 4]), "n": _log_int(rng, 2000, 1000000)}
    return {"call": call, "data": "blobs", "dim": rng.choice([2, 3]), "n": _log_int(rng, 1000, 40000)}


# ---- parameters --------------------------------------------------------------------------------
def _settings(case):
    """dc, rhoc, dm, kernel (name, parameters), metric name and wrapped flags of a case."""
    kind = case.get("kernel", "flat")
    if case["data"] == "calo":
        dc, rhoc, dm = 2.0, 4.0, 3.0
    elif case["data"] == "blobs3d":
        dc, rhoc, dm = 1.2, 8.0, 2.0
    elif case["data"] == "barrel":
        dc, rhoc, dm = 0.06, 4.0, 0.09
    else:
        dc = {1: 0.5, 2: 1.5, 3: 2.0, 4: 2.5, 5: 3.0, 6: 3.3}[case["dim"]]
        rhoc, dm = 5.0, dc
    kernel = {"flat": (0.5,), "exp": (1.0, 1.0), "gaus": (0.0, 0.5, 1.0)}[kind]
    if case["data"] == "barrel":
        kernel = {"flat": (0.5,), "exp": (25.0, 1.0), "gaus": (0.0, 0.03, 1.0)}[kind]
    wrapped = (0, 1) if case["data"] == "barrel" else ()
    return dc, rhoc, dm, kind, kernel, case.get("metric", "euclidean"), wrapped


def _metric_par(metric, dim):
    if metric == "weighted_euclidean" or metric == "weighted_chebyshev":
        return tuple(0.5 + 0.25 * d for d in range(dim))
    if metric == "periodic":
        return (0.0, 2.0 * math.pi)
    return ()


def _structs(case):
    dc, rhoc, dm, kind, kernel, metric, wrapped = _settings(case)
    params = capi.Params(dc=dc, rhoc=rhoc, dm=dm, wrapped=wrapped)
    kern = {"flat": capi.FlatKernel, "exp": capi.ExponentialKernel, "gaus": capi.GaussianKernel}[kind](*kernel)
    met = capi.Metric({"euclidean": capi.METRIC_EUCLIDEAN, "weighted_euclidean": capi.METRIC_WEIGHTED_EUCLIDEAN,
                       "periodic": capi.METRIC_PERIODIC_EUCLIDEAN, "manhattan": capi.METRIC_MANHATTAN,
                       "chebyshev": capi.METRIC_CHEBYSHEV,
                       "weighted_chebyshev": capi.METRIC_WEIGHTED_CHEBYSHEV}[metric],
                      _metric_par(metric, case["dim"]))
    return params, kern, met


# ---- inputs ------------------------------------------------------------------------------------
def _event_sizes(case):
    """Lognormal event sizes (sigma 1 around the median), as the batched and serving workloads; the
    case alone decides them, so that a captured batch keeps its shape from pass to pass."""
    lo, hi = 100, 60000 if case["data"] == "calo" else 20000
    rng = np.random.default_rng(1000 * case["median"] + case["events"])
    return np.clip(np.round(rng.lognormal(math.log(case["median"]), 1.0, size=case["events"])), lo, hi).astype(np.int64)


def _blob_count(case, n):
    """Blobs of one event and the members of each: about 740 points a blob in the 16k set."""
    return max(5, n // 1000) if case["call"] not in ("batch", "graph", "batch_host", "serve") else max(5, n // 250)


def _one_event(case, n, gen):
    """coords (dim, n) float32, weight (n,) float32 and the blob of every point (-1: noise) of a single
    event: blobs concatenated, then noise, as the reference's generator writes its sets."""
    dim, dev = case["dim"], "cuda"

    def rand(*s):
        return torch.rand(*s, generator=gen, device=dev)

    def randn(*s):
        return torch.randn(*s, generator=gen, device=dev)

    if case["data"] == "barrel":
        nb = max(8, n // 600)
        nin = int(0.85 * n)
        own = torch.arange(nin, device=dev) * nb // nin
        centre = torch.stack([6.0 * rand(nb) - 3.0, 2.0 * math.pi * rand(nb) - math.pi])
        sig = 0.02 + 0.05 * rand(nb)
        pts = centre[:, own] + randn(2, nin) * sig[own]
        noise = torch.stack([6.0 * rand(n - nin) - 3.0, 2.0 * math.pi * rand(n - nin) - math.pi])
        c = torch.cat([pts, noise], 1)
        c[1] = torch.remainder(c[1] + math.pi, 2.0 * math.pi) - math.pi
        w = -torch.log1p(-rand(n)) + 1e-3
    elif case["data"] == "blobs3d":
        nb = max(6, int(5000 * n / 4194304))
        box = 500.0 * (nb / 5000.0) ** (1.0 / 3.0)
        nin = int(0.85 * n)
        own = torch.arange(nin, device=dev) * nb // nin
        sig = 0.2 + 0.8 * rand(3, nb)
        pts = (box * rand(3, nb))[:, own] + randn(3, nin) * sig[:, own]
        c = torch.cat([pts, box * rand(3, n - nin)], 1)
        w = torch.exp(0.5 * randn(n))
    else:
        nb = _blob_count(case, n)
        box = 100.0 * (nb / 20.0) ** (1.0 / dim)
        nin = int(0.9 * n)
        own = torch.arange(nin, device=dev) * nb // nin
        c = torch.cat([(0.05 * box + 0.9 * box * rand(dim, nb))[:, own] + randn(dim, nin), box * rand(dim, n - nin)], 1)
        w = 0.5 + rand(n)
    own = torch.cat([own, torch.full((n - nin,), -1, dtype=own.dtype, device=dev)])
    return c.float().contiguous(), w.float().contiguous(), own.to(torch.int32)


def _many_events(case, gen):
    """coords (dim, n), weight (n,) and event offsets of a batch."""
    sizes = _event_sizes(case)
    off = np.concatenate([[0], np.cumsum(sizes)])
    n, E, dim, dev = int(off[-1]), len(sizes), case["dim"], "cuda"
    toff = torch.as_tensor(off, device=dev)
    ev = torch.repeat_interleave(torch.arange(E, device=dev), toff[1:] - toff[:-1], output_size=n)
    u = torch.rand(n, generator=gen, device=dev)
    if case["data"] == "calo":
        # 3-30 showers an event with exponential energies; members in proportion to the energy
        most, frac, box = 30, 0.8, 200.0
        ns = torch.randint(3, most + 1, (E,), generator=gen, device=dev)
        energy = -torch.log1p(-torch.rand(E, most, generator=gen, device=dev)) + 1e-6
        sig = 0.5 + 2.5 * torch.rand(E, most, generator=gen, device=dev)
    else:
        most, frac, box = 64, 0.9, 100.0 if dim == 4 else 60.0
        ns = torch.clamp((toff[1:] - toff[:-1]) // 250, 5, most)
        energy = torch.ones(E, most, device=dev)
        sig = torch.ones(E, most, device=dev)
    energy = energy * (torch.arange(most, device=dev)[None] < ns[:, None])
    cum = torch.cumsum(energy, 1) / energy.sum(1, keepdim=True)
    centre = box * torch.rand(E, most, dim, generator=gen, device=dev)
    rank = torch.arange(n, device=dev) - toff[ev]
    size = (toff[1:] - toff[:-1])[ev]
    is_noise = rank >= (frac * size)
    b = torch.searchsorted(cum[ev], (rank / (frac * size)).clamp(max=0.999999)[:, None].float()).squeeze(1).clamp(max=most - 1)
    b = torch.minimum(b, ns[ev] - 1)
    c = torch.empty(dim, n, device=dev)
    for d in range(dim):
        z = torch.randn(n, generator=gen, device=dev)
        noise = box * torch.rand(n, generator=gen, device=dev)
        c[d] = torch.where(is_noise, noise, centre[ev, b, d] + sig[ev, b] * z)
    w = (-torch.log1p(-u) + 1e-3) if case["data"] == "calo" else 0.5 + u
    return c.contiguous(), w.contiguous(), off.astype(np.int32)


def _inputs(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    if "events" in case:
        return _many_events(case, gen)
    return _one_event(case, case["n"], gen)


def _stream():
    return torch.cuda.current_stream().cuda_stream


def _out_tensors(names, n):
    return {k: torch.empty(n, dtype=torch.float32 if k in _FLOAT_OUT else torch.int32, device="cuda") for k in names}


def _pinned(t):
    h = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    h.copy_(t)
    return h


# ---- a case's program --------------------------------------------------------------------------
def prepare(case, seed):
    torch.cuda.init()
    params, kern, met = _structs(case)
    st = {"case": case, "params": params, "kernel": kern, "metric": met}
    call = case["call"]
    a, w, third = _inputs(case, seed)
    n = w.shape[0]
    if call == "python":
        st["table"] = np.concatenate([a.cpu().numpy(), w.cpu().numpy()[None]])
        return st
    if call == "serve":
        c, wh = a.cpu().numpy(), w.cpu().numpy()
        st["events"] = [(np.ascontiguousarray(c[:, i:j]), np.ascontiguousarray(wh[i:j]))
                        for i, j in zip(third[:-1], third[1:])]
        cfg = capi.ServerConfig(ndim=case["dim"], max_batch_events=256, max_event_points=20000,
                                device_budget_bytes=1 << 29)
        st["server"] = capi.Server(cfg, params, kern, met)
        return st
    st["ctx"] = capi.Context(torch.cuda.current_device())
    if call == "host":
        st["coords"], st["weight"] = a.cpu().numpy(), w.cpu().numpy()
    elif call == "batch_host":
        st["coords"], st["weight"], st["off"] = _pinned(a), _pinned(w), third
        st["out"] = {k: torch.empty(n, dtype=torch.int32, pin_memory=True) for k in ("cluster_index", "is_seed")}
        st["ncl"] = torch.empty(len(third) - 1, dtype=torch.int32, pin_memory=True)
    else:
        st["coords"], st["weight"] = a, w
        if call == "event":
            st["out"] = _out_tensors(_EVENT_OUT, n)
        elif call in ("batch", "graph"):
            st["off"] = third
            st["out"] = _out_tensors(_BATCH_OUT, n)
            st["ncl"] = torch.empty(len(third) - 1, dtype=torch.int32, device="cuda")
        elif call == "clusters":
            st["labels"] = third
            st["cap"] = int(third.max().item()) + 1
            st["offsets"] = torch.empty(n + 1, dtype=torch.int32, device="cuda")
            st["points"] = torch.zeros(n, dtype=torch.int32, device="cuda")
            st["centroids"] = torch.empty(st["cap"], case["dim"], device="cuda")
            st["sizes"] = torch.empty(st["cap"], dtype=torch.int32, device="cuda")
        else:
            st["labels"] = third
            st["score"] = torch.empty(n, device="cuda")
    torch.cuda.synchronize()
    if call == "graph":
        side = torch.cuda.Stream()
        st["graph"] = st["ctx"].capture_batch(a.data_ptr(), w.data_ptr(), case["dim"], third,
                                              {k: t.data_ptr() for k, t in st["out"].items()}, params, kern, met,
                                              ncl_ptr=st["ncl"].data_ptr(), stream=side.cuda_stream)
        st["side"] = side
    return st


def run(st):
    case, call = st["case"], st["case"]["call"]
    params, kern, met, dim = st["params"], st["kernel"], st["metric"], case["dim"]
    if call == "python":
        from cluestering_alpaka3_b200.clusterer import clusterer
        c = clusterer(params.dc, params.rhoc, params.dm)
        c.choose_kernel(case["kernel"], kern.par)
        return c.fit_predict(st["table"])
    if call == "serve":
        srv = st["server"]
        tickets = [srv.submit(c, w) for c, w in st["events"]]
        res = [srv.wait(t) for t in tickets]
        return {k: np.concatenate([getattr(r, k) for r in res]) for k in _EVENT_OUT}
    ctx = st["ctx"]
    if call == "host":
        r = ctx.make_clusters_host(st["coords"], st["weight"], params, kern, met, stream=_stream())
        return {k: getattr(r, k) for k in _EVENT_OUT}
    if call == "event":
        ctx.make_clusters_device(st["coords"].data_ptr(), st["weight"].data_ptr(), dim, st["weight"].shape[0],
                                 {k: t.data_ptr() for k, t in st["out"].items()}, params, kern, met, stream=_stream())
        return st["out"]
    if call == "batch":
        ctx.batch_device(st["coords"].data_ptr(), st["weight"].data_ptr(), dim, st["off"],
                         {k: t.data_ptr() for k, t in st["out"].items()}, params, kern, met,
                         ncl_ptr=st["ncl"].data_ptr(), stream=_stream())
        return {**st["out"], "n_clusters": st["ncl"]}
    if call == "graph":
        st["graph"].launch(_stream())
        return {**st["out"], "n_clusters": st["ncl"]}
    if call == "batch_host":
        ctx.batch_host(st["coords"].numpy(), st["weight"].numpy(), st["off"], params, kern, met, stream=_stream(),
                       out={k: t.numpy() for k, t in st["out"].items()}, ncl=st["ncl"].numpy())
        return {**{k: t.numpy() for k, t in st["out"].items()}, "n_clusters": st["ncl"].numpy()}
    n = st["weight"].shape[0]
    if call == "clusters":
        nc, nin = ctx.get_clusters(st["labels"].data_ptr(), n, st["offsets"].data_ptr(), st["points"].data_ptr(),
                                   stream=_stream())
        ctx.cluster_centroids_device(st["coords"].data_ptr(), st["labels"].data_ptr(), dim, n, st["cap"],
                                     st["centroids"].data_ptr(), st["sizes"].data_ptr(), stream=_stream())
        return {"offsets": st["offsets"], "points": st["points"][:nin], "centroids": st["centroids"],
                "sizes": st["sizes"], "n_clusters": nc}
    mean = ctx.silhouette_device(st["coords"].data_ptr(), st["labels"].data_ptr(), dim, n, st["score"].data_ptr(),
                                 stream=_stream())
    return {"score": st["score"][st["labels"] >= 0], "mean": mean}


# ---- bounds and exact values ---------------------------------------------------------------------
def _close_fraction(case, dc):
    """Share of its own blob's members within dc of a member (Gaussian blob, typical sigma)."""
    sigma = {"calo": 1.75, "blobs3d": 0.6, "barrel": 0.045}.get(case["data"], 1.0)
    x = dc * dc / (4.0 * sigma * sigma)
    return float(torch.special.gammainc(torch.tensor(0.5 * case["dim"], dtype=torch.float64),
                                        torch.tensor(x, dtype=torch.float64)))


def work(case):
    dim = case["dim"]
    pair = 3 * dim + 2  # difference, square, sum per coordinate; kernel value and accumulation
    if case["call"] == "clusters":
        n = case["n"]
        return {"bytes": n * 4 * (1 + 1 + dim) + (n + 1) * 4, "flops": n * dim}
    if case["call"] == "silhouette":
        n = case["n"]
        return {"bytes": n * 4 * (dim + 2), "flops": 0.9 * n * n * (3 * dim + 1)}
    dc = _settings(case)[0]
    if "events" in case:
        n = int(_event_sizes(case).sum())
        members = n / case["events"] / 8
    else:
        n = case["n"]
        members = {"barrel": 510, "blobs3d": 713}.get(case["data"], 900)
        members = min(members, n / 5)
    outs = {"python": 1, "batch_host": 2, "batch": 4, "graph": 4}.get(case["call"], 5)
    return {"bytes": n * 4 * (dim + 1 + outs), "flops": n * members * _close_fraction(case, dc) * pair}


def _pair_values(case, x, y):
    """Distances (float64) between the columns of x (dim, a) and y (dim, b)."""
    metric = case.get("metric", "euclidean")
    par = _metric_par(metric, case["dim"])
    acc = None
    for d in range(case["dim"]):
        t = (x[d][:, None] - y[d][None, :]).abs_()
        if metric == "periodic" and par[d] > 0:
            period = float(np.float32(par[d]))
            t = torch.minimum(t, (period - t).abs_())
        if metric == "manhattan":
            acc = t if acc is None else acc.add_(t)
        elif metric in ("chebyshev", "weighted_chebyshev"):
            t = t * par[d] if metric == "weighted_chebyshev" else t
            acc = t if acc is None else torch.maximum(acc, t)
        else:
            t = t.mul_(t)
            t = t.mul_(par[d]) if metric == "weighted_euclidean" else t
            acc = t if acc is None else acc.add_(t)
    return acc.sqrt_() if metric in ("euclidean", "weighted_euclidean", "periodic") else acc


def _exact_rho(case, c, w, chunk=2048):
    """Local densities of one event in 64 bits: the points are swept along the first coordinate, and
    each piece meets the points within reach of it."""
    dc, _, _, kind, kernel, metric, _ = _settings(case)
    dc = float(np.float32(dc))
    par = [float(np.float32(v)) for v in kernel]
    x, order = torch.sort(c[0].double())
    pts, wt = c.double()[:, order], w.double()[order]
    n, rho = x.shape[0], torch.empty(c.shape[1], dtype=torch.float64, device=c.device)
    reach = dc * (2.0 if metric.startswith("weighted") else 1.0) * (1 + 1e-6)
    starts = torch.arange(0, n, chunk, device=x.device)
    lo = torch.searchsorted(x, x[starts] - reach).tolist()
    hi = torch.searchsorted(x, x[torch.clamp(starts + chunk - 1, max=n - 1)] + reach, right=True).tolist()
    for k, s in enumerate(range(0, n, chunk)):
        e = min(n, s + chunk)
        step = max(1, min(e - s, (1 << 26) // max(1, hi[k] - lo[k])))
        for a in range(s, e, step):
            b = min(e, a + step)
            d = _pair_values(case, pts[:, a:b], pts[:, lo[k]:hi[k]])
            if kind == "flat":
                v = torch.full_like(d, par[0])
            elif kind == "exp":
                v = par[1] * torch.exp(-par[0] * d)
            else:
                v = par[2] * torch.exp(-(d - par[0]) ** 2 / (2 * par[1] * par[1]))
            v.masked_fill_(d > dc, 0.0)
            rows = torch.arange(a, b, device=x.device)
            v[rows - a, rows - lo[k]] = 1.0
            rho[order[a:b]] = v @ wt[lo[k]:hi[k]]
    return rho


def exact(case, seed):
    call = case["call"]
    if call in ("python", "batch_host"):
        return None  # labels and flags alone
    a, w, third = _inputs(case, seed)
    if call == "clusters":
        keep = third >= 0
        k = int(third.max().item()) + 1
        cnt = torch.bincount(third[keep].long(), minlength=k).double()
        cen = torch.stack([torch.zeros(k, dtype=torch.float64, device=a.device).index_add_(
            0, third[keep].long(), a[d][keep].double()) / cnt for d in range(case["dim"])], 1)
        return {"offsets": None, "points": None, "centroids": cen, "sizes": None, "n_clusters": None}
    if call == "silhouette":
        keep = third >= 0
        x, lab = a[:, keep].double(), third[keep].long()
        k = int(lab.max().item()) + 1
        cnt = torch.bincount(lab, minlength=k).double()
        onehot = torch.nn.functional.one_hot(lab, k).double()
        score = torch.empty(x.shape[1], dtype=torch.float64, device=a.device)
        for s in range(0, x.shape[1], 2048):
            sums = _pair_values(case, x[:, s:s + 2048], x) @ onehot
            mine = lab[s:s + 2048]
            own = sums.gather(1, mine[:, None]).squeeze(1) / (cnt[mine] - 1)
            mean = sums / cnt
            mean.scatter_(1, mine[:, None], math.inf)
            other = mean.amin(1)
            score[s:s + 2048] = (other - own) / torch.maximum(own, other)
        return {"score": score, "mean": float(score.mean().item())}
    if "events" in case:
        rho = torch.cat([_exact_rho(case, a[:, i:j], w[i:j]) for i, j in zip(third[:-1], third[1:])])
        names = _EVENT_OUT if call == "serve" else _BATCH_OUT + ("n_clusters",)
    else:
        rho = _exact_rho(case, a, w)
        names = _EVENT_OUT
    # nearest highers, their distances and the labels follow from comparisons of 32-bit densities
    return {k: rho if k == "rho" else None for k in names}
