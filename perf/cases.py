"""The joins that this engine is timed on, through its public entry points.

``listed`` holds the calls users make -- one-shot counts of resident or host
arrays in each distance form, two-set joins, pair lists, batches of joins and
the serving loop -- from a thousand points to the benchmark's sizes; ``draw``
gives further calls of the same ranges. ``prepare`` makes the inputs from a
seed (on the GPU; as numpy arrays where the call takes host data) with the
generators' distributions of ``hilbertjoin_b200.workloads``: i.i.d. U[0,1), or
a Gaussian mixture whose component weights (quantiles of an exponential) and
sigmas (log-spaced in [0.005, 0.05]) are paired at random. eps is calibrated on
the set's own first points for a mean neighbour count, as the benchmark does.
``run`` is one call; ``work`` the bytes of the inputs and outputs and the
2 d operations of every pair that no cell grid can rule out at these eps (all
pairs of uniform data, the pairs within a component of clustered data).
"""
import ctypes
import math
import random

import numpy as np
import torch

import hilbertjoin_b200 as hj
from hilbertjoin_b200.batching import batch_count
from hilbertjoin_b200.serving import Server

SAMPLE = 4096
DIMS = (8, 16, 32, 64, 128)  # of the batch and serving streams


def listed():
    return [
        # an interactive count of a small resident set: launches and latency
        _case("self_1500_d8_auto", "self", n=1500, d=8, nbrs=8, form="auto"),
        # the library's default call: a host FP64 array, plain form (an odd size of clustered points)
        _case("self_20011_d16_host_plain", "self", n=20011, d=16, data="gmm", parts=16, dtype="f64", host=True,
              nbrs=16, form="plain"),
        # a two-set join of uneven ragged sets with the dimensions reordered, as the join executable runs it
        _case("join_30011x70001_d100_auto", "join", n=30011, m=70001, d=100, nbrs=20, form="auto", reorder=True),
        # the benchmark's two-set configuration at ~20 partners per point
        _case("join_200k_d20_fp16", "join", n=200_000, m=200_000, d=20, nbrs=20, form="fp16"),
        # FP64 rows in the fastest form (the benchmark's 200k x 64 set)
        _case("self_200k_d64_f64_fp16", "self", n=200_000, d=64, dtype="f64", nbrs=32, form="fp16"),
        # the headline: 1M x 64, 32 neighbours
        _case("self_1M_d64_fp16", "self", n=1_000_000, d=64, nbrs=32, form="fp16"),
        # the largest clustered configuration: 4M x 28, 64 components, ~100 neighbours
        _case("self_4M_d28_gmm_auto", "self", n=4_000_000, d=28, data="gmm", parts=64, nbrs=100, form="auto"),
        # the other two operand formats, on clustered and on uniform data
        _case("self_300k_d32_gmm_tf32", "self", n=300_007, d=32, data="gmm", parts=16, nbrs=32, form="tf32"),
        _case("self_150k_d128_bf16x3", "self", n=150_000, d=128, nbrs=32, form="bf16x3"),
        # the pairs themselves, host FP32 points
        _case("pairs_100k_d16_host", "pairs", n=100_000, d=16, data="gmm", parts=32, host=True, nbrs=20, form="plain"),
        # many joins of uneven sizes as one batch, planned and counted in one call
        _case("batch_32_jobs", "batch", n=50_000, d=128, jobs=32, form="fp16"),
        # a burst of requests to a running server whose sets are resident
        _case("serve_64_requests", "serve", n=100_000, d=128, jobs=64, form="auto"),
    ]


def draw(rng):
    call = rng.choices(["self", "join", "pairs", "batch", "serve"], [8, 5, 2, 1, 1])[0]
    if call in ("batch", "serve"):
        return _case(None, call, n=_log(rng, 5_000, 100_000 if call == "serve" else 50_000), d=rng.choice(DIMS[1:]),
                     jobs=rng.randint(4, 32 if call == "batch" else 64), form="fp16" if call == "batch" else "auto")
    c = _case(None, call, n=_log(rng, 1_000, 1_000_000), d=_log(rng, 2, 256) if rng.random() < 0.5 else
              rng.choice((8, 16, 20, 28, 32, 64, 100, 128)), data=rng.choice(("uniform", "gmm")),
              parts=rng.randint(4, 64), dtype=rng.choice(("f32", "f32", "f64")), host=rng.random() < 0.3,
              nbrs=_log(rng, 4, 100), reorder=rng.random() < 0.25,
              form=rng.choice(("auto", "auto", "fp16", "fp16", "tf32", "bf16x3", "plain")))
    c["m"] = _log(rng, 1_000, 1_000_000) if call == "join" else 0
    if call == "pairs":
        c.update(host=True, form="plain", n=min(c["n"], 200_000), nbrs=min(c["nbrs"], 20))
    while _cost(c) > 1.0:
        c["n"], c["m"] = int(c["n"] * 0.8), int(c["m"] * 0.8)
    return c


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed * 1009 + 7)
    if case["call"] == "batch":
        return {"case": case, "jobs": _jobs(case, g, seed)}
    if case["call"] == "serve":
        return {"case": case, "served": _Served(case, g, seed)}
    means = _means(case, g)
    a = _points(case, case["n"], g, means)
    b = _points(case, case["m"], g, means) if case["call"] == "join" else None
    eps = _calibrate(a, b, case["nbrs"])
    if case["host"]:
        a, b = a.cpu().numpy(), None if b is None else b.cpu().numpy()
    # a pair list goes to the caller's buffer, with room for four times the expected pairs
    out = np.zeros((2 * case["n"] * case["nbrs"], 2), dtype=np.uint64) if case["call"] == "pairs" else None
    return {"case": case, "a": a, "b": b, "eps": eps, "out": out}


def run(state):
    c = state["case"]
    if c["call"] == "batch":
        return np.array(batch_count(state["jobs"], form=c["form"]), dtype=np.int64)
    if c["call"] == "serve":
        return state["served"].burst()
    if c["call"] == "pairs":
        return _pairs(state)
    if c["call"] == "join":
        return hj.join_count(state["a"], state["b"], state["eps"], form=c["form"], reorder_dims=c["reorder"])
    return hj.self_join_count(state["a"], state["eps"], form=c["form"], reorder_dims=c["reorder"])


def exact(case, seed):
    """Counts and pair indices are whole numbers: no rounded outputs."""
    return None


def work(case):
    c, size = case, 8 if case["dtype"] == "f64" else 4
    if c["call"] in ("batch", "serve"):
        sets = [(_dict_case(c, i), x) for i, x in enumerate(_sizes(c, 0))]
        return {"bytes": sum(4 * n * d for _, (n, d) in sets), "flops": sum(float(n) * n * d for _, (n, d) in sets)}
    pairs = float(c["n"]) * c["m"] if c["call"] == "join" else 0.5 * c["n"] * (c["n"] - 1)
    near = pairs / (c["parts"] if c["data"] == "gmm" else 1)
    out = 8 * c["n"] * c["nbrs"] if c["call"] == "pairs" else 8
    return {"bytes": size * c["d"] * (c["n"] + c["m"]) + out, "flops": 2.0 * c["d"] * near}


def _pairs(state):
    """hj_self_join_pairs of the library's C interface into the caller's buffer; returns the buffer and the count."""
    c, x, out = state["case"], state["a"], state["out"]
    opts, count = hj.Opts(), ctypes.c_uint64(0)
    hj.lib().hj_opts_init(ctypes.byref(opts))
    opts.reorder_dims = int(c["reorder"])
    fn = hj.lib().hj_self_join_pairs if c["dtype"] == "f64" else hj.lib().hj_self_join_pairs_f32
    rc = fn(x.ctypes.data, x.shape[0], x.shape[1], state["eps"], ctypes.byref(opts), out.ctypes.data, len(out),
            ctypes.byref(count), None)
    if rc != hj.OK:
        raise hj.HJError(rc, hj.lib().hj_last_error().decode())
    return out.view(np.int64), int(count.value)


# ------------------------------------------------------------------ inputs


def _case(name, call, n, d, form, m=0, data="uniform", parts=1, dtype="f32", host=False, nbrs=0, reorder=False,
          jobs=0):
    c = {"name": name} if name else {}
    return {**c, "call": call, "n": n, "m": m, "d": d, "data": data, "parts": parts, "dtype": dtype, "host": host,
            "nbrs": nbrs, "reorder": reorder, "form": form, "jobs": jobs}


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _cost(c):
    """Share of the headline's time that a drawn join may take, by the engine's
    rates: the plain form, and clustered data above 64 dims, on FP64 cores."""
    pairs = c["n"] * (c["m"] or c["n"] / 2) / (4 if c["data"] == "gmm" else 1)
    slow = c["form"] == "plain" or (c["data"] == "gmm" and c["d"] > 48)
    return pairs * max(c["d"], 32) * (60 if slow else 2) / 3e13 + c["n"] * c["nbrs"] / 4e8


def _means(c, g):
    return None if c["data"] == "uniform" else torch.rand(c["parts"], c["d"], generator=g, device="cuda",
                                                          dtype=torch.float64)


def _points(c, n, g, means):
    if means is None:
        x = torch.rand(n, c["d"], generator=g, device="cuda", dtype=torch.float64)
    else:
        k = means.shape[0]
        q = (torch.arange(k, device="cuda", dtype=torch.float64) + 0.5) / k
        sigma = (0.005 * 10.0 ** q)[torch.argsort(means[:, 0])]
        which = torch.multinomial(-torch.log1p(-q), n, replacement=True, generator=g)
        x = torch.randn(n, c["d"], generator=g, device="cuda", dtype=torch.float64)
        x = (x * sigma[which, None] + means[which]).clamp_(0.0, 1.0 - 2.0 ** -24)
    return x if c["dtype"] == "f64" else x.float()


def _calibrate(a, b, nbrs):
    """eps for about `nbrs` neighbours per point, from the sets' first points (half of a small set)."""
    s, t = (x[:max(64, min(SAMPLE, x.shape[0] // 2))].double() for x in (a, a if b is None else b))
    d2 = (s * s).sum(1)[:, None] + (t * t).sum(1)[None, :] - 2.0 * (s @ t.T)
    if b is None:
        i = torch.triu_indices(len(s), len(s), 1, device="cuda")
        d2 = d2[i[0], i[1]]
    d2 = d2.flatten()
    share = min(1.0, nbrs / max(1, (a if b is None else b).shape[0] - 1))
    k = max(1, min(d2.numel(), int(share * d2.numel())))
    return float("%.7g" % math.sqrt(max(1e-12, float(torch.kthvalue(d2, k).values))))


def _sizes(c, seed):
    """(n, d) of the sets of a batch or of a server: n log-uniform up to c["n"], d of DIMS up to c["d"]."""
    rng = random.Random(seed)
    count = c["jobs"] if c["call"] == "batch" else 16
    dims = [d for d in DIMS if d <= c["d"]]
    return [(_log(rng, min(1_000, c["n"]), c["n"]), dims[i % len(dims)]) for i in range(count)]


def _dict_case(c, i):
    return {**c, "data": "gmm" if i % 2 else "uniform", "parts": 16, "d": 0}


def _jobs(c, g, seed):
    """Joins of uneven sets: 70% self-joins, the others against a set of half the size."""
    jobs = []
    for i, (n, d) in enumerate(_sizes(c, 0)):
        k = {**_dict_case(c, i), "d": d}
        means = _means(k, g)
        a = _points(k, n, g, means)
        b = _points(k, n // 2 + 1, g, means) if i % 10 >= 7 else None
        jobs.append((a, b, _calibrate(a, b, 8 + 8 * (i % 6))))
    return jobs


class _Served:
    """A server with its resident sets and a burst of requests: each set's
    self-join, or its join with the next set of its dimension."""

    def __init__(self, c, g, seed):
        self.server = Server(form=c["form"], memory_budget_bytes=16 << 30, max_inflight=8)
        sets, self.requests = [], []
        for i, (n, d) in enumerate(_sizes(c, 0)):
            k = {**_dict_case(c, i), "d": d}
            x = _points(k, n, g, _means(k, g))
            sets.append((self.server.upload(x.cpu().numpy()), x))
        for i in range(c["jobs"]):
            ha, a = sets[i % len(sets)]
            mate = [s for s in sets if s[1].shape[1] == a.shape[1] and s[0] != ha]
            pair = mate[i % len(mate)] if mate and i % 10 >= 7 else None
            eps = _calibrate(a, None if pair is None else pair[1], 8 + 8 * (i % 6))
            self.requests.append((ha, None if pair is None else pair[0], eps))

    def burst(self):
        ids = [self.server.submit(a, b, eps) for a, b, eps in self.requests]
        return np.array([self.server.wait(i)["count"] for i in ids], dtype=np.int64)

    def __del__(self):
        if getattr(self, "server", None) is not None:
            self.server.close()
