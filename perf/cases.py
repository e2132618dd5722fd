"""The self-join work that a program using hegjoin_b200 has it do, as measurable cases.

Each case is one whole use of the library's public entry points: points in, results out.  A
program has its points on the device (or, for `host` and `serve`, in host memory) and chooses
epsilon and the number of indexed dimensions; it keeps no index between datasets, so building
the grid index and the workload order is part of a pass.

Kinds
    join     GridIndex, join and the sorted CSR of all neighbour lists
    host     the same from host memory through self_join_host
    stream   GridIndex and join_stream with per-query digests: results too large to keep
    index    GridIndex, workload order and the export of both
    serve    a stream of small requests through a running Server, each result's CSR taken

Data follows the reference generator's distribution (coordinates i.i.d. Exp(rate = 40) in
[0, 1)), or the skewed mix of 80% of that and 20% in 64 tight Gaussian clusters.  Results go
into buffers that the program keeps, sized for more pairs than it expects; what is past a
result's end stays zero.  The outputs are point ids, counts and 64-bit hashes: whole numbers,
which have no value in 64-bit floating point to be compared with.
"""
import math

import numpy as np
import torch

import hegjoin_b200 as hj

RATE = 40.0
CLUSTERS, SIGMA, CLUSTERED = 64, 0.002, 0.2
SERVE_DIMS = (2, 6, 18, 32, 90)
EPS_18D, EPS_90D, EPS_SKEW6D, EPS_2D = 0.04033349081873894, 0.20804697275161743, 0.003275492461398244, 0.002


def _case(name, kind, n, d, k, dtype, eps, neighbours, data="exp40", refine="auto"):
    return {"name": name, "kind": kind, "n": n, "d": d, "k": k, "dtype": dtype, "eps": eps,
            "neighbours": neighbours, "data": data, "refine": refine}


def listed():
    return [
        # a very small dataset: launches, allocations and host round trips are the whole cost
        _case("join_2d_f64_1k", "join", 1000, 2, 2, "f64", 0.005, 26),
        # a small sparse dataset, most cells with a point or two
        _case("join_6d_20k", "join", 20_011, 6, 6, "f32", 0.017, 42),
        # fewer indexed than data dimensions, double precision
        _case("join_5d_f64_k3_120k", "join", 120_000, 5, 3, "f64", 0.008, 39),
        # a dimension that no kernel is specialised for
        _case("join_7d_300k", "join", 300_007, 7, 6, "f32", 0.013, 46),
        # an everyday high-dimensional join that starts from host memory
        _case("host_18d_100k", "host", 100_003, 18, 6, "f32", 0.054, 44),
        # the tensor-core filter asked for by name with BF16 operands
        _case("join_32d_bf16_150k", "join", 150_001, 32, 6, "f32", 0.092, 60, refine="tc_bf16"),
        # the 18-D configuration at half its 5,000,000 points
        _case("join_18d_2500k", "join", 2_500_000, 18, 6, "f32", EPS_18D, 25),
        # the 90-D configuration, a ragged number of points
        _case("join_90d_400k", "join", 400_009, 90, 6, "f32", EPS_90D, 24),
        # the skewed 6-D configuration: millions of one-point cells and a few crowded ones
        _case("join_skew6d_4m", "join", 4_000_000, 6, 6, "f32", EPS_SKEW6D, 80, data="skewed"),
        # the 2-D configuration: thousands of neighbours per point, streamed in batches
        _case("stream_2d_f64_1m", "stream", 1_000_000, 2, 2, "f64", EPS_2D, 4700),
        # the index and workload order of the skewed 6-D configuration at its full size
        _case("index_skew6d_10m", "index", 10_000_000, 6, 6, "f32", EPS_SKEW6D, 200, data="skewed"),
        # a service with eight requests in flight, each a small join of its own shape
        {"name": "serve_small_48", "kind": "serve", "requests": 48, "n_min": 1000, "n_max": 20_000, "workers": 8},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _eps_for(rng, n, d, target):
    """An epsilon near a mean of `target` neighbours for n Exp(40) points: the quantile of a
    sample's pair distances, extended below the sample's resolution by the power law r^d."""
    g = np.random.default_rng(rng.getrandbits(32))
    x = g.exponential(1.0 / RATE, (1500, d))
    d2 = (x * x).sum(1)[:, None] + (x * x).sum(1)[None] - 2.0 * x @ x.T
    r = np.sqrt(np.maximum(d2[np.triu_indices(len(x), 1)], 0.0))
    f = target / n
    f0 = max(f, 1e-4)
    return float(np.float32(np.quantile(r, min(1.0, f0)) * (f / f0) ** (1.0 / d)))


def draw(rng):
    kind = rng.choice(["low", "low", "low", "high", "high", "high", "host", "skew", "stream", "index", "serve"])
    if kind == "serve":
        return {"kind": "serve", "requests": rng.randint(8, 64), "n_min": rng.randint(300, 2000),
                "n_max": rng.randint(5000, 30_000), "workers": rng.choice([1, 4, 8])}
    target = rng.randint(8, 96)
    if kind in ("low", "high", "host"):
        if kind == "low":
            d = rng.choice([2, 2, 3, 4, 5, 6, 7, 10, 12])
            n, dtype = _log(rng, 700, 600_000), rng.choice(["f32", "f32", "f64"])
        else:
            d = rng.choice([16, 18, 18, 24, 32, 64, 90, 120])
            n, dtype = _log(rng, 700, 200_000 if kind == "host" else 1_200_000 if d <= 18 else 250_000), "f32"
        k = min(d, 6) if rng.random() < 0.8 else min(d, rng.randint(2, 5))
        refine = rng.choice(["auto", "auto", "tc_f16", "tc_bf16"]) if d >= 16 else "auto"
        c = _case("", "host" if kind == "host" else "join", n, d, k, dtype, _eps_for(rng, n, d, target), target,
                  refine=refine)
    elif kind == "skew":
        n = _log(rng, 20_000, 3_000_000)
        c = _case("", "join", n, 6, 6, "f32", EPS_SKEW6D * rng.uniform(0.7, 1.1), 20 * n / 1e6, data="skewed")
    elif kind == "stream":
        n, eps = _log(rng, 50_000, 900_000), EPS_2D * rng.uniform(0.4, 1.0)
        c = _case("", "stream", n, 2, 2, rng.choice(["f32", "f64"]), eps, 4700 * (n / 1e6) * (eps / EPS_2D) ** 2)
    else:
        n, data = _log(rng, 20_000, 8_000_000), rng.choice(["exp40", "skewed"])
        d = 6 if data == "skewed" else rng.choice([2, 6, 18])
        n = min(n, 4_000_000) if d == 18 else n
        c = _case("", "index", n, d, min(d, 6), rng.choice(["f32", "f64"]) if d < 18 else "f32",
                  {2: EPS_2D, 6: EPS_SKEW6D * 2, 18: EPS_18D}[d], target, data=data)
    del c["name"]
    return c


def _points(case, gen):
    n, d = case["n"], case["d"]
    dtype = torch.float32 if case["dtype"] == "f32" else torch.float64
    x = torch.empty((n, d), dtype=dtype, device="cuda").exponential_(RATE, generator=gen)
    if case["data"] == "skewed":
        m = int(round(n * CLUSTERED))
        centres = torch.rand((CLUSTERS, d), dtype=dtype, device="cuda", generator=gen)
        which = torch.randint(CLUSTERS, (m,), device="cuda", generator=gen)
        x[n - m:] = centres[which] + SIGMA * torch.randn((m, d), dtype=dtype, device="cuda", generator=gen)
    return x.clamp_(0.0, 1.0 - 2.0 ** -20)


def _shapes(case):
    """(n, d, target neighbours) of each request: a function of the case alone."""
    rng = np.random.default_rng([case["requests"], case["n_min"], case["n_max"]])
    lo, hi = math.log(case["n_min"]), math.log(case["n_max"])
    return [(int(math.exp(rng.uniform(lo, hi))), int(rng.choice(SERVE_DIMS)), float(rng.uniform(4, 128)))
            for _ in range(case["requests"])]


def _requests(case, gen):
    out = []
    for n, d, target in _shapes(case):
        x = _points({"n": n, "d": d, "dtype": "f32", "data": "exp40"}, gen)
        r = torch.cdist(x[:256].double(), x.double()).reshape(-1)
        level = max(1, int(r.numel() * min(1.0, target / n)))
        eps = float(np.float32(r.kthvalue(level).values.item()))
        out.append((x.cpu().numpy(), min(d, 6), max(eps, 1e-6)))
    return out


def _room(n, neighbours):
    return int(min(n * (3.0 * neighbours + 64.0), float(n) * n))


def _ints(*shape, dtype=torch.int32):
    return torch.zeros(shape, dtype=dtype, device="cuda")


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind, n = case["kind"], case.get("n")
    if kind == "serve":
        shapes = _shapes(case)
        state = {"server": hj.Server(workers=case["workers"]), "requests": _requests(case, gen),
                 "room": [_room(m, t) for m, _, t in shapes]}
        # one buffer for all lists and one for all offsets; each request has its part
        state["all_values"] = _ints(sum(state["room"]))
        state["all_offsets"] = _ints(sum(m + 1 for m, _, _ in shapes), dtype=torch.int64)
        state["values"] = list(state["all_values"].split(state["room"]))
        state["offsets"] = list(state["all_offsets"].split([m + 1 for m, _, _ in shapes]))
    elif kind == "index":
        state = {"points": _points(case, gen), "cell_ids": _ints(n, dtype=torch.int64), "first": _ints(n),
                 "last": _ints(n), "order": _ints(n, 2)}
    elif kind == "stream":
        state = {"points": _points(case, gen)}
    else:
        state = {"points": _points(case, gen), "values": _ints(_room(n, case["neighbours"]))}
        if kind == "host":
            state["points"] = state["points"].cpu().numpy()
    torch.cuda.synchronize()
    return {"case": case, **state}


def _fill(buffer, part):
    buffer[:part.shape[0]].copy_(part)
    return buffer


def run(state):
    case = state["case"]
    if case["kind"] == "serve":
        server = state["server"]
        tickets = [server.submit(x, k, eps) for x, k, eps in state["requests"]]
        for t, off, val in zip(tickets, state["offsets"], state["values"]):
            offsets, values = server.wait(t)[0].to_csr(sort_lists=True)
            _fill(off, offsets)
            _fill(val, values)
        return {"offsets": state["all_offsets"], "values": state["all_values"]}
    k, eps = case["k"], case["eps"]
    if case["kind"] == "host":
        result = hj.self_join_host(state["points"], k, eps, refine=case["refine"])
    else:
        index = hj.GridIndex(state["points"], k, eps)
        if case["kind"] == "index":
            total = index.sort_by_workload()
            ids, first, last, lookup, _ = index.export()
            order, origin = index.workload_export()
            return {"candidates": total, "cell_ids": _fill(state["cell_ids"], ids),
                    "first": _fill(state["first"], first), "last": _fill(state["last"], last), "lookup": lookup,
                    "order": _fill(state["order"], order), "origin": origin}
        if case["kind"] == "stream":
            stats, (count, total, xor) = hj.join_stream(index, refine=case["refine"])
            return {"pairs": int(stats.total_pairs), "count": count, "sum": total, "xor": xor}
        result = hj.join(index, refine=case["refine"])
    offsets, values = result.to_csr(sort_lists=True)
    return {"offsets": offsets, "values": _fill(state["values"], values)}


def exact(case, seed):
    return None


def _candidates(n, k, eps):
    """Expected (query, candidate) pairs of the grid's 3^k stencils for Exp(40) points: per
    indexed dimension, two points fall into the same or adjacent cells of width eps with
    probability (1 - a)(1 + 2a) / (1 + a), a = exp(-40 eps)."""
    a = math.exp(-RATE * eps)
    return float(n) * n * ((1 - a) * (1 + 2 * a) / (1 + a)) ** k


def work(case):
    """Points read once and results written once; three operations per dimension for every
    candidate pair that the grid leaves (no pair of distinct points need be evaluated twice)."""
    if case["kind"] == "serve":
        shapes = _shapes(case)
        return {"bytes": float(sum(n * (4 * d + 8 + 4 * t) for n, d, t in shapes)),
                "flops": float(sum(0.3 * 0.5 * n * n * 3 * d for n, d, t in shapes))}
    n, d = case["n"], case["d"]
    points = n * d * (4 if case["dtype"] == "f32" else 8)
    if case["kind"] == "index":
        # lookup and origin per point; ids, bounds and order per cell, about 0.6 cells per point
        # where the grid is sparse
        return {"bytes": points + 8 * n + 0.6 * n * 24, "flops": 0.0}
    out = 20 * n if case["kind"] == "stream" else 8 * n + 4 * n * case["neighbours"]
    share = 1.0 - CLUSTERED if case["data"] == "skewed" else 1.0
    cand = _candidates(share * n, case["k"], case["eps"])
    if case["data"] == "skewed":
        cand += CLUSTERS * (CLUSTERED * n / CLUSTERS) ** 2 * 0.1
    return {"bytes": float(points + out), "flops": 0.5 * cand * 3 * d}
