"""The work whose speed is measured: index builds, searches and serving at the
sizes of this repository's configurations, through its public entry points.

A case is a dict of plain values:

  kind     search    one batch of device-resident queries (SearchTables.search_device)
           host      one batch of host queries, results read back as arrays (SearchTables.search)
           pipeline  the classic program: index a host dataset, then search it (HashTables.index + search)
           build     index a device-resident dataset, then search a small batch of it (HashTables.index_device)
           serve     a burst of requests of mixed size, K and T through the serving loop (Server)
  data     generator of the points (see _points)
  n d      points and dimensions; l m w: tables, projections a table, bucket width
  q k t    queries, neighbours, probes a table
  near     1: queries are points of the dataset with a little noise (look-ups of
           known items), 0: held-out draws of the same distribution
  cand     distinct candidates a query has on average, for work()
"""

from __future__ import annotations

import math

import numpy as np
import torch

import culsh_gb300 as culsh

FLT_MAX = float(np.finfo(np.float32).max)


def _case(name, kind, data, n, d, l, m, w, q, k, t, near, cand):
    return dict(name=name, kind=kind, data=data, n=n, d=d, l=l, m=m, w=float(w), q=q, k=k, t=t, near=near, cand=cand)


def listed():
    return [
        # One interactive query on a small index: latency and launches.
        _case("one_query", "host", "gauss", 100_000, 128, 8, 8, 32.0, 1, 10, 16, 0, 760),
        # The reference program's own flow at its smallest configuration:
        # host arrays, index, one classic (T = 1) search of 1,000 queries.
        _case("pipeline_100k", "pipeline", "gauss", 100_000, 128, 8, 8, 32.0, 1_000, 10, 1, 0, 156),
        # Near-duplicate look-ups: narrow buckets, most probes find nothing.
        _case("lookup_1m", "search", "int", 1_000_000, 128, 16, 12, 16.0, 10_000, 10, 16, 1, 1),
        # Multiprobe search at recall 0.9 of clustered data, sparse candidate
        # sets, ragged sizes.
        _case("sparse_1m", "search", "gauss", 1_000_003, 100, 8, 8, 28.0, 9_973, 10, 16, 0, 7_500),
        # The benchmark's headline: data without neighbourhoods at recall 0.9,
        # half of the dataset is a candidate of each query.
        _case("dense_1m", "search", "int", 1_000_000, 128, 16, 12, 825.0, 10_000, 10, 16, 0, 576_000),
        # The same data for a re-ranker that asks for 100 neighbours.
        _case("dense_1m_k100", "search", "int", 1_000_000, 128, 16, 12, 825.0, 1_000, 100, 16, 0, 573_000),
        # High-dimensional unit vectors, many probes.
        _case("sphere_d960", "search", "sphere", 1_000_000, 960, 32, 16, 2.0, 1_000, 10, 64, 0, 13_300),
        # Heavy-tailed clusters: candidate counts of a batch differ by orders
        # of magnitude.
        _case("zipf_4m", "search", "zipf", 4_000_000, 128, 20, 10, 24.0, 1_000, 50, 32, 0, 94_000),
        # Online serving of a large index: 24 requests of 1 to 4,096 queries,
        # K 10 or 100, T 1, 8 or 32.
        _case("serve_10m", "serve", "many", 10_000_000, 96, 20, 14, 36.0, 24, 100, 32, 0, 1_000),
        # Index builds: the multiprobe configuration (every point its own
        # bucket), high dimensions, the largest index.
        _case("build_1m", "build", "int", 1_000_000, 128, 16, 12, 16.0, 256, 10, 16, 1, 1),
        _case("build_d960", "build", "sphere", 1_000_000, 960, 32, 16, 0.25, 256, 10, 64, 1, 1),
        _case("build_10m", "build", "many", 10_000_000, 96, 20, 14, 5.0, 256, 10, 8, 1, 1),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One case of the listed ones' ranges."""
    kind = rng.choice(["host", "pipeline", "search", "search", "dense", "uneven", "serve", "build", "build"])
    t = rng.choice([1, 2, 5, 8, 16, 24, 32, 64])
    k = rng.choice([1, 5, 10, 10, 20, 50, 100])
    if kind == "dense":
        # integer features at a width where most points are candidates
        n, d, m = _log_int(rng, 30_000, 1_200_000), rng.randrange(24, 129), rng.randrange(8, 13)
        q = _log_int(rng, 64, max(65, min(8_000, int(1.0e9 / n))))
        return _pure("search", "int", n, d, rng.randrange(8, 17), m, 825.0 * math.sqrt(d / 128), q, k,
                     rng.choice([8, 16, 16, 24]), 0, n // 2)
    if kind == "uneven":
        n, d = _log_int(rng, 1_000_000, 4_000_000), rng.randrange(48, 129)
        return _pure("search", "zipf", n, d, rng.randrange(12, 21), rng.randrange(9, 12), 24.0 * math.sqrt(d / 128),
                     _log_int(rng, 50, 500), k, rng.choice([8, 16, 32]), 0, n // 60)
    if kind == "serve":
        n, d, m = _log_int(rng, 100_000, 4_000_000), rng.randrange(48, 129), rng.randrange(10, 15)
        return _pure("serve", "many", n, d, rng.randrange(8, 21), m, 2.6 * math.sqrt(2.0 * d), rng.randrange(6, 25),
                     max(k, 20), max(t, 4), 0, n // 5000)
    if kind == "build":
        d = rng.choice([rng.randrange(16, 129), rng.randrange(64, 257), 960])
        n = _log_int(rng, 50_000, min(4_000_000, int(4.0e8 / d)))
        data, w = (("sphere", 0.25) if d == 960 else rng.choice([("int", 16.0), ("many", 5.0), ("gauss", 8.0)]))
        return _pure("build", data, n, d, rng.randrange(4, 21), rng.randrange(6, 17), w, 256, min(k, 10), t, 1, 1)
    # clustered data at the width where neighbours share buckets: about twice
    # the distance of two points of a cluster, wider with more projections
    d = rng.choice([rng.randrange(13, 129), rng.randrange(96, 257)])
    n = _log_int(rng, 20_000, min(1_500_000, int(2.0e8 / d)))
    m = rng.randrange(6, 17)
    w = math.sqrt(2.0 * d) * min(3.2, 2.0 + max(-0.3, (m - 8) / 8))
    q = {"host": _log_int(rng, 1, 4_000), "pipeline": _log_int(rng, 100, 4_000), "search": _log_int(rng, 16, 12_000)}[kind]
    if kind == "pipeline":
        n = min(n, 200_000)
    return _pure(kind, rng.choice(["gauss", "gauss", "many"]), n, d, rng.randrange(4, 17), m, w, q, k, t, 0, n // 200)


def _pure(*a):
    c = _case("", *a)
    del c["name"]
    return c


# ---------------------------------------------------------------------------
# inputs

def _gen(seed, device="cuda"):
    return torch.Generator(device=device).manual_seed(int(seed))


def _normal(g, *shape, scale=1.0):
    return torch.randn(*shape, generator=g, device=g.device, dtype=torch.float32).mul_(scale)


def _points(case, count, seed, g):
    """`count` points of the case's distribution; its centres come from `seed`,
    the draws from the generator g.

    gauss   100 clusters, centres N(0, 10^2), noise N(0, 1)
    many    5,000 such clusters
    zipf    10,000 clusters, centres N(0, 8^2), weights falling as rank^-1.2
    int     features rounded and clamped to 0..255, N(20, 30^2), 40 % zeros
    sphere  1,000 clusters of unit vectors, noise 0.05, normalised again
    """
    d, data = case["d"], case["data"]
    out = torch.empty(count, d, dtype=torch.float32, device="cuda")
    c = _gen(seed * 7 + 1)
    if data in ("gauss", "many"):
        centres = _normal(c, 100 if data == "gauss" else 5_000, d, scale=10.0)
    elif data == "zipf":
        centres = _normal(c, 10_000, d, scale=8.0)
        weights = torch.arange(1, 10_001, dtype=torch.float64, device="cuda").pow(-1.2)
        cdf = torch.cumsum(weights / weights.sum(), 0)
    elif data == "sphere":
        centres = torch.nn.functional.normalize(_normal(c, 1_000, d), dim=1)
    step = max(1, (1 << 27) // d)   # 512 MB at a time
    for i in range(0, count, step):
        rows = min(step, count - i)
        v = _normal(g, rows, d, scale={"int": 30.0, "sphere": 0.05}.get(data, 1.0))
        if data == "int":
            v = v.add_(20.0).clamp_(min=0.0).round_().clamp_(max=255.0)
        elif data == "zipf":
            u = torch.rand(rows, generator=g, device="cuda", dtype=torch.float64)
            v += centres[torch.searchsorted(cdf, u).clamp_(max=9_999)]
        else:
            v += centres[torch.randint(centres.shape[0], (rows,), generator=g, device="cuda")]
            if data == "sphere":
                v = torch.nn.functional.normalize(v, dim=1)
        out[i:i + rows] = v
    return out


def _requests(case):
    """(queries, K, T) of a serving burst: sizes spread over 1 to 4,096."""
    if case["kind"] != "serve":
        return [(case["q"], case["k"], case["t"])]
    r = case["q"]
    return [(int(round(4096 ** (i / (r - 1)))), (10, case["k"])[i % 2], (1, 8, case["t"])[i // 2 % 3]) for i in range(r)]


def _inputs(case, seed):
    """Dataset, queries, projection (A [L, M, D], b [L, M]) of a seed."""
    g = _gen(seed)
    x = _points(case, case["n"], seed, g)
    q = sum(r[0] for r in _requests(case))
    if case["near"]:
        pick = torch.randint(case["n"], (q,), generator=g, device="cuda")
        queries = x[pick].clone()
        if case["data"] == "int":   # one feature in a hundred is off by one
            queries += (torch.rand(q, case["d"], generator=g, device="cuda") < 0.01).float()
        else:
            queries += _normal(g, q, case["d"], scale=0.002 * case["w"])
    else:
        queries = _points(case, q, seed, g)
    p = _gen(seed * 7 + 2, "cpu")
    a = torch.randn(case["l"], case["m"], case["d"], generator=p).numpy()
    b = (torch.rand(case["l"], case["m"], generator=p) * case["w"]).numpy().astype(np.float32)
    return x, queries, a, b


def prepare(case, seed):
    x, queries, a, b = _inputs(case, seed)
    torch.cuda.synchronize()
    s = {"case": case, "x": x, "queries": queries, "ht": culsh.HashTables(), "st": culsh.SearchTables()}
    s["ht"].reset(case["n"], case["d"], case["l"], case["m"], case["w"], A=a, b=b)
    kind, q, k = case["kind"], case["q"], case["k"]
    if kind in ("pipeline", "host", "serve"):
        s["queries"] = queries.cpu().numpy()
    if kind == "pipeline":
        s["x"] = x.cpu().numpy()
    elif kind != "build":
        s["ht"].index_device(x.data_ptr())
        if kind == "serve":
            s["server"] = culsh.Server(s["ht"])
            s["requests"], at = [], 0
            for rq, rk, rt in _requests(case):
                s["requests"].append((s["queries"][at:at + rq].copy(), rk, rt))
                at += rq
        else:
            s["st"].reset(s["ht"], k, case["t"])
    if kind in ("search", "build"):
        s["ids"] = torch.empty(q, k, dtype=torch.int32, device="cuda")
        s["dists"] = torch.empty(q, k, dtype=torch.float32, device="cuda")
    return s


# ---------------------------------------------------------------------------
# one pass

def run(s):
    case, ht, st = s["case"], s["ht"], s["st"]
    kind = case["kind"]
    if kind == "serve":
        srv = s["server"]
        tickets = [srv.submit(q, k, t) for q, k, t in s["requests"]]
        return [srv.wait(t) for t in tickets]
    out = {}
    if kind in ("pipeline", "build"):
        if kind == "pipeline":
            ht.index(s["x"])
        else:
            ht.index_device(s["x"].data_ptr())
        st.reset(ht, case["k"], case["t"])
        out["buckets"] = ht.getBuckets().astype(np.int64)
    if kind in ("pipeline", "host"):
        st.search(s["queries"], dataset=s["x"] if kind == "pipeline" else None)
        out["ids"], out["dists"] = st.getKnnIds(), st.getKnnDistances()
    else:
        st.search_device(s["queries"].data_ptr(), case["q"], s["ids"].data_ptr(), s["dists"].data_ptr())
        out["ids"], out["dists"] = s["ids"], s["dists"]
    out["unique"], out["nonunique"] = st.getTotalCandidates_unique(), st.getTotalCandidates_nonUnique()
    return out


def work(case):
    """Bytes read and written once and the arithmetic of the definition:
    projections of what is projected, one squared distance a candidate."""
    n, d, lm = case["n"], case["d"], case["l"] * case["m"]
    reqs = _requests(case)
    q, qk, qt = (sum(r[0] * f(r) for r in reqs) for f in (lambda r: 1, lambda r: r[1], lambda r: r[2]))
    rows = min(n, q * case["cand"])
    byt = 4 * (q * d + lm * d + rows * d) + 8 * qk + 8 * case["l"] * qt
    flops = 2.0 * q * d * lm + 3.0 * q * d * case["cand"]
    if case["kind"] in ("pipeline", "build"):   # points in, ids by bucket out
        byt += 4 * n * d + 4 * n * case["l"]
        flops += 2.0 * n * d * lm
    return {"bytes": float(byt), "flops": float(flops)}


# ---------------------------------------------------------------------------
# the same results in 64 bits

def exact(case, seed):
    x, queries, a, b = _inputs(case, seed)
    a64 = torch.from_numpy(a).to("cuda", torch.float64)
    b64 = torch.from_numpy(b).to("cuda", torch.float64)
    reqs = _requests(case)
    if case["cand"] * sum(r[0] for r in reqs) > 2.0e10:
        return None
    mult = torch.randint(-(1 << 62), 1 << 62, (case["m"],), generator=_gen(5), device="cuda", dtype=torch.int64) | 1
    tables = []
    for l in range(case["l"]):
        keys = torch.cat([_codes(part, a64[l], b64[l], case["w"]).floor().to(torch.int64).mul_(mult).sum(1)
                          for part in x.split(1 << 19)])
        tables.append(torch.sort(keys, stable=True))
    out, at = [], 0
    for rq, rk, rt in reqs:
        qs = queries[at:at + rq]
        at += rq
        dists = torch.full((rq, rk), FLT_MAX, dtype=torch.float64, device="cuda")
        probes = [_probes(_codes(qs, a64[l], b64[l], case["w"]), mult, rt) for l in range(case["l"])]
        step = max(1, min(rq, int(4.0e7 / (4 * case["cand"] + case["l"] * rt + 1))))
        for i in range(0, rq, step):
            dists[i:i + step] = _knn64(x, qs[i:i + step], tables, [p[i:i + step] for p in probes], rk)
        out.append(dists)
    kind = case["kind"]
    if kind == "serve":
        return [(None, o.cpu().numpy()) for o in out]
    got = {"buckets": None} if kind in ("pipeline", "build") else {}
    got.update(ids=None, dists=out[0], unique=None, nonunique=None)
    return got


def _codes(x, a, b, w):
    return (x.to(torch.float64) @ a.T - b) / w


def _probes(v, mult, t):
    """Keys [Q, t] of the multiprobe sequence of unfloored codes v [Q, M]: the
    home bucket, then perturbation sets in ascending order of their summed
    boundary distances."""
    home = v.floor()
    down = v - home
    deltas, order = torch.sort(torch.cat([down, 1.0 - down], 1), dim=1, stable=True)
    m = v.shape[1]
    last = min(2 * m, 64)
    sign = torch.where(order < m, -1, 1)
    unit = sign * mult[order % m]
    keys = [(home.to(torch.int64) * mult).sum(1)]
    q = torch.arange(v.shape[0], device=v.device)
    sums = torch.full((v.shape[0], t + 1), math.inf, dtype=torch.float64, device=v.device)
    sets = torch.zeros((v.shape[0], t + 1, last), dtype=torch.bool, device=v.device)
    sums[:, 0] = deltas[:, 0]
    sets[:, 0, 0] = True
    place = torch.arange(last, device=v.device)
    size = torch.ones_like(q)
    for _ in range(t - 1):
        at = sums.argmin(1)
        probe, s = sets[q, at], sums[q, at]
        keys.append(keys[0] + (probe * unit[:, :last]).sum(1))
        top = (probe * place).amax(1)
        ok = top < last - 1
        r, nt = q[ok], top[ok] + 1
        shifted = probe[ok].clone()
        shifted[torch.arange(len(r), device=v.device), nt] = True
        grown = s[ok] + deltas[r, nt]
        sums[r, at[ok]], sets[r, at[ok]] = grown, shifted
        moved = shifted.clone()
        moved[torch.arange(len(r), device=v.device), nt - 1] = False
        sums[r, size[r]], sets[r, size[r]] = grown - deltas[r, nt - 1], moved
        size[r] += 1
    return torch.stack(keys, 1)


def _knn64(x, queries, tables, probes, k):
    """Distances [Q, k] of the nearest candidates: the points of every probed
    bucket (probes: one [Q, T] of keys a table)."""
    n, nq = x.shape[0], queries.shape[0]
    q64 = queries.to(torch.float64)
    pairs = []
    for (keys, ids), probe in zip(tables, probes):
        lo = torch.searchsorted(keys, probe)
        count = (torch.searchsorted(keys, probe, right=True) - lo).reshape(-1)
        first = torch.cumsum(count, 0) - count
        slot = torch.repeat_interleave(torch.arange(count.numel(), device=x.device), count)
        at = lo.reshape(-1)[slot] + torch.arange(slot.numel(), device=x.device) - first[slot]
        pairs.append(slot.div_(probe.shape[1], rounding_mode="floor").mul_(n).add_(ids[at]))
    out = torch.full((nq, k), FLT_MAX, dtype=torch.float64, device=x.device)
    if sum(p.numel() for p in pairs) > nq * (n // 32):   # most points: a mask over the whole dataset
        mask = torch.zeros(nq * n, dtype=torch.bool, device=x.device)
        for p in pairs:
            mask[p] = True
        mask = mask.view(nq, n)
        best = out
        for i in range(0, n, 1 << 18):
            part = x[i:i + (1 << 18)].to(torch.float64)
            dist = part.square().sum(1) - 2.0 * (q64 @ part.T) + q64.square().sum(1, keepdim=True)
            dist = dist.clamp_(min=0.0).masked_fill_(~mask[:, i:i + (1 << 18)], FLT_MAX)
            dist = dist.topk(min(k, dist.shape[1]), dim=1, largest=False).values
            best = torch.cat([best, dist], 1).topk(k, dim=1, largest=False, sorted=True).values
        return best
    pair = torch.unique(torch.cat(pairs))   # sorted: by query, then id
    if not pair.numel():
        return out
    qi, xi = pair.div(n, rounding_mode="floor"), pair % n
    dist = torch.cat([(q64[qs] - x[xs].to(torch.float64)).square_().sum(1)
                      for qs, xs in zip(qi.split(1 << 20), xi.split(1 << 20))])
    by = torch.argsort(dist, stable=True)
    by = by[torch.argsort(qi[by], stable=True)]
    qi, dist = qi[by], dist[by]
    start = torch.searchsorted(qi, torch.arange(nq, device=x.device))
    rank = torch.arange(qi.numel(), device=x.device) - start[qi]
    keep = rank < k
    out[qi[keep], rank[keep]] = dist[keep]
    return out
