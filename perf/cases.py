"""Performance cases of the k-NN engine: the calls a user's program makes, over the sizes it makes them at.

A case is a dict of plain values.  `entry` names the call:

  query     DCI.query on CUDA tensors, on an index built beforehand (batch search, and the latency of one query)
  noalloc   DCI.query_noalloc into tensors of the caller (a serving loop)
  host      DCI.query_host, queries and results in host memory
  mdci      MDCI.query with one device (the class most programs construct)
  rebuild   clear + add + query: the cycle of a program whose points change between searches
  append    clear + add + append + query: points that arrive in two parts

Points and queries are drawn from one of three distributions: `latent` (randn of 32 or 64 factors through a
random linear map, plus a little noise), `mixture` (256 Gaussian clusters) and `unit` (uniform rows scaled to
unit length).
"""
import math

import torch

from dciknn_cuda_b200 import DCI, MDCI

DEFAULTS = dict(entry="query", dist="latent", dim=128, n=1_000_000, nq=1, k=10, L=2, S=10, P=100, T=10, outer=5000,
                max_cand=None, extra=0)


def _case(name, **kw):
    c = dict(DEFAULTS, **kw)
    if c["max_cand"] is None:
        c["max_cand"] = 10 * c["k"]      # what query() takes when the caller does not say
    return dict(name=name, **c)


def listed():
    return [
        # the smallest call: one query against the 2 000 x 100 example index with the default parameters
        _case("example_one_query", n=2000, dim=100, S=7),
        # the example's own cycle: index 2 000 points, ask 500 queries, clear
        _case("example_cycle", entry="rebuild", n=2000, dim=100, S=7, nq=500),
        # latency of a single query against a large index
        _case("serve_one", nq=1),
        # a serving loop's small batch, into buffers of the caller
        _case("serve_noalloc_32", entry="noalloc", nq=32),
        # the headline batch: 10 000 queries against 1M x 128
        _case("batch_10k", nq=10_000),
        # host buffers in and out; odd sizes: rows that are not a multiple of 16 bytes, ragged partitions, an odd window
        _case("host_ragged", entry="host", n=100_003, dim=50, nq=777, k=13, L=3, S=5, P=37, T=7),
        # long rows and a quota no partition can meet: every point is a candidate, the answer is the exact one
        _case("highdim_exhaustive", dist="unit", dim=960, nq=200, L=3, S=12, max_cand=10_000),
        # one shard of a clustered 10M-point set, behind the sharded class
        _case("mdci_mixture", entry="mdci", dist="mixture", n=1_250_001, dim=96, nq=1000),
        # long result lists: k = 100, 15 simple indices per composite index
        _case("large_k", n=500_001, dim=256, nq=500, k=100, S=15, outer=20_000),
        # an unsharded 10M-point index: partitions of 100 000 points, more than shared memory holds
        _case("large_partitions", dist="mixture", n=10_000_000, dim=96, nq=64),
        # points that changed: index 1M x 128 again and ask a few queries for the nearest point
        _case("rebuild_1m", entry="rebuild", nq=4, k=1),
        # points that arrive in two parts
        _case("append_stream", entry="append", n=200_000, extra=20_000, dim=64, nq=100, S=7),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    entry = rng.choice(["query", "query", "query", "noalloc", "host", "mdci", "rebuild", "append"])
    dist = rng.choice(["latent", "latent", "mixture", "unit"])
    while True:
        n = _log_int(rng, 2000, 4_000_000)
        dim = rng.choice([_log_int(rng, 16, 960), 8 * _log_int(rng, 2, 120), 64, 96, 128, 256])
        if n * dim > 1_000_000_000:
            continue
        L, S, T = rng.choice([1, 2, 2, 3]), rng.choice([5, 7, 10, 12, 15]), rng.choice([5, 7, 10, 10, 16, 20])
        P = rng.choice([20, 37, 100, 100, 100, 200, 400])
        k = rng.choice([1, 10, 10, 10, 13, 30, 100])
        nq = _log_int(rng, 1, 10_000 if entry != "noalloc" else 200)
        # no dearer than the headline batch: every query meets every point through L*S indices
        if float(nq) * n * (L * S + dim / 8) > 5e10 or n // P < 10:
            continue
        if entry == "noalloc" and n // P > 12_000:        # the fixed working array serves partitions of this size
            continue
        break
    max_cand = rng.choice([10 * k, 10 * k, 10 * k, 20 * k, 5 * k + 1])
    extra = max(1, n // rng.choice([3, 10, 50])) if entry == "append" else 0
    c = _case("", entry=entry, dist=dist, n=n, dim=dim, nq=nq, k=k, L=L, S=S, P=P, T=T,
              outer=rng.choice([5000, 5000, 20_000, 300]), max_cand=max_cand, extra=extra)
    del c["name"]
    return c


def _rows(g, n, dim, dist, shared):
    dev = shared.device
    if dist == "unit":
        z = torch.rand(n, dim, generator=g, device=dev)
        return z.div_(z.norm(dim=1, keepdim=True))
    if dist == "mixture":
        z = torch.randn(n, dim, generator=g, device=dev)
        return z.add_(shared[torch.randint(shared.shape[0], (n,), generator=g, device=dev)])
    z = torch.randn(n, shared.shape[0], generator=g, device=dev) @ shared
    return z.add_(torch.randn(n, dim, generator=g, device=dev), alpha=0.01)


def prepare(case, seed):
    dev = torch.device("cuda", 0)
    g = torch.Generator(device=dev).manual_seed(seed)
    dim, n = case["dim"], case["n"] + case["extra"]
    if case["dist"] == "mixture":
        shared = 4.0 * torch.randn(256, dim, generator=g, device=dev)
    else:
        shared = torch.randn(64 if dim >= 256 else 32, dim, generator=g, device=dev)
    data = _rows(g, n, dim, case["dist"], shared)
    query = _rows(g, case["nq"], dim, case["dist"], shared)
    args = (dim, case["L"], case["S"], case["P"], case["T"])
    st = dict(case=case)
    if case["entry"] == "mdci":
        st["index"] = MDCI(*args, devices=[0], seeds=[seed])
    else:
        st["index"] = DCI(*args, device=0, seed=seed)
    st["data"] = data[:case["n"]]
    if case["entry"] == "append":
        st["more"] = data[case["n"]:].clone()
    if case["entry"] not in ("rebuild", "append"):
        st["index"].add(st["data"])
    if case["entry"] == "host":
        query = query.cpu().pin_memory()
    if case["entry"] == "noalloc":
        st["ids"] = torch.empty(case["nq"], case["k"], dtype=torch.int32, device=dev)
        st["dists"] = torch.empty(case["nq"], case["k"], dtype=torch.float32, device=dev)
    st["query"] = query
    torch.cuda.synchronize()
    return st


def run(st):
    case, index, query = st["case"], st["index"], st["query"]
    k, outer, mc = case["k"], case["outer"], case["max_cand"]
    if case["entry"] in ("rebuild", "append"):
        index.clear()
        index.add(st["data"])
        if case["entry"] == "append":
            index.append(st["more"])
    if case["entry"] == "noalloc":
        return index.query_noalloc(query, st["ids"], st["dists"], outer, max_num_candidates=mc)
    if case["entry"] == "host":
        return index.query_host(query, k, outer, max_num_candidates=mc)
    return index.query(query, k, outer, max_num_candidates=mc)


def work(case):
    """One query reads its vector and writes k ids and distances; a batch of them reads the index once (4-byte keys
    and 2-byte ids of every entry; not at all where the quota makes every point a candidate) and once the rows that
    can become candidates, T * max_cand per partition at most.  A build reads the rows once and writes keys and ids.
    Distances: at least k candidates of every partition, or one contraction of all queries with all rows."""
    n, dim, nq, k = case["n"] + case["extra"], case["dim"], case["nq"], case["k"]
    indices, ppb = case["L"] * case["S"], -(-n // case["P"])
    per_query = min(n, case["P"] * min(ppb, case["T"] * case["max_cand"]))
    rows = min(n, nq * per_query)
    nbytes = 4.0 * nq * dim + 8.0 * nq * k + 4.0 * dim * rows
    flops = 2.0 * nq * indices * dim + 3.0 * dim * nq * min(k * case["P"], per_query)
    if case["max_cand"] < ppb:
        nbytes += 6.0 * indices * n
    else:
        flops = 2.0 * nq * n * dim
    if case["entry"] in ("rebuild", "append"):
        nbytes += 4.0 * n * dim + 8.0 * indices * n
        flops += 2.0 * n * indices * dim
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    """Ids are whole numbers, and a distance is one fixed chain of fp32 operations: the square root of
    fma(d, d, sum) over ascending coordinates.  Two correct implementations agree in every bit."""
    return "exact"
