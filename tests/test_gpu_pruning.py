"""Queries that leave out work by distance bounds (csrc/distance_bounds.cuh, csrc/prune.cuh) or answer an exhaustive
call without the index (csrc/exhaustive.cuh) against the sequential restatement: neighbour ids and distance bits
must not depend on what was left out.  Sizes sit on the edges of the 256-row and 128-query tiles, of the
32-coordinate stages, of the 32-row chunks in which groups may begin and end and of the 512-thread scan; rows that
a tensor map cannot describe (dim not a multiple of 4, a base that is not 16-byte aligned) take the variant with
ordinary loads."""
import numpy as np
import pytest
import torch

from oracle import oracle
from tests import cases

pytestmark = pytest.mark.gpu

#        rows, dim, queries, parts, L, S, T, k, max_cand, distribution
SIZES = [(2048, 32, 128, 8, 2, 4, 10, 10, 100, "latent"),      # everything a multiple of its tile
         (2049, 33, 129, 8, 2, 4, 10, 10, 30, "latent"),       # one beyond every tile; plain loads
         (2047, 31, 127, 7, 2, 3, 7, 5, 20, "latent"),
         (640, 64, 1, 2, 1, 5, 10, 1, 10, "latent"),           # one query, two partitions
         (13000, 96, 300, 200, 2, 5, 5, 3, 15, "mixture"),     # partitions of 65: several in one tile, one beyond two chunks
         (20000, 128, 260, 5, 2, 6, 10, 40, 200, "unit"),      # concentrated distances: little can be left out
         (9001, 50, 77, 9, 3, 5, 7, 13, 130, "mixture"),       # 200-byte rows
         (4000, 960, 20, 4, 2, 4, 10, 10, 60, "unit"),
         (6000, 24, 140, 30, 2, 4, 1, 7, 40, "latent"),        # windows of one point
         (3000, 16, 50, 6, 2, 4, 10, 600, 900, "latent"),      # lists longer than a partition
         # every point a candidate
         (2000, 100, 500, 100, 2, 7, 10, 10, 100, "latent"),
         (2000, 100, 1, 100, 2, 7, 10, 10, 100, "latent"),
         (511, 37, 3, 3, 1, 4, 10, 10, 1000, "latent"),        # fewer rows than threads
         (8193, 8, 1185, 10, 1, 2, 16, 1, 900, "mixture"),     # more queries than fit the scan
         (8192, 64, 129, 7, 2, 3, 7, 128, 1280, "unit"),
         (4097, 12, 40, 5, 2, 3, 10, 300, 3000, "latent"),
         (6000, 960, 9, 4, 1, 3, 10, 10, 10000, "unit"),
         (3000, 516, 300, 6, 1, 3, 10, 5, 50, "latent"),       # long rows, an odd number of query tiles taken two at a time
         (3000, 512, 256, 4, 1, 3, 10, 5, 1000, "latent")]


def _rows(rng, n, dim, dist):
    if dist == "mixture":
        return cases.mixture(rng, n, dim, centres=20)
    if dist == "unit":
        return cases.unit_uniform(rng, n, dim)
    return cases.latent_linear(rng, n, max(2, dim // 4), dim, 0.01)


def _bits(t):
    return t.cpu().numpy().view(np.uint32)


def _check(data, query, L, S, P, T, k, mc, proj, shift=0):
    from dciknn_cuda_b200 import DCI
    dim = data.shape[1]
    o = oracle.OracleDCI(dim, L, S, P, T, proj)
    o.add(data)
    oi, od = o.query(query, k, 5000, mc)
    store = torch.empty(data.size + 16, device="cuda")
    d = store[shift:shift + data.size].view(data.shape)
    d.copy_(torch.from_numpy(data))
    g = DCI(dim, L, S, P, T, proj=torch.from_numpy(proj))
    g.add(d)
    q = torch.from_numpy(query).cuda()
    for mode in (1, 0, 2):
        g.set_pruning(mode)
        ids, dists = g.query(q, k, 5000, max_num_candidates=mc, return_int_ids=True)
        assert np.array_equal(ids.cpu().numpy(), oi), mode
        assert np.array_equal(_bits(dists), od.view(np.uint32)), mode
        packed = g.query_packed(q, k, 5000, max_num_candidates=mc)
        assert torch.equal(packed & 0xFFFFFFFF, ids.to(torch.int64) & 0xFFFFFFFF), mode
    for mode in (1, 0):
        g.set_pruning(mode)
        ids, dists = torch.empty_like(ids), torch.empty_like(dists)
        g.query_noalloc(q, ids, dists, 5000, max_num_candidates=mc)
        assert np.array_equal(ids.cpu().numpy(), oi) and np.array_equal(_bits(dists), od.view(np.uint32)), mode


@pytest.mark.parametrize("size", SIZES, ids=lambda s: "%dx%d_q%d" % s[:3])
def test_answers_do_not_depend_on_what_is_left_out(size):
    n, dim, nq, P, L, S, T, k, mc, dist = size
    rng = np.random.default_rng(n + dim)
    z = _rows(rng, n + nq, dim, dist)
    _check(np.ascontiguousarray(z[:n]), np.ascontiguousarray(z[n:]), L, S, P, T, k, mc, cases.unit_rows(rng, L * S, dim))


@pytest.mark.parametrize("mc", [60, 3000])      # the traversal's quota, or every point a candidate
@pytest.mark.parametrize("kind", ["unaligned", "sorted", "duplicates", "huge", "tiny", "far", "nan"])
def test_answers_do_not_depend_on_what_is_left_out_for_unusual_rows(kind, mc):
    rng = np.random.default_rng(5)
    n, dim, nq = 3000, 32, 40
    z = _rows(rng, n + nq, dim, "latent")
    data, query = z[:n].copy(), z[n:].copy()
    if kind == "sorted":            # near rows in few partitions
        data = data[np.argsort(data[:, 0], kind="stable")].copy()
    elif kind == "duplicates":      # equal distances across partitions, ties by id
        data[n // 2:] = data[:n // 2]
        query[:20] = data[:20]
    elif kind == "huge":            # squared norms beyond the range in which bounds are formed, some beyond fp32
        data[::7] *= np.float32(1e16)
        data[3::50] *= np.float32(1e19)
        query[::5] *= np.float32(1e16)
    elif kind == "tiny":            # squares that underflow
        data *= np.float32(1e-21)
        query *= np.float32(1e-21)
    elif kind == "far":
        query *= np.float32(1000)
    elif kind == "nan":             # queries and rows without distances beside ordinary ones
        query[3] = np.nan
        data[70:90, 5] = np.nan
    proj = cases.unit_rows(rng, 8, dim)
    if kind in ("nan", "huge"):     # compared with the call that traverses every pair
        from dciknn_cuda_b200 import DCI
        g = DCI(dim, 2, 4, 6, 10, proj=torch.from_numpy(proj))
        g.add(torch.from_numpy(data).cuda())
        q = torch.from_numpy(query).cuda()
        out = []
        for mode in (2, 1, 0):
            g.set_pruning(mode)
            ids, dists = g.query(q, 10, 5000, max_num_candidates=mc, return_int_ids=True)
            out.append((ids.cpu(), dists.cpu().view(torch.int32)))
        for o in out[1:]:
            assert torch.equal(out[0][0], o[0]) and torch.equal(out[0][1], o[1])
        return
    _check(data, query, 2, 4, 6, 10, 10, mc, proj, shift=1 if kind == "unaligned" else 0)


@pytest.mark.parametrize("mc,path", [(60, "pruned"), (3000, "groups")])
def test_a_call_goes_without_the_working_memory_it_cannot_have(mc, path):
    from dciknn_cuda_b200 import DCI
    rng = np.random.default_rng(9)
    n, dim, nq, k = 6000, 32, 40, 2
    z = _rows(rng, n + nq, dim, "latent")
    g = DCI(dim, 2, 4, 6, 10, proj=torch.from_numpy(cases.unit_rows(rng, 8, dim)))
    g.add(torch.from_numpy(z[:n]).cuda())
    q = torch.from_numpy(z[n:]).cuda()
    out = []
    for limit, want in ((0, "all"), (None, path), (100, "all"), (1 << 20, path)):
        g.set_pruning(1, max_bytes=limit)
        out.append(g.query(q, k, 5000, max_num_candidates=mc, return_int_ids=True))
        assert g.last_call()["path"] == want, limit
    for ids, dists in out[1:]:
        assert torch.equal(ids, out[0][0]) and torch.equal(dists.view(torch.int32), out[0][1].view(torch.int32))


# 7 queries, k = 1: of rows that no tensor map describes the bounds cost more than the pairs that they leave out; where
# there are many queries the pairs cost far more
@pytest.mark.parametrize("n,dim,nq,k,L,S,path", [(501_175, 97, 7, 1, 2, 15, "all"), (501_175, 96, 7, 1, 2, 15, "pruned"),
                                                 (13_044, 97, 1382, 10, 3, 12, "pruned")])
def test_bounds_by_ordinary_loads_are_charged_as_such(n, dim, nq, k, L, S, path):
    from dciknn_cuda_b200 import DCI
    gen = torch.Generator(device="cuda").manual_seed(1)
    g = DCI(dim, L, S, 100, 10, seed=1)
    g.add(torch.randn(n, dim, generator=gen, device="cuda"))
    q = torch.randn(nq, dim, generator=gen, device="cuda")
    ids, dists = g.query(q, k, return_int_ids=True)
    assert g.last_call()["path"] == path
    g.set_pruning(2)
    for a, b in zip((ids, dists), g.query(q, k, return_int_ids=True)):
        assert torch.equal(a.view(torch.int32), b.view(torch.int32))


# exhaustive calls with long lists: one slice or several, both capacities of the selection buffer, as many queries as SMs
@pytest.mark.parametrize("size", [(2000, 100, 3, 100, 2, 7, 10, 1000, 10_000, "latent"), (2049, 16, 149, 20, 1, 3, 10, 513, 10_000, "mixture"),
                                  (20_011, 12, 2, 50, 1, 2, 10, 1000, 10_000, "latent"), (1025, 40, 148, 5, 1, 3, 10, 512, 10_000, "unit"),
                                  (511, 9, 5, 3, 1, 3, 10, 256, 10_000, "unit"), (40_000, 8, 5, 100, 1, 2, 10, 300, 3000, "mixture"),
                                  (70_001, 16, 20, 100, 1, 2, 10, 257, 3000, "mixture")], ids=lambda s: "%dx%d_q%d" % s[:3])
def test_exhaustive_calls_with_long_lists(size):
    n, dim, nq, P, L, S, T, k, mc, dist = size
    rng = np.random.default_rng(n + k)
    z = _rows(rng, n + nq, dim, dist)
    _check(np.ascontiguousarray(z[:n]), np.ascontiguousarray(z[n:]), L, S, P, T, k, mc, cases.unit_rows(rng, L * S, dim))


def test_exhaustive_allocation_free_call_in_two_batches():
    """300 queries against 1M rows: the bounds of all groups do not fit the built-in array at a time, and a scan of every
    row for every query would take many times as long as two batches of groups."""
    from dciknn_cuda_b200 import DCI
    gen = torch.Generator(device="cuda").manual_seed(6)
    data, q = torch.randn(1_000_000, 8, generator=gen, device="cuda"), torch.randn(300, 8, generator=gen, device="cuda")
    g = DCI(8, 1, 2, 100, 10, seed=3)
    g.add(data)
    ids, dists = torch.empty(300, 10, dtype=torch.int32, device="cuda"), torch.empty(300, 10, device="cuda")
    g.query_noalloc(q, ids, dists, 5000, max_num_candidates=20_000)
    assert g.last_call()["path"] == "groups"
    g.set_pruning(2)
    for a, b in zip((ids, dists), g.query(q, 10, 5000, max_num_candidates=20_000, return_int_ids=True)):
        assert torch.equal(a.view(torch.int32), b.view(torch.int32))


# few CTAs: each of them works through many tiles of the bounds (one and two tiles of queries at a time, ordinary loads)
# and many listed pairs, and the call takes more rounds
@pytest.mark.parametrize("max_ctas,rounds", [(1, 4), (3, 3), (40, 2)])
@pytest.mark.parametrize("size", [(4000, 96, 300, 20, 2, 5, 5, 3, 15, "mixture"), (4001, 50, 280, 20, 3, 5, 7, 3, 30, "mixture"),
                                  (3000, 516, 300, 10, 1, 3, 10, 2, 20, "mixture")], ids=lambda s: "%dx%d_q%d" % s[:3])
def test_work_is_left_out_in_every_round(size, max_ctas, rounds):
    from dciknn_cuda_b200 import DCI
    n, dim, nq, P, L, S, T, k, mc, dist = size
    rng = np.random.default_rng(n + dim)
    z = _rows(rng, n + nq, dim, dist)
    data, query, proj = np.ascontiguousarray(z[:n]), np.ascontiguousarray(z[n:]), cases.unit_rows(rng, L * S, dim)
    o = oracle.OracleDCI(dim, L, S, P, T, proj)
    o.add(data)
    oi, od = o.query(query, k, 5000, mc)
    g = DCI(dim, L, S, P, T, proj=torch.from_numpy(proj))
    g.add(torch.from_numpy(data).cuda())
    g.set_max_ctas(max_ctas)
    q = torch.from_numpy(query).cuda()
    for mode in (1, 3, 2):
        g.set_pruning(mode)
        ids, dists = g.query(q, k, 5000, max_num_candidates=mc, return_int_ids=True)
        last = g.last_call()
        assert np.array_equal(ids.cpu().numpy(), oi) and np.array_equal(_bits(dists), od.view(np.uint32)), mode
        if mode == 1:
            assert last["path"] == "pruned" and last["rounds"] >= rounds and not last["bounds_failed"]
            assert nq * k // (-(-n // P)) <= last["pairs"] < 0.6 * nq * P, last      # clustered rows: most pairs are left out
        elif mode == 3:       # the flag of a wait that ran out: everything in the first round
            assert last["bounds_failed"] and last["pairs"] == nq * P, last
        else:
            assert last["path"] == "all"


@pytest.mark.parametrize("nq", [1, 129])
def test_exhaustive_call_with_failed_bounds(nq):
    from dciknn_cuda_b200 import DCI
    rng = np.random.default_rng(4)
    n, dim, k = 6000, 40, 4
    z = _rows(rng, n + nq, dim, "latent")
    g = DCI(dim, 1, 3, 4, 10, proj=torch.from_numpy(cases.unit_rows(rng, 3, dim)))
    g.add(torch.from_numpy(z[:n]).cuda())
    q = torch.from_numpy(z[n:]).cuda()
    out = {}
    for mode in (1, 2, 3):
        g.set_pruning(mode)
        out[mode] = g.query(q, k, 5000, max_num_candidates=n, return_int_ids=True)
        assert (g.last_call()["path"], g.last_call()["bounds_failed"]) == {1: ("groups", False), 2: ("all", False), 3: ("groups", True)}[mode]
        assert torch.equal(out[mode][0], out[1][0]) and torch.equal(out[mode][1].view(torch.int32), out[1][1].view(torch.int32))


# n, dim, nq, L, S, k, max_cand, path: more pairs than the lists of one batch hold (1 GiB), more bounds than fit at a time
@pytest.mark.parametrize("n,dim,nq,L,S,k,mc,path", [(120_000, 8, 1500, 1, 3, 1000, 1100, "pruned"),
                                                    (1_000_000, 8, 2300, 1, 2, 10, 20_000, "groups")])
def test_several_batches_on_a_stream_of_its_own(n, dim, nq, L, S, k, mc, path):
    from dciknn_cuda_b200 import DCI
    gen = torch.Generator(device="cuda").manual_seed(2)
    data, q = torch.randn(n, dim, generator=gen, device="cuda"), torch.randn(nq, dim, generator=gen, device="cuda")
    g = DCI(dim, L, S, 100, 10, seed=3)
    g.add(data)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    out = []
    for mode in (1, 2):
        g.set_pruning(mode)
        with torch.cuda.stream(side):
            out.append(g.query(q, k, 5000, max_num_candidates=mc, return_int_ids=True))
        side.synchronize()
        if mode == 1:
            last = g.last_call()
            assert last["path"] == path and last["batches"] == 2 and not last["bounds_failed"], last
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1].view(torch.int32), out[1][1].view(torch.int32))


@pytest.mark.parametrize("k,mc", [(10, 100), (1, 30), (100, 5000)])
def test_queries_that_are_rows(k, mc):
    """A distance of 0 beside distances within an octave: one range of the selection's histogram holds nearly all."""
    rng = np.random.default_rng(k)
    data = cases.unit_uniform(rng, 6000, 32)
    data[3000:3010] = data[0]
    _check(data, data[:12].copy(), 1, 5, 40, 10, k, mc, cases.unit_rows(rng, 5, 32))
