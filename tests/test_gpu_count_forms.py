"""Counts that have kernels of their own (4-cycles by two-path counters,
cliques on bit matrices)
against the oracle, closed forms and the level program (an explicit launch
shape keeps the level program)."""
import os
import subprocess
import sys
from math import comb

import numpy as np
import pytest

import oracle_py as O
import subgraphmatchgpu_b200 as sme

pytestmark = pytest.mark.gpu
ALGOS = [sme.GPU_GPSM, sme.GPU_GPSM_REUSE, sme.GPU_LIGHT]


def csr_of(n, edges, both=True):
    e = np.asarray(edges, dtype=np.int64).reshape(-1, 2)
    if both:
        e = np.concatenate([e, e[:, ::-1]])
    e = np.unique(e, axis=0)
    rp = np.zeros(n + 1, np.uint64)
    np.cumsum(np.bincount(e[:, 0], minlength=n), out=rp[1:].view(np.int64))
    return rp, e[:, 1].astype(np.uint32)


def random_edges(n, m, seed):
    e = np.random.default_rng(seed).integers(0, n, (m, 2))
    return e[e[:, 0] != e[:, 1]]


# the two-path tables: a root of a warp's table (up to 640 two-paths), just
# above it, the CTA's table, direct counters
@pytest.mark.parametrize("hubs,leaves", [(2, 300), (2, 639), (2, 641), (3, 400), (8, 700), (5, 6200), (7, 9000)])
def test_cycles_of_complete_bipartite_graphs(hubs, leaves):
    edges = [(h, hubs + l) for h in range(hubs) for l in range(leaves)]
    g = sme.Graph.from_csr(*csr_of(hubs + leaves, edges))
    want = (hubs * (hubs - 1) // 2) * (leaves * (leaves - 1) // 2)
    for algo in ALGOS:
        assert g.count(1, algo) == want


@pytest.mark.parametrize("leaves", [50000, 65535, 65536, 110000])
def test_cycles_over_several_counter_ranges(leaves):
    # three hubs at the low ids of a graph of more vertices than one range of
    # 16-bit (98 304) or 32-bit counters (49 152, taken from 65 536 candidates)
    n = max(leaves + 3, 120001)
    edges = np.concatenate([np.stack([np.full(leaves, h), np.arange(n - leaves, n)], 1) for h in range(3)])
    g = sme.Graph.from_csr(*csr_of(n, edges))
    assert g.count(1) == 3 * (leaves * (leaves - 1) // 2)


def tree_with_closures(n, mids, leaves, seed):
    """Vertex 0 with `mids` neighbours, each with `leaves` more of the n, a few
    of them shared."""
    rng = np.random.default_rng(seed)
    mid = np.arange(1, mids + 1)
    far = rng.integers(mids + 1, n, mids * leaves)
    far[:: leaves // 2] = rng.choice(far, len(far[:: leaves // 2]))
    return np.concatenate([np.stack([np.zeros(mids, np.int64), mid], 1), np.stack([np.repeat(mid, leaves), far], 1)])


# a root above the hash table whose two-paths are worth its ranges of counters,
# and one whose are not: 100 ranges, 300 neighbours, about 35 000 two-paths
# asked for (paths_processed: the root alone, or the level program's paths too)
@pytest.mark.parametrize("mids,leaves,counters", [(300, 90, False), (300, 112, False), (300, 125, True), (300, 200, True),
                                                  (100, 250, True)])
def test_cycles_of_a_root_with_few_two_paths_for_its_ranges(mids, leaves, counters):
    n = 100 * 98304 + 1
    g = sme.Graph.from_csr(*csr_of(n, tree_with_closures(n, mids, leaves, leaves)))
    g.to_device(0)
    want = g.count(1, roots=[0], warp_granularity=3)
    assert want > 0
    assert g.count(1, roots=[0]) == want
    assert (sme.last_stats().paths_processed == 1) == counters
    assert g.count(1, roots=[0, 5, 0]) == 2 * want + g.count(1, roots=[5], warp_granularity=3)


def test_roots_left_by_several_chunks_of_a_task():
    # a task cut into chunks by an 80 MiB budget; every chunk leaves some roots
    # (8000 neighbours, 25 600 two-paths, five ranges) to the level program
    n, mids = 400000, 8000
    rng = np.random.default_rng(1)
    e = np.concatenate([np.stack([np.zeros(mids, np.int64), np.arange(1, mids + 1)], 1),
                        np.stack([rng.integers(1, mids + 1, 26500), rng.integers(mids + 1, n, 26500)], 1)])
    g = sme.Graph.from_csr(*csr_of(n, e))
    g.to_device(0)
    want = g.count(1, roots=[0], warp_granularity=3)
    roots = np.full(1200000, n - 1, np.uint32)
    roots[[7, 500000, 500001, 900000, 1199999]] = 0
    assert g.count(1, roots=[n - 1]) == 0
    assert g.count(1, roots=roots, mem_limit_bytes=80 << 20) == 5 * want
    s = sme.last_stats()
    assert s.batches >= 3 and s.paths_processed > len(roots) + 5 * 8000


@pytest.mark.parametrize("scale,ef", [(8, 4), (11, 9), (13, 8)])
def test_cycles_match_oracle_and_level_program(scale, ef):
    g = sme.Graph.rmat(scale, ef, seed=scale)
    rp, cl = g.csr()
    want = O.count(rp, cl, 1)
    roots = np.concatenate([np.arange(0, g.n, 3), np.arange(5), np.arange(5)])  # some of them twice
    part = g.count(1, roots=roots, warp_granularity=1)
    for resident in (False, True):
        if resident:
            g.to_device(0)
        assert g.count(1) == want
        assert g.count(1, roots=roots) == part
        assert g.count(1, root_begin=7, root_end=g.n - 3, root_stride=5) == \
            g.count(1, root_begin=7, root_end=g.n - 3, root_stride=5, warp_granularity=3)


@pytest.mark.parametrize("resident", [False, True])
def test_graphs_outside_the_contract_keep_the_level_program(resident):
    # one direction only, or a list with its own vertex: counts as before
    n = 400
    e = random_edges(n, 6000, 3)
    one_way = csr_of(n, e, both=False)
    loops = csr_of(n, np.concatenate([e, [(5, 5), (9, 9)]]))
    for rp, cl in (one_way, loops):
        g = sme.Graph.from_csr(rp, cl)
        if resident:
            g.to_device(0)
        for q in (0, 1, 3, 7):
            assert g.count(q) == g.count(q, warp_granularity=1), q


def launches(g, q, want, **kw):
    assert g.count(q, **kw) == want
    return sme.last_stats().kernel_launches


# a graph that comes with the call is checked in it: once however many chunks
# its task is cut into, and not at all where the answer changes nothing
def test_the_check_of_a_graph_that_is_not_resident():
    g = sme.Graph.rmat(10, 8, seed=6)
    o, _ = g.degree_order(orient=True)
    roots = np.full(1200000, g.n - 1, np.uint32)  # three chunks under 80 MiB
    tasks = [(g, 0, dict(roots=np.arange(0, g.n, 2)), 0), (g, 0, dict(root_begin=1), 0), (o, 0, dict(), 0),
             (g, 0, dict(), 1), (g, 3, dict(roots=np.arange(0, g.n, 2)), 1),
             (g, 1, dict(roots=roots, mem_limit_bytes=80 << 20), 1)]
    wants = [x.count(q, warp_granularity=2 if x.oriented else 3, **kw) for x, q, kw, _ in tasks]
    per_call = [launches(x, q, w, **kw) for (x, q, kw, _), w in zip(tasks, wants)]
    for x in (g, o):
        x.to_device(0)
    resident = [launches(x, q, w, **kw) for (x, q, kw, _), w in zip(tasks, wants)]
    assert sme.last_stats().batches >= 3
    assert [a - b for a, b in zip(per_call, resident)] == [c for *_, c in tasks]


# clique roots are worth the check of the lists from one in 6000 edges on
# (paths_processed counts the roots where the matrices take them)
def test_few_clique_roots_of_a_large_graph_that_is_not_resident():
    g = sme.Graph.rmat(14, 12, seed=2)
    least = -(-g.m // 6000)
    for count in (least - 1, least):
        roots = np.arange(g.n // 2, g.n // 2 + count, dtype=np.uint32)
        want = g.count(3, roots=roots, warp_granularity=3)
        assert g.count(3, roots=roots) == want
        assert (sme.last_stats().paths_processed == count) == (count == least)


# class edges of the bit matrices: a root of a complete graph of n vertices
# has n - 1 candidates
@pytest.mark.parametrize("n,ks", [(2, (3, 4)), (4, (3, 4, 5)), (5, (3, 4, 5, 6)), (33, (3, 4, 5, 6)),
                                  (34, (3, 4, 5, 6)), (65, (3, 4, 5, 6)), (130, (3, 4, 5, 6)), (257, (3, 4, 5)),
                                  (258, (3, 4, 5)), (513, (3, 4, 5)), (514, (3, 4)), (1025, (3, 4)), (1026, (3, 4)),
                                  (1500, (3,))])
def test_cliques_of_complete_graphs(n, ks):
    g = sme.Graph.clique(n)
    g.to_device(0)
    o, _ = g.degree_order(orient=True)
    for k in ks:
        q = {3: 0, 4: 3, 5: 7, 6: 11}[k]
        assert g.count(q) == comb(n, k)
        assert o.count(q) == comb(n, k)
        # root 0 has n - 1 candidates, root 1 one fewer
        assert g.count(q, roots=[1, 0, 1]) == comb(n - 1, k - 1) + 2 * comb(n - 2, k - 1)


def hub_graph(d, each=14):
    """Vertex 0 sees every other of d + 1 vertices, which hold `each` d random
    edges and a clique of 40."""
    e = np.concatenate([np.stack([np.zeros(d, np.int64), np.arange(1, d + 1)], 1), 1 + random_edges(d, each * d, d)])
    rng = np.random.default_rng(d)
    core = rng.choice(np.arange(1, d + 1), min(d, 40), replace=False)
    a, b = np.triu_indices(len(core), 1)
    e = np.concatenate([e, np.stack([core[a], core[b]], 1)])
    rp, cl = csr_of(d + 1, e)
    return sme.Graph.from_csr(rp, cl)


# few large roots are left to the level program, which spreads each over the
# device: class L of 6-cliques from 48 on, class X from 12 (32 for 6-cliques, 1
# for 4-cliques), class G from 32 (128) on
@pytest.mark.parametrize("d,q,least", [(400, 3, 1), (400, 7, 1), (400, 11, 48), (700, 3, 1), (700, 7, 12), (700, 11, 32),
                                       (1500, 3, 128), (1500, 7, 32), (1000, 11, 32), (4096, 3, 128)])
def test_few_large_roots_of_cliques(d, q, least):
    g = hub_graph(d, 14 if d < 1000 else d // 10)  # class G: a fifth of the pairs joined
    g.to_device(0)
    one = g.count(q, roots=[0], warp_granularity=1)
    assert one > 0
    for count in {1, least - 1, least} - {0}:
        roots = [0] * count + [d]
        assert g.count(q, roots=roots) == count * one
        assert (sme.last_stats().paths_processed == len(roots)) == (count >= least)


# roots of class G whose candidates are hardly joined, or joined well: the
# level program ends early on the former, the matrices do not
@pytest.mark.parametrize("joined,matrices", [(0.0, False), (0.005, False), (0.12, True)])
@pytest.mark.parametrize("q", [3, 7])
def test_large_roots_by_how_their_candidates_are_joined(q, joined, matrices):
    hubs, d = 200, 1200
    x, y = np.meshgrid(np.arange(hubs), hubs + np.arange(d))
    e = np.concatenate([np.stack([x.ravel(), y.ravel()], 1),
                        hubs + random_edges(d, int(joined * d * d / 2) + 2, 5)])
    g = sme.Graph.from_csr(*csr_of(hubs + d, e))
    g.to_device(0)
    roots = np.arange(hubs)
    assert g.count(q, roots=roots) == g.count(q, roots=roots[:1], warp_granularity=3) * hubs
    g.count(q, roots=roots)
    assert (sme.last_stats().paths_processed == hubs) == matrices


# vertex 0 sees every other vertex: a root of d candidates in every class, and
# above the last one, which keeps the level program
@pytest.mark.parametrize("d", [31, 256, 257, 700, 896, 897, 960, 961, 1024, 1025, 4096, 4097, 5000])
@pytest.mark.parametrize("q", [0, 3, 7, 11])
def test_cliques_of_a_hub_root(d, q):
    g = hub_graph(d)
    g.to_device(0)
    want = g.count(q, warp_granularity=1)
    assert want > 0
    assert g.count(q) == want
    roots = [0, 3, 0, d]
    assert g.count(q, roots=roots) == g.count(q, roots=roots, warp_granularity=1)


def bipartite_with_cliques(d, a, b):
    """K_{d,d} with a clique of `a` vertices on its left and one of b on its
    right side; `count(k)` of its k-cliques: any clique of either side (up to
    one vertex outside the planted ones) with any of the other."""
    left, right = np.meshgrid(np.arange(d), d + np.arange(d))
    e = [np.stack([left.ravel(), right.ravel()], 1)]
    for at, size in ((0, a), (d + 7, b)):
        x, y = np.triu_indices(size, 1)
        e.append(np.stack([at + x, at + y], 1))
    side = lambda size, i: (1, d)[i] if i < 2 else comb(size, i)
    return csr_of(2 * d, np.concatenate(e)), lambda k: sum(side(a, i) * side(b, k - i) for i in range(k + 1))


# every root of a graph whose lists stay long when they are cut to the higher
# (degree, id): d candidates for each vertex of one side, in every class
@pytest.mark.parametrize("d", [20, 200, 300, 700, 897, 1000, 1024, 1200])
@pytest.mark.parametrize("q", [0, 3, 7, 11])
def test_cliques_of_every_root_with_long_oriented_lists(d, q):
    csr, count = bipartite_with_cliques(d, 6, 5)
    g = sme.Graph.from_csr(*csr)
    g.to_device(0)
    want = count(sme.query_vertex_count(q))
    assert want > 0
    assert g.count(q) == want
    assert sme.last_stats().paths_processed == g.n  # the matrices counted it
    o, _ = g.degree_order(orient=True)
    assert o.count(q, root_stride=1) == want


def best_ms(g, q, **kw):
    counts = set()
    ms = []
    for _ in range(7):
        counts.add(g.count(q, **kw))
        ms.append(sme.last_stats().device_ms)
    return counts, min(ms)


# many roots of 600 candidates without an edge among them: the matrices are all
# the work, and each is built once
def test_many_roots_with_empty_neighbourhoods():
    csr, _ = bipartite_with_cliques(600, 0, 0)
    g = sme.Graph.from_csr(*csr)
    g.to_device(0)
    roots = np.random.default_rng(3).integers(0, g.n, 3000)
    got, ms = best_ms(g, 7, roots=roots)
    want, level_ms = best_ms(g, 7, roots=roots, warp_granularity=3)
    assert got == want == {0}
    assert ms < 1.2 * level_ms


# a budget that has no room for the scratch of the largest class: roots of more
# than 1024 (6-cliques: 896) candidates go to the level program, and with them
# a whole task whose lists were cut by (degree, id)
@pytest.mark.parametrize("n,budget", [(1100, 100), (1100, 300), (1100, 580), (1100, 640), (1024, 300)])
def test_cliques_without_room_for_the_largest_class(n, budget):
    g = sme.Graph.clique(n)
    g.to_device(0)
    kw = dict(mem_limit_bytes=budget << 20)
    fits = n <= 1025 or budget >= 640  # twice the scratch's 298 MiB
    assert g.count(0, **kw) == comb(n, 3)
    assert (sme.last_stats().paths_processed == n) == fits
    roots = [0] * 130 + [n - 300]  # enough for the largest class
    assert g.count(3, roots=roots, **kw) == 130 * comb(n - 1, 3) + comb(299, 3)
    assert (sme.last_stats().paths_processed == len(roots)) == fits


def test_cycles_without_room_for_the_range_queue():
    # 62 narrow ranges a root: the queue of 100 000 roots takes 50 MB
    n = 62 * 49152
    g = sme.Graph.from_csr(*csr_of(n, np.concatenate([random_edges(3000, 20000, 4), [(5, n - 1)]])))
    g.to_device(0)
    roots = np.arange(100000, dtype=np.uint32)
    want = g.count(1, warp_granularity=3)
    for budget, counters in ((76, False), (400, True)):
        assert g.count(1, roots=roots, mem_limit_bytes=budget << 20) == want
        assert (sme.last_stats().paths_processed == len(roots)) == counters


@pytest.mark.parametrize("resident", [False, True])
def test_cliques_of_skewed_graphs(resident):
    g = sme.Graph.rmat(14, 12, seed=2)
    o, _ = g.degree_order(orient=True)
    renumbered, _ = g.degree_order(orient=False)
    for x in (g, o, renumbered) if resident else ():
        x.to_device(0)
    for q in (0, 3, 7):
        want = g.count(q, warp_granularity=3)
        assert [x.count(q, a) for x in (g, o, renumbered) for a in ALGOS] == [want] * 9
        part = dict(root_begin=5, root_end=g.n - 9, root_stride=3)
        assert g.count(q, **part) == g.count(q, warp_granularity=3, **part)
        assert o.count(q, **part) == o.count(q, warp_granularity=2, **part)


def test_batched_cycles_and_cliques():
    # 4-cycles by counters (one range of w and several), cliques on oriented
    # lists; graphs outside their contract, and oriented ones, as they are
    graphs, queries = [], []

    def add(g, *qs):
        for q in qs:
            graphs.append(g)
            queries.append(q)

    add(sme.Graph.er(64, 6.0, seed=1), 1, 0, 3)
    add(sme.Graph.ba(700, 9, seed=2), 1, 0, 3, 7, 2)
    add(sme.Graph.ba(4096, 6, seed=3), 1)
    add(sme.Graph.ba(4097, 6, seed=4), 1, 3)
    add(sme.Graph.rmat(14, 4, seed=5), 1, 0)
    add(sme.Graph.clique(40), 1, 0, 3, 7, 11)
    add(sme.Graph.clique(2), 1, 0, 3)
    add(sme.Graph.rmat(10, 8, seed=6).degree_order(orient=True)[0], 0, 3, 7)
    e = random_edges(300, 4000, 8)
    add(sme.Graph.from_csr(*csr_of(300, e, both=False)), 1, 0, 3)
    add(sme.Graph.from_csr(*csr_of(300, np.concatenate([e, [(4, 4)]]))), 1, 0)
    hub = [(h, 2 + l) for h in range(2) for l in range(9000)]  # two hubs, three ranges
    add(sme.Graph.from_csr(*csr_of(9002, hub)), 1)
    want = [g.count(q, warp_granularity=1) if not g.oriented else g.count(q, warp_granularity=2)
            for g, q in zip(graphs, queries)]
    assert want[-1] == 9000 * 8999 // 2
    # self loops: the batched plan checks every pair it orders, as before
    for kw in (dict(), dict(autotune=False, granularity=1), dict(autotune=False, use_graph=False)):
        plan = sme.BatchPlan(graphs, queries, **kw)
        for _ in range(2):
            assert plan.run()[0].tolist() == want, kw
    only = sme.BatchPlan(graphs[:1], [1])  # nothing for the depth-first kernel
    assert only.run()[0].tolist() == want[:1]


# a large flat graph: its roots' few two-paths are not worth a pass over every
# range of counters (the same graph with a loop is always searched depth first)
def test_batched_cycles_of_a_large_flat_graph():
    n = 1 << 19
    e = random_edges(n, 2 * n, 11)
    ms, counts = [], []
    for extra in ([], [(n, n)]):
        g = sme.Graph.from_csr(*csr_of(n + 1, np.concatenate([e, extra]) if extra else e))
        plan = sme.BatchPlan([g], [1])
        runs = [plan.run() for _ in range(7)]
        counts += [int(c[0]) for c, _ in runs]
        ms.append(min(t for _, t in runs))
        plan.close()
    assert counts == [g.count(1, warp_granularity=1)] * 14
    assert ms[0] < 2.5 * ms[1]


@pytest.mark.parametrize("n", [5, 12, 20, 65, 130])
def test_houses_of_complete_graphs(n):
    g = sme.Graph.clique(n)
    g.to_device(0)
    assert g.count(4) == 60 * comb(n, 5)  # 5! placements, two of them alike


@pytest.mark.parametrize("scale,ef,seed", [(9, 8, 1), (11, 6, 2), (12, 8, 3)])
def test_houses_match_the_level_program(scale, ef, seed):
    g = sme.Graph.rmat(scale, ef, seed=seed)
    g.to_device(0)
    want = g.count(4, warp_granularity=1)
    assert [g.count(4, a) for a in ALGOS] == [want] * 3
    roots = np.concatenate([np.arange(0, g.n, 3), [0, 1, 0]])  # some twice
    assert g.count(4, roots=roots) == g.count(4, roots=roots, warp_granularity=3)


# roots of the most neighbours the counters take and one more; several ranges
# of counters; a root just under the least number of paths
@pytest.mark.parametrize("d,n", [(1024, 1100), (1025, 1100), (700, 98304), (700, 98305), (900, 250000), (12, 200000)])
def test_houses_of_a_hub_root(d, n):
    rng = np.random.default_rng(d)
    near = np.sort(rng.choice(np.arange(1, n), d, replace=False))
    e = np.concatenate([np.stack([np.zeros(d, np.int64), near], 1), near[random_edges(d, 6 * d, 7)],
                        np.stack([rng.choice(near, 20 * d), rng.integers(1, n, 20 * d)], 1)])
    rp, cl = csr_of(n, e[e[:, 0] != e[:, 1]])
    g = sme.Graph.from_csr(rp, cl)
    g.to_device(0)
    roots = [0, int(near[0]), int(near[-1]), int(near[d // 2]), 0]
    want = g.count(4, roots=roots, warp_granularity=1)
    assert want > 0
    assert g.count(4, roots=roots) == want


@pytest.mark.parametrize("cap", [0, 1, 1000, 90000, 300000])
def test_enumeration_copies_up_to_the_capacity(cap):
    # 161 700 triangles (1.9 MB: the staged copy), and below its threshold
    g = sme.Graph.clique(100)
    out = np.full((max(cap, 1), 3), 0xFFFFFFFF, np.uint32)
    import ctypes as C
    n = C.c_uint64()
    o = sme.opts(0)
    st = sme.lib().sme_enumerate(g.handle, C.byref(o), out.ctypes.data, cap, C.byref(n))
    assert n.value == comb(100, 3)
    assert st == (0 if cap >= n.value else 8)
    got = out[:min(cap, n.value)]
    assert len(np.unique(got.astype(np.int64) @ [10000, 100, 1])) == len(got)
    assert (got < 100).all() and (got[:, 0] < got[:, 1]).all() and (got[:, 1] < got[:, 2]).all()
    assert (out[min(cap, n.value):] == 0xFFFFFFFF).all()


def test_enumeration_over_several_staging_halves():
    g = sme.Graph.clique(60)  # 487 635 4-cliques, 7.8 MB
    inst = g.enumerate(3)
    key = np.sort(inst.astype(np.int64) @ [216000, 3600, 60, 1])
    assert len(np.unique(key)) == comb(60, 4) == len(inst)


def test_staging_takes_no_more_threads_than_the_process_may_use():
    code = """
import os, sys
os.sched_setaffinity(0, {sorted(os.sched_getaffinity(0))[0]})
sys.path.insert(0, sys.argv[1])
import subgraphmatchgpu_b200 as sme
threads = lambda: len(os.listdir("/proc/self/task"))
g = sme.Graph.clique(60)
g.enumerate(0)  # 410 KB: a plain copy
before = threads()
assert len(g.enumerate(3)) == 487635  # 7.8 MB: staged
print(before, threads())
"""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    env = {k: v for k, v in os.environ.items() if not k.startswith("OMP")}
    r = subprocess.run([sys.executable, "-c", code, root], capture_output=True, text=True, timeout=300, env=env)
    assert r.returncode == 0, r.stderr
    before, after = map(int, r.stdout.split())
    assert after == before
