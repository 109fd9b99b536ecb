"""Workloads of the subgraph-enumeration engine, called as a user's program calls it.

Each case is a plain dict.  `kind` says which entry point it goes through:

  count      Graph.count on one graph: resident on the device, copied to it by
             the call (`place` "host" / "packed") or left in host memory and
             streamed under a device budget (`place` "external")
  enumerate  Graph.enumerate: every instance, in a canonical order
  batch      BatchPlan.run: many small graphs, one prepared plan
  serve      Server.submit / wait: a closed loop of requests of mixed patterns
             on resident and attached graphs

Graphs are undirected (both directions stored, sorted lists, no self loops,
no isolated vertices) and made from the seed: R-MAT with a/b/c =
.57/.19/.19 (skewed, the shape of social and web graphs), Erdos-Renyi (flat)
or Barabasi-Albert.  A root task is a block of vertices of degree <= 1024, the
unit in which a program that shares a large graph's enumeration out hands it
to the engine.  Every output is a whole number, so results are exact.
"""
import math
import random

import numpy as np
import torch

import subgraphmatchgpu_b200 as sme

TRIANGLE, CYCLE4, DIAMOND, CLIQUE4, HOUSE, CLIQUE5 = 0, 1, 2, 3, 4, 7
HUB = 1024  # root blocks hold vertices up to this degree


def _case(kind, name=None, **kw):
    c = {} if name is None else {"name": name}
    c |= {"kind": kind, "graph": "rmat", "edges": 0, "scale": 0, "query": 0, "algo": sme.GPU_LIGHT,
          "roots": 0, "place": "resident", "oriented": False, "budget_mb": 0, "items": 0}
    return c | kw


def listed():
    return [
        # one triangle count on a small resident graph (16 384-vertex R-MAT,
        # edge factor 8): a call's fixed cost
        _case("count", "triangle s14", scale=14, edges=8 << 14, query=TRIANGLE),
        # the plain BFS plan on a mid-sized graph: 4-cycles of a
        # Barabasi-Albert graph of odd size
        _case("count", "4-cycle ba gpsm", graph="ba", scale=15, edges=9 * 30011, query=CYCLE4, algo=sme.GPU_GPSM),
        # root blocks of a large resident graph (R-MAT scale 20, edge factor
        # 16), the sizes that the repository's benchmark steps through
        _case("count", "4-clique s20 roots", scale=20, edges=16 << 20, query=CLIQUE4, roots=16384),
        _case("count", "4-cycle s20 roots", scale=20, edges=16 << 20, query=CYCLE4, roots=512),
        # the house on a block of roots: `!=` conditions and ranked counts
        _case("count", "house s18 roots", scale=18, edges=16 << 18, query=HOUSE, roots=1024),
        # a graph in host memory, copied by the call as packed lists: a
        # diamond block on the large graph
        _case("count", "diamond s20 packed", scale=20, edges=16 << 20, query=DIAMOND, roots=8192, place="packed"),
        # a whole mid-sized graph, hubs included, under the reuse plan
        _case("count", "4-clique s18 reuse", scale=18, edges=16 << 18, query=CLIQUE4, algo=sme.GPU_GPSM_REUSE),
        # 5-cliques of the degree-ordered, oriented graph
        _case("count", "5-clique s17 oriented", scale=17, edges=16 << 17, query=CLIQUE5, oriented=True),
        # adjacency lists (7 MB) stay in host memory and stream through a
        # device budget whose list cache is below their size
        _case("count", "4-clique s16 external", scale=16, edges=16 << 16, query=CLIQUE4, place="external",
              budget_mb=13),
        # all 4-cliques as instances, into a buffer of fixed capacity
        _case("enumerate", "4-clique s13 enumerate", scale=13, edges=8 << 13, query=CLIQUE4),
        # 512 small graphs, half Erdos-Renyi, half Barabasi-Albert, one plan
        _case("batch", "batch 512", items=512),
        # 64 requests in a closed loop over four slots: patterns of three to
        # five vertices, half on resident graphs, half on attached ones
        _case("serve", "serve 64", scale=18, edges=16 << 18, items=64),
    ]


def _odd(rng, lo, hi):
    """A whole number, log-uniform over [lo, hi]."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _light(kind):
    """Patterns counted on whole graphs; a flat graph has few dense ones."""
    return [TRIANGLE, CYCLE4] if kind == "er" else [TRIANGLE, DIAMOND, CLIQUE4]


def draw(rng):
    pick = rng.choice(["whole", "whole", "roots", "roots", "host", "external", "oriented", "plan", "enumerate",
                       "batch", "serve"])
    if pick == "whole":  # light patterns on a whole resident graph of any size
        kind = rng.choice(["rmat", "er", "ba"])
        scale = rng.randint(10, 18 if kind == "rmat" else 16)
        return _case("count", graph=kind, scale=scale, edges=_odd(rng, 6 << scale, 16 << scale),
                     query=rng.choice(_light(kind)))
    if pick == "roots":  # heavier patterns on a block of roots
        q = rng.choice([CYCLE4, CLIQUE4, DIAMOND, HOUSE, CLIQUE5])
        scale = rng.randint(15, 18 if q in (HOUSE, CLIQUE5) else 20)
        most = {CYCLE4: 512, CLIQUE4: 16384, DIAMOND: 8192, HOUSE: 1024, CLIQUE5: 4096}[q]
        return _case("count", scale=scale, edges=_odd(rng, 6 << scale, 16 << scale), query=q,
                     roots=_odd(rng, most // 64, most))
    if pick == "host":
        scale = rng.randint(12, 20)
        return _case("count", scale=scale, edges=_odd(rng, 6 << scale, 16 << scale),
                     query=rng.choice([TRIANGLE, DIAMOND, CLIQUE4]), roots=_odd(rng, 256, 8192),
                     place=rng.choice(["host", "packed"]))
    if pick == "external":
        scale = rng.randint(12, 16)
        return _case("count", scale=scale, edges=_odd(rng, 8 << scale, 16 << scale),
                     query=rng.choice([TRIANGLE, CLIQUE4]), place="external", budget_mb=rng.randint(13, 48))
    if pick == "oriented":
        scale = rng.randint(12, 17)
        return _case("count", graph=rng.choice(["rmat", "ba"]), scale=scale,
                     edges=_odd(rng, 4 << scale, 16 << scale), query=rng.choice([TRIANGLE, CLIQUE4, CLIQUE5]),
                     oriented=True)
    if pick == "plan":  # the other two plans
        kind, scale = rng.choice(["rmat", "er", "ba"]), rng.randint(10, 16)
        return _case("count", graph=kind, scale=scale, edges=_odd(rng, 6 << scale, 10 << scale),
                     query=rng.choice(_light(kind)), algo=rng.choice([sme.GPU_GPSM, sme.GPU_GPSM_REUSE]))
    if pick == "enumerate":
        kind, scale = rng.choice(["rmat", "er"]), rng.randint(9, 13)
        return _case("enumerate", graph=kind, scale=scale, edges=_odd(rng, 4 << scale, 8 << scale),
                     query=TRIANGLE if kind == "er" else rng.choice([TRIANGLE, CLIQUE4]))
    if pick == "batch":
        return _case("batch", items=_odd(rng, 64, 512))
    scale = rng.randint(16, 18)
    return _case("serve", scale=scale, edges=_odd(rng, 8 << scale, 16 << scale), items=_odd(rng, 8, 64))


# ------------------------------------------------------------------ inputs --
def _csr(u, v, n):
    """Undirected CSR of an edge list: both directions, no self loops, no
    parallel edges, isolated vertices dropped with an order-preserving
    relabel.  Numpy row_ptrs (uint64) and cols (uint32)."""
    keep = u != v
    u, v = u[keep], v[keep]
    key = torch.unique(torch.cat([u * n + v, v * n + u]))
    src, dst = key // n, key % n
    deg = torch.bincount(src, minlength=n)
    new = torch.cumsum(deg > 0, 0) - 1
    rp = torch.cat([deg.new_zeros(1), torch.cumsum(deg[deg > 0], 0)])
    return rp.cpu().numpy().astype(np.uint64), new[dst].to(torch.int32).cpu().numpy().view(np.uint32)


def _make_graph(kind, scale, edges, seed):
    """One graph of about `edges` undirected edges on at most 2^scale vertices."""
    n = 1 << scale
    if kind == "ba":  # every new vertex brings `attach` edges
        attach = max(2, round(edges / n))
        return sme.Graph.ba(max(attach + 2, edges // attach), attach, seed=seed)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    if kind == "er":
        u = torch.randint(0, n, (edges,), generator=gen, device="cuda")
        v = torch.randint(0, n, (edges,), generator=gen, device="cuda")
    else:
        u = torch.zeros(edges, dtype=torch.int64, device="cuda")
        v = torch.zeros(edges, dtype=torch.int64, device="cuda")
        for _ in range(scale):
            r = torch.rand(edges, generator=gen, device="cuda")
            u = 2 * u + (r >= 0.76)
            v = 2 * v + (((r >= 0.57) & (r < 0.76)) | (r >= 0.95))
    return sme.Graph.from_csr(*_csr(u, v, n))


def _graph_of(case, seed):
    return _make_graph(case["graph"], case["scale"], case["edges"], seed)


def prepare(case, seed):
    if case["kind"] == "batch":
        # graph sizes log-uniform over 64..4096 vertices, average degree 4..32
        rng = random.Random(seed)
        graphs, queries = [], []
        for i in range(case["items"]):
            n, d = int(round(2 ** rng.uniform(6, 12))), rng.uniform(4, 32)
            s = seed * 100003 + i
            graphs.append(sme.Graph.er(n, d, seed=s) if i % 2 == 0 else
                          sme.Graph.ba(n, max(1, round(d / 2)), seed=s))
            queries.append(rng.choice([TRIANGLE, CYCLE4, DIAMOND, CLIQUE4]))
        return {"case": case, "plan": sme.BatchPlan(graphs, queries)}
    if case["kind"] == "serve":
        rng = random.Random(seed)
        srv = sme.Server(slots=4, mem_budget_bytes=4 << 30)
        resident = [_make_graph("rmat", case["scale"] - d, case["edges"] >> d, seed + d) for d in (0, 2, 4)]
        gids = [srv.add_graph(g) for g in resident]
        requests = []
        for i in range(case["items"]):
            q = rng.choice([TRIANGLE, CYCLE4, DIAMOND, CLIQUE4, HOUSE, CLIQUE5])
            if rng.random() < 0.5:  # 256..8192 vertices, average degree 8
                n = _odd(rng, 256, 8192)
                requests.append((q, {"attached": sme.Graph.er(n, 8.0, seed=seed * 100003 + i)}))
            else:
                k = rng.randrange(3)
                rp, _ = resident[k].csr()
                block = _roots(rp, 64, seed * 131 + i)
                requests.append((q, {"gid": gids[k], "roots": block}))
        return {"case": case, "server": srv, "requests": requests, "keep": resident}
    g = _graph_of(case, seed)
    opts = {"algo": case["algo"]}
    if case["roots"]:
        opts["roots"] = _roots(g.csr()[0], case["roots"], seed)
    if case["oriented"]:
        g, _ = g.degree_order(orient=True)
    if case["place"] == "resident":
        g.to_device(0)
    elif case["place"] == "packed":
        g.pack()
    elif case["place"] == "external":
        opts["mode"] = sme.EXTERNAL_GPU
        opts["mem_limit_bytes"] = case["budget_mb"] << 20
    return {"case": case, "graph": g, "n": g.n, "opts": opts}


def _roots(row_ptrs, count, seed):
    low = np.flatnonzero(np.diff(row_ptrs.astype(np.int64)) <= HUB)
    return np.random.default_rng(seed).permutation(low)[:count].astype(np.uint32)


def _capacity(case):
    return 48 * case["edges"]


def _keys(inst, n, cap):
    key = torch.full((cap,), torch.iinfo(torch.int64).max, dtype=torch.int64, device="cuda")
    k = torch.zeros(len(inst), dtype=torch.int64, device="cuda")
    for i in range(inst.shape[1]):
        k = k * n + inst[:, i]
    key[:len(k)] = torch.sort(k).values
    return key


# --------------------------------------------------------------------- run --
def run(state):
    case = state["case"]
    if case["kind"] == "batch":
        return state["plan"].run()[0].view(np.int64)
    if case["kind"] == "serve":
        srv = state["server"]
        ids = [srv.submit(q, **kw) for q, kw in state["requests"]]
        return np.array([srv.wait(i)[0] for i in ids], dtype=np.int64)
    if case["kind"] == "enumerate":
        # the engine gives instances in no fixed order: as one key each,
        # sorted, on the device, the unused capacity after them
        inst = state["graph"].enumerate(case["query"], cap=_capacity(case), **state["opts"])
        return _keys(torch.from_numpy(inst.view(np.int32)).cuda(), state["n"], _capacity(case))
    return state["graph"].count(case["query"], **state["opts"])


# -------------------------------------------------------------------- work --
def work(case):
    """Each list and row pointer read once (nominal sizes), the counts or the
    instances' buffer written once.  Enumeration is bound by the
    search itself, whose size only a run tells."""
    if case["kind"] == "batch":
        mean_n = (4096 - 64) / math.log(64)
        return {"bytes": case["items"] * (mean_n * (18 * 4 + 4) + 8), "flops": 0}
    n, m = 1 << case["scale"], 2 * case["edges"]
    if case["oriented"]:
        m //= 2
    size = 8 * n + 4 * m
    if case["kind"] == "serve":
        return {"bytes": size * (1 + 1 / 4 + 1 / 16) + case["items"] / 2 * 1e5, "flops": 0}
    if case["kind"] == "enumerate":
        return {"bytes": size + 8 * _capacity(case), "flops": 0}
    return {"bytes": size + 4 * case["roots"] + 8, "flops": 0}


def tolerance(case):
    return "exact"


# ------------------------------------------------------------------- exact --
def exact(case, seed):
    """Counts from the adjacency matrix in 64 bits, instances by extension
    over it; None where the matrix is too large or the task is a block."""
    if case["kind"] not in ("count", "enumerate") or case["roots"] or case["oriented"] or case["graph"] == "ba":
        return None
    if case["scale"] > 14 or case["query"] not in (TRIANGLE, CYCLE4, DIAMOND, CLIQUE4):
        return None
    rp, cl = (torch.from_numpy(x.astype(np.int64)).cuda() for x in _graph_of(case, seed).csr())
    n = len(rp) - 1
    src = torch.repeat_interleave(torch.arange(n, device="cuda"), rp[1:] - rp[:-1])
    adj = torch.zeros(n, n, dtype=torch.float64, device="cuda")
    adj[src, cl] = 1
    if case["kind"] == "count" and case["query"] != CLIQUE4:
        common = adj @ adj  # common neighbours of every pair
        common.fill_diagonal_(0)
        if case["query"] == TRIANGLE:
            return int((common * adj).sum().item()) // 6
        pairs = common * (common - 1) / 2
        if case["query"] == CYCLE4:  # both diagonals of a cycle see it
            return int(pairs.sum().item()) // 4
        return int((pairs * adj).sum().item()) // 2
    up = torch.triu(adj, 1) > 0  # neighbours above each vertex
    del adj
    rows, total = torch.nonzero(up), 0
    keys = []
    for i in range(0, len(rows), 4096):
        part = rows[i:i + 4096]
        both = up[part[:, 0]] & up[part[:, 1]]
        at = torch.nonzero(both)
        part = torch.cat([part[at[:, 0]], at[:, 1:]], 1)
        if case["query"] == CLIQUE4:
            grown = []
            for j in range(0, len(part), 16384):
                p = part[j:j + 16384]
                at = torch.nonzero(up[p[:, 0]] & up[p[:, 1]] & up[p[:, 2]])
                grown.append(torch.cat([p[at[:, 0]], at[:, 1:]], 1))
            part = torch.cat(grown) if grown else part.new_zeros(0, 4)
        total += len(part)
        if case["kind"] == "enumerate":
            keys.append(part)
    return _keys(torch.cat(keys), n, _capacity(case)) if case["kind"] == "enumerate" else total
