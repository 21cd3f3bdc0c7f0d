"""The work users have this framework do, as measurable cases.

A case is a dict of plain values.  Its kind names the entry point it goes
through:

  pivot    Context.run_pivot     the plain form, one pivot per call
  batch    Context.run_batch     up to 64 given pivots in one multi-source pass
  sampled  Context.run_sampled   the sampling loop, heuristics 0..6
  serve    Server                requests of several users on resident graphs
  job      Graph.from_edges ...  one whole job: edge list in, betweenness out

Graphs: `kron` is the Graph500 R-MAT shape (edge factor 16 unless given), drawn
from the seed here with torch and handed over as a CSC or an edge list; from
scale 22 on it comes from the framework's own Graph500 generator.  `grid` is
the framework's 4-neighbour grid (2% of edges dropped, 0.01% long-range edges).
"""
import random

import numpy as np
import torch

import axbc_gb300 as ax

EDGEFACTOR = 16


def listed():
    return [
        # the smallest call: one pivot of the plain form on a graph of a
        # thousand vertices, leaves folded away (-H 1)
        dict(name="pivot_s10_H1", kind="pivot", graph="kron", n=1 << 10, pivots=1, H=1, directed=False),
        # the plain form on an ordinary graph, as a host program in the
        # reference's manner drives it: pivot after pivot, bc read at the end
        dict(name="pivot4_s18", kind="pivot", graph="kron", n=1 << 18, pivots=4, H=0, directed=False),
        # an odd-sized directed graph (-U), pivots fewer than a warp has lanes
        dict(name="batch17_dir_n50021", kind="batch", graph="kron", n=50021, pivots=17, H=0, directed=True),
        # one full-width pass on a mid-size graph
        dict(name="batch64_s18_H1", kind="batch", graph="kron", n=1 << 18, pivots=64, H=1, directed=False),
        # the Graph500 scale-14 configuration: uniform sampling, 256 rounds
        dict(name="sampled_z0_s14", kind="sampled", graph="kron", n=1 << 14, z=0, nbfs=256, W=32, H=0,
             bader_c=0, nchecks=1),
        # the reference's sequential form (one pivot per snapshot, its default
        # width) with the mixture heuristic, on a small odd-sized graph
        dict(name="sampled_z6_W1_n5003", kind="sampled", graph="kron", n=5003, z=6, nbfs=24, W=1, H=0,
             bader_c=0, nchecks=1),
        # the scale-20 configuration: degree-weighted sampling, leaves folded,
        # full-width rounds
        dict(name="sampled_z1_s20_H1", kind="sampled", graph="kron", n=1 << 20, z=1, nbfs=256, W=64, H=1,
             bader_c=0, nchecks=1),
        # the headline configuration on its own graph: scale 23, betweenness-
        # weighted sampling in rounds of 32 (128 rounds of its 1024)
        dict(name="sampled_z3_s23", kind="sampled", graph="kron", n=1 << 23, z=3, nbfs=128, W=32, H=0,
             bader_c=0, nchecks=1),
        # the mesh configuration: 2048^2 grid, dependency-weighted sampling with
        # Bader's stop: hundreds of narrow levels each way
        dict(name="sampled_z4_grid2048", kind="sampled", graph="grid", n=2048 * 2048, z=4, nbfs=2048, W=64, H=0,
             bader_c=1, nchecks=8),
        # many pivots on a mesh (road-network-like): wide pass, many levels
        dict(name="batch32_grid512", kind="batch", graph="grid", n=512 * 512, pivots=32, H=0, directed=False),
        # one job from an edge list: ingest, clustering-coefficient sampling,
        # betweenness out
        dict(name="job_z2_s16_H1", kind="job", graph="kron", n=1 << 16, z=2, nbfs=64, W=32, H=1,
             bader_c=0, nchecks=1),
        # the serving configuration cut to twelve requests on three resident
        # graphs (two power-law, one mesh), mixed heuristics and stops
        dict(name="serve12", kind="serve", graph="mix", n=1 << 16, requests=12, nbfs=192, W=8),
    ]


def draw(rng):
    kind = rng.choice(["pivot", "batch", "batch", "sampled", "sampled", "sampled", "job", "serve"])

    def size(lo, hi):  # vertices, spread over the logarithm, mostly not powers of two
        n = int(round(2.0 ** rng.uniform(lo, hi)))
        return 1 << (n.bit_length() - 1) if rng.random() < 0.25 else n

    def side(lo, hi):
        return int(round(2.0 ** rng.uniform(lo, hi))) ** 2

    grid = rng.random() < 0.25
    if kind == "pivot":
        if grid:
            return dict(kind=kind, graph="grid", n=side(5, 8), pivots=rng.randint(1, 4), H=0, directed=False)
        return dict(kind=kind, graph="kron", n=size(10, 18), pivots=rng.randint(1, 4), H=rng.randint(0, 1),
                    directed=False)
    if kind == "batch":
        if grid:
            return dict(kind=kind, graph="grid", n=side(5, 9), pivots=rng.randint(1, 64), H=0, directed=False)
        directed = rng.random() < 0.3
        return dict(kind=kind, graph="kron", n=size(10, 20), pivots=rng.randint(1, 64),
                    H=0 if directed else rng.randint(0, 1), directed=directed)
    if kind == "sampled":
        if grid:
            return dict(kind=kind, graph="grid", n=side(6, 9), z=rng.randint(0, 1), nbfs=rng.randint(8, 64),
                        W=rng.choice([8, 32, 64]), H=0, bader_c=rng.randint(0, 1), nchecks=rng.randint(1, 16))
        n = size(12, 20)
        return dict(kind=kind, graph="kron", n=n, z=rng.choice([0, 1, 3, 4, 5, 6]) if n <= 1 << 16
                    else rng.choice([0, 1, 3, 4, 5]), nbfs=rng.randint(32, 128), W=rng.choice([8, 16, 32, 50, 64]),
                    H=rng.randint(0, 1), bader_c=rng.randint(0, 1), nchecks=rng.randint(1, 16))
    if kind == "job":
        return dict(kind=kind, graph="kron", n=size(10, 16), z=rng.choice([0, 1, 2, 3]), nbfs=rng.randint(16, 64),
                    W=rng.choice([8, 32, 64]), H=rng.randint(0, 1), bader_c=0, nchecks=1)
    return dict(kind=kind, graph="mix", n=size(12, 16), requests=rng.randint(4, 12), nbfs=rng.randint(64, 192),
                W=rng.choice([8, 32]))


# ---------------------------------------------------------------- inputs
def _edges(n, seed, device):
    """R-MAT edges (Graph500 initiator) as int64 vectors u, v: ids scrambled by
    a random permutation, folded into [0, n) when n is no power of two."""
    g = torch.Generator(device=device)
    g.manual_seed(1_000_003 * int(seed) + n)
    scale = max(1, (n - 1).bit_length())
    ne = n * EDGEFACTOR
    u = torch.zeros(ne, dtype=torch.int64, device=device)
    v = torch.zeros(ne, dtype=torch.int64, device=device)
    for _ in range(scale):
        r = torch.rand(ne, generator=g, device=device)
        u = 2 * u + (r >= 0.76)
        v = 2 * v + (((r >= 0.57) & (r < 0.76)) | (r >= 0.95))
    perm = torch.randperm(1 << scale, generator=g, device=device)
    return perm[u] % n, perm[v] % n


def _csc(n, seed, directed, H, device):
    """(col, row, reach) of the kron graph: column c lists, ascending, the r of
    its edges (r, c); H = 1 folds degree-1 vertices into their neighbours."""
    u, v = _edges(n, seed, device)
    keep = u != v
    u, v = u[keep], v[keep]
    if not directed:
        u, v = torch.cat([u, v]), torch.cat([v, u])
    key = torch.unique(v * n + u)
    c, r = key // n, key % n
    reach = torch.zeros(n, dtype=torch.int64, device=device)
    if H:
        deg = torch.bincount(c, minlength=n)
        leaf = deg == 1
        hang = leaf[c] & ~leaf[r]  # edges (r, c) with c a leaf of r
        reach.index_add_(0, r[hang], torch.ones_like(r[hang]))
        keep = ~leaf[c] & ~leaf[r]
        c, r = c[keep], r[keep]
    col = torch.zeros(n + 1, dtype=torch.int64, device=device)
    col[1:] = torch.cumsum(torch.bincount(c, minlength=n), 0)
    return col, r, reach


def _pivots(deg, k, seed):
    """k distinct pivots among the vertices that have edges."""
    cand = np.flatnonzero(deg > 0)
    return np.random.RandomState((1009 * int(seed) + 7) % (1 << 32)).choice(cand, size=min(k, len(cand)),
                                                              replace=False).astype(np.uint32)


def _graph(case, seed):
    """(Graph, degrees on the host)."""
    n, H = case["n"], case.get("H", 0)
    if case["graph"] == "grid":
        G = ax.Graph.grid(round(n ** 0.5), 0.02, 1e-4, seed=7 + int(seed))
        return G, G.deg()
    if n >= 1 << 22:
        G = ax.Graph.kronecker(n.bit_length() - 1, EDGEFACTOR, 23 + int(seed), 24 + int(seed), H=H)
        return G, G.deg()
    col, row, reach = _csc(n, seed, case.get("directed", False), H, "cuda")
    col = col.cpu().numpy().astype(np.uint32)
    G = ax.Graph.from_csc(col, row.cpu().numpy().astype(np.uint32), reach.cpu().numpy().astype(np.uint32))
    return G, np.diff(col)


def _requests(case, seed, graphs):
    """The requests' parameters: graph, heuristic, a round budget or Bader's stop."""
    mix, r = random.Random(11), random.Random(int(seed))  # the mix of requests; their seeds
    out = []
    for _ in range(case["requests"]):
        if mix.random() < 0.5:
            stop = dict(nbfs=int(round(16 * (case["nbfs"] / 16.0) ** mix.random())), bader_c=0, nchecks=1)
        else:
            stop = dict(nbfs=case["nbfs"], bader_c=1, nchecks=mix.randint(4, 16))
        gid = mix.randrange(graphs)
        # on the mesh (the last graph) there are no triangles, and path counts
        # that wrap to 0 leave no usable weights: uniform or degree sampling
        z = mix.choice([0, 1] if gid == graphs - 1 else [0, 1, 2, 3, 4, 5])
        out.append(dict(graph_id=gid, z=z, W=case["W"], seed=r.randrange(1, 1 << 30), **stop))
    return out


def prepare(case, seed):
    kind = case["kind"]
    if kind == "job":
        u, v = _edges(case["n"], seed, "cuda")
        return dict(case=case, seed=int(seed), edges=torch.stack([u, v], 1).cpu().numpy().astype(np.uint64))
    if kind == "serve":
        small = max(256, case["n"] >> 2)
        side = max(16, round((case["n"] >> 2) ** 0.5))
        graphs = [_graph(dict(graph="kron", n=case["n"]), seed)[0], _graph(dict(graph="kron", n=small), seed)[0],
                  _graph(dict(graph="grid", n=side * side), seed)[0]]
        srv = ax.Server()
        for g in graphs:
            srv.add_graph(g)
        return dict(case=case, server=srv, n=[g.n for g in graphs], requests=_requests(case, seed, len(graphs)))
    G, deg = _graph(case, seed)
    st = dict(case=case, seed=int(seed), graph=G, ctx=ax.Context(G))
    if kind in ("pivot", "batch"):
        st["pivots"] = _pivots(deg, case["pivots"], seed)
        st["p"] = np.full(len(st["pivots"]), 1.0 / case["n"])
    return st


# ---------------------------------------------------------------- one pass
def _padded(values, size, fill):
    out = np.full(size, fill, np.asarray(fill).dtype)
    out[:len(values)] = values
    return out


def _sampled(ctx, case, seed):
    r = ctx.run_sampled(z=case["z"], nbfs=case["nbfs"], bader_c=case["bader_c"], nchecks=case["nchecks"],
                        H=case["H"], seed=4343543 + seed, W=case["W"])
    return dict(bc=ctx.bc(), pivots=_padded(r["pivots"], case["nbfs"], -1), probs=_padded(r["probs"], case["nbfs"], 0.0),
                counts=np.array([r["nrounds"], r["skipped"], r["dropped"], r["ui_end"], r["te"]], np.int64))


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "serve":
        srv = state["server"]
        ids = [srv.submit(**q) for q in state["requests"]]
        out = []
        for rid, q in zip(ids, state["requests"]):
            srv.wait(rid)
            bc, piv, _ = srv.result(rid, state["n"][q["graph_id"]])
            srv.release(rid)
            out.append(dict(bc=bc, pivots=_padded(piv, q["nbfs"], -1)))
        return out
    if kind == "job":
        G = ax.Graph.from_edges(state["edges"], case["n"], H=case["H"])
        ctx = ax.Context(G)
        out = _sampled(ctx, case, state["seed"])
        ctx.close()
        G.close()
        return out
    ctx = state["ctx"]
    if kind == "sampled":
        return _sampled(ctx, case, state["seed"])
    ctx.reset()
    if kind == "pivot":
        stats = [ctx.run_pivot(v, p, case["H"]) for v, p in zip(state["pivots"], state["p"])]
    else:
        stats = ctx.run_batch(state["pivots"], state["p"], case["H"])
    return dict(bc=ctx.bc(), stats=np.array([[s["nvisited"], s["all"], s["te"], s["levels"]] for s in stats], np.int64))


def work(case):
    """The graph read once (offsets and adjacency entries, 4 bytes each) and the
    betweenness vector written once; per pivot and adjacency entry one path-count
    addition forward, one multiplication and one addition backward."""
    def entries(graph, n, directed=False):
        if graph == "grid":
            return 4 * n
        return (1 if directed else 2) * EDGEFACTOR * n * 9 // 10  # repeated edges left out

    if case["kind"] == "serve":
        n = case["n"]
        b = sum(4 * entries(g, k) + 8 * k for g, k in (("kron", n), ("kron", n >> 2), ("grid", n >> 2)))
        return dict(bytes=b + 4 * n * case["requests"] / 2.0,
                    flops=3.0 * entries("kron", n) / 2 * case["nbfs"] / 3 * case["requests"])
    n = case["n"]
    m = entries(case["graph"], n, case.get("directed", False))
    pivots = case.get("pivots", case.get("nbfs", 1))
    if case["graph"] == "grid" and case.get("bader_c"):
        pivots = 1  # the stop holds after the first round
    b = 4.0 * m + 8.0 * n
    if case["kind"] == "job":
        b += 16.0 * EDGEFACTOR * n
    return dict(bytes=b, flops=3.0 * m * pivots)


# ---------------------------------------------------------------- 64 bits
def _drand48(seed):
    x = ((seed & 0xFFFFFFFF) << 16) | 0x330E
    while True:
        x = (0x5DEECE66D * x + 0xB) & 0xFFFFFFFFFFFF
        yield x >> 17


def _uniform_pivots(case, seed, deg):
    """The pivots of the uniform heuristic (-z 0): the reference's draw order."""
    n = case["n"]
    r = _drand48(4343543 + int(seed))
    for _ in range(case["nchecks"] + 1):
        next(r)
    lim = (n * n) & 0xFFFFFFFF
    used, out = set(), []
    for _ in range(min(case["nbfs"], n)):
        bad, v = 0, None
        while bad <= lim:
            v = next(r) % (n + 1)
            if v not in used:
                break
            bad += 1
            v = None
        if v is None:
            continue
        if v < n:
            used.add(v)
            if deg[v] > 0:
                out.append(v)
    return out


def _brandes(col, row, reach, pivots, H):
    """bc of the pivots (p = 1/n each) in float64, level by level."""
    dev = row.device
    n = len(col) - 1
    src = torch.repeat_interleave(torch.arange(n, device=dev), col[1:] - col[:-1])
    bc = torch.zeros(n, dtype=torch.float64, device=dev)
    reach = reach.double()
    for v0 in pivots:
        v0 = int(v0)
        lvl = torch.full((n,), -1, dtype=torch.int32, device=dev)
        sigma = torch.zeros(n, dtype=torch.float64, device=dev)
        lvl[v0], sigma[v0] = 0, 1.0
        steps = []
        L = 0
        while True:
            e = torch.nonzero((lvl[src] == L) & (lvl[row] == -1)).view(-1)
            if e.numel() == 0:
                break
            c, u = src[e], row[e]
            sigma.index_add_(0, u, sigma[c])
            L += 1
            lvl[u] = L
            steps.append((c, u))
        delta = reach.clone()
        depths = steps[::-1] if len(steps) == 1 else steps[:0:-1]
        for c, u in depths:
            delta.index_add_(0, c, (delta[u] + 1.0) / sigma[u] * sigma[c])
        term = delta * (reach[v0] + 1.0) * n
        term[v0] = 0.0
        bc += term
        if float(reach[v0]) > 0:
            total = float((lvl >= 0).sum()) + float(reach[v0])
            if H:
                total += float(reach[lvl > 0].sum())
            bc[v0] += float(reach[v0]) * (total - 2.0)
    return bc


def exact(case, seed):
    """bc in 64 bits.  None for grids, whose path counts wrap at 2^32 by the
    reference's definition, for graphs too large to enumerate here, and for the
    heuristics whose pivots depend on rounded weights."""
    if case["graph"] != "kron" or case["n"] > 1 << 18:
        return None
    if case["kind"] in ("pivot", "batch"):
        col, row, reach = _csc(case["n"], seed, case["directed"], case["H"], "cuda")
        piv = _pivots(np.diff(col.cpu().numpy()), case["pivots"], seed)
        return dict(bc=_brandes(col, row, reach, piv, case["H"]).cpu().numpy(), stats=None)
    if case["kind"] == "sampled" and case["z"] == 0 and not case["bader_c"]:
        col, row, reach = _csc(case["n"], seed, False, case["H"], "cuda")
        piv = _uniform_pivots(case, seed, np.diff(col.cpu().numpy()))
        return dict(bc=_brandes(col, row, reach, piv, case["H"]).cpu().numpy(),
                    pivots=None, probs=_padded(np.full(len(piv), 1.0 / case["n"]), case["nbfs"], 0.0), counts=None)
    return None
