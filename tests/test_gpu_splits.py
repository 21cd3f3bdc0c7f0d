"""Batched passes at the degrees where the kernels split a vertex's adjacency
differently (subgroups of 8 and 16 lanes, chunks of 32, several warps above 128
neighbours, spans above 1024), at pass widths around one and two mask words, with
every level pushed, pulled or chosen, against the oracle bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DEGREES = [1, 2, 7, 8, 9, 15, 16, 17, 31, 32, 33, 63, 64, 65, 127, 128, 129, 159, 160, 161, 255, 256, 257, 383, 384,
           385, 1023, 1024, 1025, 1057, 2047, 2048, 2049]


def hub_graph(orc, undirected):
    """Vertex i < len(DEGREES) has exactly DEGREES[i] neighbours among the rest,
    which form a path with a few chords."""
    rng = np.random.default_rng(11)
    h, rest = len(DEGREES), 3000
    e = [np.stack([np.full(d, i), h + rng.choice(rest, d, replace=False)], 1) for i, d in enumerate(DEGREES)]
    chain = np.arange(h, h + rest - 1)
    e.append(np.stack([chain, chain + 1], 1))
    e.append(h + rng.integers(0, rest, size=(200, 2)))
    e = np.concatenate(e).astype(np.uint64)
    if not undirected:  # both directions occur, lists differ between them
        back = e[rng.random(len(e)) < 0.6]
        e = np.concatenate([e, back[:, ::-1]])
    return orc.pipeline(e, h + rest, undirected, 0)


@pytest.mark.parametrize("factor", [8.0, 0.0, 1e30])
@pytest.mark.parametrize("k", [1, 31, 32, 33, 64])
@pytest.mark.parametrize("undirected", [True, False])
def test_degree_edges(axbc, orc, undirected, k, factor):
    g = hub_graph(orc, undirected)
    ctx = axbc.Context(axbc.Graph.from_csc(g.col, g.row, g.reach))
    ctx.set_tuning(8.0, factor)
    rng = np.random.default_rng(k)
    piv = rng.choice(np.flatnonzero(g.deg > 0), k, replace=False).astype(np.uint32)
    p = np.full(k, 1.0 / g.n)
    for _ in range(2):  # the second pass starts from the first one's buffers
        ctx.reset()
        ctx.run_batch(piv, p)
    want, delta_last, _ = orc.bc_pivots(g, piv, p)
    assert np.array_equal(ctx.bc(), want) and np.array_equal(ctx.delta(), delta_last)
    for s in {0, k // 2, k - 1}:
        _, lvl, sigma, delta, _ = orc.bc_pivot(g, int(piv[s]), p[s])
        gs, gl, gd = ctx.batch_source(s)
        assert np.array_equal(gs, sigma) and np.array_equal(gl, lvl) and np.array_equal(gd, delta), s


@pytest.mark.parametrize("n", [3, 65, 66, 67, 129, 2048, 2049, 2051])
def test_clustering_of_complete_graphs(axbc, n):
    # a vertex's higher neighbours number up to n - 1: every table size, and
    # more members than a block's table holds.  A fan of leaves around vertex 0
    # makes the graph's largest degree exceed 64, so that ranks exist
    u, v = np.triu_indices(n, 1)
    leaves = 80
    e = np.concatenate([np.stack([u, v], 1), np.stack([np.zeros(leaves, int), n + np.arange(leaves)], 1)])
    lcc = axbc.Graph.from_edges(e.astype(np.uint64), n + leaves).lcc()
    d = np.float32(n - 1 + leaves)
    want = np.concatenate([[np.float32((n - 1) * (n - 2)) / (d * (d - 1))], np.ones(n - 1), np.zeros(leaves)])
    assert np.array_equal(lcc, want.astype(np.float32))


@pytest.mark.parametrize("H", [0, 1])
def test_clustering_of_a_power_law_graph(axbc, orc, H):
    e = axbc.kron_edges(12, 16)
    g = orc.pipeline(e.astype(np.uint64), 1 << 12, True, H)
    assert np.array_equal(axbc.Graph.from_csc(g.col, g.row, g.reach).lcc(), orc.lcc(g))
    # a self-loop or a repeated entry takes the general count
    col, row = g.col.copy(), g.row.copy()
    v = int(np.flatnonzero(g.deg > 2)[5])
    row[col[v]] = row[col[v] + 1]
    h = orc.CSC(col, row)
    assert np.array_equal(axbc.Graph.from_csc(col, row).lcc(), orc.lcc(h))


@pytest.mark.parametrize("factor", [8.0, 0.0, 1e30])
@pytest.mark.parametrize("undirected", [True, False])
def test_plain_pivots_at_degree_edges(axbc, orc, undirected, factor):
    g = hub_graph(orc, undirected)
    ctx = axbc.Context(axbc.Graph.from_csc(g.col, g.row, g.reach))
    ctx.set_tuning(factor, 8.0)
    rng = np.random.default_rng(3)
    for v in rng.choice(np.flatnonzero(g.deg > 0), 6, replace=False):
        for profiled in (False, True):  # one launch, then level by level
            ctx.profile(profiled)
            ctx.reset()
            st = ctx.run_pivot(int(v), 1.0 / g.n, 1)
            want, lvl, sigma, delta, stats = orc.bc_pivot(g, int(v), 1.0 / g.n, 1)
            assert np.array_equal(ctx.bc(), want) and np.array_equal(ctx.delta(), delta)
            assert np.array_equal(ctx.levels(), lvl) and np.array_equal(ctx.sigma(), sigma)
            assert st == stats


def sparse_graph(kind, rng):
    """Graphs without a vertex of more than 64 neighbours: their passes run a
    cluster of blocks per pivot, unless a level is too wide."""
    if kind.startswith("grid"):
        side = int(kind[4:])
        i = np.arange(side * side).reshape(side, side)
        e = [np.stack([i[:, :-1].ravel(), i[:, 1:].ravel()], 1), np.stack([i[:-1].ravel(), i[1:].ravel()], 1)]
        return np.concatenate(e), side * side
    if kind == "path":
        return np.stack([np.arange(699), np.arange(1, 700)], 1), 700
    if kind == "ladders":  # every degree up to 64, three components
        e = [np.stack([np.full(d, 3 * d), 300 + rng.choice(900, d, replace=False)], 1) for d in range(1, 40)]
        chain = np.arange(300, 1199)
        return np.concatenate(e + [np.stack([chain, chain + 1], 1), [[1250, 1251]]]), 1300
    n = 6000  # "wide": levels of thousands of vertices
    return rng.integers(0, n, size=(4 * n, 2)), n


@pytest.mark.parametrize("undirected", [True, False])
@pytest.mark.parametrize("k", [1, 2, 33, 64])
@pytest.mark.parametrize("kind", ["grid40", "path", "ladders", "wide"])
def test_mesh_passes(axbc, orc, kind, k, undirected):
    rng = np.random.default_rng(17)
    e, n = sparse_graph(kind, rng)
    g = orc.pipeline(e.astype(np.uint64), n, undirected, 0)
    assert g.deg.max() <= 64
    ctx = axbc.Context(axbc.Graph.from_csc(g.col, g.row, rng.integers(0, 3, n).astype(np.uint32)))
    g = orc.CSC(g.col, g.row, ctx.graph.csc()[2])
    piv = rng.choice(n, k, replace=False).astype(np.uint32)
    p = rng.random(k) + 0.1
    for _ in range(2):
        ctx.reset()
        stats = ctx.run_batch(piv, p, 1)
    want, delta_last, _ = orc.bc_pivots(g, piv, p, 1)
    assert np.array_equal(ctx.bc(), want, equal_nan=True) and np.array_equal(ctx.delta(), delta_last, equal_nan=True)
    levels = ctx.level_stats()
    total = 0
    for s in range(k):
        _, lvl, sigma, delta, st = orc.bc_pivot(g, int(piv[s]), p[s], 1)
        assert stats[s] == st
        total += st["nvisited"]
        if s in (0, k - 1):
            gs, gl, gd = ctx.batch_source(s)
            assert np.array_equal(gs, sigma) and np.array_equal(gl, lvl)
            assert np.array_equal(gd, delta, equal_nan=True)
    assert int(levels["count"].sum()) == total


def test_mesh_pass_on_several_blocks(axbc, orc):
    e, n = sparse_graph("grid300", None)  # wide enough for clusters of two and more
    g = orc.pipeline(e.astype(np.uint64), n, True, 0)
    ctx = axbc.Context(axbc.Graph.from_csc(g.col, g.row))
    for k in (1, 3):
        piv = np.array([12, 44850, 89999][:k], np.uint32)
        p = np.full(k, 0.5)
        ctx.reset()
        ctx.run_batch(piv, p)
        want, delta_last, _ = orc.bc_pivots(g, piv, p)
        assert np.array_equal(ctx.bc(), want, equal_nan=True) and np.array_equal(ctx.delta(), delta_last, equal_nan=True)


@pytest.mark.parametrize("nchecks", [0, 1, 31, 32, 33, 70])
@pytest.mark.parametrize("z", [0, 1, 3, 5])
def test_sampler_windows_and_many_check_vertices(axbc, orc, z, nchecks):
    # rounds around the 64- and 256-value windows with many repeated draws, and
    # more check vertices than the replay keeps in shared memory
    rng = np.random.default_rng(5)
    e = rng.integers(0, 300, size=(2400, 2))
    g = orc.pipeline(e.astype(np.uint64), 320, True, 0)
    G = axbc.Graph.from_csc(g.col, g.row, g.reach)
    for W, c in ((1, 1), (16, 0), (17, 2), (64, 1)):
        ctx = axbc.Context(G)
        got = ctx.run_sampled(z=z, nbfs=300, bader_c=c, nchecks=nchecks, seed=77 + W, W=W)
        want = orc.run(g, z=z, nbfs=300, bader_c=c, nchecks=nchecks, seed=77 + W, W=W)
        assert np.array_equal(got["checks"], want["checks"]) and np.array_equal(got["pivots"], want["pivots"])
        assert np.array_equal(got["probs"], want["probs"], equal_nan=True)
        for k in ("nrounds", "skipped", "dropped", "ui_end", "te", "stopped"):
            assert got[k] == want[k], (W, c, k)
        assert np.array_equal(ctx.bc(), want["bc"], equal_nan=True)


@pytest.mark.parametrize("undirected", [True, False])
@pytest.mark.parametrize("leaves", [65, 254, 255, 256, 510, 511, 512, 513, 1300])
def test_ingest_of_a_hub_among_isolated_vertices(axbc, orc, leaves, undirected):
    # adjacency runs around the 512 entries a warp renumbers, with vertices
    # without entries before, between and after the linked ones
    n = 3 * leaves + 40
    hub = 17
    spokes = 20 + 3 * np.arange(leaves)
    e = np.concatenate([np.stack([np.full(leaves, hub), spokes], 1), np.stack([spokes[:-1], spokes[1:]], 1)[::7],
                        [[hub, hub], [spokes[3], spokes[3]], [hub, spokes[0]]]]).astype(np.uint64)
    want = orc.pipeline(e, n, undirected, 0)
    graph = axbc.Graph.from_edges(e, n, undirected=undirected, H=0)
    col, row, reach = graph.csc()
    assert np.array_equal(col, want.col) and np.array_equal(row, want.row) and not reach.any()
    ctx = axbc.Context(graph)
    piv = np.array([hub, spokes[0], spokes[-1]], np.uint32)
    ctx.run_batch(piv, np.full(3, 0.25))
    assert np.array_equal(ctx.bc(), orc.bc_pivots(want, piv, np.full(3, 0.25))[0])
