"""One-launch passes that cannot run, or give up, as the host sees it (failures
injected on the host; no kernel fails): what the call then does, and that the
context's next pass has the oracle's bits."""
import numpy as np
import pytest

from test_gpu_splits import hub_graph

pytestmark = pytest.mark.gpu
FAIL_WAIT, FAIL_CLUSTER, FAIL_COOP = 0, 1, 2


def failing(axbc, kind, n, call):
    axbc.lib().axbc_inject_pass_failures(kind, n)
    try:
        return call()
    finally:
        axbc.lib().axbc_inject_pass_failures(kind, 0)


def pass_of(ctx, orc, g, piv, p):
    """A batched pass's bc and last dependencies against the oracle's."""
    ctx.reset()
    ctx.run_batch(piv, p)
    want, delta_last, _ = orc.bc_pivots(g, piv, p)
    assert np.array_equal(ctx.bc(), want, equal_nan=True)
    assert np.array_equal(ctx.delta(), delta_last, equal_nan=True)


@pytest.mark.parametrize("undirected", [True, False])
@pytest.mark.parametrize("k", [31, 64])
def test_span_arrivals_start_at_zero_after_a_wait_ran_out(axbc, orc, k, undirected):
    # hubs of 1025 to 2049 neighbours: two and three spans, the last to arrive
    # adds them up.  Other pivots in the second pass, so that span sums left by
    # the first are wrong for it
    g = hub_graph(orc, undirected)
    ctx = axbc.Context(axbc.Graph.from_csc(g.col, g.row, g.reach))
    ctx.set_persistent(1)
    piv = np.random.default_rng(k).permutation(np.flatnonzero(g.deg > 0)).astype(np.uint32)
    p = np.full(k, 1.0 / g.n)
    with pytest.raises(axbc.AxbcError) as ex:
        failing(axbc, FAIL_WAIT, 1, lambda: ctx.run_batch(piv[:k], p))
    assert ex.value.status == 4
    pass_of(ctx, orc, g, piv[k:2 * k], p)
    pass_of(ctx, orc, g, piv[2 * k:3 * k], p)


def grid(orc, side):
    i = np.arange(side * side).reshape(side, side)
    e = np.concatenate([np.stack([i[:, :-1].ravel(), i[:, 1:].ravel()], 1), np.stack([i[:-1].ravel(), i[1:].ravel()], 1)])
    return orc.pipeline(e.astype(np.uint64), side * side, True, 0)


@pytest.mark.parametrize("skip", [0, 1, 2])
@pytest.mark.parametrize("first", [1, 8])
def test_mesh_pass_without_room_for_its_vectors(axbc, orc, first, skip):
    # the vectors of a pass of 33 pivots replace those of the first pass; each of
    # their three allocations is refused in turn
    g = grid(orc, 40)
    ctx = axbc.Context(axbc.Graph.from_csc(g.col, g.row, g.reach))
    piv = np.random.default_rng(1).choice(g.n, 66, replace=False).astype(np.uint32)
    p = np.full(33, 0.25)
    pass_of(ctx, orc, g, piv[:first], p[:first])
    vector = 8 * g.n + 4 * (g.n + 2)  # levels, queue, level starts of one pivot
    bare = ctx.bytes - (1 if first == 1 else 8) * vector
    axbc.lib().axbc_inject_alloc_failure_after(skip)
    try:
        ctx.run_batch(piv[:33], p)
    finally:
        axbc.lib().axbc_inject_alloc_failure_after(-1)
    assert (ctx.bytes - bare) % (8 * g.n) == 0  # level masks of the batched form, no vectors
    want, delta_last, _ = orc.bc_pivots(g, np.concatenate([piv[:first], piv[:33]]), np.full(first + 33, 0.25))
    assert np.array_equal(ctx.bc(), want, equal_nan=True) and np.array_equal(ctx.delta(), delta_last, equal_nan=True)
    ctx.run_batch(piv[33:], p)
    assert (ctx.bytes - bare) % (8 * g.n) == 0  # not tried again
    pass_of(ctx, orc, g, piv[33:], p)  # but after a reset
    assert (ctx.bytes - bare - 64 * vector) % (8 * g.n) == 0


@pytest.mark.parametrize("k", [2, 40])
def test_vectors_of_a_mesh_pass_go_when_a_level_is_too_wide(axbc, orc, k):
    rng = np.random.default_rng(17)
    n = 6000
    g = orc.pipeline(rng.integers(0, n, size=(4 * n, 2)).astype(np.uint64), n, True, 0)
    G = axbc.Graph.from_csc(g.col, g.row, g.reach)
    piv = rng.choice(n, k, replace=False).astype(np.uint32)
    held = []
    for mode in (0, 1):  # the mesh form is tried first; the batched form at once
        ctx = axbc.Context(G)
        ctx.set_persistent(mode)
        pass_of(ctx, orc, g, piv, np.full(k, 0.5))
        pass_of(ctx, orc, g, piv, np.full(k, 0.5))
        held.append(ctx.bytes)
    assert held[0] == held[1]


def mesh_blocks(axbc, ctx, blocks):
    """Set the blocks per pivot of later mesh passes; those of the last one."""
    import ctypes
    used = ctypes.c_int()
    assert axbc.lib().axbc_ctx_mesh_blocks(ctx._h, blocks, ctypes.byref(used)) == 0
    return used.value


@pytest.mark.parametrize("refused", [1, 2, 4, 5])
def test_mesh_pass_on_the_largest_cluster_that_fits(axbc, orc, refused):
    g = grid(orc, 40)
    ctx = axbc.Context(axbc.Graph.from_csc(g.col, g.row, g.reach))
    piv = np.array([0, 820, 1599], np.uint32)
    mesh_blocks(axbc, ctx, 16)
    failing(axbc, FAIL_CLUSTER, refused, lambda: pass_of(ctx, orc, g, piv, np.full(3, 0.5)))
    assert mesh_blocks(axbc, ctx, 16) == 16 >> refused  # 5: none fits, the batched form
    pass_of(ctx, orc, g, piv[1:], np.full(2, 0.5))
    assert mesh_blocks(axbc, ctx, 0) == 16 >> refused


@pytest.mark.parametrize("undirected", [True, False])
@pytest.mark.parametrize("k", [1, 2, 3])
@pytest.mark.parametrize("blocks", [1, 2, 4, 8, 16])
def test_mesh_pass_on_clusters_of_each_size(axbc, orc, blocks, k, undirected):
    # levels around the threads of a block and of every cluster, and the padding
    # (isolated vertices) that keeps them from being too wide
    rng = np.random.default_rng(7)
    width = [1, 2, 31, 500, 1023, 1024, 1025, 2047, 2048, 2049, 4097, 8193, 16385, 16384, 9000, 33, 1, 1]
    first, n = np.cumsum([0] + width), 280000
    e = []
    for i in range(len(width) - 1):
        child = np.arange(width[i + 1])
        e += [np.stack([first[i] + parent, first[i + 1] + child], 1)
              for parent in (child % width[i], rng.integers(0, width[i], width[i + 1]))]
    e = np.concatenate(e)
    if not undirected:
        e = np.concatenate([e[:, ::-1], e[rng.random(len(e)) < 0.1]])
    g = orc.pipeline(e.astype(np.uint64), n, undirected, 0)
    G = axbc.Graph.from_csc(g.col, g.row, rng.integers(0, 3, n).astype(np.uint32))
    g = orc.CSC(g.col, g.row, G.csc()[2])
    ctx = axbc.Context(G)
    mesh_blocks(axbc, ctx, blocks)
    piv = np.array([0, 1, 0][:k], np.uint32)
    for _ in range(2):
        pass_of(ctx, orc, g, piv, np.full(k, 0.5))
        assert mesh_blocks(axbc, ctx, blocks) == blocks
    for s in range(k):
        _, lvl, sigma, delta, _ = orc.bc_pivot(g, int(piv[s]), 0.5)
        gs, gl, gd = ctx.batch_source(s)
        assert np.array_equal(gs, sigma) and np.array_equal(gl, lvl) and np.array_equal(gd, delta, equal_nan=True)


@pytest.mark.parametrize("blocks", [1, 2, 8, 16])
def test_too_wide_a_level_on_clusters_then_the_batched_form(axbc, orc, blocks):
    rng = np.random.default_rng(17)
    n = 60000  # a random graph: levels of tens of thousands of vertices
    g = orc.pipeline(rng.integers(0, n, size=(3 * n, 2)).astype(np.uint64), n, True, 0)
    ctx = axbc.Context(axbc.Graph.from_csc(g.col, g.row, g.reach))
    mesh_blocks(axbc, ctx, blocks)
    piv = rng.choice(n, 6, replace=False).astype(np.uint32)
    for k in (2, 6):
        pass_of(ctx, orc, g, piv[:k], np.full(k, 0.5))
        assert mesh_blocks(axbc, ctx, blocks) == 0


@pytest.mark.parametrize("d", [2, 4, 16])
@pytest.mark.parametrize("n", [65535, 65536, 70001])
def test_a_graph_too_wide_is_tried_once(axbc, orc, n, d):
    # from 65536 vertices on by a forward sweep of its first pivot, below by the
    # pass itself; then the batched form for every context of the graph
    rng = np.random.default_rng(n)
    e = np.stack([np.repeat(np.arange(n), d // 2), rng.integers(0, n, n * (d // 2))], 1)
    g = orc.pipeline(e.astype(np.uint64), n, True, 0)
    assert g.deg.max() <= 64
    G = axbc.Graph.from_csc(g.col, g.row, g.reach)
    piv = rng.choice(np.flatnonzero(g.deg > 0), 5, replace=False).astype(np.uint32)
    lvl = [orc.bc_pivot(g, int(v), 0.5)[1] for v in piv]
    wide = max(np.bincount(x[x >= 0]).max() for x in lvl) > max(2048, n // 16)
    assert wide == (d > 2)  # one random neighbour each: levels of a few thousand
    made = []
    for _ in range(3):
        ctx = axbc.Context(G)
        before = ctx.launches
        pass_of(ctx, orc, g, piv, np.full(5, 0.5))
        made.append(ctx.launches - before)
        assert (mesh_blocks(axbc, ctx, 0) == 0) == wide
    if not wide:
        assert made[1] == made[2] == made[0] - (2 if n >= 1 << 16 else 0)  # the trial
        return
    assert made[1] == made[2] == made[0] - 2  # a reset and the attempt


@pytest.mark.parametrize("k", [2, 9])
@pytest.mark.parametrize("side", [255, 256, 300])
def test_a_mesh_passes_its_trial(axbc, orc, side, k):
    g = grid(orc, side)
    G = axbc.Graph.from_csc(g.col, g.row, np.random.default_rng(3).integers(0, 2, g.n).astype(np.uint32))
    g = orc.CSC(g.col, g.row, G.csc()[2])
    for _ in range(2):
        ctx = axbc.Context(G)
        pass_of(ctx, orc, g, np.random.default_rng(k).choice(g.n, k, replace=False).astype(np.uint32), np.full(k, 0.5))
        assert mesh_blocks(axbc, ctx, 0) > 0


@pytest.mark.parametrize("z", [0, 1, 2, 3, 5])
@pytest.mark.parametrize("n", [7, 8, 9, 15, 16, 17, 22, 23, 31, 32, 33, 50])
def test_rounds_dropped_after_n_squared_rejections(axbc, orc, n, z):
    # n^2 rejections drop a round: fewer and more than a window's 64 and 256
    # draws.  Half the vertices have no neighbour, so that some heuristics run
    # out of vertices to draw
    rng = np.random.default_rng(n)
    half = max(4, n // 2)
    e = np.concatenate([rng.integers(0, half, size=(2 * n, 2)), [[0, 1], [1, 2], [0, 2]]])
    g = orc.pipeline(e.astype(np.uint64), n, True, 0)
    G = axbc.Graph.from_csc(g.col, g.row, g.reach)
    for W in (1, 7, 64):
        ctx = axbc.Context(G)
        got = ctx.run_sampled(z=z, nbfs=n, bader_c=0, nchecks=1, seed=n + W, W=W)
        want = orc.run(g, z=z, nbfs=n, bader_c=0, nchecks=1, seed=n + W, W=W)
        assert np.array_equal(got["pivots"], want["pivots"])
        assert np.array_equal(got["probs"], want["probs"], equal_nan=True)
        for k in ("nrounds", "skipped", "dropped", "ui_end", "te"):
            assert got[k] == want[k], (W, k)
        assert np.array_equal(ctx.bc(), want["bc"], equal_nan=True)


@pytest.mark.parametrize("skip", range(4))
def test_plain_pivot_without_room_for_its_one_launch(axbc, orc, skip):
    # the level-by-level form's buffers are there; the four beside them are not
    g = hub_graph(orc, True)
    ctx = axbc.Context(axbc.Graph.from_csc(g.col, g.row, g.reach))
    ctx.profile(True)
    ctx.run_pivot(1, 0.5)
    ctx.profile(False)
    piv = np.flatnonzero(g.deg > 0)[::400].astype(np.uint32)
    for v in (int(x) for x in piv):
        ctx.reset()
        axbc.lib().axbc_inject_alloc_failure_after(skip)
        try:
            st = ctx.run_pivot(v, 0.5, 1)
        finally:
            axbc.lib().axbc_inject_alloc_failure_after(-1)
        want, lvl, sigma, delta, stats = orc.bc_pivot(g, v, 0.5, 1)
        assert np.array_equal(ctx.bc(), want) and np.array_equal(ctx.delta(), delta) and st == stats
        assert np.array_equal(ctx.levels(), lvl) and np.array_equal(ctx.sigma(), sigma)


@pytest.mark.parametrize("skip", range(9))
def test_pass_of_one_pivot_without_room_for_its_one_launch(axbc, orc, skip):
    g = hub_graph(orc, True)
    ctx = axbc.Context(axbc.Graph.from_csc(g.col, g.row, g.reach))
    piv = np.flatnonzero(g.deg > 0)[::400].astype(np.uint32)
    pass_of(ctx, orc, g, piv[:5], np.full(5, 0.5))
    axbc.lib().axbc_inject_alloc_failure_after(skip)
    try:
        pass_of(ctx, orc, g, piv[5:6], np.full(1, 0.5))
    finally:
        axbc.lib().axbc_inject_alloc_failure_after(-1)
    _, lvl, sigma, delta, _ = orc.bc_pivot(g, int(piv[5]), 0.5)
    gs, gl, gd = ctx.batch_source(0)
    assert np.array_equal(gs, sigma) and np.array_equal(gl, lvl) and np.array_equal(gd, delta)
    pass_of(ctx, orc, g, piv[6:7], np.full(1, 0.5))


def pivot_of(ctx, orc, g, v, H=1):
    """A plain pivot's bc, vectors and statistics against the oracle's."""
    ctx.reset()
    st = ctx.run_pivot(v, 0.5, H)
    want, lvl, sigma, delta, stats = orc.bc_pivot(g, v, 0.5, H)
    assert np.array_equal(ctx.bc(), want) and np.array_equal(ctx.delta(), delta) and st == stats
    assert np.array_equal(ctx.levels(), lvl) and np.array_equal(ctx.sigma(), sigma)


def plain_launches(ctx, v):
    before = ctx.launches
    ctx.run_pivot(v, 0.5)
    return ctx.launches - before


@pytest.mark.parametrize("undirected", [True, False])
def test_plain_pivot_without_a_cooperative_launch(axbc, orc, undirected):
    g = hub_graph(orc, undirected)
    G = axbc.Graph.from_csc(g.col, g.row, g.reach)
    v = int(np.flatnonzero(g.deg > 0)[700])
    ctx = axbc.Context(G)
    assert plain_launches(ctx, v) == 1
    failing(axbc, FAIL_COOP, 1, lambda: pivot_of(ctx, orc, g, v))
    assert plain_launches(ctx, v) > 5  # not asked for again
    pivot_of(ctx, orc, g, v)
    ctx = axbc.Context(G)
    ctx.set_persistent(-1)  # the caller wants none
    pivot_of(ctx, orc, g, v)
    assert plain_launches(ctx, v) > 5
    ctx.set_persistent(0)
    pivot_of(ctx, orc, g, v)
    assert plain_launches(ctx, v) == 1


@pytest.mark.parametrize("undirected", [True, False])
@pytest.mark.parametrize("k", [1, 31, 64])
def test_passes_without_a_cooperative_launch(axbc, orc, k, undirected):
    g = hub_graph(orc, undirected)
    ctx = axbc.Context(axbc.Graph.from_csc(g.col, g.row, g.reach))
    piv = np.random.default_rng(k).permutation(np.flatnonzero(g.deg > 0)).astype(np.uint32)
    p = np.full(k, 1.0 / g.n)
    failing(axbc, FAIL_COOP, 1, lambda: pass_of(ctx, orc, g, piv[:k], p))
    pass_of(ctx, orc, g, piv[k:2 * k], p)
    ctx.set_persistent(1)  # asked for by name: an error, as before
    with pytest.raises(axbc.AxbcError) as ex:
        ctx.run_batch(piv[:k], p)
    assert ex.value.status == 2
    ctx.set_persistent(0)
    pass_of(ctx, orc, g, piv[:k], p)


@pytest.mark.parametrize("undirected", [True, False])
def test_plain_pivot_after_a_wait_that_ran_out(axbc, orc, undirected):
    g = hub_graph(orc, undirected)
    ctx = axbc.Context(axbc.Graph.from_csc(g.col, g.row, g.reach))
    v = np.flatnonzero(g.deg > 0)
    failing(axbc, FAIL_WAIT, 1, lambda: pivot_of(ctx, orc, g, int(v[9])))
    pivot_of(ctx, orc, g, int(v[-1]))
    assert plain_launches(ctx, int(v[9])) == 1


@pytest.mark.parametrize("undirected", [True, False])
@pytest.mark.parametrize("H", [0, 1])
@pytest.mark.parametrize("k,fails", [(1, 1), (1, 2), (31, 1), (64, 1)])
def test_passes_start_again_after_a_wait_that_ran_out(axbc, orc, k, fails, H, undirected):
    # the roots have their numbers of the view already; with one pivot the plain
    # form's launch fails first, then the persistent loop's
    g = hub_graph(orc, undirected)
    reach = np.random.default_rng(2).integers(0, 3, g.n).astype(np.uint32)
    ctx = axbc.Context(axbc.Graph.from_csc(g.col, g.row, reach))
    g = orc.CSC(g.col, g.row, reach)
    piv = np.random.default_rng(k).permutation(np.flatnonzero(g.deg > 0)).astype(np.uint32)
    p = np.full(k, 1.0 / g.n)
    for i in range(3):  # the failing pass first, between others and after itself
        q = piv[k * i:k * i + k]
        ctx.reset()
        stats = failing(axbc, FAIL_WAIT, fails if i < 2 else 0, lambda: ctx.run_batch(q, p, H))
        want, delta_last, _ = orc.bc_pivots(g, q, p, H)
        assert np.array_equal(ctx.bc(), want) and np.array_equal(ctx.delta(), delta_last)
        for s in (0, k - 1):
            _, lvl, sigma, delta, st = orc.bc_pivot(g, int(q[s]), p[s], H)
            gs, gl, gd = ctx.batch_source(s)
            assert stats[s] == st
            assert np.array_equal(gs, sigma) and np.array_equal(gl, lvl) and np.array_equal(gd, delta)


def test_sampled_runs_and_requests_go_on_after_waits_that_ran_out(axbc, orc):
    e = axbc.kron_edges(10, 16).astype(np.uint64)
    g = orc.pipeline(e, 1024, True, 0)
    G = axbc.Graph.from_csc(g.col, g.row, g.reach)
    for z, W, c in ((0, 32, 0), (3, 1, 0), (2, 64, 1)):
        prm = dict(z=z, nbfs=48, bader_c=c, nchecks=4, seed=3, W=W)
        want = orc.run(g, **prm)
        ctx = axbc.Context(G)
        got = failing(axbc, FAIL_WAIT, 3, lambda: ctx.run_sampled(**prm))
        assert np.array_equal(got["pivots"], want["pivots"]) and got["te"] == want["te"]
        assert np.array_equal(ctx.bc(), want["bc"], equal_nan=True)
        srv = axbc.Server()
        gid = srv.add_graph(G)

        def serve():
            rid = srv.submit(gid, **prm)
            assert srv.wait(rid, timeout_ms=60000)["state"] == "done"
            return srv.result(rid, G.n)[0]
        assert np.array_equal(failing(axbc, FAIL_WAIT, 3, serve), want["bc"], equal_nan=True)
        srv.close()


def long_path(orc, n, hub=70):
    """A path of n vertices, with leaves that make its second one a hub."""
    c = np.arange(n)
    e = np.concatenate([np.stack([c[:-1], c[1:]], 1), np.stack([np.ones(hub, int), n + np.arange(hub)], 1)])
    return orc.pipeline(e.astype(np.uint64), n + hub, True, 0)


def test_deepest_pass_of_one_pivot(axbc, orc):
    for n, fits in ((65533, True), (65534, False)):
        g = long_path(orc, n)
        ctx = axbc.Context(axbc.Graph.from_csc(g.col, g.row, g.reach))
        one, p = np.zeros(1, np.uint32), np.full(1, 0.5)
        if fits:
            pass_of(ctx, orc, g, one, p)
        else:
            with pytest.raises(axbc.AxbcError) as ex:
                ctx.run_batch(one, p)
            assert ex.value.status == 5
        pass_of(ctx, orc, g, np.full(1, n // 2, np.uint32), p)


def test_too_deep_a_pass_is_refused_at_the_limit(axbc, orc):
    # and not at the end of a traversal twenty times as deep
    import time
    took = []
    for n in (70000, 1400000):
        g = long_path(orc, n)
        ctx = axbc.Context(axbc.Graph.from_csc(g.col, g.row, g.reach))
        for _ in range(2):
            t = time.perf_counter()
            with pytest.raises(axbc.AxbcError) as ex:
                ctx.run_batch(np.zeros(1, np.uint32), np.full(1, 0.5))
            t = time.perf_counter() - t
            assert ex.value.status == 5
        took.append(t)
    assert took[1] < 5 * took[0], took


@pytest.mark.parametrize("first", [1, 3])
def test_no_source_of_a_failed_pass(axbc, orc, first):
    # a mesh pass of 599 levels, then a pass that fails where only ten level
    # masks exist: there is no source to read, neither the old nor a new one
    g = grid(orc, 300)
    ctx = axbc.Context(axbc.Graph.from_csc(g.col, g.row, g.reach))
    piv = np.array([0, 44850, 89999], np.uint32)
    pass_of(ctx, orc, g, piv[:first], np.full(first, 0.5))
    assert ctx.batch_source(0)[1].max() == 598
    ctx.set_persistent(-1)
    axbc.lib().axbc_inject_alloc_failures(1)
    try:
        with pytest.raises(axbc.AxbcError) as ex:
            ctx.run_batch(piv, np.full(3, 0.5))
    finally:
        axbc.lib().axbc_inject_alloc_failures(0)
    assert ex.value.status == 3
    with pytest.raises(axbc.AxbcError) as ex:
        ctx.batch_source(0)
    assert ex.value.status == 1
    pass_of(ctx, orc, g, piv, np.full(3, 0.5))
    assert np.array_equal(ctx.batch_source(1)[1], orc.bc_pivot(g, 44850, 0.5)[1])


def test_one_launch_forms_from_two_threads(axbc, orc):
    # contexts of two threads: grids of blocks that wait for one another, each
    # wide enough for the whole device, launched at the same time
    import threading
    import time
    made = []
    for scale, seed in ((12, 3), (14, 4)):
        e = axbc.kron_edges(scale, 16, seed, seed + 1).astype(np.uint64)
        g = orc.pipeline(e, 1 << scale, True, 0)
        piv = np.flatnonzero(g.deg > 0)[::97][:24].astype(np.uint32)
        made.append((g, axbc.Graph.from_csc(g.col, g.row, g.reach), piv, np.full(len(piv), 0.5)))
    got, failed = {}, []

    def work(i):
        try:
            g, G, piv, p = made[i]
            ctx = axbc.Context(G)
            for v in piv:
                ctx.run_pivot(int(v), 0.5)
            a = ctx.bc()
            ctx.reset()
            for _ in range(8):
                ctx.run_batch(piv, p, 0, stats=False)
                ctx.run_batch(piv[:1], p[:1], 0, stats=False)
            got[i] = a, ctx.bc()
        except Exception as ex:  # reported by the test's thread
            failed.append(ex)

    t0 = time.perf_counter()
    threads = [threading.Thread(target=work, args=(i,)) for i in (0, 1)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed
    assert time.perf_counter() - t0 < 3.5  # no wait ran out (about 4 s) on the way
    for i, (g, _, piv, p) in enumerate(made):
        assert np.array_equal(got[i][0], orc.bc_pivots(g, piv, p)[0])
        order = np.concatenate([np.concatenate([piv, piv[:1]])] * 8)
        assert np.array_equal(got[i][1], orc.bc_pivots(g, order, np.full(len(order), 0.5))[0])
