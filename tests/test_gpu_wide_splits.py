"""The splits of larger graphs at the degrees where they change hands: parts of
128 positions from 2^18 adjacency entries on and of 512 from 2^25, the backward
by warps with its combine from 2^22 entries (2^21 at two mask words) on, and the
step launches, against the oracle bit for bit.  The graphs are the hubs of every
edge degree among filler that makes up the entries."""
import functools

import numpy as np
import pytest

from test_gpu_splits import DEGREES

pytestmark = pytest.mark.gpu


@functools.lru_cache(maxsize=2)
def filled_graph(orc, entries, undirected):
    """Hubs of exactly DEGREES[i] neighbours (each way, where edges have one) on a
    path, vertices of 1 to 12 neighbours, and random filler of `entries` entries
    on which both hang."""
    rng = np.random.default_rng(11)
    h, path, small = len(DEGREES), 3000, 4800
    core = max(5000, entries // 40)
    at_path, at_small = h, h + path
    at_core = at_small + small
    e = [np.stack([np.full(d, i), at_path + rng.choice(path, d, replace=False)], 1) for i, d in enumerate(DEGREES)]
    c = at_path + np.arange(path)
    e.append(np.stack([c[:-1], c[1:]], 1))
    e.append(np.stack([rng.choice(c, 300), at_core + rng.integers(0, core, 300)], 1))
    v = np.repeat(at_small + np.arange(small), 1 + np.arange(small) % 12)
    e.append(np.stack([v, at_core + rng.integers(0, core, len(v))], 1))
    fill = int(entries * 1.04) // (2 if undirected else 1)
    e.append(at_core + rng.integers(0, core, size=(fill, 2)))
    if not undirected:  # out-lists of the same degrees, other entries; most of the rest both ways
        back = np.concatenate(e[h:-1])
        e += [np.stack([at_path + rng.choice(path, d, replace=False), np.full(d, i)], 1) for i, d in enumerate(DEGREES)]
        e.append(back[rng.random(len(back)) < 0.6, ::-1])
    e = np.concatenate(e)
    g = orc.pipeline(e.astype(np.uint64), at_core + core, undirected, 0)
    assert len(g.row) >= entries and np.array_equal(g.deg[:h], DEGREES)
    return g


def check(axbc, orc, g, k, mode, factor):
    ctx = axbc.Context(axbc.Graph.from_csc(g.col, g.row, g.reach))
    ctx.set_tuning(8.0, factor)
    ctx.set_persistent(mode)
    rng = np.random.default_rng(k)
    linked = np.flatnonzero(g.deg > 0)
    piv = np.concatenate([linked[linked < len(DEGREES)][-3:], rng.choice(linked, 61, replace=False)])[:k].astype(np.uint32)
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


# the same loop, the steps, and the rule's choice, at 2^18 entries; then the steps
# with tiles (below the line) and with the backward by warps (above it)
@pytest.mark.parametrize("factor", [8.0, 0.0, 1e30])
@pytest.mark.parametrize("k,mode", [(1, -1), (1, 1), (31, -1), (32, 0), (33, 0), (64, -1)])
@pytest.mark.parametrize("undirected", [True, False])
def test_parts_of_128(axbc, orc, undirected, k, mode, factor):
    check(axbc, orc, filled_graph(orc, (1 << 18) + 1000, undirected), k, mode, factor)


@pytest.mark.parametrize("factor", [8.0, 0.0, 1e30])
@pytest.mark.parametrize("k", [2, 32, 33, 64])
@pytest.mark.parametrize("undirected", [True, False])
def test_step_launches_around_the_backward_by_warps(axbc, orc, undirected, k, factor):
    # two mask words: by warps; one: in tiles
    check(axbc, orc, filled_graph(orc, (1 << 21) + 1000, undirected), k, 0, factor)


@pytest.mark.parametrize("factor", [8.0, 0.0, 1e30])
@pytest.mark.parametrize("k", [2, 32, 64])
@pytest.mark.parametrize("undirected", [True, False])
def test_backward_by_warps_at_both_widths(axbc, orc, undirected, k, factor):
    check(axbc, orc, filled_graph(orc, (1 << 22) + 1000, undirected), k, 0, factor)


@pytest.mark.parametrize("k", [3, 33])
def test_parts_of_512(axbc, orc, k):
    check(axbc, orc, filled_graph(orc, (1 << 25) + 1000, True), k, 0, 8.0)
