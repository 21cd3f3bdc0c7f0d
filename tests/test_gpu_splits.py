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
