"""One-launch passes that cannot run, or give up, as the host sees it (failures
injected on the host; no kernel fails): what the call then does, and that the
context's next pass has the oracle's bits."""
import numpy as np
import pytest

from test_gpu_splits import hub_graph

pytestmark = pytest.mark.gpu
FAIL_WAIT = 0


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
