"""Failure detection without a GPU fault: the device waits of this library are bounded, and a wait
that runs out sets the context's status word, returns, and is reported by the call that made it.
The wait here polls a tile flag that nothing ever publishes."""
import os

import numpy as np
import pytest

import axoncuda_b200 as ax
from conftest import GOLDEN
from oracle import oracle as O

pytestmark = pytest.mark.gpu
AXC_EINTERNAL, AXC_EOVERFLOW = 10, 11
DEV_SPIN_LIMIT = 3


@pytest.mark.parametrize("spin_limit", [1, 1000, 100000])
def test_bounded_wait_gives_up_and_the_context_recovers(ctx, spin_limit):
    rc = ax.lib().axc_selftest_bounded_wait(ctx._h, spin_limit)
    assert rc == AXC_EINTERNAL
    assert f"status word = {DEV_SPIN_LIMIT}" in ax.lib().axc_last_error(ctx._h).decode()
    # the status word was cleared and the context still partitions correctly
    g = ax.read(os.path.join(GOLDEN, "snn_4x64.snn"))
    p = ax.params_incc(16, 64, 1 << 20, cnc=4, rfr=8)
    part, st = ctx.partition(g, p)
    ref, K, _, _ = O.partition(g.n, g.off, g.pins, g.nsrc, g.w, 0, omega=16, delta=64, max_parts=1 << 20,
                               cnc=4, rfr=8, ipm=1)
    np.testing.assert_array_equal(part, ref)
    assert st.valid == 1


def test_bounded_wait_rejects_a_zero_limit(ctx):
    assert ax.lib().axc_selftest_bounded_wait(ctx._h, 0) == 1  # AXC_EINVAL


@pytest.mark.parametrize("hyperedges", [0, 1, 300])
def test_evaluate_refuses_a_partition_id_without_a_count(ctx, hyperedges):
    """Ids up to 2^32 - 2 have a partition count; 2^32 - 1 is refused on the host, before any kernel would
    index by it."""
    n = 400
    g = ax.Hypergraph(n, np.arange(hyperedges + 1, dtype=np.uint64) * n, np.tile(np.arange(n, dtype=np.uint32), hyperedges),
                      np.ones(hyperedges, np.uint32), np.ones(hyperedges, np.float32))
    part = np.zeros(n, np.uint32)
    part[7] = 0xFFFFFFFF
    with pytest.raises(ax.AxcError) as err:
        ctx.evaluate(g, ax.params_kway(2, 0.1), part)
    assert err.value.code == AXC_EOVERFLOW
    part[7] = 1
    st = ctx.evaluate(g, ax.params_kway(2, 0.1), part)
    assert st.num_parts == 2 and st.connectivity == hyperedges
