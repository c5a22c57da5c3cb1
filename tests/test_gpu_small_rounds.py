"""The rounds of small constrained levels in one launch against the oracle, on both sides of what takes
a level there (256 partitions, 8192 nodes, hyperedges of 128 pins); and the dedupe and incidence lists of
hyperedges on both sides of a warp's packing and tables, with duplicate pins."""
import numpy as np
import pytest

import axoncuda_b200 as ax
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nodes,fanout,K", [(32, 5, 2), (1024, 20, 255), (2048, 127, 40), (2048, 128, 40),
                                            (8192, 20, 256), (8192, 20, 257), (8196, 20, 256)])
@pytest.mark.parametrize("rounds", [1, 5])
def test_small_level_rounds_match_oracle(ctx, nodes, fanout, K, rounds):
    g = ax.gen_snn(4, nodes // 4, fanout, 0.0, fanout, 0.7, nodes + K)
    off, pins, nsrc = O.dedupe(g.off, g.pins, g.nsrc)
    g = ax.Hypergraph(g.n, off, pins, nsrc, g.w)
    rng = np.random.default_rng(K)
    part = rng.integers(0, K, g.n).astype(np.uint32)
    ns = rng.integers(1, 3, g.n).astype(np.uint32)
    omega, delta = 2 * g.n // K + 8, 6 * g.n * fanout // K + 200
    out, ran = ctx.stage_refine(g, part, K, ns, omega, delta, True, rounds, 3)
    o = O.refine(g.n, g.off, g.pins, g.nsrc, O.wfx(g.w), ns, part, K, omega, delta, True, rounds, 3)
    np.testing.assert_array_equal(out, o)
    assert 1 <= ran <= rounds and (out != part).any()


@pytest.mark.parametrize("lengths", [[1, 2, 3], [31, 32, 33], [1, 32, 64, 2], [16, 16, 5, 300], [255, 256, 257],
                                     [2047, 2048, 2049, 3], [1, 4, 9000, 2]])
@pytest.mark.parametrize("count", [1, 33, 4000])
def test_construct_of_packed_hyperedges_matches_oracle(ctx, lengths, count):
    if count * max(lengths) > 2_000_000:
        count = 33
    rng = np.random.default_rng(count + lengths[0])
    n = 50
    lens = np.resize(lengths, count)
    off = np.concatenate([[0], np.cumsum(lens)]).astype(np.uint64)
    pins = rng.integers(0, n if max(lengths) < 256 else 6000, int(off[-1])).astype(np.uint32)
    nsrc = np.minimum(rng.integers(1, 4, count), lens).astype(np.uint32)
    g = ax.Hypergraph(int(pins.max()) + 1, off, pins, nsrc, np.ones(count, np.float32))
    out = ctx.stage_construct(g)
    o_off, o_pins, o_nsrc = O.dedupe(g.off, g.pins, g.nsrc)
    expect = (o_off, o_pins, o_nsrc) + tuple(O.touching(g.n, o_off, o_pins, o_nsrc))
    for a, b in zip(out, expect):
        np.testing.assert_array_equal(a, b)
