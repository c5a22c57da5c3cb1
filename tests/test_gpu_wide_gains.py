"""Gains above 256 partitions against the oracle, on both sides of every table choice: sums by partition
(one word, or two where a node's weights pass 2^32) and bit planes up to 4096 partitions, the
sampled rule's tables by partition and hashed, with equal and unequal weights, and its exact pass
from bitmaps and hash tables. Sorts and scans of the pipeline at their tile bounds through the
incidence lists."""
import numpy as np
import pytest

import axoncuda_b200 as ax
from oracle import oracle as O
from test_gpu_parity import census_entries_per_node

pytestmark = pytest.mark.gpu


def weigh(g, weights, seed):
    rng = np.random.default_rng(seed)
    g.w = {"unit": np.ones(g.e), "third": np.full(g.e, 1 / 3), "quarters": rng.integers(0, 64, g.e) / 4.0,
           "heavy": rng.integers(1, 16000, g.e)}[weights].astype(np.float32)
    return g


def check_gains(ctx, g, K, omega, delta, encourage, discount, seed):
    rng = np.random.default_rng(seed)
    part = rng.integers(0, K, g.n).astype(np.uint32)
    ns = rng.integers(1, 3, g.n).astype(np.uint32)
    tgt, gain = ctx.stage_gains(g, part, K, ns, omega, delta, encourage, discount)
    o_tgt, o_gain = O.gains(g.n, g.off, g.pins, g.nsrc, O.wfx(g.w), ns, part, K, omega, delta, encourage, discount)
    np.testing.assert_array_equal(tgt, o_tgt)
    np.testing.assert_array_equal(gain, o_gain)
    assert (tgt != 0xFFFFFFFF).any()
    return part


# dense hyperedges: bit planes with equal weights at every lane count (16 to 128 words), tables
# otherwise; sparse ones: tables only
@pytest.mark.parametrize("weights", ["unit", "third", "quarters", "heavy"])
@pytest.mark.parametrize("K", [257, 512, 513, 1500, 2500, 4096])
def test_gains_by_partition_match_oracle(ctx, K, weights):
    g = weigh(ax.gen_snn(4, 700, 150, 0.7, 600, 0.7, K), weights, K)
    check_gains(ctx, g, K, 1 << 20 if K % 2 else 2 * g.n // K + 4, 500, 1, 1, K)


@pytest.mark.parametrize("weights", ["unit", "heavy"])
@pytest.mark.parametrize("K", [300, 3000])
def test_gains_of_sparse_hyperedges_match_oracle(ctx, K, weights):
    g = weigh(ax.gen_circuit(3000, 90000, 2, 40, 2.2, 0.5, 0.05, 7), weights, 7)
    check_gains(ctx, g, K, 1 << 20, 1 << 20, 0, 1, K)


# 12,288 / 12,289 and 16,384 / 16,385 partitions: the last tables by partition, and the last bitmaps
@pytest.mark.parametrize("K,weights,delta", [(5000, "quarters", 1 << 20), (5001, "heavy", 120), (12288, "quarters", 100),
                                             (12289, "quarters", 1 << 20), (16384, "unit", 110), (16385, "unit", 1 << 20),
                                             (16385, "heavy", 100), (40000, "third", 100)])
def test_sampled_gains_by_table_match_oracle(ctx, K, weights, delta):
    g = weigh(ax.gen_snn(4, 1200, 90, 0.5, 400, 0.7, 41), weights, K)
    part = check_gains(ctx, g, K, 5, delta, 1, 2, K)
    assert (census_entries_per_node(g, part) > 4096).any()


@pytest.mark.parametrize("pins", [1, 1023, 1024, 8192, 8193, 12289, 524288, 524289, 700001])
def test_incidence_lists_at_sort_tile_bounds(ctx, pins):
    """One hyperedge per pin pair, so that the sort holds exactly `pins` elements."""
    rng = np.random.default_rng(pins)
    e = (pins + 1) // 2
    off = np.minimum(np.arange(e + 1) * 2, pins).astype(np.uint64)
    n = 3 * pins + 5
    p = rng.choice(n, pins, replace=False).astype(np.uint32)
    g = ax.Hypergraph(n, off, p, np.minimum(1, np.diff(off.astype(np.int64))).astype(np.uint32), np.ones(e, np.float32))
    _, _, _, toff, touch, nin = ctx.stage_construct(g)
    o_toff, o_touch, o_nin = O.touching(g.n, g.off, g.pins, g.nsrc)
    np.testing.assert_array_equal(toff, o_toff)
    np.testing.assert_array_equal(touch, o_touch)
    np.testing.assert_array_equal(nin, o_nin)


@pytest.mark.parametrize("K,omega,delta", [(4097, 3, 1 << 20), (5000, 4, 200), (8000, 3, 110), (12289, 5, 110),
                                           (16385, 2, 1 << 20)])
def test_sampled_candidate_bands_match_oracle(ctx, K, omega, delta):
    g = weigh(ax.gen_snn(4, 1200, 120, 0.5, 400, 0.7, K), "unit", K)
    check_gains(ctx, g, K, omega, delta, 1, 2, K)
