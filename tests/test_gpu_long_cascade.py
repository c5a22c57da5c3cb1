"""Rounds on levels of long hyperedges against the oracle: movers on both sides of every kernel's limit
(512 or 64 for a warp, 2048, 4096 or 1024 for the wide kernel, the block kernel's 2048 and beyond),
with partitions by index and hashed, few (sweeps) and many (events)."""
import numpy as np
import pytest

import axoncuda_b200 as ax
from oracle import oracle as O

pytestmark = pytest.mark.gpu

LENGTHS = [129, 200, 257, 500, 513, 700, 1025, 1500, 2049, 3000, 4097, 4990, 5990]


def with_long_hyperedges(seed, n=6000, e=9000):
    """A netlist of n nodes, whose nets make most nodes movers, and long hyperedges over it."""
    g = ax.gen_circuit(n, e, 2, 40, 2.3, 0.9, 0.05, seed)
    rng = np.random.default_rng(seed)
    off, pins, nsrc = list(g.off[:-1]), [g.pins], list(g.nsrc)
    at = int(g.off[-1])
    for length in LENGTHS * 2:
        off.append(at)
        m = int(rng.integers(1, 4))
        p = rng.choice(g.n, length, replace=False).astype(g.pins.dtype)
        p[:m].sort()
        p[m:].sort()
        pins.append(p)
        nsrc.append(m)
        at += length
    off.append(at)
    w = np.concatenate([g.w, rng.integers(1, 9, 2 * len(LENGTHS)) / 2.0]).astype(np.float32)
    return ax.Hypergraph(g.n, np.asarray(off, np.uint64), np.concatenate(pins), np.asarray(nsrc, np.uint32), w)


# 65,536 and 65,537 partitions: the last whose targets fit a node's state, and the first beyond
@pytest.mark.parametrize("encourage,K,delta", [(False, 3, 1 << 20), (False, 40, 1 << 20), (False, 250, 1 << 20),
                                               (True, 4, 9000), (True, 200, 1500), (True, 256, 1500), (True, 257, 1500),
                                               (True, 1024, 400), (True, 1025, 400), (True, 1500, 1 << 20),
                                               (True, 65536, 400), (True, 65537, 400)])
def test_rounds_of_long_hyperedges_match_oracle(ctx, encourage, K, delta):
    g = with_long_hyperedges(K) if K < 65536 else with_long_hyperedges(K, 70000, 80000)
    rng = np.random.default_rng(K)
    part = rng.integers(0, K, g.n).astype(np.uint32)
    ns = rng.integers(1, 3, g.n).astype(np.uint32)
    omega, rounds = 3 * g.n // K + 8, 3 if K < 65536 else 1
    out, ran = ctx.stage_refine(g, part, K, ns, omega, delta, encourage, rounds, 3)
    o = O.refine(g.n, g.off, g.pins, g.nsrc, O.wfx(g.w), ns, part, K, omega, delta, encourage, rounds, 3)
    np.testing.assert_array_equal(out, o)
    assert (out != part).any()
