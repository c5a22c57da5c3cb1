"""Levels whose largest nodes have far more incidences than the mean, against the oracle: hubs on both sides
of what a group of lanes, a warp or a block takes, at mean degrees that give a node 4, 8 and 32 lanes."""
import numpy as np
import pytest

import axoncuda_b200 as ax
from oracle import oracle as O

pytestmark = pytest.mark.gpu
HUBS = [256, 257, 512, 513, 2048, 2049, 4096, 4097, 8192, 8193, 20000]


def hub_graph(n, mean, weighted):
    """Node i is in HUBS[i] 2-pin nets; nets of 2 to 12 pins over all nodes up to the mean degree."""
    rng = np.random.default_rng(n)
    nets = [np.array([h, v], np.uint32) for h, d in enumerate(HUBS) for v in len(HUBS) + rng.integers(0, n - len(HUBS), d)]
    P = 2 * len(nets)
    while P < mean * n:
        p = np.unique(len(HUBS) + rng.integers(0, n - len(HUBS), rng.integers(2, 13))).astype(np.uint32)
        nets.append(rng.permutation(p))
        P += len(p)
    nets = [nets[i] for i in rng.permutation(len(nets))]
    off = np.concatenate([[0], np.cumsum([len(p) for p in nets])]).astype(np.uint64)
    w = rng.integers(1, 16000, len(nets)) if weighted else np.ones(len(nets))
    return ax.Hypergraph(n, off, np.concatenate(nets), np.ones(len(nets), np.uint32), w.astype(np.float32))


@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("n,mean", [(20000, 5), (10000, 16), (2500, 60)])
@pytest.mark.parametrize("K", [40, 300, 5000])
def test_gains_of_hubs_match_oracle(ctx, n, mean, K, weighted):
    g = hub_graph(n, mean, weighted)
    rng = np.random.default_rng(K)
    part = rng.integers(0, K, g.n).astype(np.uint32)
    ns = rng.integers(1, 3, g.n).astype(np.uint32)
    omega, delta = 3 * g.n // K + 8, 1 << 20
    tgt, gain = ctx.stage_gains(g, part, K, ns, omega, delta, True, 1)
    o_tgt, o_gain = O.gains(g.n, g.off, g.pins, g.nsrc, O.wfx(g.w), ns, part, K, omega, delta, True, 1)
    np.testing.assert_array_equal(tgt, o_tgt)
    np.testing.assert_array_equal(gain, o_gain)
    assert (tgt != 0xFFFFFFFF).any()


@pytest.mark.parametrize("n,mean", [(20000, 5), (6000, 16), (2500, 60)])
@pytest.mark.parametrize("encourage,K", [(True, 2), (True, 40), (True, 300), (False, 3), (False, 40)])
def test_rounds_with_hubs_match_oracle(ctx, n, mean, encourage, K):
    g = hub_graph(n, mean, False)
    rng = np.random.default_rng(K)
    part = rng.integers(0, K, g.n).astype(np.uint32)
    ns = rng.integers(1, 3, g.n).astype(np.uint32)
    omega, delta = 3 * g.n // K + 8, (g.P if encourage else 0x7FFFFFFF)
    out, ran = ctx.stage_refine(g, part, K, ns, omega, delta, encourage, 3, 3)
    o = O.refine(g.n, g.off, g.pins, g.nsrc, O.wfx(g.w), ns, part, K, omega, delta, encourage, 3, 3)
    np.testing.assert_array_equal(out, o)
    assert (out != part).any()
