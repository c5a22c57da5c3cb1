"""Rating against the oracle on both sides of its choices: tables by node (up to 8192 nodes with the
shared inbound counts, 16,384 without) or hashed, the counts kept or not by the level's largest
inbound count, and candidates whose whole contribution is zero."""
import numpy as np
import pytest

import axoncuda_b200 as ax
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("slack", [-200, -1, 0, None])
@pytest.mark.parametrize("nodes", [2048, 8192, 8196, 16384, 16388])
def test_rating_forms_match_oracle(ctx, nodes, slack):
    g = ax.gen_snn(4, nodes // 4, 90, 0.5, 300, 0.7, nodes)
    off, pins, nsrc = O.dedupe(g.off, g.pins, g.nsrc)
    rng = np.random.default_rng(nodes)
    w = np.where(rng.random(g.e) < 0.3, 0.0, rng.integers(1, 9, g.e) / 4.0).astype(np.float32)
    g = ax.Hypergraph(g.n, off, pins, nsrc, w)
    nin = O.touching(g.n, g.off, g.pins, g.nsrc)[2]
    delta = (1 << 31) - 1 if slack is None else 2 * int(nin.max()) + slack
    ns = rng.integers(1, 3, g.n).astype(np.uint32)
    pairs, scores = ctx.stage_rating(g, ns, 3, delta, 4)
    o_pairs, o_scores = O.rating(g.n, g.off, g.pins, g.nsrc, O.wfx(g.w), ns, 3, delta, 4)
    np.testing.assert_array_equal(pairs, o_pairs)
    np.testing.assert_array_equal(scores, o_scores)
    assert (pairs != 0xFFFFFFFF).any()


def hub_pair(nodes, nets, weight, hub_nets):
    """Nodes 0 and 1 joined by `nets` 2-pin nets of the given weight (node 0 their source); node 0 in
    `hub_nets` further nets of 128 pins. Sizes of 1 for the two and 3 for the rest: with a limit
    of 3 each of them has the other as its only candidate."""
    rng = np.random.default_rng(nets)
    pins = [np.array([0, 1], np.uint32)] * nets
    for _ in range(hub_nets):
        pins.append(np.concatenate([[2 + rng.integers(nodes - 2)], [0], 2 + rng.permutation(nodes - 2)[:126]]).astype(np.uint32))
    off, p, nsrc = O.dedupe(np.cumsum([0] + [len(x) for x in pins]).astype(np.uint64), np.concatenate(pins),
                            np.ones(len(pins), np.uint32))
    w = np.array([weight] * nets + [1.0] * hub_nets, np.float32)
    ns = np.full(nodes, 3, np.uint32)
    ns[:2] = 1
    return ax.Hypergraph(nodes, off, p, nsrc, w), ns


# Sums of the pair's contributions (weight * 2^17 each): 2^32, which wraps to zero, and on both sides of it.
# 12 and 30 nets: a block's tables; 80: a heavy node's.
@pytest.mark.parametrize("hub_nets", [12, 30, 80])
@pytest.mark.parametrize("binding", [False, True])
@pytest.mark.parametrize("nets,weight", [(4, 8192.0), (32, 1024.0), (8, 8192.0), (31, 1024.0), (33, 1024.0)])
def test_wrapped_scores_match_oracle(ctx, nets, weight, binding, hub_nets):
    g, ns = hub_pair(1500, nets, weight, hub_nets)
    nin = O.touching(g.n, g.off, g.pins, g.nsrc)[2]
    delta = 2 * int(nin.max()) - 1 if binding else (1 << 31) - 1
    pairs, scores = ctx.stage_rating(g, ns, 3, delta, 4)
    o_pairs, o_scores = O.rating(g.n, g.off, g.pins, g.nsrc, O.wfx(g.w), ns, 3, delta, 4)
    assert o_pairs[0] == 1 and o_pairs[4] == 0
    np.testing.assert_array_equal(pairs, o_pairs)
    np.testing.assert_array_equal(scores, o_scores)


@pytest.mark.parametrize("binding", [False, True])
@pytest.mark.parametrize("nodes", [2048, 8192, 16384])
def test_large_weights_match_oracle(ctx, nodes, binding):
    """Weights of zero and up to the fixed-point limit on hyperedges that repeat one another."""
    g = ax.gen_snn(4, nodes // 4, 40, 0.5, 120, 0.7, nodes)
    off, pins, nsrc = O.dedupe(g.off, g.pins, g.nsrc)
    lens = np.tile(np.diff(off.astype(np.int64)), 2)
    rng = np.random.default_rng(nodes)
    w = rng.choice([0.0, 1.0, 64.0, 8192.0, 16384.0], len(lens)).astype(np.float32)
    g = ax.Hypergraph(g.n, np.concatenate([[0], np.cumsum(lens)]).astype(np.uint64), np.tile(pins, 2), np.tile(nsrc, 2), w)
    nin = O.touching(g.n, g.off, g.pins, g.nsrc)[2]
    delta = 2 * int(nin.max()) - 1 if binding else (1 << 31) - 1
    ns = np.ones(g.n, np.uint32)
    pairs, scores = ctx.stage_rating(g, ns, 2, delta, 16)
    o_pairs, o_scores = O.rating(g.n, g.off, g.pins, g.nsrc, O.wfx(g.w), ns, 2, delta, 16)
    np.testing.assert_array_equal(pairs, o_pairs)
    np.testing.assert_array_equal(scores, o_scores)
