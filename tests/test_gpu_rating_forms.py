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
