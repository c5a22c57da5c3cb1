"""The kernel timer's bytes belong to the launches it times: each rating and k-way gains kernel counts its
own model over the nodes it was given, and nothing where another kernel took them."""
import numpy as np
import pytest

import axoncuda_b200 as ax
from oracle import oracle as O

pytestmark = pytest.mark.gpu
NO_LIMIT = 0x7FFFFFFF


def timed(ctx, kernel, call):
    ctx.profile_kernel(kernel)
    try:
        ctx.profile_read()
        out = call()
        return ctx.profile_read(), out
    finally:
        ctx.profile_kernel(None)


def dense_network(nodes, fanout, seed):
    g = ax.gen_snn(4, nodes // 4, fanout, 0.0, 0, 1.0, seed)
    off, pins, nsrc = O.dedupe(g.off, g.pins, g.nsrc)
    return ax.Hypergraph(g.n, off, pins, nsrc, np.ones(g.e, np.float32))


# up to 16,384 nodes the block tiers' tables are by node (k_rate_direct), above they are hashed (k_rate_block)
@pytest.mark.parametrize("nodes,kernel,other", [(2048, "k_rate_direct", "k_rate_block"),
                                                (17000, "k_rate_block", "k_rate_direct")])
def test_rating_bytes_count_the_launched_kernel(ctx, nodes, kernel, other):
    g = dense_network(nodes, 60, nodes)
    length = np.diff(g.off.astype(np.int64))
    visits = np.bincount(g.pins, weights=np.repeat(np.where(length <= 128, length, 0), length), minlength=g.n)
    assert visits.max() <= 8192 and (visits > 2048).any()  # no heavy node; tables beyond the first try's
    listed = visits > 256  # the others are a warp's
    kt, _ = timed(ctx, kernel, lambda: ctx.stage_rating(g, np.ones(g.n, np.uint32), 3, NO_LIMIT, 4))
    assert kt.launches > 0
    assert kt.bytes == 4 * int(visits[listed].sum()) + 8 * 4 * int(listed.sum())
    kt, _ = timed(ctx, other, lambda: ctx.stage_rating(g, np.ones(g.n, np.uint32), 3, NO_LIMIT, 4))
    assert (kt.launches, kt.bytes) == (0, 0)


# equal weights, more than 8 partitions and dense: bit planes; else a group of lanes per node. Levels of at
# most 1024 nodes take a block per node.
@pytest.mark.parametrize("nodes,fanout,K,kernel", [(4000, 80, 40, "k_kway_planes"), (4000, 80, 8, "k_kway_gain"),
                                                   (4000, 10, 40, "k_kway_gain"), (800, 80, 40, "k_kway_planes_block"),
                                                   (800, 80, 8, "k_kway_gain_block")])
def test_kway_bytes_count_the_launched_kernel(ctx, nodes, fanout, K, kernel):
    g = dense_network(nodes, fanout, K)
    part = np.random.default_rng(K).integers(0, K, g.n).astype(np.uint32)

    def refine():
        return ctx.stage_refine(g, part, K, np.ones(g.n, np.uint32), 2 * g.n // K + 8, NO_LIMIT, False, 2, 3)

    for name in ("k_kway_gain", "k_kway_gain_block", "k_kway_planes", "k_kway_planes_block"):
        kt, (_, ran) = timed(ctx, name, refine)
        if name != kernel:
            assert (kt.launches, kt.bytes) == (0, 0), name
            continue
        words = 1 if K <= 32 else 2
        assert kt.launches == ran
        assert kt.bytes == ran * ((8 + 4 * words) * g.P + 16 * g.n)
