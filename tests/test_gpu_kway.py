"""K-way refinement through the per-hyperedge records and the per-copy ranking, and the cascade of
short hyperedges mover by mover, against the oracle: whole levels (axc_stage_refine) at the partition
counts where the records and the lane groups change width, on levels ranked by one block (at most
8192 nodes) and larger ones, with hyperedges on both sides of every length limit, hub nodes and
weights; and whole partitions, whose multi-start refines several copies at once."""
import numpy as np
import pytest

import axoncuda_b200 as ax
from oracle import oracle as O

pytestmark = pytest.mark.gpu
NO_LIMIT = 0x7FFFFFFF


def netlist(n, weights, seed, long_nets=True):
    """Short local nets, nets of 8, 9, 64, 65, 128, 129, 1024, 1025 and 5000 pins (the lengths where
    kernels change), and a hub node on a third of the short nets."""
    rng = np.random.default_rng(seed)
    g = ax.gen_circuit(n, n + n // 10, 2, 64, 2.5, 0.9, 0.02, seed)
    nets = [g.pins[int(a):int(b)] for a, b in zip(g.off[:-1], g.off[1:])]
    nets = [np.append(p, np.uint32(7)) if i % 3 == 0 and 7 not in p else p for i, p in enumerate(nets)]
    if long_nets:
        for size in sorted({min(n, s) for s in (1, 8, 9, 64, 65, 128, 129, 1024, 1025, 5000)}):
            nets += [rng.choice(n, size, replace=False).astype(np.uint32) for _ in range(3)]
    off = np.concatenate([[0], np.cumsum([len(p) for p in nets])]).astype(np.uint64)
    w = {"unit": np.ones(len(nets)), "quarters": rng.integers(0, 64, len(nets)) / 4.0,
         "heavy": rng.integers(1, 16000, len(nets))}[weights]
    nsrc = rng.integers(0, 2, len(nets)).astype(np.uint32)
    return ax.Hypergraph(n, off, np.concatenate(nets), nsrc, w.astype(np.float32))


def check_refine(ctx, g, K, encourage, omega, delta, rounds, seed=3):
    rng = np.random.default_rng(K)
    part = rng.integers(0, K, g.n).astype(np.uint32)
    ns = rng.integers(1, 4, g.n).astype(np.uint32)
    out, ran = ctx.stage_refine(g, part, K, ns, omega, delta, encourage, rounds, seed)
    o = O.refine(g.n, g.off, g.pins, g.nsrc, O.wfx(g.w), ns, part, K, omega, delta, encourage, rounds, seed)
    np.testing.assert_array_equal(out, o)
    assert 1 <= ran <= rounds and (out != part).any()


@pytest.mark.parametrize("n,weights", [(900, "unit"), (3000, "quarters"), (8192, "unit"), (9000, "heavy")])
@pytest.mark.parametrize("K", [2, 4, 5, 9, 17, 33, 65, 129, 256, 257])
def test_kway_levels_match_oracle(ctx, n, weights, K):
    g = netlist(n, weights, n)
    check_refine(ctx, g, K, False, int(2.2 * n / K) + 3, NO_LIMIT, 3)


@pytest.mark.parametrize("encourage,K,delta", [(True, 40, 900), (True, 400, 300), (True, 400, NO_LIMIT),
                                               (False, 300, 1 << 20)])
@pytest.mark.parametrize("n", [2000, 9000])
def test_cascade_by_movers_matches_oracle(ctx, n, encourage, K, delta):
    """Inbound-constrained and hashed levels: the same short and long hyperedges in one level."""
    g = netlist(n, "quarters", n + 1)
    check_refine(ctx, g, K, encourage, int(2.2 * n / K) + 8, delta * n // 1000 if delta < 1000 else delta, 3)


@pytest.mark.parametrize("k,weights", [(1, "unit"), (3, "quarters"), (40, "unit"), (100, "quarters"), (200, "unit"),
                                       (300, "quarters")])
def test_multistart_matches_oracle(ctx, k, weights):
    g = netlist(2500, weights, 11)
    p = ax.params_kway(k, 0.1, cnc=4, rfr=4)
    part, _ = ctx.partition(g, p)
    o, _, _, _ = O.partition(g.n, g.off, g.pins, g.nsrc, g.w, 1, k=k, eps=p.eps, cnc=4, rfr=4)
    np.testing.assert_array_equal(part, o)


def test_multistart_without_moves(ctx):
    """Hyperedges of zero weight propose no move in any copy."""
    g = netlist(600, "unit", 5, long_nets=False)
    g.w[:] = 0
    p = ax.params_kway(4, 0.1, cnc=4, rfr=4)
    part, _ = ctx.partition(g, p)
    o, _, _, _ = O.partition(g.n, g.off, g.pins, g.nsrc, g.w, 1, k=4, eps=p.eps, cnc=4, rfr=4)
    np.testing.assert_array_equal(part, o)


def dense_network(n, hubs):
    """Equal weights and at least 48 incidences per node on average, where gains count in bit planes; `hubs`
    nodes are in two hyperedges of three."""
    g = ax.gen_snn(4, n // 4, 90, 0.3, 200, 0.7, n)
    rng = np.random.default_rng(n)
    nets = []
    for a, b in zip(g.off[:-1], g.off[1:]):
        p = g.pins[int(a):int(b)]
        nets.append(np.concatenate([p, [v for v in range(hubs) if v not in p and rng.random() < 0.67]]).astype(np.uint32))
    off = np.concatenate([[0], np.cumsum([len(p) for p in nets])]).astype(np.uint64)
    off, pins, nsrc = O.dedupe(off, np.concatenate(nets), g.nsrc)
    g = ax.Hypergraph(g.n, off, pins, nsrc, np.full(g.e, 1 / 3, np.float32))
    assert g.P >= 48 * g.n
    return g


# one to eight words of partitions; a block per node (at most 1024 nodes), and a warp per node with the
# hubs' more than 1024 incidences in blocks
@pytest.mark.parametrize("n,hubs", [(800, 0), (3200, 3)])
@pytest.mark.parametrize("K", [8, 9, 32, 33, 64, 65, 128, 129, 256])
def test_kway_planes_match_oracle(ctx, n, hubs, K):
    g = dense_network(n, hubs)
    deg = np.bincount(g.pins, minlength=g.n)
    assert (deg > 1024).sum() == hubs
    check_refine(ctx, g, K, False, int(2.2 * n / K) + 3, NO_LIMIT, 3)


@pytest.mark.parametrize("hub_degree", [131055, 131056, 131063, 131064])
def test_kway_planes_at_their_capacity_match_oracle(ctx, hub_degree):
    """A node of 2^17 incidences: the last whose eighth a block's counters hold, and the first that sums
    by partition instead. All its neighbours are in one partition, where the counters reach their limit."""
    n, K = 2000, 40
    rng = np.random.default_rng(hub_degree)
    pins = np.zeros((hub_degree, 2), np.uint32)
    pins[:, 1] = 1 + rng.integers(0, n // 2, hub_degree)
    g = ax.Hypergraph(n, np.arange(hub_degree + 1, dtype=np.uint64) * 2, pins.ravel(), np.ones(hub_degree, np.uint32),
                      np.ones(hub_degree, np.float32))
    part = np.where(np.arange(n) <= n // 2, 5, rng.integers(0, K, n)).astype(np.uint32)
    part[0] = 7
    ns = np.ones(n, np.uint32)
    out, ran = ctx.stage_refine(g, part, K, ns, n, NO_LIMIT, False, 3, 3)
    o = O.refine(g.n, g.off, g.pins, g.nsrc, O.wfx(g.w), ns, part, K, n, NO_LIMIT, False, 3, 3)
    np.testing.assert_array_equal(out, o)
    assert out[0] == 5
