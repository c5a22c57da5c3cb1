"""The work that users have this partitioner do, as cases that can be timed and compared.

A case is one call of a public entry point on a seeded synthetic hypergraph: `partition` (host
buffers in and out, what the command line does), `partition_device` (the hypergraph and the result
stay in device memory), `batch` (many small jobs through the executor's lanes) or `evaluate` (the
metrics and the validity of a given partition). The hypergraphs are those of the benchmark, the
tests, the batched and the serving workloads: circuit netlists (local nets of 2 to 64 pins, no
sources) and layered spiking networks (one source per hyperedge, fixed or lognormal fan-out), at
their sizes and smaller, odd ones among them. The results are whole numbers and must stay the same.
"""
import ctypes as C
import math
import random

import numpy as np
import torch

import axoncuda_b200 as ax

ARENA_BYTES = 12 << 30
LANES = 16
NET_PINS = 4.02   # mean pins of a net: sizes 2..64 with P(s) ~ s^-2.5
JOB_SEEDS = 1000  # a batch's jobs take consecutive generator seeds from seed * JOB_SEEDS

_ctx = None


def context():
    """The one context of this process, as a program keeps it for all its calls."""
    global _ctx
    if _ctx is None:
        _ctx = ax.Context(0, ARENA_BYTES)
        _ctx.serve_configure(LANES, 24 << 30)
    return _ctx


def circuit(nodes, mode, call="partition", weighted=False, **params):
    return dict(call=call, net="circuit", nodes=nodes, nets=nodes + nodes // 10, mode=mode, weighted=weighted, **params)


def snn(layers, width, fanout, mode, sigma=0.0, p_next=1.0, call="partition", weighted=False, **params):
    return dict(call=call, net="snn", layers=layers, width=width, fanout=fanout, sigma=sigma, p_next=p_next, mode=mode,
                weighted=weighted, **params)


def kway(k, cnc=4, rfr=16):
    return dict(k=k, eps=0.03, cnc=cnc, rfr=rfr)


def incc(omega, delta, cnc=4, rfr=16, ipm=1):
    return dict(omega=omega, delta=delta, max_parts=1 << 20, cnc=cnc, rfr=rfr, ipm=ipm)


def listed():
    cases = {
        # the smallest call: a tool that partitions one small network and waits for the answer
        "snn_4x64_incc": snn(4, 64, 8, "incc", **incc(16, 64, rfr=8)),
        # a mid-size netlist with net weights and the command line's default of 16 candidates
        "circuit_21k_k8_weighted": circuit(21013, "kway", weighted=True, **kway(8, cnc=16)),
        # the benchmark's layered network on a small neuromorphic target
        "snn_8x512_incc": snn(8, 512, 64, "incc", **incc(128, 1024)),
        # the benchmark's netlist: its line, the same from device memory in more parts
        "circuit_200k_k2": circuit(200000, "kway", **kway(2)),
        "circuit_200k_k64": circuit(200000, "kway", call="partition_device", **kway(64)),
        # a serving request of the inbound-constrained kind
        "circuit_120k_incc": circuit(120007, "incc", **incc(256, 2048)),
        # the large layered network's generator at a hundredth and a tenth of its neurons
        "snn_20x500_incc": snn(20, 500, 256, "incc", sigma=0.8, p_next=0.7, **incc(1024, 4096)),
        "snn_20x5000_incc": snn(20, 5000, 256, "incc", sigma=0.8, p_next=0.7, **incc(1024, 4096)),
        "snn_20x5000_k128": snn(20, 5000, 256, "kway", sigma=0.8, p_next=0.7, **kway(128)),
        # a large netlist into a few parts
        "circuit_1m_k16": circuit(1000003, "kway", **kway(16)),
        # the batched workload: netlists and layered networks of uneven size, half and half
        "batch_24": dict(call="batch", jobs=24, nodes_min=1000, nodes_max=30000, kinds_seed=5),
        # grading a partition of a large netlist
        "evaluate_1m_k64": circuit(1000003, "kway", call="evaluate", weighted=True, **kway(64)),
    }
    return [dict(case, name=name) for name, case in cases.items()]


def log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["circuit_kway", "circuit_kway", "circuit_incc", "snn_incc", "snn_incc_lognormal",
                       "snn_kway", "batch", "evaluate"])
    weighted = rng.random() < 0.3
    cnc = rng.choice([4, 4, 16])
    if kind == "circuit_kway":
        call = rng.choice(["partition", "partition_device"])
        k = rng.choice([2, 3, 8, 16, 32, 64])
        nodes = log_int(rng, 1500, 800000 if k <= 16 else 180000)
        return circuit(nodes, "kway", call=call, weighted=weighted, **kway(k, cnc=cnc))
    if kind == "circuit_incc":
        return circuit(log_int(rng, 1500, 110000), "incc", weighted=weighted,
                       **incc(rng.choice([128, 256, 1024]), rng.choice([1024, 2048, 4096]), cnc=cnc))
    if kind == "snn_incc":
        return snn(rng.randint(3, 10), log_int(rng, 40, 900), rng.randint(8, 64), "incc", weighted=weighted,
                   **incc(rng.choice([64, 128, 256]), rng.choice([512, 1024, 2048]), cnc=cnc, ipm=rng.randint(0, 1)))
    if kind == "snn_incc_lognormal":
        return snn(rng.randint(5, 20), log_int(rng, 80, 450), 256, "incc", sigma=0.8, p_next=0.7, weighted=weighted,
                   **incc(1024, 4096))
    if kind == "snn_kway":
        return snn(rng.randint(5, 20), log_int(rng, 100, 4500), 256, "kway", sigma=0.8, p_next=0.7, weighted=weighted,
                   **kway(rng.choice([2, 8, 32, 128])))
    if kind == "batch":
        return dict(call="batch", jobs=rng.randint(4, 20), nodes_min=1000, nodes_max=log_int(rng, 4000, 30000),
                    kinds_seed=rng.randrange(1 << 20))
    return circuit(log_int(rng, 2000, 900000), "kway", call="evaluate", weighted=weighted, **kway(rng.choice([2, 16, 64, 300])))


def hypergraph(case, seed):
    if case["net"] == "circuit":
        g = ax.gen_circuit(case["nodes"], case["nets"], 2, 64, 2.5, 0.9, 0.02, seed)
    else:
        g = ax.gen_snn(case["layers"], case["width"], case["fanout"], case["sigma"], 2048, case["p_next"], seed)
    if case["weighted"]:
        rng = np.random.default_rng(seed)
        g.w = (rng.integers(1, 65, g.e) / 4.0).astype(np.float32)
    return g


def parameters(case):
    if case["mode"] == "kway":
        return ax.params_kway(case["k"], case["eps"], cnc=case["cnc"], rfr=case["rfr"])
    return ax.params_incc(case["omega"], case["delta"], case["max_parts"], cnc=case["cnc"], rfr=case["rfr"],
                          ipm=case["ipm"])


def batch_cases(case):
    """The jobs of a batch: netlists and layered networks in turn, k from {2, 8, 32}."""
    rng = random.Random(case["kinds_seed"])
    jobs = []
    for i in range(case["jobs"]):
        nodes = log_int(rng, case["nodes_min"], case["nodes_max"])
        p = kway(rng.choice([2, 8, 32]))
        if i % 2 == 0:
            jobs.append(circuit(nodes, "kway", **p))
        else:
            jobs.append(snn(8, max(nodes // 8, 65), 64, "kway", **p))
    return jobs


def prepare(case, seed):
    ctx = context()
    if case["call"] == "batch":
        jobs = [(hypergraph(c, seed * JOB_SEEDS + i), parameters(c)) for i, c in enumerate(batch_cases(case))]
        return dict(case=case, ctx=ctx, jobs=jobs)
    g, p = hypergraph(case, seed), parameters(case)
    state = dict(case=case, ctx=ctx, g=g, p=p)
    if case["call"] == "evaluate":
        # runs of neighbouring ids with some nodes elsewhere, as partitions of local netlists are
        rng = np.random.default_rng(seed + 1)
        part = (np.arange(g.n, dtype=np.uint64) * case["k"] // g.n).astype(np.uint32)
        moved = rng.random(g.n) < 0.1
        part[moved] = rng.integers(0, case["k"], int(moved.sum()))
        state["part"] = part
    if case["call"] == "partition_device":
        def on_gpu(a, like):
            return torch.from_numpy(a.view(like)).cuda()

        dev = dict(off=on_gpu(g.off, np.int64), pins=on_gpu(g.pins, np.int32), nsrc=on_gpu(g.nsrc, np.int32),
                   w=torch.from_numpy(g.w).cuda(), part=torch.empty(g.n, dtype=torch.int32, device="cuda"))
        torch.cuda.synchronize()
        state.update(dev=dev, hg=ax.HGraph(
            g.n, g.e, C.cast(dev["off"].data_ptr(), C.POINTER(C.c_uint64)),
            C.cast(dev["pins"].data_ptr(), C.POINTER(C.c_uint32)),
            C.cast(dev["nsrc"].data_ptr(), C.POINTER(C.c_uint32)),
            C.cast(dev["w"].data_ptr(), C.POINTER(C.c_float)), None))
    return state


def metrics(st):
    """What the call reports of a partition, in whole numbers."""
    return np.array([st.num_parts, st.connectivity_fx, st.cutnet_fx, st.soed_fx, st.max_part_size,
                     st.max_part_inbound, st.valid], dtype=np.int64)


def run(state):
    ctx, call = state["ctx"], state["case"]["call"]
    if call == "batch":
        return [(part.view(np.int32), metrics(st)) for part, st in ctx.partition_batch(state["jobs"])]
    if call == "evaluate":
        return metrics(ctx.evaluate(state["g"], state["p"], state["part"]))
    if call == "partition_device":
        part, st = state["dev"]["part"], ax.Stats()
        rc = ax.lib().axc_partition_device(ctx._h, C.byref(state["hg"]), C.byref(state["p"]),
                                           C.cast(part.data_ptr(), C.POINTER(C.c_uint32)), C.byref(st))
        if rc:
            raise ax.AxcError(rc, "axc_partition_device")
        return part, np.array([st.num_parts], dtype=np.int64)
    part, st = ctx.partition(state["g"], state["p"])
    return part.view(np.int32), metrics(st)


def one_work(case):
    """Bytes of a call: offsets, pins, source counts and weights read once, the partition written once."""
    if case["net"] == "circuit":
        nodes, edges = case["nodes"], case["nets"]
        pins = edges * NET_PINS
    else:
        nodes, edges = case["layers"] * case["width"], (case["layers"] - 1) * case["width"]
        mean = case["fanout"] * math.exp(case["sigma"] ** 2 / 2)
        pins = edges * (1 + min(mean, 0.9 * case["width"] * (case["layers"] - 1)))
    return 8 * (edges + 1) + 4 * pins + 8 * edges + 4 * nodes


def work(case):
    """The bytes alone: all arithmetic is on integers, a few operations per pin and pass."""
    jobs = batch_cases(case) if case["call"] == "batch" else [case]
    return {"bytes": float(sum(one_work(c) for c in jobs)), "flops": 0.0}


def tolerance(case):
    return "exact"


def exact(case, seed):
    """The metrics of a given partition in plain numpy; a partition itself has no other source."""
    if case["call"] != "evaluate":
        return None
    state = prepare(case, seed)
    g, part, k = state["g"], state["part"].astype(np.int64), case["k"]
    length = np.diff(g.off).astype(np.int64)
    hedge = np.repeat(np.arange(g.e, dtype=np.int64), length)
    pair = hedge * k + part[g.pins]
    lam = np.bincount(np.unique(pair) // k, minlength=g.e)
    dest = np.arange(g.P, dtype=np.int64) - np.repeat(g.off[:-1].astype(np.int64), length) >= g.nsrc[hedge]
    inbound = np.bincount(np.unique(pair[dest]) % k, minlength=k)
    wfx = np.minimum(np.floor(g.w.astype(np.float64) * ax.FIXED_POINT_SCALE), 2.0 ** 32 - 1).astype(np.int64)
    size = np.bincount(part, minlength=k)
    omega = ax.kway_omega(g.n, k, case["eps"])
    valid = bool((size > 0).all() and size.max() <= omega and inbound.max() <= 0x7FFFFFFF)
    return np.array([(size > 0).sum(), (wfx * (lam - 1)).sum(), (wfx * (lam > 1)).sum(),
                     (wfx * (lam - 1) * length).sum(), size.max(), inbound.max(), valid], dtype=np.int64)
