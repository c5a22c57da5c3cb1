"""What a partition takes of the arena: arenas of these many bytes have held these partitions since before the
levels kept lists of long hyperedges, states of two words per node and weights per node."""
import numpy as np
import pytest

import axoncuda_b200 as ax

pytestmark = pytest.mark.gpu


def netlist(n, seed):
    return ax.gen_circuit(n, n + n // 10, 2, 64, 2.5, 0.9, 0.02, seed)


CASES = {
    # 179,406 parts: most nodes' gains by tables, none by candidates
    "many parts": (lambda: netlist(400000, 5), ax.params_incc(3, 40, 1 << 20, cnc=4, rfr=8), 263444992),
    # copies of 5000 parts each
    "5000 parts": (lambda: netlist(100000, 4), ax.params_kway(5000, 0.05, cnc=4, rfr=8), 505680640),
    "few hyperedges": (lambda: ax.Hypergraph(500000, np.array([0, 3, 5], np.uint64), np.array([1, 2, 3, 7, 9], np.uint32),
                                             np.ones(2, np.uint32), np.ones(2, np.float32)),
                       ax.params_incc(100, 100, 1 << 20, cnc=4, rfr=8), 94133760),
}


@pytest.mark.parametrize("case", CASES)
def test_partition_fits_the_arena_it_fitted(case):
    make, p, arena = CASES[case]
    g = make()
    with ax.Context(0, arena) as ctx:
        part, st = ctx.partition(g, p)
    assert st.valid == 1 and st.device_bytes_peak <= arena
