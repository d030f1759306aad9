"""A stream of symbolic apply! calls, one launch per call and no
synchronisation in between, as a user's loop of apply!(state, gate) issues
them.  Each launch is a programmatic dependent of the launch before it on the
stream (knob "gates_pdl", on by default); the kernel reads the rows only after
its predecessor has completed, so the calls keep their order, also next to
plain launches of other kernels and when the stream is replayed from a CUDA
graph.  Bit-exact with phases against the oracle's sequence."""
import ctypes

import numpy as np
import pytest
import torch

import oracle
from qcb200 import ops as O
from qcb200._lib import check, ptr
from test_gpu_tableau import rand_tab

pytestmark = pytest.mark.gpu

G1 = ["H", "S", "SDAG", "X", "Y", "Z", "SQRTX", "SQRTY", "HXY", "CXYZ"]
G2 = ["CNOT", "CPHASE", "SWAP", "ZCY", "XCX", "YCZ", "ISWAP", "SQRTZZ", "CXSWAP", "INVSQRTYY"]


def random_gates(n, count, rng):
    gates = []
    for _ in range(count):
        if rng.random() < 0.4:
            gates.append(O.Op(O.OP[G1[rng.integers(len(G1))]], int(rng.integers(1, n + 1))))
        else:
            a, b = rng.choice(np.arange(1, n + 1), 2, replace=False)
            gates.append(O.Op(O.OP[G2[rng.integers(len(G2))]], int(a), int(b)))
    return gates


@pytest.mark.parametrize("pdl", [1, 0])
def test_single_gate_calls_in_a_stream(qcb, pdl):
    n = 1000
    rng = np.random.default_rng(500 + pdl)
    t = rand_tab(n, n, rng)
    gates = random_gates(n, 300, rng)
    lib = qcb.lib()
    check(lib.qcb_tune_set(b"gates_pdl", pdl))
    try:
        g = t.copy().to_gpu()
        h = g._need_dev().handle
        side = torch.cuda.Stream()
        sp = ctypes.c_void_p(side.cuda_stream)
        ph, xz = t.phases.copy(), t.xzs.copy()
        for k, op in enumerate(gates):
            arr = O.to_array([op])
            check(lib.qcb_apply_gates(h, ptr(arr), 1, 1, sp))
            ph, xz = oracle.apply_gates(ph, xz, n, arr, True)
            if k % 25 == 24:
                # a plain launch of another kernel in between: row s <- row 1 * row s
                s_row = 2 + k % 50
                check(lib.qcb_mul_rows(h, s_row, 1, h, 1, 0, 0, 0, 1, None, sp))
                ph, xz = oracle.mul_rows(ph, xz, None, None, s_row, 1, 1, 0)
        side.synchronize()
        g.to_cpu()
        assert np.array_equal(g.xzs, xz) and np.array_equal(g.phases, ph)
    finally:
        check(lib.qcb_tune_set(b"gates_pdl", 1))


def test_single_gate_calls_replayed_from_a_graph(qcb):
    n = 700
    rng = np.random.default_rng(77)
    t = rand_tab(n, n, rng)
    gates = [O.to_array([op]) for op in random_gates(n, 120, rng)]
    lib = qcb.lib()
    g = t.copy().to_gpu()
    h = g._need_dev().handle
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        cs = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
        for arr in gates:
            check(lib.qcb_apply_gates(h, ptr(arr), 1, 1, cs))
    ph, xz = t.phases.copy(), t.xzs.copy()
    for _ in range(3):
        graph.replay()
        for arr in gates:
            ph, xz = oracle.apply_gates(ph, xz, n, arr, True)
    torch.cuda.synchronize()
    del graph
    g.to_cpu()
    assert np.array_equal(g.xzs, xz) and np.array_equal(g.phases, ph)


@pytest.mark.parametrize("n,rows,count,local", [
    (1, 1, 8, 1), (2, 33, 9, 2), (63, 31, 7, 63), (64, 64, 200, 64), (65, 65, 470, 65), (200, 32, 481, 3),
    (130, 257, 4100, 130), (500, 1000, 9000, 500), (3000, 40, 700, 3000), (70, 5, 5000, 2)])
def test_gate_lists_by_levels(qcb, n, rows, count, local):
    """Gate lists of the bit-sliced kernel: around the shortest such list, the
    two parameter sizes and several launches, wide levels and chains on few
    qubits (`local`: the gates touch the first that many), ragged rows and
    words; the row-per-thread kernel takes the shorter ones."""
    rng = np.random.default_rng(n + count)
    t = rand_tab(rows, n, rng)
    arr = O.to_array(random_gates(local, count, rng) if local > 1 else
                     [O.Op(O.OP[G1[rng.integers(len(G1))]], 1) for _ in range(count)])
    for phases in (True, False):
        g = t.copy().to_gpu()
        qcb.apply_(g, arr, phases=phases)
        g.to_cpu()
        ph, xz = oracle.apply_gates(t.phases, t.xzs, n, arr, phases)
        assert np.array_equal(g.xzs, xz) and np.array_equal(g.phases, ph)


def test_gate_list_replayed_from_a_graph(qcb):
    n, rng = 300, np.random.default_rng(5)
    t = rand_tab(n, n, rng)
    arr = O.to_array(random_gates(n, 900, rng))
    want = arr.copy()
    g = t.copy().to_gpu()
    h = g._need_dev().handle
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        check(qcb.lib().qcb_apply_gates(h, ptr(arr), len(arr), 1, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    arr[:] = 0  # the list is borrowed for the call only
    ph, xz = t.phases.copy(), t.xzs.copy()
    for _ in range(2):
        graph.replay()
        ph, xz = oracle.apply_gates(ph, xz, n, want, True)
    torch.cuda.synchronize()
    del graph
    g.to_cpu()
    assert np.array_equal(g.xzs, xz) and np.array_equal(g.phases, ph)


@pytest.mark.parametrize("n,rows", [(5000, 70), (20_000, 33), (30_000, 5)])
@pytest.mark.parametrize("count", [12, 13, 14, 51, 52, 53])
def test_gate_lists_on_wide_tableaux(qcb, n, rows, count):
    """Around the shortest list that runs bit-sliced on wide tableaux (13 gates
    on 5000 qubits, 52 on 20000; above about 28000 none does)."""
    rng = np.random.default_rng(n + count)
    t = rand_tab(rows, n, rng)
    arr = O.to_array(random_gates(n, count, rng))
    g = t.copy().to_gpu()
    qcb.apply_(g, arr)
    g.to_cpu()
    ph, xz = oracle.apply_gates(t.phases, t.xzs, n, arr, True)
    assert np.array_equal(g.xzs, xz) and np.array_equal(g.phases, ph)
