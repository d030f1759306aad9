"""Host threads with a handle and a stream of their own: calls on tableaux of
different sizes at the same time, which share the kernels' launch attributes."""
import ctypes
import threading

import numpy as np
import pytest
import torch

import oracle
from qcb200 import Tableau, ops as O
from qcb200._lib import check, ptr

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def qcb():
    import qcb200

    qcb200.ensure_init(0)
    return qcb200


def run_threads(jobs, times):
    """jobs: functions of a stream pointer, each called `times` times by a
    thread of its own, all at once; the first error of each."""
    errors, gate = [None] * len(jobs), threading.Barrier(len(jobs))

    def body(k):
        st = torch.cuda.Stream()
        try:
            gate.wait()
            for _ in range(times):
                jobs[k](ctypes.c_void_p(st.cuda_stream))
        except Exception as e:  # noqa: BLE001
            errors[k] = e
        st.synchronize()

    threads = [threading.Thread(target=body, args=(k,)) for k in range(len(jobs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    return errors


def random_rows(rows, n, rng):
    return Tableau.from_bits(rng.integers(0, 4, rows), rng.random((rows, n)) < 0.5, rng.random((rows, n)) < 0.5)


def test_dense_apply_of_two_sizes_at_once(qcb):
    """Operators on 1000 and on 800 qubits (64 and 52 KB of tables)."""
    rng = np.random.default_rng(1)
    jobs, tabs, times = [], [], 400
    for n in (1000, 800):
        op = qcb.CliffordOperator(qcb.tensor_pow(qcb.tCNOT(), n // 2).tab).to_gpu()
        t = random_rows(40, n, rng)
        g = t.copy().to_gpu()
        tabs.append((t, g, op))
        jobs.append(lambda st, g=g, op=op: check(qcb.lib().qcb_apply_dense(g.dev.handle, op.tab.dev.handle, 1, st)))
    assert run_threads(jobs, times) == [None, None]
    for t, g, op in tabs:  # tCNOT twice is the identity
        g.to_cpu()
        assert np.array_equal(g.xzs, t.xzs) and np.array_equal(g.phases, t.phases)


def test_gate_lists_on_two_widths_at_once(qcb):
    """Slices of 160 and 48 KB (20000 and 6000 qubits), two threads of each."""
    rng = np.random.default_rng(2)
    jobs, tabs, times = [], [], 4000
    for n in (20000, 6000, 20000, 6000):
        arr = O.to_array([O.sCNOT(2 * k + 1, 2 * k + 2) for k in range(60)])
        t = random_rows(20, n, rng)
        g = t.copy().to_gpu()
        tabs.append((t, g))
        jobs.append(lambda st, g=g, arr=arr: check(qcb.lib().qcb_apply_gates(g.dev.handle, ptr(arr), len(arr), 1, st)))
    assert run_threads(jobs, times) == [None] * 4
    for t, g in tabs:  # CNOTs twice are the identity
        g.to_cpu()
        assert np.array_equal(g.xzs, t.xzs) and np.array_equal(g.phases, t.phases)


def test_canonicalize_of_two_heights_at_once(qcb):
    """Views of 8192 and 5100 rows (128 and 80 KB of row lists)."""
    rng = np.random.default_rng(3)
    jobs, tabs = [], []
    for rows in (8192, 5100):
        t = random_rows(rows, 130, rng)
        g = qcb.Stabilizer(t.copy()).to_gpu()
        tabs.append((t, g))
        jobs.append(lambda st, g=g, rows=rows: check(qcb.lib().qcb_canonicalize(g.tab.dev.handle, 1, rows, 0, None, None, st)))
    assert run_threads(jobs, 100) == [None, None]
    for t, g in tabs:  # without phases, the canonical form is its own
        _, xz, _, _ = oracle.canonicalize(t.phases, t.xzs, 130, False)
        g.to_cpu()
        assert np.array_equal(g.tab.xzs, xz)


def test_permutations_of_two_widths_at_once(qcb):
    """Rows of 50000 and 26000 qubits (98 and 51 KB of staging), two threads of each."""
    jobs, tabs, rng = [], [], np.random.default_rng(4)
    for n in (50_000, 26_000, 50_000, 26_000):
        perm = np.arange(n, 0, -1, dtype=np.uint32)
        t = random_rows(3, n, rng)
        g = t.copy().to_gpu()
        tabs.append((t, g))
        jobs.append(lambda st, g=g, perm=perm: check(qcb.lib().qcb_permutesystems(g.dev.handle, ptr(perm), st)))
    assert run_threads(jobs, 2000) == [None] * 4
    for t, g in tabs:  # an even number of reversals
        g.to_cpu()
        assert np.array_equal(g.xzs, t.xzs)
