"""Calls whose device scratch is not there (test knob "scratch_limit") or that
end in the middle (test knob "fail_call")."""
import ctypes

import numpy as np
import pytest
import torch

import oracle
from qcb200 import circuits, ops as O, randoms
from test_gpu_tableau import rand_tab

pytestmark = pytest.mark.gpu


@pytest.fixture
def no_scratch(qcb):
    def limit(kb):
        qcb.check(qcb.lib().qcb_tune_set(b"scratch_limit", kb))

    yield limit
    limit(0)


@pytest.mark.parametrize("rows,n", [(16, 20), (40, 300), (64, 65), (100, 100), (600, 600), (1100, 200), (1000, 1000)])
@pytest.mark.parametrize("phases", [True, False])
def test_canonicalize_without_scratch(qcb, no_scratch, rows, n, phases):
    """Where there is no room for a copy of the rows, the kernels in one
    cluster's shared memory canonicalize the view."""
    rng = np.random.default_rng(rows + n)
    t = rand_tab(rows, n, rng) if rows != n else randoms.random_stabilizer(n, rng).tab
    s = qcb.Stabilizer(t.copy()).to_gpu()
    no_scratch(1)
    _, rx, rz = qcb.canonicalize_(s, phases=phases, ranks=True)
    no_scratch(0)
    s.to_cpu()
    ph, xz, orx, orz = oracle.canonicalize(t.phases, t.xzs, n, phases)
    assert (rx, rz) == (orx, orz)
    assert np.array_equal(s.tab.xzs, xz) and np.array_equal(s.tab.phases, ph)


def pool_used():
    """Bytes in use of device 0's stream-ordered pool."""
    cu = ctypes.CDLL("libcuda.so.1")
    pool, used = ctypes.c_void_p(), ctypes.c_uint64()
    assert cu.cuDeviceGetDefaultMemPool(ctypes.byref(pool), 0) == 0
    assert cu.cuMemPoolGetAttribute(pool, 7, ctypes.byref(used)) == 0  # CU_MEMPOOL_ATTR_USED_MEM_CURRENT
    return used.value


def memory_in_use():
    """(bytes of the pool in use, bytes of the device in use outside the pool's reserve)"""
    cu = ctypes.CDLL("libcuda.so.1")
    torch.cuda.synchronize()
    pool, res = ctypes.c_void_p(), ctypes.c_uint64()
    assert cu.cuDeviceGetDefaultMemPool(ctypes.byref(pool), 0) == 0
    assert cu.cuMemPoolGetAttribute(pool, 5, ctypes.byref(res)) == 0  # CU_MEMPOOL_ATTR_RESERVED_MEM_CURRENT
    free, total = torch.cuda.mem_get_info()
    return pool_used(), total - free - res.value


def failing_calls(qcb, call, most=200):
    """`call` with its first, second, ... checked CUDA call failing, until it
    makes them all; how many failed."""
    for k in range(1, most):
        qcb.check(qcb.lib().qcb_tune_set(b"fail_call", k))
        try:
            call()
            failed = False
        except qcb.QCBError:
            failed = True
        finally:
            qcb.check(qcb.lib().qcb_tune_set(b"fail_call", 0))
        if not failed:
            return k - 1
    raise AssertionError("the call never succeeds")


def batch_jobs(qcb, specs):
    jobs = []
    for d, rounds, p, shots in specs:
        arr = O.to_array(circuits.rotated_surface_code_memory(d, rounds, p))
        qmax, bmax = O.affected_counts(arr)
        jobs.append((qcb.PauliFrame(shots, qmax, bmax, init=False), qcb.Program(arr), 5))
    return jobs


@pytest.mark.parametrize("specs", [[(3, 3, 1e-3, 2000)], [(9, 9, 5e-3, 400_000), (3, 1, 1e-3, 100)]])
def test_failing_batch_create_gives_its_memory_back(qcb, specs):
    """qcb_batch_create with every one of its CUDA calls failing in turn; the
    second batch's noise scratch lies outside the pool (above 64 MB)."""
    jobs = batch_jobs(qcb, specs)
    qcb.Batch(jobs).run().status()  # warm: modules, pools
    before = memory_in_use()
    assert failing_calls(qcb, lambda: qcb.Batch(jobs)) >= 5
    after = memory_in_use()
    assert after[0] == before[0] and abs(after[1] - before[1]) < 16 << 20


def test_batch_without_noise_scratch(qcb, no_scratch):
    """Without room for the noise scratch the jobs' noise is drawn in the walk."""
    jobs = batch_jobs(qcb, [(5, 3, 4e-3, 20_000), (3, 2, 1e-2, 3000)])
    records = []
    for kb in (0, 1):
        no_scratch(kb)
        b = qcb.Batch(jobs)
        no_scratch(0)
        b.run().status()
        records.append([f.record_planes() for f, *_ in jobs])
    assert all(np.array_equal(a, b) for a, b in zip(*records))


@pytest.mark.parametrize("what", ["dense", "canonicalize", "canonicalize_ranks"])
def test_failing_calls_give_their_scratch_back(qcb, what):
    """apply! of a dense operator and canonicalize! by panels with every one of
    their CUDA calls failing in turn; the last one, which makes them all, is
    right."""
    n, rng = 130, np.random.default_rng(8)
    t = rand_tab(90, n, rng)
    op = qcb.random_clifford(n, rng)
    op.to_gpu()
    s = qcb.Stabilizer(t.copy()).to_gpu()

    def call():
        if what == "dense":
            qcb.check(qcb.lib().qcb_apply_dense(s.tab.dev.handle, op.tab.dev.handle, 1, None))
        else:
            qcb.canonicalize_(s, ranks=what != "canonicalize")

    call()  # warm
    torch.cuda.synchronize()
    before = pool_used()
    assert failing_calls(qcb, lambda: (s.tab.dev.upload(t.phases, t.xzs), call())) >= 5
    torch.cuda.synchronize()
    assert pool_used() == before
    s.to_cpu()
    if what == "dense":
        ph, xz = oracle.apply_dense(t.phases, t.xzs, n, op.tab.phases, op.tab.xzs, True)
    else:
        ph, xz, _, _ = oracle.canonicalize(t.phases, t.xzs, n, True)
    assert np.array_equal(s.tab.xzs, xz) and np.array_equal(s.tab.phases, ph)


def pool_peak(call):
    """Bytes of the pool in use at most during `call`, beyond those before."""
    cu = ctypes.CDLL("libcuda.so.1")
    pool, zero, high = ctypes.c_void_p(), ctypes.c_uint64(0), ctypes.c_uint64()
    assert cu.cuDeviceGetDefaultMemPool(ctypes.byref(pool), 0) == 0
    torch.cuda.synchronize()
    before = pool_used()
    assert cu.cuMemPoolSetAttribute(pool, 8, ctypes.byref(zero)) == 0  # CU_MEMPOOL_ATTR_USED_MEM_HIGH
    call()
    torch.cuda.synchronize()
    assert cu.cuMemPoolGetAttribute(pool, 8, ctypes.byref(high)) == 0
    return high.value - before


@pytest.mark.parametrize("rows,n", [(36_000, 7424), (49_000, 4928), (900_000, 1000), (5_000_000, 64)])
def test_dense_apply_scratch_is_bounded(qcb, rows, n):
    """The partial products of all runs of qubits take at most 256 MB."""
    rng = np.random.default_rng(rows)
    W = 2 * ((n + 63) // 64)
    t = qcb.DeviceTableau(rows, n)
    t.upload(np.zeros(rows, np.uint8), np.repeat(rng.integers(0, 2**63, (1000, W), dtype=np.uint64), rows // 1000, axis=0))
    op = qcb.DeviceTableau(2 * n, n)
    op.upload(np.zeros(2 * n, np.uint8), rng.integers(0, 2**63, (2 * n, W), dtype=np.uint64))
    peak = pool_peak(lambda: qcb.check(qcb.lib().qcb_apply_dense(t.handle, op.handle, 1, None)))
    assert 0 < peak <= (256 << 20) + (1 << 20)


@pytest.mark.parametrize("n,rows,kb", [(1000, 1000, 200), (1000, 777, 100), (300, 500, 30), (2100, 700, 400), (4097, 200, 400),
                                       (64, 5000, 40)])
@pytest.mark.parametrize("phases", [True, False])
def test_dense_apply_in_slabs(qcb, no_scratch, n, rows, kb, phases):
    """Several slabs of rows, the last one ragged, with one and more runs of
    qubits each, where only kb KB of scratch are there."""
    rng = np.random.default_rng(n + rows)
    state = rand_tab(rows, n, rng)
    c = rand_tab(2 * n, n, rng)
    s, op = state.copy().to_gpu(), c.copy().to_gpu()
    before = qcb.lib().qcb_launch_count()
    no_scratch(kb)
    qcb.check(qcb.lib().qcb_apply_dense(s.dev.handle, op.dev.handle, int(phases), None))
    no_scratch(0)
    assert qcb.lib().qcb_launch_count() - before >= 4 + phases  # two slabs at least
    s.to_cpu()
    ph, xz = oracle.apply_dense(state.phases, state.xzs, n, c.phases, c.xzs, phases)
    assert np.array_equal(s.xzs, xz) and np.array_equal(s.phases, ph)


@pytest.mark.parametrize("n,rows", [(48, 70), (64, 9), (65, 100), (1000, 130), (2048, 33), (2049, 40), (4100, 20), (30, 20_000)])
@pytest.mark.parametrize("phases", [True, False])
def test_dense_apply_without_scratch(qcb, no_scratch, n, rows, phases):
    """Without room for the partial products of one group of rows, a warp a row
    multiplies its images."""
    rng = np.random.default_rng(n + rows)
    state = rand_tab(rows, n, rng)
    c = rand_tab(2 * n, n, rng)
    s, op = state.copy().to_gpu(), c.copy().to_gpu()
    no_scratch(1)
    qcb.check(qcb.lib().qcb_apply_dense(s.dev.handle, op.dev.handle, int(phases), None))
    no_scratch(0)
    s.to_cpu()
    ph, xz = oracle.apply_dense(state.phases, state.xzs, n, c.phases, c.xzs, phases)
    assert np.array_equal(s.xzs, xz) and np.array_equal(s.phases, ph)


def test_a_refused_allocation_is_reported_once(qcb):
    """A frame and a tableau larger than the device are refused with QCB_EOOM;
    the call after it is not affected (its launch reported the same error)."""
    t = rand_tab(10, 100, np.random.default_rng(3))
    arr = O.to_array([O.sHadamard(1)])
    g = t.copy().to_gpu()
    for make in (lambda: qcb.PauliFrame(2**40, 100, 100, init=False), lambda: qcb.DeviceTableau(2**31 - 1, 10_000)):
        with pytest.raises(qcb.QCBError, match="memory"):
            make()
        qcb.apply_(g, arr)
    g.to_cpu()
    assert np.array_equal(g.xzs, t.xzs) and np.array_equal(g.phases, t.phases)  # H twice
