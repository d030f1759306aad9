"""project! at the benchmarked tableau configuration: uniformly random
stabilizer states (random_stabilizer(n), Bravyi-Maslov) of n = 1000, 2000
and 4000 qubits, Stabilizer kind (src/project_trace_reset.jl:276-308), 1,000
random Paulis of weight ~ U{1..n}, bit for bit with phases against the
oracle.

  * chain: the 1,000 Paulis projected in order on one state by one call; some
    Paulis repeat the one before (that one is in the stabilizer group after
    its projection), which takes the commuting branch (canonicalize! +
    generate!, a determined result);
  * independent: each Pauli projected on a fresh copy of the state.
"""
import numpy as np
import pytest

import oracle
from qcb200 import randoms
from qcb200.tableau import Tableau

pytestmark = pytest.mark.gpu

K = 1000


def config_inputs(n, seed):
    rng = np.random.default_rng(seed)
    s = randoms.random_stabilizer(n, rng)
    ps = randoms.random_paulis(K, n, rng)
    return s.tab, ps


@pytest.mark.parametrize("n", [1000, 2000, 4000])
def test_project_chain_stabilizer(qcb, n):
    tab, ps = config_inputs(n, 31 + n)
    repeats = list(range(100, K, 100 if n < 4000 else 250))
    for j in repeats:
        ps.xzs[j], ps.phases[j] = ps.xzs[j - 1], ps.phases[j - 1]
    st = qcb.Stabilizer(tab.copy()).to_gpu()
    _, anti, res = qcb.project_(st, ps.copy().to_gpu())
    st.to_cpu()
    ph, xz = tab.phases.copy(), tab.xzs.copy()
    outs = []
    for j in range(K):
        code, ph, xz, _, a, r = oracle.project("Stabilizer", ph, xz, n, ps.xzs[j], ps.phases[j])
        assert code == 0
        outs.append((a, None if r < 0 else r))
    assert list(zip(anti, res)) == outs
    assert np.array_equal(st.tab.xzs, xz) and np.array_equal(st.tab.phases, ph)
    # the repeated Paulis commute with the state and are determined
    assert all(anti[j] == 0 and res[j] is not None for j in repeats)
    assert sum(a != 0 for a in anti) >= K - len(repeats) - 5


@pytest.mark.parametrize("n", [1000, 2000, 4000])
def test_project_independent_stabilizer(qcb, n):
    tab, ps = config_inputs(n, 77 + n)
    pristine = qcb.Stabilizer(tab.copy()).to_gpu()
    work = qcb.Stabilizer(tab.copy()).to_gpu()
    lib = qcb.lib()
    k = 200 if n == 4000 else K
    for j in range(k):
        qcb.check(lib.qcb_tableau_copy(work.tab.dev.handle, pristine.tab.dev.handle, None))
        p = Tableau(ps.phases[j:j + 1].copy(), n, ps.xzs[j:j + 1].copy())
        _, a, r = qcb.project_(work, qcb.PauliOperator(p.phases, n, p.xzs).to_gpu())
        code, ph, xz, _, oa, orr = oracle.project("Stabilizer", tab.phases, tab.xzs, n, ps.xzs[j], ps.phases[j])
        assert (a, r) == (oa, None if orr < 0 else orr), j
        if j % 50 == 0:
            work.to_cpu()
            assert np.array_equal(work.tab.xzs, xz) and np.array_equal(work.tab.phases, ph), j


def test_project_after_a_commuting_pauli_in_the_cluster_kernel(qcb):
    """A Pauli whose result is the product of stabilizer rows, followed by
    others, on a tableau over several CTAs of one cluster: the partial
    products of the CTAs are read before the next Pauli overwrites them."""
    n, k = 1100, 70
    rng = np.random.default_rng(1230)
    d = randoms.random_destabilizer(n, rng)
    ps = randoms.random_paulis(k, n, rng, phases=True)
    for j in (0, 30, 64):
        src = (ps.xzs[j - 1], ps.phases[j - 1]) if j else (d.tab.xzs[n], d.tab.phases[n])
        ps.xzs[j], ps.phases[j] = src
    st = qcb.Destabilizer(d.tab.copy()).to_gpu()
    qcb.check(qcb.lib().qcb_tune_set(b"project_grid", 2))
    try:
        _, anti, res = qcb.project_(st, ps.copy().to_gpu())
    finally:
        qcb.check(qcb.lib().qcb_tune_set(b"project_grid", 0))
    st.to_cpu()
    ph, xz, outs = d.tab.phases.copy(), d.tab.xzs.copy(), []
    for j in range(k):
        code, ph, xz, _, a, v = oracle.project("Destabilizer", ph, xz, n, ps.xzs[j], ps.phases[j])
        outs.append((a, None if v < 0 else v))
    assert list(zip(anti, res)) == outs
    assert np.array_equal(st.tab.xzs, xz) and np.array_equal(st.tab.phases, ph)


@pytest.mark.parametrize("kind", ["Stabilizer", "MixedStabilizer", "Destabilizer", "MixedDestabilizer"])
@pytest.mark.parametrize("n,k,commuting", [(7, 64, ()), (64, 33, ()), (96, 130, (100,)), (97, 64, (63,)), (130, 200, (70, 71, 140)),
                                           (1088, 65, ()), (1100, 130, (0, 64))])
def test_project_by_panels(qcb, kind, n, k, commuting):
    """Runs of Paulis by panels: ragged panels, views around the search's
    window and rows per thread, Paulis that commute in between (repeats of the
    one before, or a stabilizer row), low ranks with logical operators, and
    without a result; against the oracle."""
    rng = np.random.default_rng(n + k)
    d = randoms.random_destabilizer(n, rng)
    ps = randoms.random_paulis(k, n, rng, phases=True)
    for j in commuting:
        src = (ps.xzs[j - 1], ps.phases[j - 1]) if j else (d.tab.xzs[n], d.tab.phases[n])
        ps.xzs[j], ps.phases[j] = src
    rank = 0
    if kind in ("Stabilizer", "MixedStabilizer"):
        tab = Tableau(d.tab.phases[n:].copy(), n, d.tab.xzs[n:].copy())
        if kind == "MixedStabilizer":
            rank = max(1, n - n // 8)
            tab.xzs[rank:], tab.phases[rank:] = 0, 0
    else:
        tab = d.tab
        rank = n - n // 4 if kind == "MixedDestabilizer" else 0
    for keep in (True, False):
        st = getattr(qcb, kind)(tab.copy(), rank if kind.startswith("Mixed") else None).to_gpu()
        _, anti, res = qcb.project_(st, ps.copy().to_gpu(), keep_result=keep)
        st.to_cpu()
        ph, xz, r, outs = tab.phases.copy(), tab.xzs.copy(), rank, []
        for j in range(k):
            code, ph, xz, r, a, v = oracle.project(kind, ph, xz, n, ps.xzs[j], ps.phases[j], r, keep, True)
            assert code == 0
            outs.append((a, None if v < 0 else v))
        assert list(zip(anti, res)) == outs
        assert np.array_equal(st.tab.xzs, xz) and np.array_equal(st.tab.phases, ph)
        if kind.startswith("Mixed"):
            assert st.rank == r


@pytest.mark.parametrize("kind", ["Stabilizer", "Destabilizer", "MixedDestabilizer"])
def test_projectrand_by_panels(qcb, kind):
    """The random signs of projectrand! in a run by panels equal those of one
    call per Pauli (the other kernels) with the same draws."""
    n, k = 150, 100
    rng = np.random.default_rng(11)
    d = randoms.random_destabilizer(n, rng)
    ps = randoms.random_paulis(k, n, rng, phases=True)
    ps.xzs[80], ps.phases[80] = ps.xzs[79], ps.phases[79]
    tab = d.tab if kind != "Stabilizer" else Tableau(d.tab.phases[n:].copy(), n, d.tab.xzs[n:].copy())
    rank = n - 9 if kind == "MixedDestabilizer" else None
    a = getattr(qcb, kind)(tab.copy(), rank).to_gpu()
    b = getattr(qcb, kind)(tab.copy(), rank).to_gpu()
    _, ra = qcb.projectrand_(a, ps.copy().to_gpu(), rng=np.random.default_rng(3))
    draws = 2 * np.random.default_rng(3).integers(0, 2, size=k)

    class Draw:
        def __init__(self, v):
            self.v = v

        def integers(self, lo, hi, size):
            return np.array([self.v // 2])

    rb = []
    for j in range(k):
        p = qcb.PauliOperator(ps.phases[j:j + 1].copy(), n, ps.xzs[j:j + 1].copy()).to_gpu()
        rb.append(qcb.projectrand_(b, p, rng=Draw(int(draws[j])))[1])
    a.to_cpu()
    b.to_cpu()
    assert ra == rb and a == b
