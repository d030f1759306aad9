"""project! of runs in which Paulis commute with the state: trials by panels that
end at once, early or after some panels, and the kernels that take the run then;
against the oracle."""
import numpy as np
import pytest

import oracle
from qcb200 import Tableau, randoms

pytestmark = pytest.mark.gpu


def state_of(qcb, kind, n, d):
    """(state, tableau, rank) of a kind from a random destabilizer."""
    if kind in ("Stabilizer", "MixedStabilizer"):
        tab = Tableau(d.tab.phases[n:].copy(), n, d.tab.xzs[n:].copy())
        rank = 0
        if kind == "MixedStabilizer":
            rank = n - n // 8
            tab.xzs[rank:], tab.phases[rank:] = 0, 0
    else:
        tab, rank = d.tab, n - n // 4 if kind == "MixedDestabilizer" else 0
    return getattr(qcb, kind)(tab.copy(), rank if kind.startswith("Mixed") else None), tab, rank


def paulis(d, n, k, commuting, rng):
    """k random Paulis; those at `commuting` repeat the one before (the first: a stabilizer row)."""
    ps = randoms.random_paulis(k, n, rng, phases=True)
    for j in commuting:
        src = (ps.xzs[j - 1], ps.phases[j - 1]) if j else (d.tab.xzs[n], d.tab.phases[n])
        ps.xzs[j], ps.phases[j] = src
    return ps


@pytest.mark.parametrize("kind", ["Stabilizer", "MixedStabilizer", "Destabilizer", "MixedDestabilizer"])
@pytest.mark.parametrize("n,k,commuting", [(40, 80, (0,)), (40, 80, (1,)), (70, 100, (7, 70)), (70, 100, (8, 71)), (70, 150, (9, 75, 76)),
                                           (100, 40, tuple(range(0, 40, 2))), (33, 200, tuple(range(1, 200, 4))),
                                           (64, 64, tuple(range(64))), (50, 140, (0, 64, 128)), (40, 300, (5,)), (40, 300, (250, 251)),
                                           (40, 400, (300,)), (40, 400, (256,)), (40, 400, (320, 390)), (150, 290, (0, 280)), (20, 257, (256,)), (20, 320, (319,))])
def test_runs_that_end_early(qcb, kind, n, k, commuting):
    rng = np.random.default_rng(n + k + len(commuting))
    d = randoms.random_destabilizer(n, rng)
    ps = paulis(d, n, k, commuting, rng)
    for keep in (True, False):
        st, tab, rank = state_of(qcb, kind, n, d)
        st.to_gpu()
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


def test_runs_without_room_for_the_panels(qcb):
    """Without room for the panels' copy of the rows the other kernels project the run."""
    n, k = 60, 90
    rng = np.random.default_rng(6)
    d = randoms.random_destabilizer(n, rng)
    ps = paulis(d, n, k, (40, 41), rng)
    out = []
    for kb in (0, 1):
        st = qcb.Destabilizer(d.tab.copy()).to_gpu()
        qcb.check(qcb.lib().qcb_tune_set(b"scratch_limit", kb))
        try:
            _, anti, res = qcb.project_(st, ps.copy().to_gpu())
        finally:
            qcb.check(qcb.lib().qcb_tune_set(b"scratch_limit", 0))
        st.to_cpu()
        out.append((anti, res, st.tab.xzs.tolist(), st.tab.phases.tolist()))
    assert out[0] == out[1]
