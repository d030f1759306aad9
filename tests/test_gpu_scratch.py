"""Calls whose device scratch is not there (test knob "scratch_limit")."""
import numpy as np
import pytest

import oracle
from qcb200 import randoms
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
