"""Kernels that start while their predecessors drain."""
import numpy as np
import pytest

from demystification_dfn_b200 import networks
from demystification_dfn_b200.simulation import Simulation

pytestmark = pytest.mark.gpu


def test_wait_limit_does_not_cover_the_kernel_before():
    """A K.V that starts beside a stage kernel of several milliseconds (a
    Newton solve that uses up 20 000 iterations) waits for it without spending
    its own limit: 1024 polls (a K.V of this size needs fewer than 64) are
    enough, and the steps are those of the default limit."""
    p = networks.single_fault(n_el=2000, length=20e3, mode="modeIII", tol=1e-6)
    kw = dict(pressure="tridiag", formulation="newton", newton_maxit=20000, newton_tol=1e-300)
    got = []
    for polls in (None, 1024):
        with Simulation(p, **kw) as s:
            s.set_wait_limit(polls)
            rep = s.solve_steps(2)
            assert rep["newton_fail"] > 0 and rep["newton_iters"] > 100000
            got.append(s.state())
    assert got[0]["time"] == got[1]["time"] and np.array_equal(got[0]["Y"], got[1]["Y"])
