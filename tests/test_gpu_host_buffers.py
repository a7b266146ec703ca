"""Callers' host buffers: what a call that fails leaves in them."""
import ctypes

import numpy as np
import pytest

from demystification_dfn_b200 import _lib, networks
from demystification_dfn_b200.layout import ptr
from demystification_dfn_b200.simulation import Simulation

pytestmark = pytest.mark.gpu

DFN_ERR_TIMEOUT = 10


def _device_kernel(sim):
    """K.V on device arrays: returns without a look at the error flag."""
    import torch

    v = torch.ones(sim.N, dtype=torch.float64, device="cuda")
    out = torch.empty(2 * sim.N, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    _lib.check(sim.lib.dfn_kernel_device(sim.h, v.data_ptr(), out.data_ptr(), out[sim.N:].data_ptr()), sim.lib)
    sim.lib.dfn_set_graphs(sim.h, 1)   # waits for the handle's stream
    return out


@pytest.mark.parametrize("buffers", ["pageable", "pinned", "one of each"])
def test_expired_wait_leaves_the_callers_state_buffers(buffers):
    """A K.V whose wait expired and that nobody has asked about: the next read
    of the state reports it and leaves the caller's arrays as they were; the
    one after that (the flag is reported once) fills them."""
    import torch

    p = networks.small_network(seed=33, n_faults=4, tol=1e-6)
    with Simulation(p, pressure="tridiag", gemv="tma") as s:
        s.solve_steps(2)
        ref = s.state()
        Y = torch.full((3 * s.N,), -7.0, dtype=torch.float64, pin_memory=buffers != "pageable").numpy()
        P = torch.full((s.N,), -7.0, dtype=torch.float64, pin_memory=buffers == "pinned").numpy()
        t = ctypes.c_double(-7.0)
        args = (s.h, ptr(Y), ptr(P), ctypes.byref(t), None, None)
        s.set_wait_limit(0)
        _device_kernel(s)
        assert s.lib.dfn_get_state(*args) == DFN_ERR_TIMEOUT
        assert (Y == -7.0).all() and (P == -7.0).all() and t.value == -7.0
        s.set_wait_limit(None)
        assert s.lib.dfn_get_state(*args) == 0
        assert np.array_equal(Y, ref["Y"]) and np.array_equal(P, ref["P"]) and t.value == ref["time"]
