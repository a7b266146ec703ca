"""Callers' host buffers: staged or direct, delivered or left as they were."""
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


def _array(n, pinned):
    import torch

    return torch.full((n,), -7.0, dtype=torch.float64, pin_memory=pinned).numpy()


def _all_calls(p, pinned, **kw):
    """Every entry point that moves host buffers, on buffers of one kind (or of
    alternating kinds); what each delivered."""
    turn = [0]

    def new(n, like=None):
        turn[0] += 1
        a = _array(n, pinned if isinstance(pinned, bool) else turn[0] % 2 == 0)
        if like is not None:
            a[:] = like
        return a

    out = {}
    with Simulation(p, **kw) as s:
        N, lib, h = s.N, s.lib, s.h
        rng = np.random.default_rng(N)
        v = rng.normal(size=N)
        Y0, P0 = s.arrays.Y0(), s.arrays.P + 1e5

        def call(name, *args):
            _lib.check(getattr(lib, name)(h, *args), lib)

        sT, sN = new(N), new(N)
        call("dfn_kernel", ptr(new(N, v)), ptr(sT), ptr(sN))
        Yd, Pt, Pd = new(3 * N), new(N), new(N)
        call("dfn_set_state", ptr(new(3 * N, Y0)), ptr(new(N, P0)), 0.0, 100.0, 0)
        call("dfn_friction_law", 1.0, 3 * N, ptr(new(3 * N, Y0)), ptr(Yd))
        call("dfn_compute_P", 10.0, ptr(Pt), ptr(Pd), None)
        call("dfn_solve_steps", 2, None)
        Y, P, slip = new(3 * N), new(N), new(N)
        call("dfn_get_state", ptr(Y), ptr(P), None, None, None)
        call("dfn_get_slip", 0, ptr(slip))
        snap = [new(N) for _ in range(6)]
        call("dfn_get_snapshot", *[ptr(a) for a in snap], None)
        host = [new(N) for _ in range(5)]
        call("dfn_step_host", ptr(new(3 * N, Y0)), ptr(new(N, P0)), 0.0, 100.0, *[ptr(a) for a in host], None)
        Y2, P2 = new(3 * N), new(N)
        call("dfn_get_state", ptr(Y2), None, None, None, None)
        call("dfn_get_state", None, ptr(P2), None, None, None)
        out.update(sT=sT, sN=sN, Yd=Yd, Pt=Pt, Pd=Pd, Y=Y, P=P, slip=slip, Y2=Y2, P2=P2)
        out.update({"snap%d" % i: a for i, a in enumerate(snap)}, **{"host%d" % i: a for i, a in enumerate(host)})
        # nothing of a later call reached an earlier one's buffers
        assert np.array_equal(host[0], Y2[:N]) and np.array_equal(host[2], P2)
    return out


@pytest.mark.parametrize("n_el", [2, 3, 9, 33, 200, 1404])
def test_buffers_of_either_kind_get_the_same(n_el):
    """Pageable buffers go through the staging memory as far as it reaches (the
    vectors of the smallest networks and the last ones of a step do not fit,
    nor do both results of the pressure for two elements), pinned ones do not."""
    p = networks.single_fault(n_el=n_el, length=10.0 * n_el, mode="modeII", tol=1e-6)
    ref = _all_calls(p, True, pressure="tridiag")
    for pinned in (False, "alternating"):
        got = _all_calls(p, pinned, pressure="tridiag")
        for k in ref:
            assert np.array_equal(ref[k], got[k]), k


@pytest.mark.parametrize("n", [20_000, 30_000, 140_000])
def test_buffers_larger_than_the_staging_memory(n):
    """20 000 elements: the state fits the staging memory, a step's vectors do in
    part; 30 000: the state does not, single vectors do; 140 000: none does."""
    p = networks.single_fault(n_el=n, length=10.0 * n, mode="modeIII", kernel="hmatrix", tol=1e-6)
    kw = dict(pressure="tridiag", storage="fp32", hmat_leaf=64, hmat_eta=2.0, hmat_eps=1e-4)
    ref, got = (_all_calls(p, pinned, **kw) for pinned in (True, False))
    for k in ref:
        assert np.array_equal(ref[k], got[k]), k


def test_call_after_one_that_delivered_nothing():
    """A pressure solve that meets its iteration cap leaves its buffers as they
    were, and the next calls do not see its staged copies."""
    p = networks.single_fault(n_el=300, length=3000.0, mode="modeIII", tol=1e-300)
    q = networks.single_fault(n_el=300, length=3000.0, mode="modeIII", tol=1e-6)
    v = np.random.default_rng(0).normal(size=300)
    with Simulation(q, pressure="cg") as s:
        ref = s.kernel(v)
    with Simulation(p, pressure="cg") as s:
        for pinned in (False, True):
            Pt, Pd, ier = _array(300, pinned), _array(300, pinned), ctypes.c_int32(-1)
            _lib.check(s.lib.dfn_compute_P(s.h, 5000.0, ptr(Pt), ptr(Pd), ctypes.byref(ier)), s.lib)
            assert ier.value == 1 and (Pt == -7.0).all() and (Pd == -7.0).all()
            got = s.kernel(v)
            assert np.array_equal(got[0], ref[0]) and np.array_equal(got[1], ref[1])
            assert (Pt == -7.0).all() and (Pd == -7.0).all()
