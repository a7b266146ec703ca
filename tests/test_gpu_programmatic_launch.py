"""Kernels that start while their predecessors drain."""
import numpy as np
import pytest

from demystification_dfn_b200 import learned, networks
from demystification_dfn_b200.ensemble import Ensemble
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


def _same(a, b):
    assert a["time"] == b["time"] and np.array_equal(a["Y"], b["Y"]) and np.array_equal(a["P"], b["P"])


@pytest.mark.parametrize("kind", ["hmatrix", "hmatrix_cg", "newton", "newton_mlp", "bf16x2", "batch", "tensor_cores",
                                  "fp64_shared"])
def test_steps_in_one_call_or_one_by_one_elsewhere(kind):
    """The same steps back to back on the device or with a host synchronisation
    after each, bit for bit, in the kernel chains other than the FP64 one of a
    single network."""
    net = networks.fault_network(n_faults=60, box=2000.0, seed=5, tol=1e-6,
                                 kernel="hmatrix" if "hmatrix" in kind else "direct")
    one = {
        "hmatrix": dict(storage="fp32", pressure="tridiag", hmat_leaf=32, hmat_eta=2.0, hmat_eps=1e-6),
        "hmatrix_cg": dict(storage="fp64", pressure="cg", hmat_leaf=32, hmat_eta=2.0, hmat_eps=1e-6),
        "newton": dict(formulation="newton", pressure="cg"),
        "newton_mlp": dict(formulation="newton", guess="mlp", pressure="tridiag"),
        "bf16x2": dict(storage="bf16x2", pressure="cg"),
    }
    if kind in one:
        with Simulation(net, **one[kind]) as a, Simulation(net, **one[kind]) as b:
            if kind == "newton_mlp":
                for s in (a, b):
                    s.set_mlp(learned.init_weights(1))
            a.solve_steps(12)
            for _ in range(12):
                b.solve_steps(1)
            _same(a.state(), b.state())
        return
    if kind == "batch":
        ps = [networks.small_network(seed=s, n_faults=3 + s % 3, tol=1e-6) for s in range(9)]
        kw = dict(pressure="cg")
    else:
        ps = networks.shared_geometry_ensemble(9, base=net, seed=1)
        kw = dict(storage={"tensor_cores": "bf16x2_tc"}.get(kind, kind), pressure="tridiag")
    with Ensemble(ps, **kw) as a, Ensemble(ps, **kw) as b:
        a.solve(n_steps=12)
        for _ in range(12):
            b.solve(n_steps=1)
        for i in range(len(ps)):
            _same(a.state(i), b.state(i))


@pytest.mark.parametrize("form,count", [("v", 60), ("newton", 60), ("v", 330)])
def test_large_batch_steps_like_each_network_alone(form, count):
    """More than 56 832 elements take the stage kernel that loads where it
    needs, fewer the one that loads ahead of its wait; more than 303 104 let
    the blocks of the commit walk. Some members reject steps; bit for bit."""
    ps = [networks.fault_network(n_faults=50, box=1750.0, seed=i % 5, mode="modeIII", tol=1e-6 if form == "v" else 1e-10)
          for i in range(count)]
    kw = dict(storage="bf16x2", pressure="cg", formulation=form)
    with Ensemble(ps, **kw) as e:
        total = sum(e.n_elements)
        assert total > (303104 if count > 60 else 56832)
        reps = e.solve(n_steps=10)
        got = [e.state(i) for i in range(count)]
    assert any(r["rejected"] for r in reps)
    for j in range(5):
        with Simulation(ps[j], **kw) as s:
            assert s.N <= 56832
            rep = s.solve_steps(10)
            ref = s.state()
        for i in range(j, count, 5):
            assert reps[i]["rejected"] == rep["rejected"]
            _same(got[i], ref)
