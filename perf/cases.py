"""The work that users of this framework have it do, as measurable cases.

``listed()`` names the cases, ``draw(rng)`` gives others of the same ranges,
``prepare`` builds what a program holds before the call (problem arrays, the
handle with its kernel matrices, the state), ``run`` makes one pass through
the public entry points and returns whole results, ``work`` counts the bytes
and operations that no implementation can avoid and ``exact`` computes the
results again in 64 bits with plain torch and numpy.

The fault geometry of a case is fixed by its sizes (made once per process);
the seed gives the friction parameters, the initial slip rates, the fault
that carries the pressure step and the vectors handed to the operators.

Runs of one network (``steps`` and ``host_steps``) start every pass from the
same state, as a program does that holds its state in its own arrays and has
a stretch of steps made from it; ensembles go on from where they are, since
their states live in the handle.
"""
import dataclasses
import functools
import math

import numpy as np
import torch

from demystification_dfn_b200 import learned, networks
from demystification_dfn_b200.ensemble import Ensemble
from demystification_dfn_b200.layout import build_arrays
from demystification_dfn_b200.simulation import Simulation

HMAT = dict(hmat_leaf=64, hmat_eta=2.0)


def listed():
    return [
        # the smallest networks: a handful of faults, where launches are all there is
        dict(name="steps_small_network", kind="steps", faults=4, mode="modeII", store="fp64", pressure="cg", steps=20),
        # one straight fault, 40 km in 10 m elements, fluid injection: the reference's own example problem
        dict(name="steps_single_fault", kind="steps", faults=1, elements=4000, mode="modeIII", store="fp64",
             pressure="tridiag", steps=16),
        # the 800-fault network of the benchmark, FP64, with the reference's CG for the pore pressure
        dict(name="steps_network_800", kind="steps", faults=800, mode="modeII", store="fp64", pressure="cg", steps=8),
        # a caller that owns the state: step by step with host arrays in and the output snapshot back
        dict(name="host_steps_network", kind="host_steps", faults=203, mode="modeII", store="bf16x2", pressure="cg",
             steps=4),
        # the operators by themselves, for a program with a time integrator of its own:
        # stress transfer of a slip-rate vector (ragged size) ...
        dict(name="stress_transfer", kind="kernel", faults=317, mode="modeII", store="fp64", pressure="cg"),
        # ... and the whole right-hand side (pressure, stress transfer, friction)
        dict(name="right_hand_side", kind="rhs", faults=61, mode="modeIII", store="fp32", pressure="cg"),
        # 4000 faults in 20 km x 20 km under tectonic load, hierarchical matrix with FP32 factors: the largest network
        dict(name="steps_hmatrix_4000", kind="hmatrix_steps", faults=4000, mode="modeII", store="fp32", pressure="cg",
             eps=1e-6, steps=8),
        # many distinct networks at once, dense kernels, friction law solved for the slip rate
        dict(name="ensemble_dense", kind="ensemble", faults=0, count=24, mode="modeII", store="fp32",
             pressure="tridiag", form="newton", steps=8),
        # the same with hierarchical matrices
        dict(name="ensemble_hmatrix", kind="ensemble_hmatrix", faults=0, count=24, mode="modeII", store="fp32",
             pressure="tridiag", form="newton", eps=1e-5, steps=8),
        # 64 realisations of one network sharing its kernel matrix: tensor cores ...
        dict(name="shared_tensor_cores", kind="shared", faults=800, count=64, mode="modeII", store="bf16x2_tc",
             pressure="tridiag", form="v", steps=16),
        # ... and in FP64 (fewer, ragged members)
        dict(name="shared_fp64", kind="shared", faults=400, count=50, mode="modeII", store="fp64_shared",
             pressure="tridiag", form="v", steps=8),
        # training the network that proposes the start of the friction solve
        dict(name="train_guess", kind="train", samples=49_999, batch=4096, epochs=2),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["steps", "steps", "steps", "host_steps", "kernel", "rhs", "hmatrix_steps", "ensemble",
                       "ensemble_hmatrix", "shared", "shared", "train"])
    if kind == "train":
        return dict(kind=kind, samples=_log(rng, 500, 49_999), batch=rng.choice([512, 1000, 4096]),
                    epochs=rng.randint(1, 2))
    c = dict(kind=kind, mode=rng.choice(["modeII", "modeIII"]), store=rng.choice(["fp64", "fp32", "bf16x2"]),
             pressure=rng.choice(["cg", "tridiag"]), steps=rng.randint(2, 8))
    if kind in ("steps", "host_steps", "kernel", "rhs"):
        if rng.random() < 0.3:
            c.update(faults=1, elements=_log(rng, 33, 8000))
        else:
            c.update(faults=_log(rng, 2, 700))
        if kind in ("kernel", "rhs"):
            del c["steps"]
        return c
    c["store"] = "fp32"
    if kind == "hmatrix_steps":
        return dict(c, faults=_log(rng, 250, 2500), eps=rng.choice([1e-5, 1e-6]), steps=rng.randint(2, 4))
    c.update(count=_log(rng, 2, 20), pressure="tridiag", form=rng.choice(["v", "newton"]))
    if kind == "ensemble":
        return dict(c, faults=_log(rng, 10, 200), store=rng.choice(["fp64", "fp32", "bf16x2"]))
    if kind == "ensemble_hmatrix":
        return dict(c, faults=_log(rng, 50, 250), eps=rng.choice([1e-5, 1e-6]))
    tc = rng.random() < 0.5
    return dict(c, store="bf16x2_tc" if tc else "fp64_shared", count=_log(rng, 2, 130), form="v",
                faults=_log(rng, 10, 500 if tc else 200))


# ---------------------------------------------------------------------------
# problems


@functools.lru_cache(maxsize=4)
def _geometry(kind, faults, elements, count, mode):
    """Problem arrays of a case's networks (one, or `count` distinct ones)."""
    kernel = "hmatrix" if "hmatrix" in kind else "direct"
    if kind.startswith("ensemble"):
        n = {} if faults == 0 else dict(n_faults=faults)   # 0: 100 to 400 faults each
        return [build_arrays(networks.ensemble_member(i, mode=mode, kernel=kernel, **n)) for i in range(count)]
    if faults == 1:
        return [build_arrays(networks.single_fault(n_el=elements, length=10.0 * elements, mode=mode, kernel=kernel))]
    if kind == "hmatrix_steps":
        p = networks.fault_network(n_faults=faults, box=20000.0 * math.sqrt(faults / 4000), mode=mode, kernel=kernel,
                                   tol=1e-6, v_load=1e-9)
    elif faults < 10:
        p = networks.small_network(n_faults=faults, mode=mode)
    else:
        p = networks.fault_network(n_faults=faults, box=7000.0 * math.sqrt(faults / 800), mode=mode)
    return [build_arrays(p)]


def _geo(case):
    return _geometry(case["kind"], case["faults"], case.get("elements", 0), case.get("count", 1), case["mode"])


def _realisation(base, rng):
    """The network `base` with friction parameters, initial state and pressure step of its own."""
    F, N = len(base.fault_nb_element), base.N
    real = ~base.fake_mask
    of = np.repeat(np.arange(F), base.fault_nb_element)
    ch = {}
    for k in ("a", "b"):
        v = getattr(base, k).copy()
        v[real] *= np.exp(rng.normal(0.0, 0.02, F))[of]
        ch[k] = v
    V = base.V.copy()
    V[real] *= np.exp(rng.normal(0.0, 0.1, int(real.sum())))
    theta = base.theta.copy()
    theta[real] = np.log(base.V0[real] / V[real])
    P = np.zeros(N)
    if len(base.src_fault) == 0:
        f = int(rng.integers(F))
        s, n = int(base.fault_first[f]), int(base.fault_nb_element[f])
        P[s:s + max(1, n // 2)] = 10e6
    Q = base.src_Q * float(np.exp(rng.normal(0.0, 0.1)))
    return dataclasses.replace(base, V=V, theta=theta, P=P, src_Q=Q, _keep=[], **ch)


def _problems(case, seed):
    rng = np.random.default_rng(seed)
    g = _geo(case)
    if case["kind"] == "shared":
        g = [g[0]] * case["count"]
    return [_realisation(b, rng) for b in g]


def _slip_rates(arr, rng):
    """A slip-rate vector in the middle of a run: some faults slip much faster than the rest."""
    v = arr.V * np.exp(rng.normal(0.0, 3.0, arr.N))
    v[arr.fake_mask] = 0.0
    return v


def _samples(case, seed):
    """Inputs and targets as recorded from the friction solves: seven smooth inputs, a correction that sets in
    where radiation damping does."""
    rng = np.random.default_rng(seed)
    x = rng.normal(0.0, 0.5, (case["samples"], 7)).astype(np.float32)
    t = (0.3 * np.tanh(2.0 * x[:, 0] - x[:, 1]) + 0.1 * x[:, 2] * x[:, 6]).astype(np.float32)
    return x, t, learned.init_weights(int(rng.integers(1 << 30)))


def prepare(case, seed):
    kind = case["kind"]
    if kind == "train":
        x, t, w = _samples(case, seed)
        return dict(case=case, x=x, t=t, w=w)
    probs = _problems(case, seed)
    kw = dict(storage=case["store"], pressure=case["pressure"], formulation=case.get("form", "v"))
    if "hmatrix" in kind:
        kw.update(HMAT, hmat_eps=case["eps"])
    if kind in ("ensemble", "ensemble_hmatrix", "shared"):
        return dict(case=case, ens=Ensemble(probs, max_step=CAP, **kw))
    p = probs[0]
    st = dict(case=case, sim=Simulation(p, **kw), Y=p.Y0(), P=p.P.copy())
    rng = np.random.default_rng(seed + 1)
    if kind == "kernel":
        st["v"] = _slip_rates(p, rng)
    elif kind == "rhs":
        st["Y"][:p.N] = _slip_rates(p, rng)
    elif kind == "host_steps":
        st["out"] = [np.empty(p.N) for _ in range(5)]
    return st


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "train":
        w, loss = learned.train(state["x"], state["t"], weights=state["w"], epochs=case["epochs"],
                                batch=case["batch"], lr=2e-3, seed=0)
        return dict(weights=w, loss=loss)
    if kind in ("ensemble", "ensemble_hmatrix", "shared"):
        ens = state["ens"]
        ens.solve(n_steps=case["steps"])
        s = [ens.state(i) for i in range(ens.B)]
        return dict(_blocks([q["Y"] for q in s]), P=np.concatenate([q["P"] for q in s]),
                    slip=np.concatenate([ens.slip(i) for i in range(ens.B)]),
                    time=np.array([q["time"] for q in s]), t_try=np.array([q["t_try"] for q in s]))
    sim = state["sim"]
    if kind == "kernel":
        return sim.kernel(state["v"])
    if kind == "rhs":
        return _blocks([sim.friction_law(DT_RHS, state["Y"])])
    if kind == "host_steps":
        # V, theta, P and tractions come back; the state of the next step is made from them
        Y, P, t, tt = state["Y"], state["P"], 0.0, T_FIRST
        V0, Dc = sim.arrays.V0, sim.arrays.Dc
        out = state["out"]
        for _ in range(case["steps"]):
            rep = sim.step_host(Y, P, t, tt, out)
            t, tt = rep.time, rep.t_try
            Y = np.concatenate([out[0], np.log(out[1] * (V0 / Dc)), out[4]])
            P = out[2]
        return dict(V=out[0].copy(), theta=out[1].copy(), P=out[2].copy(), tT=out[3].copy(), tN=out[4].copy(),
                    time=t, t_try=tt)
    sim.set_state(state["Y"], state["P"], 0.0, T_FIRST)
    sim.solve_steps(case["steps"])
    s = sim.state()
    return dict(_blocks([s["Y"]]), P=s["P"], time=s["time"], t_try=s["t_try"])


def _blocks(Ys):
    """The blocks of the state vectors: slip rate (or slip), log-state, normal traction."""
    return {k: np.concatenate([Y.reshape(3, -1)[j] for Y in Ys]) for j, k in enumerate(("first", "psi", "sigma"))}


DT_RHS = 50.0     # s: offset of the right-hand side from the step start
T_FIRST = 100.0   # s: first trial step, as solve() begins
CAP = 600.0       # s: largest step of the ensembles, so that one pass costs what the next does

# ---------------------------------------------------------------------------
# what a pass cannot do without

_ENTRY = {"fp64": 8, "fp32": 4, "bf16x2": 4, "bf16x2_tc": 4, "fp64_shared": 8}


def _matrix_values(case, N):
    """Stored values of one network's kernel matrices: all of them, or for a hierarchical matrix of these leaf
    sizes and tolerances about 300 (1e-5) or 360 (1e-6) per element, component and level of the cluster tree."""
    comps = 2 if case["mode"] == "modeII" else 1
    if "hmatrix" in case["kind"]:
        per = (300 if case["eps"] > 5e-6 else 360) * max(1.0, math.log2(N / 64))
        return comps * N * min(N, per)
    return comps * N * N


def work(case):
    if case["kind"] == "train":
        n = case["samples"] * case["epochs"]
        return {"bytes": 32.0 * n, "flops": 6.0 * n * (7 * 64 + 64 * 64 + 64)}
    sizes = [a.N for a in _geo(case)]
    vals = sum(_matrix_values(case, N) for N in sizes)
    members = case["count"] if case["kind"] == "shared" else 1
    elements = sum(sizes) * members
    rhs = 6 * case["steps"] if "steps" in case else 1      # an accepted step takes at least six right-hand sides
    state = elements * 8 * (3 if case["kind"] == "kernel" else 20)   # vectors of a right-hand side
    products = 3 if case["store"] == "bf16x2_tc" else 1    # hi hi, hi lo, lo hi
    return {"bytes": float(rhs * (vals * _ENTRY[case["store"]] + state)),
            "flops": float(rhs * 2 * vals * members * products)}


# ---------------------------------------------------------------------------
# the same results in 64 bits


def _cuda():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _stiffness(arr):
    """K_T and K_N (None in mode III) of one network, with their elastic prefactor, [N, N] in FP64."""
    dev = _cuda()
    nd = torch.tensor(arr.node, dtype=torch.float64, device=dev)
    mid, d = 0.5 * (nd[1:] + nd[:-1]), nd[1:] - nd[:-1]
    tan = d / d.norm(dim=1, keepdim=True)
    nrm = torch.stack([-tan[:, 1], tan[:, 0]], 1)
    KT = torch.empty(arr.N, arr.N, dtype=torch.float64, device=dev)
    KN = torch.empty_like(KT) if arr.fracture_mode == 2 else None
    pref = arr.mu / (2 * math.pi) if KN is None else arr.mu / math.pi * (1 - arr.cs ** 2 / arr.cp ** 2)
    for r0 in range(0, arr.N, 512):
        r = slice(r0, min(arr.N, r0 + 512))
        x = mid[r, None, 0] - nd[None, :, 0]
        y = mid[r, None, 1] - nd[None, :, 1]
        r2 = x * x + y * y
        if KN is None:
            w = (tan[r, 0, None] * x + tan[r, 1, None] * y) / r2
            KT[r] = pref * (w[:, 1:] - w[:, :-1])
            continue
        gx, gy = x / r2, y / r2
        n1, n2 = nrm[r, 0, None], nrm[r, 1, None]
        c2, s2 = n2 * n2 - n1 * n1, 2 * n1 * n2
        cos2, sin2 = (y * y - x * x) / r2, 2 * x * y / r2
        q, w = s2 * sin2 + c2 * cos2, s2 * cos2 - c2 * sin2
        l1, l2 = nrm[None, :, 0], nrm[None, :, 1]
        a, b = q * gx, q * gy
        KT[r] = pref * (l2 * (a[:, :-1] - a[:, 1:]) - l1 * (b[:, :-1] - b[:, 1:]))
        a, b = gx - gy * w, gy + gx * w
        KN[r] = pref * (l1 * (a[:, :-1] - a[:, 1:]) + l2 * (b[:, :-1] - b[:, 1:]))
    return KT, KN


class _Network:
    """One network's right-hand side, pressure step and adaptive Cash-Karp steps in FP64."""

    A = (0.2, 0.3, 0.6, 1.0, 0.875)
    B = ((0.2,), (3 / 40, 9 / 40), (0.3, -0.9, 1.2), (-11 / 54, 2.5, -70 / 27, 35 / 27),
         (1631 / 55296, 175 / 512, 575 / 13824, 44275 / 110592, 253 / 4096))
    C = (37 / 378, 0.0, 250 / 621, 125 / 594, 0.0, 512 / 1771)
    DC = (37 / 378 - 2825 / 27648, 0.0, 250 / 621 - 18575 / 48384, 125 / 594 - 13525 / 55296, -277 / 14336,
          512 / 1771 - 0.25)

    def __init__(self, arr, K, pressure="cg", form="v", cap=86400.0):
        self.arr, self.K, self.cg, self.form, self.cap = arr, K, pressure == "cg", form, cap
        dev = K[0].device
        self.t = {k: torch.tensor(getattr(arr, k), dtype=torch.float64, device=dev)
                  for k in ("a", "b", "Dc", "f0", "V0", "normal_loading_dot", "shear_loading_dot")}
        self.fake = torch.tensor(arr.fake_mask, device=dev)
        self.eta = arr.mu / (2 * arr.cs)
        self.Y = torch.tensor(arr.Y0(), dtype=torch.float64, device=dev)
        self.P = arr.P.astype(np.float64).copy()
        self.time, self.t_try = 0.0, T_FIRST
        N = arr.N
        kx = np.zeros(N + 1)
        p = arr.permeability
        both = p[1:] + p[:-1]
        kx[1:N] = np.where(both > 0, 2 * p[1:] * p[:-1] / np.where(both > 0, both, 1), 0.0)
        ds2 = ((arr.node[1:] - arr.node[:-1]) ** 2).sum(1)
        c = arr.porosity * arr.dyn_viscosity * (arr.fluid_comp + arr.rock_comp)
        self.v = (kx[:-1] + kx[1:]) / (c * ds2)
        self.u, self.w = np.zeros(N), np.zeros(N)
        self.u[1:] = kx[1:N] / (c * ds2[:-1])
        self.w[:-1] = kx[1:N] / (c * ds2[1:])
        self.src = np.zeros(N)
        self.tb, self.te = (arr.src_t_beg, arr.src_t_end) if len(arr.src_Q) else (np.array([1e300]), np.array([1e300]))
        for f, i, q in zip(arr.src_fault, arr.src_index, arr.src_Q):   # one source per fault at most
            e = int(arr.fault_first[f - 1] + i - 1)
            self.src[e] += q / (arr.porosity * (arr.fluid_comp + arr.rock_comp)) / math.sqrt(ds2[e])
        L = int(arr.fault_nb_element.max())
        at = arr.fault_first[:, None] + np.arange(L)[None]
        self.inside = np.arange(L)[None] < arr.fault_nb_element[:, None]
        self.at = np.where(self.inside, at, 0)
        if form == "newton":
            q = self.t
            V, psi, sig = self.Y[:N].clone(), self.Y[N:2 * N], self.Y[2 * N:]
            Cf = torch.exp((q["f0"] + q["b"] * psi) / q["a"])
            w = torch.asinh(V * Cf / (2 * q["V0"]))
            self.tau0 = self.eta * V - (sig + self._dev(self.P)) * q["a"] * w
            self.tau0[self.fake] = 0.0
            self.Y[:N] = 0.0
        self.slip = torch.zeros(N, dtype=torch.float64, device=dev)

    def _dev(self, x):
        return torch.as_tensor(x, dtype=torch.float64, device=self.Y.device)

    def stress(self, x):
        return self.K[0] @ x, (self.K[1] @ x if self.K[1] is not None else torch.zeros_like(x))

    def pressure(self, dt):
        """Implicit step from the committed pressure: (P, dP/dt, converged)."""
        t = self.time + dt
        b = self.P + (dt * self.src if np.any((t >= self.tb) & (t < self.te)) else 0.0)
        x, ok = self._cg(dt, b) if self.cg else (self._thomas(dt, b), True)
        return x, ((x - self.P) / dt if dt >= 1e-9 else np.zeros_like(x)), ok

    def _thomas(self, dt, b):
        at, on = self.at, self.inside
        A1, A2, A3 = -dt * self.u[at], 1 + dt * self.v[at], -dt * self.w[at]
        r = b[at]
        A2[~on], A1[~on], A3[~on] = 1.0, 0.0, 0.0
        L = at.shape[1]
        c, d = np.zeros_like(A1), np.zeros_like(A1)
        cp, dp = np.zeros(len(at)), np.zeros(len(at))
        for k in range(L):
            den = A2[:, k] - A1[:, k] * cp
            cp, dp = A3[:, k] / den, (r[:, k] - A1[:, k] * dp) / den
            c[:, k], d[:, k] = cp, dp
        x = np.zeros(len(at))
        out = b.copy()
        for k in range(L - 1, -1, -1):
            x = np.where(on[:, k], d[:, k] - c[:, k] * x, 0.0)
            out[at[on[:, k], k]] = x[on[:, k]]
        return out

    def _cg(self, dt, b):
        D = 1 + dt * self.v
        s1, s3 = -dt * self.u / D, -dt * self.w / D

        def mul(v):
            m = v.copy()
            m[1:] += s1[1:] * v[:-1]
            m[:-1] += s3[:-1] * v[1:]
            return m

        x = self.P.copy()
        r = b / D - mul(x)
        p, rr, it = r.copy(), r @ r, 0
        while np.abs(r).max() >= self.arr.tol_solver:
            it += 1
            m = mul(p)
            al = rr / (p @ m)
            x, r = x + al * p, r - al * m
            new = r @ r
            p, rr = r + (new / rr) * p, new
            if it > 200:
                return x, False
        return x, True

    def rhs(self, Y, Pt, Pd, tt=0.0):
        N, q = self.arr.N, self.t
        psi, sig = Y[N:2 * N], Y[2 * N:]
        Pt = self._dev(Pt)
        T, Nn = self.stress(Y[:N])
        self.T = T
        if self.form == "v":
            V, Pd = Y[:N], self._dev(Pd)
            ds = Nn + q["normal_loading_dot"]
            Bq, Cq = V / (2 * q["V0"]), torch.exp((q["f0"] + q["b"] * psi) / q["a"])
            D = 1 / torch.sqrt(1 / (Cq * Cq) + Bq * Bq)
            heal = q["V0"] / q["Dc"] * torch.exp(-psi) - V.abs() / q["Dc"]
            num = (q["shear_loading_dot"] + T + (ds + Pd) * q["a"] * torch.asinh(Bq * Cq)
                   + Bq * D * (sig + Pt) * q["b"] * heal)
            dV = num / (self.eta - D * (sig + Pt) * q["a"] / (2 * q["V0"]))
        else:
            ds = torch.zeros_like(psi)
            tau = self.tau0 + T + q["shear_loading_dot"] * tt
            s = -(sig + Nn + q["normal_loading_dot"] * tt + Pt)
            lnA = torch.log(2 * q["V0"]) - (q["f0"] + q["b"] * psi) / q["a"]
            sa = torch.where(s > 0, s * q["a"], torch.ones_like(s))
            lz = torch.log(tau.abs() / self.eta) - lnA
            wr = torch.copysign(torch.where(lz > 20, lz + math.log(2), torch.asinh(torch.exp(lz.clamp(max=20)))), tau)
            w = tau / sa
            w = torch.where((wr.abs() < w.abs()), wr, w)
            for _ in range(60):
                e = torch.exp(lnA + w.abs() - math.log(2))
                z = torch.exp(-2 * w.abs())
                g = tau - self.eta * torch.copysign(e * (1 - z), w) - sa * w
                w = w + (g / (self.eta * e * (1 + z) + sa)).clamp(-10, 10)
            V = torch.copysign(torch.exp(lnA + w.abs() - math.log(2)) * (1 - torch.exp(-2 * w.abs())), w)
            V = torch.where(s > 0, V, tau / self.eta)
            heal = q["V0"] / q["Dc"] * torch.exp(-psi) - V.abs() / q["Dc"]
            dV = V
        out = torch.stack([dV, heal, ds])
        out[:, self.fake] = 0.0
        return out.reshape(-1)

    def step(self):
        newton = self.form == "newton"
        Pt, Pd, ok = self.pressure(self.t_try)
        while not ok:
            self.t_try /= 2
            Pt, Pd, ok = self.pressure(self.t_try)
        h, eps = self.t_try, self.arr.tol_solver
        k = [self.rhs(self.Y, self.P if newton else Pt, Pd, self.time)]
        scale = self.Y.abs() + (k[0] * h).abs() + eps
        while True:
            k, V = k[:1], [self.Y[:self.arr.N]]
            full = self.pressure(h)
            for c, row in zip(self.A, self.B):
                y = self.Y + h * sum(b * x for b, x in zip(row, k))
                V.append(y[:self.arr.N])
                if newton:
                    k.append(self.rhs(y, self.P + c * (full[0] - self.P), 0.0, self.time + c * h))
                else:
                    Pt, Pd, _ = full if c == 1.0 else self.pressure(c * h)
                    k.append(self.rhs(y, Pt, Pd))
            err = (h * sum(c * x for c, x in zip(self.DC, k)) / scale).abs().max().item() / eps
            if err <= 1.0:
                break
            h = max(0.9 * h * err ** -0.25, 0.1 * h)
        self.Y = self.Y + h * sum(c * x for c, x in zip(self.C, k))
        self.slip = self.slip + h * sum(c * x for c, x in zip(self.C, V))
        if full[2]:
            self.P = full[0]
        self.time += h
        self.t_try = min(0.9 * h * err ** -0.2 if err > float(np.float32(1.89e-4)) else 5 * h, self.cap)


def _train64(case, x, t, w):
    """The training pass in FP64 (same sample order and minibatches, Adam)."""
    n, order = len(t), list(range(len(t)))
    s, m64 = 1442695040888963407, (1 << 64) - 1
    for i in range(n - 1, 0, -1):
        s = (s * 6364136223846793005 + 1442695040888963407) & m64
        j = (s >> 33) % (i + 1)
        order[i], order[j] = order[j], order[i]
    dev = _cuda()
    x, t = (torch.tensor(v[order], dtype=torch.float64, device=dev) for v in (x, t))
    w = torch.tensor(w, dtype=torch.float64, device=dev, requires_grad=True)
    m, v = torch.zeros_like(w), torch.zeros_like(w)
    step, loss = 0, [0.0, 0.0]
    for ep in range(case["epochs"]):
        total = 0.0
        for b in range(0, n, case["batch"]):
            xb, tb = x[b:b + case["batch"]], t[b:b + case["batch"]]
            o = 0
            W1, b1, W2, b2, W3, b3 = (w[o1:o2] for o1, o2 in ((0, 448), (448, 512), (512, 4608), (4608, 4672),
                                                              (4672, 4736), (4736, 4737)))
            h = torch.nn.functional.silu(xb @ W1.reshape(7, 64) + b1)
            h = torch.nn.functional.silu(h @ W2.reshape(64, 64) + b2)
            sq = ((h @ W3 + b3 - tb) ** 2).sum()
            (g,) = torch.autograd.grad(sq / len(tb), w)
            total += sq.item()
            step += 1
            m, v = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g
            upd = 2e-3 * (m / (1 - 0.9 ** step)) / (torch.sqrt(v / (1 - 0.999 ** step)) + 1e-8)
            w = (w - upd).detach().requires_grad_()
        if ep == 0:
            loss[0] = total / n
        loss[1] = total / n
    return dict(weights=w.detach().cpu().numpy(), loss=np.array(loss))


def exact(case, seed):
    kind = case["kind"]
    if kind == "train":
        return _train64(case, *_samples(case, seed))
    if kind == "hmatrix_steps" and case["faults"] > 800:
        return None   # a dense kernel matrix of that size does not fit
    probs = _problems(case, seed)
    p = probs[0]
    if kind in ("ensemble", "ensemble_hmatrix", "shared"):
        K = _stiffness(p) if kind == "shared" else None
        nets = []
        for q in probs:
            n = _Network(q, K or _stiffness(q), case["pressure"], case["form"], CAP)
            for _ in range(case["steps"]):
                n.step()
            n.K = None
            nets.append(n)
        newton = case["form"] == "newton"
        return dict(_blocks([n.Y.cpu().numpy() for n in nets]), P=np.concatenate([n.P for n in nets]),
                    slip=np.concatenate([(n.Y[:n.arr.N] if newton else n.slip).cpu().numpy() for n in nets]),
                    time=np.array([n.time for n in nets]), t_try=np.array([n.t_try for n in nets]))
    net = _Network(p, _stiffness(p), case["pressure"])
    rng = np.random.default_rng(seed + 1)
    if kind == "kernel":
        return tuple(s.cpu().numpy() for s in net.stress(net._dev(_slip_rates(p, rng))))
    if kind == "rhs":
        net.Y[:p.N] = net._dev(_slip_rates(p, rng))
        Pt, Pd, _ = net.pressure(DT_RHS)
        return _blocks([net.rhs(net.Y, Pt, Pd).cpu().numpy()])
    for _ in range(case["steps"]):
        net.step()
    Y, N = net.Y.cpu().numpy(), p.N
    if kind == "host_steps":
        return dict(V=Y[:N], theta=p.Dc / p.V0 * np.exp(Y[N:2 * N]), P=net.P, tT=net.T.cpu().numpy(), tN=Y[2 * N:],
                    time=net.time, t_try=net.t_try)
    return dict(_blocks([Y]), P=net.P, time=net.time, t_try=net.t_try)
