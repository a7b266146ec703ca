"""Rounding of the friction law."""
import numpy as np
import pytest

from demystification_dfn_b200 import networks
from demystification_dfn_b200.layout import build_arrays
from demystification_dfn_b200.simulation import Simulation

pytestmark = pytest.mark.gpu


def test_root_of_the_friction_denominator_is_rounded_correctly():
    """dV = loading / (mu/2cs - D s a / 2V0) with D = 1/sqrt(1/C^2 + B^2):
    parameters that are powers of two, rates whose B = V / 2V0 squares exactly
    and 1/C^2, the stress transfer and the healing term far below half a unit
    of what they are added to, so that every operation but 1/|B|, the sum and
    the last division is exact and the result is known to the bit."""
    n = 4000
    ar = build_arrays(networks.single_fault(n_el=n, length=10.0 * n, mode="modeIII", q_kgs=0.0))
    V0, a, s, load = 2.0 ** -20, 2.0 ** -7, -2.0 ** 26, 2.0 ** 30
    ar.a[:] = ar.b[:] = a
    ar.f0[:] = 0.5
    ar.V0[:] = V0
    ar.P[:] = 0.0
    ar.shear_loading_dot[:] = load
    ar.normal_loading_dot[:] = 0.0
    rng = np.random.default_rng(0)
    B = rng.integers(2 ** 25, 2 ** 26, n) * 2.0 ** -78     # 26 bits
    Y = np.concatenate([2 * V0 * B, np.full(n, 64.0), np.full(n, s)])
    with Simulation(ar, pressure="tridiag") as sim:
        dV = sim.friction_law(1.0, Y)[:n]
    den = ar.mu / (2 * ar.cs) - (1.0 / B) * s * a / (2 * V0)
    assert np.array_equal(dV, load / den)
