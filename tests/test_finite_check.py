"""CPU check of the test for finite values that guards the states handed in."""
import ctypes

import numpy as np
import pytest

from demystification_dfn_b200 import build_arrays, networks
from demystification_dfn_b200.layout import to_c


def _create(lib, a):
    h = ctypes.c_void_p()
    st = lib.dfn_create(ctypes.byref(to_c(a)), None, ctypes.byref(h))
    if st == 0:
        lib.dfn_destroy(h)
    return st


@pytest.mark.parametrize("n_el", [2, 7, 8, 9, 16, 23])
@pytest.mark.parametrize("bad", [np.nan, -np.nan, np.inf, -np.inf])
def test_every_position_is_looked_at(lib, n_el, bad):
    a = build_arrays(networks.single_fault(n_el=n_el, length=10.0 * n_el))
    for k in range(n_el):
        keep = a.theta[k]
        a.theta[k] = bad
        assert _create(lib, a) == 4, k
        a.theta[k] = keep
    a.theta[0], a.theta[-1] = np.inf, -np.inf      # no cancelling
    assert _create(lib, a) == 4


@pytest.mark.parametrize("n_el", [2, 7, 8, 9, 23])
def test_extreme_finite_values_pass(lib, n_el):
    a = build_arrays(networks.single_fault(n_el=n_el, length=10.0 * n_el))
    for v in (np.finfo(float).max, -np.finfo(float).max, 5e-324, -0.0):
        a.theta[:] = v
        assert _create(lib, a) != 4
