"""Roe's flux on an exactly sonic uniform state: Harten's fix is le + lam^2/le with le = 0 and
lam = 0 there, which must give the wave speed 0, not 0/0 -- the flux of equal states is the
exact flux."""
import ctypes as C

import numpy as np
import pytest

from hyperboliconvergence_gb300 import _capi
from hyperboliconvergence_gb300._capi import FLUX, check


@pytest.mark.parametrize("flux", ["roe", "roe_face"])
@pytest.mark.parametrize("u", [1.0, -1.0])
def test_sonic_uniform_state(flux, u):
    lib = _capi.load()
    # gamma = 2, rho = 2, p = 1: the sound speed, its averages and their roots are exactly 1
    species = np.array([2.0, 287.058, 0.3, 1.0, 1.0])
    face = np.array([1.5, 0.0, 0.0, 1.0, 0.0, 0.0, 1.0])
    q = np.array([u, 0.25, 2.0, 1.0])
    out = np.empty(5)
    ptr = lambda a: a.ctypes.data_as(C.POINTER(C.c_double))  # noqa: E731
    check(lib.hc_flux_eval(FLUX[flux], 0, 0, ptr(species), ptr(face), ptr(q), ptr(q), ptr(out)))
    m = 2.0 * u
    h = 1.0 / (2.0 - 1.0) + 0.5 * (u * u + 0.25 * 0.25)
    want = 1.5 * np.array([m * u + 1.0, m * 0.25, m, m * h, abs(u) + 1.0])
    assert np.allclose(out, want, rtol=1e-14, atol=0)
