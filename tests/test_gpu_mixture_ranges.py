"""The NASA-7 mixture over its temperature ranges: species whose ranges meet at different temperatures, and
states whose temperature solve starts in one range and ends in another.

The reference here is numpy in extended precision. Tolerances: the temperature solve stops at
|e_ref - e(T)| <= 1e-8 J/kg, so |dT| <= 1e-8 / c_v; what the rounding of e_ref = E/rho - |u|^2/2 (a few
ulps of E/rho) adds is bounded by 8 eps |E/rho| / c_v. Properties at a given T take 64 eps of the sum of
their terms' magnitudes.
"""
import numpy as np
import pytest

from ablate_b200 import _lib as L
from ablate_b200 import fv

pytestmark = pytest.mark.gpu

RU = np.longdouble("8314.46261815324")
MID = [400.0, 1000.0, 1000.0, 700.0, 1500.0]
EPS = np.finfo(float).eps


def _eos(ns):
    rng = np.random.default_rng(ns)
    species = []
    for k in range(ns):
        low = [rng.uniform(2.5, 4.0), rng.uniform(1e-4, 6e-4), -rng.uniform(0, 5e-8), rng.uniform(0, 3e-12), 0.0, rng.uniform(-3e4, 1e4), 1.0]
        high = [low[0] * rng.uniform(1.0, 1.1), low[1] * rng.uniform(0.8, 1.0), low[2] * 0.5, low[3], 1e-17, 0.0, 1.0]
        t = MID[k % len(MID)]
        h = lambda a: a[0] * t + a[1] * t ** 2 / 2 + a[2] * t ** 3 / 3 + a[3] * t ** 4 / 4 + a[4] * t ** 5 / 5
        high[5] = low[5] + h(low) - h(high)  # the enthalpy is continuous at T_mid, c_p is not
        species.append({"name": f"S{k}", "composition": {"X": rng.uniform(2.0, 44.0)}, "T_ranges": [200.0, t, 3500.0], "low": low, "high": high})
    return fv.TChem(species, atomic_weights={"X": 1.0})


def _terms(eos, T):
    """(e_k, c_v,k, |terms of h_k|) in J/kg, extended precision, shape (n, ns)."""
    T = np.asarray(T, np.longdouble)[:, None]
    r = RU / eos.mw.astype(np.longdouble)

    def h(a, t):
        parts = [a[:, 0] * t, a[:, 1] * t ** 2 / 2, a[:, 2] * t ** 3 / 3, a[:, 3] * t ** 4 / 4, a[:, 4] * t ** 5 / 5, a[:, 5] + 0 * t]
        return r * sum(parts), r * sum(abs(p) for p in parts)

    lo, hi = eos.nasa7[:, 1:8].astype(np.longdouble), eos.nasa7[:, 8:15].astype(np.longdouble)
    low = T < eos.nasa7[:, 0]
    href = h(lo, np.full((1, 1), np.longdouble("298.15")))[0]
    hv = np.where(low, h(lo, T)[0], h(hi, T)[0])
    mag = np.where(low, h(lo, T)[1], h(hi, T)[1]) + abs(href)
    cp = r * np.where(low, lo[:, 0] + T * (lo[:, 1] + T * (lo[:, 2] + T * (lo[:, 3] + T * lo[:, 4]))),
                      hi[:, 0] + T * (hi[:, 1] + T * (hi[:, 2] + T * (hi[:, 3] + T * hi[:, 4]))))
    return hv - href - r * T, cp - r, mag


@pytest.mark.parametrize("ns", [1, 2, 5, 9, 16, 53])
def test_temperature_across_ranges(ns):
    eos = _eos(ns)
    rng = np.random.default_rng(100 + ns)
    edges = np.array([m * f for m in sorted(set(MID)) for f in (1 - 1e-12, 1.0, 1 + 1e-12)])
    T = np.concatenate([edges, np.geomspace(205.0, 3400.0, 120)])
    n = T.size
    Y = rng.dirichlet(np.ones(ns), n)
    Y[:, -1] = 1.0 - Y[:, :-1].sum(1)
    e, cv, mag = _terms(eos, T)
    rho = rng.uniform(0.05, 5.0, n)
    vel = rng.uniform(-300.0, 300.0, (n, 3))
    U = np.empty((n, 5 + ns))
    U[:, 0] = rho
    U[:, 1] = rho * ((e * Y).sum(1).astype(float) + 0.5 * (vel ** 2).sum(1))
    U[:, 2:5] = rho[:, None] * vel
    U[:, 5:] = rho[:, None] * Y
    phys, keep = fv.make_physics(eos, [])
    cvm = (cv * Y).sum(1).astype(float)
    got = fv.eos_property(phys, 3, L.PROP_TEMPERATURE, U)[:, 0]
    # the fractions are rebuilt from rho Y: an ulp each, times the species' energies
    bound = (1e-8 + 8 * EPS * np.abs(U[:, 1] / rho) + 8 * EPS * (mag * Y).sum(1).astype(float)) / cvm + 4 * EPS * T
    assert np.all(np.abs(got - T) <= bound), (np.abs(got - T) / bound).max()
    # properties at T: e_s, h, c_v, c_p, a
    R = (RU / eos.mw * Y).sum(1).astype(float)
    es = (e * Y).sum(1).astype(float)
    scale = 64 * EPS * (mag * Y).sum(1).astype(float)
    at = lambda p: fv.eos_property(phys, 3, p, U, T)[:, 0]
    assert np.all(np.abs(at(L.PROP_INTERNAL_SENSIBLE_ENERGY) - es) <= scale)
    assert np.all(np.abs(at(L.PROP_SENSIBLE_ENTHALPY) - (es + R * T)) <= scale)
    np.testing.assert_allclose(at(L.PROP_CV), cvm, rtol=64 * EPS)
    np.testing.assert_allclose(at(L.PROP_CP), cvm + R, rtol=64 * EPS)
    np.testing.assert_allclose(at(L.PROP_SPEED_OF_SOUND), np.sqrt((cvm + R) / cvm * R * T), rtol=64 * EPS)
