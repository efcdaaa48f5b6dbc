"""The two forms of the tangent's face pass, with the value (F asked for) and without it.

* The status word: a residual that is not finite sets it in both forms, whether a face flux overflows, or only
  the sum of finite ones over the cell's volume; large fluxes that cancel do not. The direction is zero there,
  so that every tangent is an exact zero and only the value can be at fault.
* The 64-species instance (run-time loops): F is the RHS's and dF the same in both forms, with minmod and van
  Leer; five species padded into it against their own instance, and the 53 species of gri30.
"""
import dataclasses

import numpy as np
import pytest

from ablate_b200 import _lib as L
from ablate_b200 import fv
from ablate_b200.mesh import box_mesh
from ablate_b200.workloads import Workload
from tests import rhs_cases as R
from tests.test_gpu_species_counts import _solver

pytestmark = pytest.mark.gpu

H = 2.0 ** -20  # edge of the cells


def _gas(dim, flux, recon, limiter, exponent, noise):
    """A gas of energy density 10^exponent at Mach 0.1: its energy flux over a face is about
    0.1 * 10^(1.5 exponent) H^(dim-1), and 1/V is H^-dim."""
    shape = (9, 7, 5)[:dim]
    mesh = box_mesh(shape, upper=tuple(H * n for n in shape), periodic=(True,) * dim)
    rng = np.random.default_rng(4)
    n = mesh.n_cells
    E = 10.0 ** exponent * (1.0 + noise * rng.standard_normal(n))
    U = np.zeros((n, 2 + dim))
    U[:, 0], U[:, 1] = 1.0 + noise * rng.standard_normal(n), E
    U[:, 2] = 0.1 * np.sqrt(0.56 * E)
    eos = fv.PerfectGas({"gamma": 1.4, "Rgas": 287.0})
    return Workload("large", mesh, eos, [fv.NavierStokesTransport({}, eos, flux)], recon, limiter, U, "large")


@pytest.mark.parametrize("dim,flux,recon,limiter", [(2, fv.Ausm(), "upwind", "none"), (3, fv.AusmpUp(0.3), "leastsquares", "minmod")])
@pytest.mark.parametrize("exponent,noise,status", [(5.0, 0.05, L.OK),          # ordinary
                                                   (210.0, 0.05, L.ERR_NAN),   # rho u H overflows
                                                   (204.0, 0.05, L.ERR_NAN),   # finite fluxes, their sum over V overflows
                                                   (204.0, 0.0, L.OK)])        # and the same fluxes cancelling
def test_a_residual_that_is_not_finite_sets_the_status(dim, flux, recon, limiter, exponent, noise, status):
    w = _gas(dim, flux, recon, limiter, exponent, noise)
    s = w.solver()
    dU = np.zeros_like(w.U)
    if exponent < 10:
        dU = np.random.default_rng(5).standard_normal(w.U.shape) * np.abs(w.U).mean(0) * 1e-2
    dF, dF2, F = (np.zeros_like(w.U) for _ in range(3))
    with np.errstate(all="ignore"):
        s.ComputeJVP(0.0, w.U, dU, dF2, F)
        assert s.Status() == status
        s.ComputeJVP(0.0, w.U, dU, dF)
    assert s.Status() == status
    assert bool(np.isfinite(F).all()) == (status == L.OK)
    scale = np.abs(dF2).max(0)
    assert np.all(np.abs(dF - dF2) <= 64 * np.finfo(float).eps * scale)
    s.close()


@pytest.mark.parametrize("limiter", ["minmod", "vanleer"])
@pytest.mark.parametrize("name,instance", [("species3d_ns5", 64), ("gri30_box3d", None)])
def test_the_64_species_tangent_with_and_without_its_value(name, instance, limiter):
    w = dataclasses.replace(R.case(name), limiter=limiter)
    s = _solver(w, instance)
    owned = w.mesh.cell_kind == L.CELL_OWNED
    dU = np.random.default_rng(3).standard_normal(w.U.shape) * np.abs(w.U).mean(0) * 1e-3
    F0, F, dF, dF2 = (np.zeros_like(w.U) for _ in range(4))
    s.ComputeRHSFunction(0.0, w.U, F0, L.PRECISION_FP64)
    s.ComputeJVP(0.0, w.U, dU, dF)
    s.ComputeJVP(0.0, w.U, dU, dF2, F)
    assert s.Status() == L.OK
    s.close()
    pairs = [("F against the RHS", F, F0, 1e-12), ("dF with F", dF2, dF, 1e-13)]
    if instance:
        exact = _solver(w)
        dFx, Fx = np.zeros_like(w.U), np.zeros_like(w.U)
        exact.ComputeJVP(0.0, w.U, dU, dFx, Fx)
        assert exact.Status() == L.OK
        exact.close()
        pairs += [("F against the exact instance", F, Fx, 1e-12), ("dF against the exact instance", dF2, dFx, 1e-12)]
    for what, a, b, tol in pairs:
        for block, e in R.block_errors(a, b, owned, 5).items():
            assert e <= tol, f"{what}, {block}: {e:.3e}"
