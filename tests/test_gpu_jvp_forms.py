"""The two forms of the tangent's face pass, with the value (F asked for) and without it.

* The 64-species instance (run-time loops): F is the RHS's and dF the same in both forms, with minmod and van
  Leer; five species padded into it against their own instance, and the 53 species of gri30.
"""
import dataclasses

import numpy as np
import pytest

from ablate_b200 import _lib as L
from tests import rhs_cases as R
from tests.test_gpu_species_counts import _solver

pytestmark = pytest.mark.gpu


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
