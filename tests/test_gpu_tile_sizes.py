"""The face passes on meshes around the limits of the tile size (it follows from the cell count: 32 cells per
tile on the smallest meshes, up to 256 on large ones): last tiles of one cell, and one cell more than a wave
of tiles. The RHS against the oracle (1e-12, the FP64 bar), the adjoint as the transpose of the tangent, and
the tangent with and without its value."""
import numpy as np
import pytest

from ablate_b200 import _lib as L
from ablate_b200 import fv, workloads
from ablate_b200.mesh import box_mesh
from ablate_b200.workloads import Workload, initial_aux
from oracle import oracle as orc

pytestmark = pytest.mark.gpu

SHAPES = [(8, 4, 1), (11, 3, 1), (8, 8, 4), (43, 3, 2), (37, 32, 16), (61, 25, 13), (37, 32, 32), (53, 35, 21), (19, 73, 55)]
# a wave of tiles on 148 SMs and a little more: three CTAs per SM with five species, two with nine
SPECIES_SHAPES = [((37, 24, 16), 5), ((29, 35, 14), 5), ((37, 32, 24), 5), ((29, 28, 35), 5), ((37, 16, 16), 9), ((27, 27, 13), 9),
                  ((37, 32, 16), 9), ((61, 25, 13), 9)]


def _workload(shape, ns):
    mesh = box_mesh(shape, periodic=(False, True, False) if min(shape) > 2 else (False,) * 3, order="morton")
    rng = np.random.default_rng(sum(shape) + ns)
    n = mesh.n_cells
    vel = 60.0 + 20.0 * rng.standard_normal((n, 3))
    if ns:
        eos = workloads.synthetic_mixture(ns, 7)
        T = 700.0 + 200.0 * np.sin(6 * mesh.cell_centroid[:, 0]) + 10.0 * rng.standard_normal(n)
        U = workloads.mixture_state(eos, 1.0 + 0.1 * rng.random(n), vel, T, rng.dirichlet(np.full(ns, 3.0), n))
        flux, tr = fv.AusmpUp(0.3), fv.ConstantLewis(1.8e-5, 0.72, 1.0)
        procs = [fv.NavierStokesTransport({}, eos, flux, tr), fv.SpeciesTransport(eos, flux, tr)]
        return Workload("tiles", mesh, eos, procs, "leastsquares", "vanleer", U, "tiles")
    eos = fv.PerfectGas({"gamma": 1.4, "Rgas": 287.0})
    rho = 1.0 + 0.1 * rng.random(n)
    U = np.concatenate([rho[:, None], (2.5e5 * (1 + 0.02 * rng.standard_normal(n)) + 0.5 * rho * (vel ** 2).sum(1))[:, None], rho[:, None] * vel], 1)
    procs = [fv.NavierStokesTransport({}, eos, fv.AusmpUp(0.3), fv.Constant(k=0.025, mu=1.8e-5))]
    return Workload("tiles", mesh, eos, procs, "leastsquares", "minmod", U, "tiles")


@pytest.mark.parametrize("shape,ns", [(shape, ns) for shape in SHAPES for ns in (0, 5)] + SPECIES_SHAPES)
def test_passes_around_the_tile_limits(shape, ns):
    if ns and np.prod(shape) > 40000:
        pytest.skip("with species the tile size stops at 128 cells")
    w = _workload(shape, ns)
    owned = w.mesh.cell_kind == L.CELL_OWNED
    phys, keep = w.physics()
    ref, _ = orc.rhs(w.mesh, phys, w.U, initial_aux(w))
    s = w.solver()
    F = np.zeros_like(w.U)
    s.ComputeRHSFunction(0.0, w.U, F)
    assert np.linalg.norm(F[owned] - ref[owned]) <= 1e-12 * np.linalg.norm(ref[owned])
    assert np.all(F[~owned] == 0.0)
    rng = np.random.default_rng(3)
    scale = np.abs(w.U).mean(0)
    v = 1e-2 * scale * rng.standard_normal(w.U.shape)
    wt = rng.standard_normal(w.U.shape) / scale * owned[:, None]
    Jv, Jv2, F2, Jw = (np.zeros_like(w.U) for _ in range(4))
    s.ComputeJVP(0.0, w.U, v, Jv)
    s.ComputeJVP(0.0, w.U, v, Jv2, F2)
    s.ComputeVJP(0.0, w.U, wt, Jw)
    assert s.Status() == L.OK
    assert np.linalg.norm(Jv - Jv2) <= 1e-13 * np.linalg.norm(Jv)
    assert np.linalg.norm(F2[owned] - F[owned]) <= 1e-12 * np.linalg.norm(F[owned])
    # the dot-product test, to the magnitude of its terms
    terms = np.abs(wt * Jv).sum() + np.abs(Jw * v).sum()
    assert abs((wt * Jv).sum() - (Jw * v).sum()) <= 1e-12 * terms
    s.close()
