"""A cell with more faces than a CTA has threads, or a 64-bit word has bits: the passes put no limit of their own
on a cell's faces. A hub of n sides inside a ring of n cells, ghosts outside; the RHS against the oracle (1e-12,
the FP64 bar), and the adjoint as the transpose of the tangent."""
import numpy as np
import pytest

from ablate_b200 import _lib as L
from ablate_b200 import fv
from ablate_b200.mesh import Mesh
from ablate_b200.workloads import Workload, initial_aux
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def _wheel(n):
    r1, r2, r3 = 1.0, 1.3, 1.6  # hub rim, ring's outside, ghost centroids at (r2 + r3) / 2
    th = 2 * np.pi * np.arange(n) / n
    mid = th + np.pi / n

    def at(r, a):
        return np.stack([r * np.cos(a), r * np.sin(a), np.zeros(n)], 1)

    ring = 1 + np.arange(n)
    area = lambda r: 0.5 * n * r * r * np.sin(2 * np.pi / n)
    cells = np.concatenate([np.stack([np.zeros(n, int), ring], 1), np.stack([ring, np.roll(ring, -1)], 1), np.stack([ring, ring + n], 1)])
    # radial faces between ring cell i and i + 1 lie at the angle between their middles
    chord = 2 * np.sin(np.pi / n)
    tangent = np.stack([-np.sin(th), np.cos(th), np.zeros(n)], 1)
    normal = np.concatenate([chord * r1 * at(1.0, mid), (r2 - r1) * np.roll(tangent, -1, 0), chord * r2 * at(1.0, mid)])
    apothem = np.cos(np.pi / n)
    fcen = np.concatenate([at(r1 * apothem, mid), np.roll(at(0.5 * (r1 + r2), th), -1, 0), at(r2 * apothem, mid)])
    ccen = np.concatenate([np.zeros((1, 3)), at(0.5 * (r1 + r2) * apothem, mid), at(0.5 * (r2 + r3), mid)])
    vol = np.concatenate([[area(r1)], np.full(n, (area(r2) - area(r1)) / n), np.full(n, (area(r3) - area(r2)) / n)])
    kind = np.concatenate([np.full(n + 1, L.CELL_OWNED), np.full(n, L.CELL_BOUNDARY)]).astype(np.uint8)
    return Mesh(2, cells.astype(np.int32), normal, fcen, ccen, vol, kind, n_interior=n + 1)


@pytest.mark.parametrize("n", [64, 65, 300])
def test_a_cell_with_many_faces(n):
    mesh = _wheel(n)
    rng = np.random.default_rng(n)
    m = mesh.n_cells
    rho, vel = 1.0 + 0.1 * rng.random(m), 60.0 + 20.0 * rng.standard_normal((m, 2))
    U = np.concatenate([rho[:, None], (2.5e5 * (1 + 0.05 * rng.standard_normal(m)) + 0.5 * rho * (vel ** 2).sum(1))[:, None], rho[:, None] * vel], 1)
    eos = fv.PerfectGas({"gamma": 1.4, "Rgas": 287.0})
    w = Workload("wheel", mesh, eos, [fv.NavierStokesTransport({}, eos, fv.AusmpUp(0.3), fv.Constant(k=0.025, mu=1.8e-5))], "leastsquares", "minmod", U, "wheel")
    phys, keep = w.physics()
    ref, _ = orc.rhs(mesh, phys, U, initial_aux(w))
    owned = mesh.cell_kind == L.CELL_OWNED
    s = w.solver()
    F, Jv, Jw = (np.zeros_like(U) for _ in range(3))
    s.ComputeRHSFunction(0.0, U, F)
    for k in range(4):
        assert np.linalg.norm(F[owned, k] - ref[owned, k]) <= 1e-12 * np.linalg.norm(ref[owned, k])
    scale = np.abs(U).mean(0)
    v = 1e-2 * scale * rng.standard_normal(U.shape)
    wt = rng.standard_normal(U.shape) / scale * owned[:, None]
    s.ComputeJVP(0.0, U, v, Jv)
    s.ComputeVJP(0.0, U, wt, Jw)
    assert s.Status() == L.OK
    terms = np.abs(wt * Jv).sum() + np.abs(Jw * v).sum()
    assert abs((wt * Jv).sum() - (Jw * v).sum()) <= 1e-12 * terms
    s.close()
