"""The SSP-RK3 step, whose stages are taken in the face pass, against the same step driven from the host
through the ghost fill, the RHS and the stage entry point. The arithmetic per row is the same; a multiply-add
may be contracted differently, and the three stages carry that on: 16 ulps of a row's largest component
cover it."""
import numpy as np
import pytest

from ablate_b200 import _lib as L
from ablate_b200 import distributed as D
from ablate_b200 import fv
from ablate_b200.workloads import initial_aux
from tests import rhs_cases as R

pytestmark = pytest.mark.gpu


def _entry_points(torch, ref, V, dt, precision, st):
    """The step on V, whose ghosts are filled, through the entry points."""
    A, B, F = V.clone(), V.clone(), torch.empty_like(V)

    def stage(a, b, Us, out):
        F.zero_()
        ref.ComputeRHSDevice(0.0, Us.data_ptr(), F.data_ptr(), precision, st)
        ref.RkStageDevice(a, V.data_ptr(), b, Us.data_ptr(), dt, F.data_ptr(), out.data_ptr(), st)

    stage(0.0, 1.0, V, A)
    ref.FillGhostsDevice(A.data_ptr(), st)
    stage(0.75, 0.25, A, B)
    ref.FillGhostsDevice(B.data_ptr(), st)
    stage(1.0 / 3.0, 2.0 / 3.0, B, V)
    ref.NormalizeSpeciesDevice(V.data_ptr(), st)
    ref.FillGhostsDevice(V.data_ptr(), st)


@pytest.mark.parametrize("name,precision", [("sod2d_ausm_upwind", L.PRECISION_FP64), ("tgv3d_mixed_check", L.PRECISION_FP64),
                                            ("tgv3d_mixed_check", L.PRECISION_MIXED), ("walled_channel3d", L.PRECISION_FP64),
                                            ("box1d_visc", L.PRECISION_FP64), ("shear3d_ns5", L.PRECISION_FP64),
                                            ("tets3d_ns9", L.PRECISION_FP64)])
@pytest.mark.parametrize("cfl_step", [False, True])
def test_staged_step_matches_the_entry_points(name, precision, cfl_step):
    torch = pytest.importorskip("torch")
    w = R.case(name)
    U0 = torch.from_numpy(np.ascontiguousarray(w.U)).cuda()
    st = torch.cuda.current_stream().cuda_stream
    step, ref = w.solver(), w.solver()
    for s in (step, ref):
        if w.boundary is not None:
            s.SetBoundary(*w.boundary)
    V = U0.clone()
    ref.FillGhostsDevice(V.data_ptr(), st)
    dt = ref.CflTimeStepDevice(V.data_ptr(), 0.4, st)
    _entry_points(torch, ref, V, dt, precision, st)

    G = U0.clone()
    if cfl_step:
        time = torch.full((), 0.25, dtype=torch.float64, device="cuda")
        step.StepCflDevice(L.STEP_SSPRK3, 0.4, G.data_ptr(), precision, time.data_ptr(), st)
        assert float(time) == 0.25 + dt
    else:
        step.StepDevice(L.STEP_SSPRK3, 0.0, dt, G.data_ptr(), precision, st)
    assert step.Status() == L.OK
    bound = 16 * np.finfo(float).eps * torch.maximum(V.abs().amax(0), V.abs())
    assert bool(((G - V).abs() <= bound).all())
    step.close()
    ref.close()


@pytest.mark.parametrize("name", ["box2d_ausmpup_vanleer_suth", "walled_channel3d", "species3d_ns5", "tets3d_ns9"])
def test_staged_step_of_a_partition_keeps_its_halo_rows(name):
    # one domain of three: its halo rows are neither owned nor filled from a condition, and every stage reads
    # the caller's. A step of a NaN state first: whatever the stages' buffers held, NaN is what is left in them
    torch = pytest.importorskip("torch")
    w = R.case(name)
    d = D.submesh(w.mesh, D.partition_cells(w.mesh, 3), 1)
    kinds = set(d.mesh.cell_kind.tolist())
    assert {L.CELL_OWNED, L.CELL_HALO} <= kinds
    st = torch.cuda.current_stream().cuda_stream
    U0 = torch.from_numpy(np.ascontiguousarray(w.U[d.gid])).cuda()
    step, ref = (fv.FiniteVolumeSolver(d.mesh, w.eos, w.processes, w.petscfv_type, w.limiter) for _ in range(2))
    for s in (step, ref):
        if w.boundary is not None:
            s.SetBoundary(w.boundary[0], w.boundary[1][d.gid])
    G = torch.full_like(U0, float("nan"))
    step.StepDevice(L.STEP_SSPRK3, 0.0, 1e-9, G.data_ptr(), L.PRECISION_FP64, st)
    assert step.Status() != L.OK
    for s in (step, ref):
        s.SetAux(initial_aux(w)[d.gid])  # the NaN state's temperatures are no guesses
    V, G = U0.clone(), U0.clone()
    ref.FillGhostsDevice(V.data_ptr(), st)
    dt = ref.CflTimeStepDevice(V.data_ptr(), 0.4, st)
    _entry_points(torch, ref, V, dt, L.PRECISION_FP64, st)
    step.StepDevice(L.STEP_SSPRK3, 0.0, dt, G.data_ptr(), L.PRECISION_FP64, st)
    assert step.Status() == L.OK and ref.Status() == L.OK
    halo = torch.from_numpy(np.isin(d.mesh.cell_kind, [L.CELL_HALO, L.CELL_HALO_OUTER])).cuda()
    assert torch.equal(G[halo], U0[halo])
    bound = 16 * np.finfo(float).eps * torch.maximum(V.abs().amax(0), V.abs())
    assert bool(((G - V).abs() <= bound).all())
    step.close()
    ref.close()
