"""The work a program has this framework do, as cases that can be timed and checked.

Every case drives a ``FiniteVolumeSolver`` through its public methods. ``flow`` names the mesh and the
physics (all of them generators or variants of ``ablate_b200/workloads.py``), ``n`` the size, ``op`` the
call and ``precision`` the arithmetic asked for:

  flow   sod    2D Euler on n x n quads, outflow ghosts, AUSM, first order
         tgv    3D Navier-Stokes on an n^3 periodic box, AUSM+up, least squares + minmod
         wall   the same physics in an n^3 channel with inlet, outflow and walls (ghost cells)
         shear  3D Euler + ns NASA-7 species on an n^3 box, AUSM+up, least squares + minmod
         tets   3D Navier-Stokes + ns NASA-7 species with constant-Lewis diffusion on about n Delaunay
                tetrahedra, AUSM+up, least squares + van Leer
  op     rhs    one right-hand side on device-resident rows (the stage of an explicit time stepper)
         host   one right-hand side on host arrays (the drop-in call of a CPU time stepper)
         march  ``steps`` SSP-RK3 steps at CFL 0.5 with the step size kept on the device
         step   one SSP-RK3 step of given size (three right-hand sides, each from the temperatures of the
                stage before it, and the species normalisation)
         jvp    one Jacobian-vector product (the operator of a matrix-free Newton-Krylov solve)
         vjp    one vector-Jacobian product (one stage of an adjoint march)
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from ablate_b200 import _lib as L
from ablate_b200 import fv, workloads
from ablate_b200.mesh import box_mesh, delaunay_mesh

RU = 8314.46261815324  # J/(kmol K)
TREF = 298.15          # K, reference of the sensible enthalpies
AIR = {"gamma": 1.4, "Rgas": 287.0}
MU, PRANDTL = 1.8e-5, 0.72
CP_AIR = AIR["gamma"] * AIR["Rgas"] / (AIR["gamma"] - 1.0)


def listed():
    return [
        # the smallest call: a 2D shock problem on a coarse grid, all launch latency
        {"name": "sod_rhs_32", "flow": "sod", "n": 32, "ns": 0, "op": "rhs", "precision": "fp64"},
        # the 2D shock problem marched in time: dozens of short launches back to back
        {"name": "sod_march_256", "flow": "sod", "n": 256, "ns": 0, "op": "march", "steps": 10, "precision": "fp64"},
        # the ordinary explicit stage of a 3D viscous flow, in both precisions
        {"name": "tgv_rhs_112", "flow": "tgv", "n": 112, "ns": 0, "op": "rhs", "precision": "fp64"},
        {"name": "tgv_mixed_64", "flow": "tgv", "n": 64, "ns": 0, "op": "rhs", "precision": "mixed"},
        # a bounded domain of odd size: ghost cells, partly filled tiles, spacing not exact in binary
        {"name": "wall_rhs_45", "flow": "wall", "n": 45, "ns": 0, "op": "rhs", "precision": "fp64"},
        # the Krylov operator of an implicit step, and one stage of an adjoint march
        {"name": "wall_jvp_64", "flow": "wall", "n": 64, "ns": 0, "op": "jvp", "precision": "fp64"},
        {"name": "wall_vjp_72", "flow": "wall", "n": 72, "ns": 0, "op": "vjp", "precision": "fp64"},
        # a time step of a five-species shear layer, and its adjoint
        {"name": "shear_step_64", "flow": "shear", "n": 64, "ns": 5, "op": "step", "precision": "fp64"},
        {"name": "shear_vjp_56", "flow": "shear", "n": 56, "ns": 5, "op": "vjp", "precision": "fp64"},
        # reacting-flow transport on tetrahedra: nine species, diffusion, cones of four faces
        {"name": "tets_rhs_200k", "flow": "tets", "n": 200_000, "ns": 9, "op": "rhs", "precision": "fp64"},
        {"name": "tets_jvp_60k", "flow": "tets", "n": 60_000, "ns": 9, "op": "jvp", "precision": "fp64"},
        # the drop-in call: PETSc's vectors are host memory, copied in and out on each call
        {"name": "tgv_host_48", "flow": "tgv", "n": 48, "ns": 0, "op": "host", "precision": "fp64"},
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    flow = rng.choice(["sod", "tgv", "wall", "shear", "tets"])
    case = {"flow": flow, "ns": 0, "precision": "fp64"}
    if flow == "sod":
        case.update(op=rng.choice(["rhs", "march"]), n=size(16, 512))
        if case["op"] == "march":
            case["steps"] = 10
    elif flow in ("tgv", "wall"):
        case["op"] = rng.choice(["rhs", "rhs", "host", "jvp", "vjp"])
        case["n"] = size(8, {"rhs": 112, "host": 80}.get(case["op"], 88))
        if case["op"] == "rhs":
            case["precision"] = rng.choice(["fp64", "mixed"])
    elif flow == "shear":
        # 5 and 9 species have kernels of their own; 4 and 7 run padded in them
        case["ns"] = rng.choice([4, 5, 5, 7, 9])
        # a step is compiled for the counts with kernels of their own
        case["op"] = rng.choice(["rhs", "jvp", "vjp"] + (["step"] if case["ns"] in (5, 9) else []))
        case["n"] = size(8, 72 if case["op"] in ("rhs", "step") else 56)
    else:
        case["op"] = rng.choice(["rhs", "jvp", "vjp"])
        case["ns"] = rng.choice([5, 9])
        case["n"] = size(1500, 200_000 if case["op"] == "rhs" else 60_000)
    return case


# ---------------------------------------------------------------------------------------------------
# inputs: the mesh follows from the case, the state and the species data from the seed
# ---------------------------------------------------------------------------------------------------
@functools.lru_cache(maxsize=8)
def _mesh(flow, n):
    if flow == "sod":
        return box_mesh((n, n), order="morton")
    if flow == "tgv":
        return box_mesh((n, n, n), periodic=(True, True, True), order="morton")
    if flow == "wall":
        return box_mesh((n, n, n), periodic=(False, False, True), order="morton")
    if flow == "shear":
        return box_mesh((n, n, n), periodic=(True, False, True), order="morton")
    return delaunay_mesh(n)


def _gas_state(rho, vel, p):
    return np.concatenate([rho[:, None], (p / (AIR["gamma"] - 1.0) + 0.5 * rho * (vel ** 2).sum(1))[:, None], rho[:, None] * vel], 1)


def _fill_outflow(mesh, U):
    ghost = mesh.cell_kind[mesh.face_cells[:, 1]] == L.CELL_BOUNDARY
    U[mesh.face_cells[ghost, 1]] = U[mesh.face_cells[ghost, 0]]
    return U


def _mixture_case(mesh, eos, T, Y, vel):
    Y = Y / Y.sum(1, keepdims=True)
    rho = 101325.0 / (RU * T * (Y / eos.mw).sum(1))
    return _fill_outflow(mesh, workloads.mixture_state(eos, rho, vel, T, Y))


def _state(case, mesh, seed):
    """(state rows, equation of state) of a case."""
    rng = np.random.default_rng(seed)
    x, nc, flow = mesh.cell_centroid, mesh.n_cells, case["flow"]
    if flow == "sod":
        rho, p = np.where(x[:, 0] < 0.5, 1.0, 0.125), np.where(x[:, 0] < 0.5, 1e5, 1e4)
        for _ in range(8):
            c, a = rng.uniform(0.1, 0.9, 2), rng.uniform(-0.01, 0.01)
            rho = rho * (1.0 + a * np.exp(-((x[:, :2] - c) ** 2).sum(1) / (2 * 0.05 ** 2)))
        return _fill_outflow(mesh, _gas_state(rho, np.zeros((nc, 2)), p)), fv.PerfectGas(AIR)
    if flow == "tgv":
        # the vortex, with noise on the density and pressure as well (a symmetric state ties the limiter)
        return workloads.tgv_state(mesh, seed=seed) * (1.0 + 0.002 * rng.standard_normal((nc, 1))), fv.PerfectGas(AIR)
    if flow == "wall":
        # the inlet flow at Mach 0.3 with 0.5 % noise; no-slip ghosts at y = 0 and 1, outflow ghosts at x
        rho0, V = 101325.0 / (287.0 * 300.0), 0.3 * math.sqrt(1.4 * 287.0 * 300.0)
        rho = rho0 * (1.0 + 0.005 * rng.standard_normal(nc))
        vel = 0.005 * V * rng.standard_normal((nc, 3))
        vel[:, 0] += V
        U = _fill_outflow(mesh, _gas_state(rho, vel, np.full(nc, 101325.0)))
        wall = (x[:, 1] < 0.0) | (x[:, 1] > 1.0)
        U[wall, 2:] *= -1.0
        return U, fv.PerfectGas(AIR)
    ns = case["ns"]
    eos = workloads.synthetic_mixture(ns, seed + 1)
    if flow == "shear":
        t = 0.5 * (1.0 + np.tanh((x[:, 1] - 0.5) / 0.02))
        Y = 0.02 * rng.uniform(0.0, 1.0, (nc, ns))
        Y[:, 0] += 1.0 - t
        Y[:, 1] += t
        vel = rng.standard_normal((nc, 3))
        vel[:, 0] += 50.0 + 100.0 * t
        return _mixture_case(mesh, eos, 300.0 + 600.0 * t, Y, vel), eos
    # layered composition around a hot core, with cell-to-cell noise
    r2 = ((x[:, 1] - 0.1) ** 2 + (x[:, 2] - 0.1) ** 2) / 0.01
    T = 300.0 + 2200.0 * np.exp(-2.0 * r2) * (0.6 + 0.4 * np.sin(2 * np.pi * x[:, 0])) ** 2
    T = np.clip(T * (1.0 + 0.02 * rng.standard_normal(nc)), 300.0, 2500.0)
    Y = np.stack([1.2 + np.cos(2 * np.pi * (k + 1) * x[:, 0] + k) for k in range(ns)], 1)
    Y = 0.8 * Y / Y.sum(1, keepdims=True) + 0.2 * rng.dirichlet(np.full(ns, 2.0), nc)
    vel = np.stack([30.0 * np.sin(10 * np.pi * x[:, 1]), 10.0 * np.cos(2 * np.pi * x[:, 0]), np.full(nc, 5.0)], 1)
    return _mixture_case(mesh, eos, T, Y, vel + 2.0 * rng.standard_normal((nc, 3))), eos


def _solver(case, mesh, eos):
    flow = case["flow"]
    if flow == "sod":
        return fv.FiniteVolumeSolver(mesh, eos, [fv.NavierStokesTransport({"cfl": 0.5}, eos, fv.Ausm())], "upwind", "none")
    flux = fv.AusmpUp(0.3)
    if flow in ("tgv", "wall"):
        ns = fv.NavierStokesTransport({"cfl": 0.5}, eos, flux, fv.Constant(k=MU * CP_AIR / PRANDTL, mu=MU))
        return fv.FiniteVolumeSolver(mesh, eos, [ns], "leastsquares", "minmod")
    tr = fv.ConstantLewis(MU, PRANDTL, 1.0) if flow == "tets" else None
    procs = [fv.NavierStokesTransport({"cfl": 0.5}, eos, flux, tr), fv.SpeciesTransport(eos, flux, tr)]
    return fv.FiniteVolumeSolver(mesh, eos, procs, "leastsquares", "vanleer" if flow == "tets" else "minmod")


def _direction(U, seed):
    """A perturbation (jvp) or weight (vjp) of the rows, each component at its own scale."""
    rng = np.random.default_rng(seed + 77)
    return rng.standard_normal(U.shape) * np.abs(U).mean(0)


def _weight(U, seed):
    rng = np.random.default_rng(seed + 78)
    return rng.standard_normal(U.shape) / np.abs(U).mean(0)


def _dt(case):
    return 1e-4 / case["n"]  # about CFL 0.2 at the shear layer's fastest sound speed


def prepare(case, seed):
    mesh = _mesh(case["flow"], case["n"])
    U, eos = _state(case, mesh, seed)
    s = {"case": case, "solver": _solver(case, mesh, eos)}
    s["prec"] = L.PRECISION_MIXED if case["precision"] == "mixed" else L.PRECISION_FP64
    if case["op"] == "host":
        s["U"], s["F"] = U, np.zeros_like(U)
        return s
    s["U"] = torch.from_numpy(U).cuda()
    s["out"] = torch.empty_like(s["U"])
    if case["ns"]:
        # the temperatures of a running computation: those of the state before a small change
        rng = np.random.default_rng(seed + 5)
        before = s["U"] * torch.from_numpy(1.0 + 1e-3 * rng.standard_normal((U.shape[0], 1))).cuda()
        s["solver"].ComputeRHSDevice(0.0, before.data_ptr(), s["out"].data_ptr(), s["prec"], torch.cuda.current_stream().cuda_stream)
    if case["op"] == "jvp":
        s["dir"] = torch.from_numpy(_direction(U, seed)).cuda()
    elif case["op"] == "vjp":
        s["dir"] = torch.from_numpy(_weight(U, seed)).cuda()
    elif case["op"] == "march":
        s["time"] = torch.zeros((), dtype=torch.float64, device="cuda")
    return s


def run(s):
    solver, op = s["solver"], s["case"]["op"]
    if op == "host":
        s["F"].fill(0.0)
        return solver.ComputeRHSFunction(0.0, s["U"], s["F"], s["prec"])
    stream = torch.cuda.current_stream().cuda_stream
    U, out = s["U"], s["out"]
    if op in ("march", "step"):
        out.copy_(U)
        if op == "step":
            solver.StepDevice(L.STEP_SSPRK3, 0.0, _dt(s["case"]), out.data_ptr(), s["prec"], stream)
            return out
        s["time"].zero_()
        for _ in range(s["case"]["steps"]):
            solver.StepCflDevice(L.STEP_SSPRK3, 0.5, out.data_ptr(), s["prec"], s["time"].data_ptr(), stream)
        return {"U": out, "time": s["time"]}
    out.zero_()
    if op == "rhs":
        solver.ComputeRHSDevice(0.0, U.data_ptr(), out.data_ptr(), s["prec"], stream)
    elif op == "jvp":
        solver.ComputeJVPDevice(0.0, U.data_ptr(), s["dir"].data_ptr(), out.data_ptr(), 0, stream)
    else:
        solver.ComputeVJPDevice(0.0, U.data_ptr(), s["dir"].data_ptr(), out.data_ptr(), stream)
    return out


# ---------------------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------------------
def _counts(case):
    """(cells, faces) of a case, without building its mesh."""
    n = case["n"]
    if case["flow"] == "sod":
        return n * n, 2 * n * (n + 1)
    if case["flow"] == "tets":
        return n, 2 * n
    return n ** 3, 3 * n ** 3


def work(case):
    dim, ns = (2 if case["flow"] == "sod" else 3), case["ns"]
    nc = 2 + dim + ns
    cells, faces = _counts(case)
    # one right-hand side reads the rows, 1/V and per face its two cells and its normal, and writes the rows
    mesh_bytes = cells * 8 + faces * (8 + 8 * dim)
    row = cells * nc * 8
    face = 150 + 20 * ns if case["flow"] == "sod" or case["flow"] == "shear" else 250 + 60 * ns
    if ns:
        face += 2 * 4 * 13 * ns  # four evaluations of the mixture's energy per side
    cell = 0 if case["flow"] == "sod" else 2 * dim * nc * (2 * dim + 12)
    flops = faces * face + cells * (cell + 8 * nc)
    op = case["op"]
    if op in ("rhs", "host"):
        return {"bytes": 2 * row + mesh_bytes, "flops": flops}
    if op in ("march", "step"):
        stages = 3 * case.get("steps", 1)
        # each stage reads the rows and writes them advanced; the mesh is read by each
        return {"bytes": stages * (2 * row + mesh_bytes), "flops": stages * flops}
    return {"bytes": 3 * row + mesh_bytes, "flops": 3 * flops}


def tolerance(case):
    """About four times the largest error against ``exact`` over the ranges of ``draw``. The mixed path
    states 1e-6; a mixture's temperature is solved to 1e-8 J/kg, which its cancelling sums amplify."""
    op, species = case["op"], case["ns"] > 0
    if case["precision"] == "mixed":
        return {"rel": 1e-6}
    if op == "march":
        return {"rel": 1e-15}
    if op == "step":
        return {"rel": 1e-14}
    if case["flow"] == "sod":
        return {"rel": 2e-14}
    if op == "vjp":
        return {"rel": 1e-12 if species else 2e-13}
    return {"rel": 4e-12 if species else 1e-12}


# ---------------------------------------------------------------------------------------------------
# the same results in plain torch, 64 bits
# ---------------------------------------------------------------------------------------------------
class _Geometry:
    """Dense per-cell face lists (every interior cell has the same number of faces on these meshes),
    face offsets and least-squares weights."""

    def __init__(self, mesh, device, gradients):
        t = lambda a, dtype=torch.float64: torch.from_numpy(np.ascontiguousarray(a)).to(device, dtype)
        dim = mesh.dim
        fc = t(mesh.face_cells, torch.int64)
        self.dim, self.n_own, self.n_cells = dim, mesh.n_interior, mesh.n_cells
        self.Lc, self.Rc = fc[:, 0], fc[:, 1]
        self.normal = t(mesh.face_normal[:, :dim])
        cen, cc = t(mesh.face_centroid[:, :dim]), t(mesh.cell_centroid[:, :dim])
        shift = 0.0 if mesh.face_shift is None else t(mesh.face_shift[:, :dim])
        self.dxL, self.dxR = cen - cc[self.Lc], cen - shift - cc[self.Rc]
        self.ivol = 1.0 / t(mesh.cell_volume[:self.n_own])
        nf, K = fc.shape[0], 2 * dim if mesh.shape else dim + 1
        cell = torch.cat([self.Lc, self.Rc])
        face = torch.arange(nf, device=device).repeat(2)
        side = torch.arange(2, device=device).repeat_interleave(nf)
        keep = cell < self.n_own
        cell, face, side = cell[keep], face[keep], side[keep]
        order = torch.argsort(cell, stable=True)
        self.face, side = face[order].view(self.n_own, K), side[order].view(self.n_own, K)
        self.sign = torch.where(side == 1, 1.0, -1.0).to(torch.float64)
        self.nbr = torch.where(side == 0, self.Rc[self.face], self.Lc[self.face])
        dx = self.dxL - self.dxR  # right minus left centroid
        self.rmin = torch.where((side == 0)[..., None], self.dxL[self.face], self.dxR[self.face]).norm(dim=2).amin(1)
        if not gradients:
            return
        self.v = -self.sign[..., None] * dx[self.face]
        inner = (self.nbr < self.n_own).to(torch.float64)[..., None]
        self.ws, self.wa = _pinv(self.v * inner) * inner, _pinv(self.v)
        # a ghost cell's gradient is along the line to its one neighbour
        gf = torch.nonzero(self.Rc >= self.n_own).squeeze(1)
        gf = gf[torch.argsort(self.Rc[gf])]
        self.g_int = self.Lc[gf]
        self.g_w = -dx[gf] / (dx[gf] ** 2).sum(1, keepdim=True)


def _pinv(B):
    """Pseudo-inverse of each cell's neighbour offsets B (n, K, 3), as weights (n, K, 3): by the normal
    equations, refined by Newton-Schulz steps; by eigenvectors where the offsets span fewer directions."""
    A = B.transpose(1, 2) @ B
    r0, r1, r2 = A.unbind(1)
    det = (r0 * torch.linalg.cross(r1, r2)).sum(1)
    scale = (A.diagonal(dim1=1, dim2=2).sum(1) / 3.0) ** 3
    inv = torch.stack([torch.linalg.cross(r1, r2), torch.linalg.cross(r2, r0), torch.linalg.cross(r0, r1)], 1) / det[:, None, None]
    low = torch.nonzero(~(det > 1e-10 * scale)).squeeze(1)
    if low.numel():
        e, V = torch.linalg.eigh(A[low].cpu())
        ie = torch.where(e > 1e-14 * e[:, -1:], 1.0 / e, torch.zeros_like(e))
        inv[low] = (V @ (ie[:, :, None] * V.transpose(1, 2))).to(A.device)
    X = inv @ B.transpose(1, 2)
    for _ in range(2):
        X = 2.0 * X - X @ (B @ X)
    return X.transpose(1, 2).contiguous()


class _Gas:
    def __init__(self, case, eos, device):
        self.ns = case["ns"]
        if not self.ns:
            return
        c = torch.from_numpy(eos.nasa7).to(device)
        self.tm, self.a = c[:, 0], (c[:, 1:8], c[:, 8:15])
        self.imw = 1.0 / torch.from_numpy(eos.mw).to(device)
        self.href = self.h_molar(torch.full((1,), TREF, dtype=torch.float64, device=device))[0] * self.imw

    def coefficients(self, T):
        low = (T[:, None] < self.tm)[..., None]
        return torch.where(low, self.a[0], self.a[1]).unbind(2)

    def h_molar(self, T):
        a, t = self.coefficients(T), T[:, None]
        return RU * (t * (a[0] + t * (a[1] / 2 + t * (a[2] / 3 + t * (a[3] / 4 + t * (a[4] / 5))))) + a[5])

    def cp_mass(self, T):
        a, t = self.coefficients(T), T[:, None]
        return RU * (a[0] + t * (a[1] + t * (a[2] + t * (a[3] + t * a[4])))) * self.imw

    def e_species(self, T):
        return self.h_molar(T) * self.imw - self.href - RU * T[:, None] * self.imw

    def fractions(self, rho, rhoY):
        y = (rhoY[:, :-1] / rho[:, None]).clamp(0.0, 1.0)
        s = y.sum(1, keepdim=True)
        over = s > 1.0
        return torch.cat([torch.where(over, y / s, y), torch.where(over, torch.zeros_like(s), 1.0 - s)], 1)

    def temperature(self, e, Y):
        with torch.no_grad():
            T = torch.full_like(e, 1000.0)
            for _ in range(40):
                cv = (Y * (self.cp_mass(T) - RU * self.imw)).sum(1)
                T = (T - ((self.e_species(T) * Y).sum(1) - e) / cv).clamp(1.0, 1e5)
            cv = (Y * (self.cp_mass(T) - RU * self.imw)).sum(1)
        # one more step carries the derivatives (implicit function theorem)
        return T - ((self.e_species(T) * Y).sum(1) - e) / cv

    def decode(self, U, dim):
        """(e, a, p) of state rows."""
        rho, vel = U[:, 0], U[:, 2:2 + dim] / U[:, :1]
        e = U[:, 1] / rho - 0.5 * (vel ** 2).sum(1)
        if not self.ns:
            p = (AIR["gamma"] - 1.0) * rho * e
            return vel, e, torch.sqrt(AIR["gamma"] * p / rho), p
        Y = self.fractions(rho, U[:, 2 + dim:])
        T = self.temperature(e, Y)
        cp, R = (Y * self.cp_mass(T)).sum(1), RU * (Y * self.imw).sum(1)
        return vel, (self.e_species(T) * Y).sum(1), torch.sqrt(cp / (cp - R) * R * T), rho * R * T

    def aux(self, U, dim):
        """(T, u, Y) of cell rows."""
        rho = U[:, :1]
        vel = U[:, 2:2 + dim] / rho
        e = U[:, 1] / U[:, 0] - 0.5 * (vel ** 2).sum(1)
        if not self.ns:
            return torch.cat([(e * (AIR["gamma"] - 1.0) / AIR["Rgas"])[:, None], vel], 1)
        T = self.temperature(e, self.fractions(U[:, 0], U[:, 2 + dim:]))
        return torch.cat([T[:, None], vel, U[:, 2 + dim:] / rho], 1)


def _ausm(uL, aL, rL, pL, uR, aR, rR, pR):
    mL, mR = uL / aL, uR / aR
    subL, subR = mL.abs() <= 1.0, mR.abs() <= 1.0
    mp = torch.where(subL, 0.25 * (mL + 1.0) ** 2, 0.5 * (mL + mL.abs()))
    mm = torch.where(subR, -0.25 * (mR - 1.0) ** 2, 0.5 * (mR - mR.abs()))
    pp = torch.where(subL, 0.25 * (mL + 1.0) ** 2 * (2.0 - mL), 0.5 * (1.0 + torch.sign(mL)))
    pm = torch.where(subR, 0.25 * (mR - 1.0) ** 2 * (2.0 + mR), 0.5 * (1.0 - torch.sign(mR)))
    m = mp + mm
    left = m >= 0.0
    return torch.where(left, m * aL * rL, m * aR * rR), pR * pm + pL * pp, left


def _ausm_up(uL, aL, rL, pL, uR, aR, rR, pR, minf=0.3):
    r12, a12 = 0.5 * (rL + rR), 0.5 * (aL + aR)
    mL, mR = uL / a12, uR / a12
    mbar2 = (uL ** 2 + uR ** 2) / (2.0 * a12 ** 2)
    mo = torch.sqrt(torch.clamp(torch.clamp(mbar2, min=minf ** 2), max=1.0))
    fa = mo * (2.0 - mo)
    al = 3.0 / 16.0 * (-4.0 + 5.0 * fa ** 2)
    p2 = lambda m: 0.25 * (m + 1.0) ** 2
    m2 = lambda m: -0.25 * (m - 1.0) ** 2
    subL, subR = mL.abs() < 1.0, mR.abs() < 1.0
    mp = torch.where(subL, p2(mL) * (1.0 - 2.0 * m2(mL)), 0.5 * (mL + mL.abs()))
    mm = torch.where(subR, m2(mR) * (1.0 + 2.0 * p2(mR)), 0.5 * (mR - mR.abs()))
    pp = torch.where(subL, p2(mL) * ((2.0 - mL) - 16.0 * al * mL * m2(mL)), 0.5 * (1.0 + torch.sign(mL)))
    pm = torch.where(subR, m2(mR) * ((-2.0 - mR) + 16.0 * al * mR * p2(mR)), 0.5 * (1.0 - torch.sign(mR)))
    m12 = mp + mm - 0.25 / fa * torch.clamp(1.0 - 0.25 * mbar2, min=0.0) * (pR - pL) / (r12 * a12 ** 2)
    left = m12 > 0.0
    p12 = pp * pL + pm * pR - 0.75 * pp * pm * r12 * fa * a12 ** 2 * (mR - mL)
    return a12 * m12 * torch.where(left, rL, rR), p12, left


def _limited(g, case, un, uc, G):
    """Least-squares gradient G (cells, components, 3) times the smallest limiter factor over the faces."""
    den = torch.einsum("ncd,nkd->nkc", G, g.v)
    dif = un - uc[:, None]
    flat = den == 0.0  # a component without a gradient: factor 0
    f = 0.5 * dif / torch.where(flat, torch.ones_like(den), den)
    if case["flow"] == "tets":
        lim = 4.0 * f * (1.0 - f)
    else:
        lim = 4.0 * torch.clamp(torch.minimum(f, 1.0 - f), max=0.25)
    # at f = 0 (an outflow ghost equal to its cell) the factor's derivative is 0
    lim = torch.where(lim > 0.0, lim, torch.zeros_like(lim))
    phi = torch.where(flat, torch.zeros_like(lim), lim).amin(1)
    # a field whose gradient is steeper than 1e10 where its factor is 0 is cancelled
    steep = (phi == 0.0) & (G.detach().abs().amax(2) > 1e10)
    ne = 2 + g.dim
    drop = torch.cat([steep[:, :ne].any(1, keepdim=True).expand(-1, ne), steep[:, ne:].any(1, keepdim=True).expand(-1, phi.shape[1] - ne)], 1)
    return G * torch.where(drop, torch.zeros_like(phi), phi)[..., None]


def _rhs(g, gas, case, U):
    dim, ns, nb = g.dim, gas.ns, g.n_cells - g.n_own
    ne = 2 + dim
    cL, cR = U[g.Lc], U[g.Rc]
    if case["flow"] == "sod":
        uL, uR = cL, cR
    else:
        uc, un = U[:g.n_own], U[g.nbr]
        G = _limited(g, case, un, uc, torch.einsum("nkd,nkc->ncd", g.ws, un - uc[:, None]))
        G = torch.cat([G, G.new_zeros(nb, *G.shape[1:])])
        uL = cL + torch.einsum("fcd,fd->fc", G[g.Lc], g.dxL)
        uR = cR + torch.einsum("fcd,fd->fc", G[g.Rc], g.dxR)
    area = g.normal.norm(dim=1)
    unit = g.normal / area[:, None]
    (vL, eL, aL, pL), (vR, eR, aR, pR) = gas.decode(uL, dim), gas.decode(uR, dim)
    calc = _ausm if case["flow"] == "sod" else _ausm_up
    mf, p12, left = calc((vL * unit).sum(1), aL, uL[:, 0], pL, (vR * unit).sum(1), aR, uR[:, 0], pR)
    mA = mf * area
    up = torch.where(left[:, None], uL, uR)
    vel = torch.where(left[:, None], vL, vR)
    H = torch.where(left, eL + pL / uL[:, 0], eR + pR / uR[:, 0]) + 0.5 * (vel ** 2).sum(1)
    flux = [mA[:, None], (H * mA)[:, None], vel * mA[:, None] + p12[:, None] * g.normal]
    if ns:
        flux.append(mA[:, None] * up[:, ne:] / up[:, :1])
    flux = torch.cat(flux, 1)
    if case["flow"] in ("tgv", "wall", "tets"):
        A = gas.aux(U, dim)
        GA = torch.einsum("nkd,nkc->ncd", g.wa, A[g.nbr] - A[:g.n_own, None])
        if nb:
            GA = torch.cat([GA, (A[g.g_int] - A[g.n_own:])[:, :, None] * g.g_w[:, None]])
        Gf, Af, Uf = 0.5 * (GA[g.Lc] + GA[g.Rc]), 0.5 * (A[g.Lc] + A[g.Rc]), 0.5 * (cL + cR)
        if ns:
            cp = (gas.fractions(Uf[:, 0], Uf[:, ne:]) * gas.cp_mass(Af[:, 0])).sum(1)
            k = MU * cp / PRANDTL
        else:
            k = torch.full_like(mA, MU * CP_AIR / PRANDTL)
        gv = Gf[:, 1:1 + dim]
        tau = MU * (gv + gv.transpose(1, 2) - 2.0 / 3.0 * torch.diag_embed(gv.diagonal(dim1=1, dim2=2).sum(1, keepdim=True).expand(-1, dim)))
        tn = torch.einsum("fcd,fd->fc", tau, g.normal)
        en = (Af[:, 1:1 + dim] * tn).sum(1) + k * (Gf[:, 0] * g.normal).sum(1)
        dif = [torch.zeros_like(en)[:, None], -en[:, None], -tn]
        if ns:
            # rho D = k / cp = mu / Pr at Lewis number 1
            yn = -MU / PRANDTL * torch.einsum("fcd,fd->fc", Gf[:, 1 + dim:], g.normal)
            hs = gas.h_molar(Af[:, 0]) * gas.imw - gas.href
            dif[1] = dif[1] + (yn * hs).sum(1, keepdim=True)
            dif.append(yn)
        flux = flux + torch.cat(dif, 1)
    F = (g.sign[..., None] * flux[g.face]).sum(1) * g.ivol[:, None]
    return torch.cat([F, F.new_zeros(nb, F.shape[1])])


def _outflow(g, U):
    if g.n_cells == g.n_own:
        return U
    ghost = torch.nonzero(g.Rc >= g.n_own).squeeze(1)
    U = U.clone()
    U[g.Rc[ghost]] = U[g.Lc[ghost]]
    return U


def _ssprk3(g, gas, case, U, dt):
    own = torch.arange(g.n_cells, device=U.device)[:, None] < g.n_own
    stage = lambda a, b, V: _outflow(g, torch.where(own, a * U + b * (V + dt * _rhs(g, gas, case, V)), V))
    U = _outflow(g, U)
    U1 = stage(0.0, 1.0, U)
    U1 = stage(0.75, 0.25, U1)
    U1 = stage(1.0 / 3.0, 2.0 / 3.0, U1)
    if gas.ns:
        rho, k = U1[:, :1], 2 + g.dim
        y = (U1[:, k:-1] / rho).clamp(0.0, 1.0)
        s = y.sum(1, keepdim=True)
        y = torch.where(s > 1.0, torch.cat([y / s, torch.zeros_like(s)], 1), torch.cat([y, 1.0 - s], 1))
        U1 = _outflow(g, torch.cat([U1[:, :k], torch.where(own, rho * y, U1[:, k:])], 1))
    return U1


def exact(case, seed):
    mesh = _mesh(case["flow"], case["n"])
    rows, eos = _state(case, mesh, seed)
    device = "cuda" if torch.cuda.is_available() else "cpu"
    g, gas = _Geometry(mesh, device, case["flow"] != "sod"), _Gas(case, eos, device)
    U, op = torch.from_numpy(rows).to(device), case["op"]
    if op == "jvp":
        # J d through two reverse passes: d/dw of <w^T J, d>
        U.requires_grad_(True)
        d = torch.from_numpy(_direction(rows, seed)).to(device)
        w = torch.zeros_like(U, requires_grad=True)
        (wJ,) = torch.autograd.grad((w * _rhs(g, gas, case, U)).sum(), U, create_graph=True)
        return torch.autograd.grad((wJ * d).sum(), w)[0]
    if op == "vjp":
        U.requires_grad_(True)
        w = torch.from_numpy(_weight(rows, seed)).to(device)
        return torch.autograd.grad((w * _rhs(g, gas, case, U)).sum(), U)[0]
    with torch.no_grad():
        if op == "step":
            return _ssprk3(g, gas, case, U, _dt(case))
        if op == "march":
            time = torch.zeros((), dtype=torch.float64, device=device)
            for _ in range(case["steps"]):
                vel, _, a, _ = gas.decode(U[:g.n_own], g.dim)
                dt = (0.5 * 2.0 * g.rmin / (a + vel.abs().sum(1))).amin()
                U, time = _ssprk3(g, gas, case, U, dt), time + dt
            return {"U": U, "time": time}
        F = _rhs(g, gas, case, U)
    return F.cpu().numpy() if op == "host" else F
