"""Performance cases of the framework: the calls a user's program makes, at the sizes it makes them.

Seven kinds of call, each over the range of grids it meets (30x10x10 elements, the plain
cantilever, to 256x128x128, the large one; aspect ratios near 2:1:1, ragged sizes among them):

  apply    K u on a problem handle, FP64 or FP32 (the matrix-free operator by itself)
  solve    K U = F for one load: Jacobi-PCG, MG-PCG with the default hierarchy, or FP64
           PCG with the FP32 multigrid preconditioner
  batch    K U_k = F_k for several loads at once
  simp     one iteration of the 3D design loop on device arrays
  simp2d   one iteration of the 2D design loop
  adjoint  the differentiable objective, forward and backward, through autograd
  update   what follows a solve: element energies, sensitivities, filter, OC update

Density fields are sums of 16 cosines with seeded wave numbers and phases ("late": clipped to
[1e-3, 1], so that some elements are inactive; "mid" and "early": milder contrast, as in the
earlier iterations of a run).  Grids of the design loop and of the mixed-precision solver have
sizes that coarsen (multiples of 2 or 4), as a program would choose them; the other kinds take
odd sizes too.  Everything is made from the seed on the device.
"""
import math

import numpy as np
import torch

from topologyoptimization_b200 import Problem, adjoint, mesh, worker2d
from topologyoptimization_b200 import _native as N

E0, EMIN, NU = 1.0, 1e-9, 0.3


def listed():
    return [
        # one operator apply on the plain cantilever's grid: launch latency
        {"name": "apply_f64_30x10x10", "kind": "apply", "nx": 30, "ny": 10, "nz": 10, "dtype": "f64"},
        # the operator microbenchmark's grid
        {"name": "apply_f64_128x64x64", "kind": "apply", "nx": 128, "ny": 64, "nz": 64, "dtype": "f64"},
        # the operator of the FP32 preconditioner on the large grid
        {"name": "apply_f32_256x128x128", "kind": "apply", "nx": 256, "ny": 128, "nz": 128, "dtype": "f32"},
        # the plain cantilever's FE solve with the default Jacobi solver
        {"name": "solve_cg_30x10x10", "kind": "solve", "nx": 30, "ny": 10, "nz": 10, "solver": "cg"},
        # a desktop-sized FE solve with the default multigrid hierarchy
        {"name": "solve_mgpcg_64x32x32", "kind": "solve", "nx": 64, "ny": 32, "nz": 32, "solver": "mgpcg"},
        # a mid-sized FE solve with the mixed-precision solver, coarse levels of odd size
        {"name": "solve_mixed_150x74x78", "kind": "solve", "nx": 150, "ny": 74, "nz": 78, "solver": "mixed", "stage": "mid"},
        # eight load cases of one design
        {"name": "batch8_160x80x80", "kind": "batch", "nx": 160, "ny": 80, "nz": 80, "nrhs": 8},
        # an iteration of the design loop with the worker's defaults (projection, MG-PCG)
        {"name": "simp_mgpcg_60x20x20", "kind": "simp", "nx": 60, "ny": 20, "nz": 20, "solver": "mgpcg"},
        # an iteration of the design loop on the large grid with the mixed-precision solver
        {"name": "simp_mixed_256x128x128", "kind": "simp", "nx": 256, "ny": 128, "nz": 128, "solver": "mixed",
         "stage": "late"},
        # an iteration of the 2D worker
        {"name": "simp2d_300x100", "kind": "simp2d", "nx": 300, "ny": 100},
        # the differentiable displacement objective with an output spring (two solves)
        {"name": "adjoint_96x48x48", "kind": "adjoint", "nx": 96, "ny": 48, "nz": 48},
        # the design update after a solve, a grid with a ragged edge on every axis
        {"name": "update_201x99x103", "kind": "update", "nx": 201, "ny": 99, "nz": 103, "rmin": 2.5},
    ]


# smallest and largest element count of each kind's grids
_RANGE = {"apply": (3e3, 4.1e6), "cg": (3e3, 2.5e4), "mgpcg": (3e3, 1.5e5), "mixed": (3e4, 2.5e6), "batch": (3e4, 9e5),
          "simp mgpcg": (3e3, 8e4), "simp mixed": (3e4, 3e6), "simp2d": (1.5e3, 2.9e4), "adjoint": (3e4, 2.4e5),
          "update": (3e3, 4.1e6)}


def draw(rng):
    kind = rng.choice(["apply", "apply", "apply", "solve", "solve", "solve", "batch", "simp", "simp", "simp2d", "adjoint",
                       "update"])
    case = {"kind": kind}
    if kind == "apply":
        case["dtype"] = rng.choice(["f64", "f32"])
    elif kind == "solve":
        case["solver"] = rng.choice(["cg", "mgpcg", "mixed"])
    elif kind == "simp":
        case["solver"] = rng.choice(["mgpcg", "mixed"])
    elif kind == "batch":
        case["nrhs"] = rng.randint(2, 8)
    elif kind == "update":
        case["rmin"] = rng.choice([1.5, 2.0, 2.5, 3.0])
    lo, hi = _RANGE[{"solve": case.get("solver"), "simp": "simp " + case.get("solver", "")}.get(kind, kind)]
    nel = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    if kind == "simp2d":
        r = rng.uniform(0.3, 0.6)
        case["nx"] = max(4, round(math.sqrt(nel / r)))
        case["ny"] = max(4, round(r * case["nx"]))
        return case
    ry, rz = rng.uniform(0.4, 0.6), rng.uniform(0.4, 0.6)
    nx = (nel / (ry * rz)) ** (1 / 3)
    mixed = case.get("solver") == "mixed"
    if mixed:
        case["stage"] = "mid" if kind == "solve" else rng.choice(["mid", "late"])
    # a design loop's grid has even sizes: with odd ones the default hierarchy may not converge
    step = (2 if case["stage"] == "mid" else 4) if mixed else 2 if kind == "simp" else 1
    nx, ny, nz = (max(4, step * round(n / step)) for n in (nx, ry * nx, rz * nx))
    case.update(nx=max(8, nx), ny=ny, nz=nz)
    return case


# ---- inputs ------------------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _cosines(dims, seed):
    """Sum of 16 cosines over the element centres, unit variance; x fastest."""
    rng = np.random.default_rng(int(seed))
    S = torch.zeros(tuple(reversed(dims)), dtype=torch.float64, device="cuda")
    axes = [(torch.arange(n, dtype=torch.float64, device="cuda") + 0.5) * (2 * math.pi / n) for n in dims]
    for _ in range(16):
        k = rng.integers(1, 5, size=len(dims))
        a = float(rng.uniform(0, 2 * math.pi))
        arg = torch.full((), a, dtype=torch.float64, device="cuda")
        for i, t in enumerate(axes):
            shape = [1] * len(dims)
            shape[len(dims) - 1 - i] = -1
            arg = arg + (float(k[i]) * t).reshape(shape)
        S += torch.cos(arg)
    return S / math.sqrt(8)


def _density(dims, seed, stage):
    S = _cosines(dims, seed)
    mean, amp, floor = {"late": (0.5, 0.25, 1e-3), "mid": (0.5, 0.15, 0.1), "early": (0.4, 0.1, 0.1)}[stage]
    return torch.clamp(mean + amp * S, floor, 1.0).float().reshape(-1)


def _dims(case):
    return (case["nx"], case["ny"], case["nz"])


def _design(case, seed, stage, load):
    """Design and preserved mask: the elements under the support and the load stay solid."""
    nx, ny, nz = _dims(case)
    pres = torch.zeros((nz, ny, nx), dtype=torch.uint8, device="cuda")
    pres[:, :, 0] = 1
    if load == "line":
        pres[0, :, nx - 1] = 1
    else:
        pres[nz - 1, ny - 1, nx - 1] = 1
    pres = pres.reshape(-1)
    x = _density(_dims(case), seed, stage)
    x[pres == 1] = 1.0
    return x, pres


def _load(case, load):
    nx, ny, nz = _dims(case)
    if load == "point":
        return mesh.load_vector(nx, ny, nz, "down").astype(np.float64)
    F = np.zeros(mesh.ndof(nx, ny, nz))
    F[3 * mesh.node_id(nx, np.arange(ny + 1), 0, ny, nz) + 2] = -1.0
    return F


def _mg(solver):
    if solver == "mixed":
        return N.default_mg_opts(coarse_direct=1, safe_omega=1, chebyshev=1, cheb_ratio=16.0, max_levels=6)
    return N.default_mg_opts()


def _solve_opts(solver, tol):
    if solver == "mixed":
        return N.default_solve_opts(precond=N.PREC_MG, precision=N.F32_PRECOND, max_iter=2000, tol=tol, ref_epsilon=0)
    prec = N.PREC_MG if solver == "mgpcg" else N.PREC_JACOBI
    return N.default_solve_opts(precond=prec, max_iter=400 if solver == "mgpcg" else 2000, tol=tol, ref_epsilon=0)


def _setting(case):
    """(stage, load, penal, tol) of a case with a solve: the mixed solver takes a developed
    design, the default ones one of the first iterations."""
    if case.get("solver") == "mixed":
        return case["stage"], "line", 3.0, 1e-8
    if case["kind"] == "simp":
        return "early", "point", 2.0, 2e-5
    return "early", "line", 2.0, 1e-8


def _point_loads(case, seed):
    """Unit point loads in random directions at random nodes of the face z = nz."""
    nx, ny, nz = _dims(case)
    F = np.zeros((case["nrhs"], mesh.ndof(nx, ny, nz)))
    rng = np.random.default_rng(int(seed))
    for k in range(case["nrhs"]):
        n = int(mesh.node_id(int(rng.integers(0, nx + 1)), int(rng.integers(0, ny + 1)), nz, ny, nz))
        d = rng.standard_normal(3)
        F[k, 3 * n:3 * n + 3] = d / np.linalg.norm(d)
    return torch.from_numpy(F).cuda()


def _bending(case, seed):
    """A displacement field: a bending cantilever with a seeded perturbation of its nodes."""
    nx, ny, nz = _dims(case)
    d = {"dtype": torch.float64, "device": "cuda"}
    X = torch.arange(nx + 1, **d).reshape(-1, 1, 1)
    Y = torch.arange(ny + 1, **d).reshape(1, -1, 1)
    Z = torch.arange(nz + 1, **d).reshape(1, 1, -1)
    L = float(nx)
    U = torch.empty((nx + 1, ny + 1, nz + 1, 3), **d)
    w = -(X * X) * (3 * L - X) / (L ** 3)
    dw = -(6 * L * X - 3 * X * X) / (L ** 3)
    U[..., 0] = -(Z - nz / 2) * dw
    U[..., 1] = 0.3 * (Y - ny / 2) * (Z - nz / 2) * (L - X) / L ** 2
    U[..., 2] = w + 0.0 * Y + 0.0 * Z
    U += 0.02 / L * torch.randn(U.shape, generator=_gen(seed + 1), **d)
    return U.reshape(-1)


def _output_dof(case):
    nx, ny, nz = _dims(case)
    return int(3 * mesh.node_id(nx, ny // 2, nz, ny, nz) + 2)


def _problem(case, solver, support="left"):
    nx, ny, nz = _dims(case)
    return Problem(nx, ny, nz, mesh.fixed_mask(nx, ny, nz, support), nu=NU, mg=_mg(solver))


def _apply_inputs(case, seed):
    nx, ny, nz = _dims(case)
    x = (1e-3 + (1 - 1e-3) * torch.rand(nx * ny * nz, generator=_gen(seed), dtype=torch.float64, device="cuda")).float()
    u = torch.randn(mesh.ndof(nx, ny, nz), generator=_gen(seed + 1), dtype=torch.float64, device="cuda")
    u[:3 * (ny + 1) * (nz + 1)] = 0.0
    return x, u.float() if case["dtype"] == "f32" else u


def _beta_2d(case):
    return 2.0


def _inputs_2d(case, seed):
    nx, ny = case["nx"], case["ny"]
    x = torch.clamp(0.45 + 0.12 * _cosines((nx, ny), seed), 0.1, 1.0).float()  # [y, x]
    x = x.t().contiguous().reshape(-1)  # the 2D worker's order: y fastest
    pres = np.zeros(nx * ny, np.uint8)
    pres[mesh.constraint_elements2d(nx, ny, "left")] = 1
    pres[mesh.force_elements2d(nx, ny, "down")] = 1
    pres = torch.from_numpy(pres).cuda()
    x[pres == 1] = 1.0
    return x, pres


def _volfrac(x):
    """The volume the design has: OC keeps it."""
    return float(x.double().mean())


# ---- prepare and run ---------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind}
    if kind == "simp2d":
        nx, ny = case["nx"], case["ny"]
        x, s["pres"] = _inputs_2d(case, seed)
        P = worker2d.Problem2D(nx, ny, mesh.fixed_mask2d(nx, ny, "left"), nu=NU)
        P.set_load(mesh.load_vector2d(nx, ny, "down").astype(np.float64))
        s["opts"] = N.SimpOpts2D(volfrac=_volfrac(x), penal=2.0, rmin=1.5, E0=E0, Emin=EMIN, beta=_beta_2d(case),
                                 use_projection=1, cg_tol=2e-3, cg_max_iter=worker2d.MAX_CG_ITERATIONS)
        s.update(P=P, x0=x, x=x.clone())
        return s
    if kind == "apply":
        P = _problem(case, "mgpcg")
        x, u = _apply_inputs(case, seed)
        P.set_densities(x, 3.0, E0, EMIN)
        s.update(P=P, u=u, out=torch.empty_like(u), call=P.apply_f32_dev if case["dtype"] == "f32" else P.apply_dev)
        return s
    if kind == "batch":
        P = _problem(case, "mixed", "bottom-corners")
        P.set_densities(torch.full((P.nel,), 0.2, device="cuda"), 3.0, E0, EMIN)
        F = _point_loads(case, seed)
        s.update(P=P, F=F, U=torch.zeros_like(F), opts=_solve_opts("mixed", 1e-8))
        return s
    if kind == "update":
        P = _problem(case, "mgpcg")
        x = _density(_dims(case), seed, "late")
        f = {"dtype": torch.float32, "device": "cuda"}
        s.update(P=P, x=x, U=_bending(case, seed), rmin=case["rmin"], volfrac=_volfrac(x), energy=torch.empty(P.nel, **f),
                 dc=torch.empty(P.nel, **f), dcn=torch.empty(P.nel, **f), xnew=torch.empty(P.nel, **f))
        return s
    if kind == "adjoint":
        P = _problem(case, "mixed")
        P.set_spring(_output_dof(case), 0.1)
        P.set_load(_load(case, "line"))
        x, _ = _design(case, seed, "early", "line")
        l = torch.zeros(P.ndof, dtype=torch.float64, device="cuda")
        l[_output_dof(case)] = 1.0
        s.update(P=P, x=x.double(), l=l, design=adjoint.design_opts(penal=3.0, E0=E0, Emin=EMIN, filter_radius=2.0),
                 opts=N.default_solve_opts(precond=N.PREC_MG, max_iter=2000, tol=1e-8, ref_epsilon=0))
        return s
    stage, load, penal, tol = _setting(case)
    P = _problem(case, case["solver"])
    P.set_load(_load(case, load))
    x, pres = _design(case, seed, stage, load)
    if kind == "solve":
        P.set_densities(x, penal, E0, EMIN)
        s.update(P=P, U=torch.zeros(P.ndof, dtype=torch.float64, device="cuda"), opts=_solve_opts(case["solver"], tol))
        return s
    proj = case["solver"] != "mixed"
    s["opts"] = N.SimpOpts(volfrac=_volfrac(x), penal=penal, rmin=1.5, E0=E0, Emin=EMIN, beta=2.0 if proj else 1.0,
                           use_projection=int(proj), guard_sensitivities=int(not proj),
                           solve=_solve_opts(case["solver"], tol))
    s.update(P=P, x0=x, x=x.clone(), pres=pres)
    return s


def run(s):
    P, kind = s["P"], s["kind"]
    if kind == "apply":
        s["call"](s["u"], s["out"])
        return s["out"]
    if kind == "solve":
        P.solve_dev(s["U"], s["opts"])
        return s["U"]
    if kind == "batch":
        P.solve_multi_dev(s["F"], s["U"], s["opts"])
        return s["U"]
    if kind in ("simp", "simp2d"):
        s["x"].copy_(s["x0"])  # the step updates the design in place
        info = P.simp_step_dev(s["x"], s["opts"], s["pres"])
        return {"x": s["x"], "compliance": info.compliance, "change": info.change}
    if kind == "update":
        P.element_energy_dev(s["U"], s["energy"])
        P.sensitivity_dev(s["x"], s["x"], s["energy"], 3.0, E0, 1.0, False, s["dc"])
        P.filter_sens_dev(s["rmin"], s["x"], s["dc"], s["dcn"])
        change, _, _ = P.oc_update_dev(s["x"], s["dcn"], s["xnew"], s["volfrac"])
        return {"energy": s["energy"], "dc": s["dc"], "dcn": s["dcn"], "x": s["xnew"], "change": change}
    x = s["x"].detach().requires_grad_(True)
    J = adjoint.FEObjective().apply(x, P, s["design"], s["opts"], s["l"])
    J.backward()
    return {"J": J.detach(), "grad": x.grad}


def work(case):
    """Inputs read once, outputs written once (a solve's iterations are not counted)."""
    if case["kind"] == "simp2d":
        nel, ndof = case["nx"] * case["ny"], mesh.ndof2d(case["nx"], case["ny"])
        return {"bytes": 8 * nel + 16 * ndof, "flops": 2 * 64 * nel}
    nx, ny, nz = _dims(case)
    nel, ndof = nx * ny * nz, mesh.ndof(nx, ny, nz)
    if case["kind"] == "apply":
        return {"bytes": (4 if case["dtype"] == "f32" else 8) * (2 * ndof + nel), "flops": 140 * nel}
    if case["kind"] == "update":
        return {"bytes": 8 * ndof + 20 * nel, "flops": 140 * nel}
    k = case.get("nrhs", 1)
    return {"bytes": 8 * nel + 16 * ndof * k, "flops": 140 * nel * k}


# ---- the same in plain 64-bit torch -------------------------------------------------------
def _hex_ke():
    """Element matrix of the reference: 2x2x2 Gauss points in natural coordinates, unit
    Jacobian (js/optimizer-worker-3d.js lk())."""
    f = E0 / ((1 + NU) * (1 - 2 * NU))
    C = np.zeros((6, 6))
    C[:3, :3] = f * NU
    C[range(3), range(3)] = f * (1 - NU)
    C[range(3, 6), range(3, 6)] = f * (1 - 2 * NU) / 2
    sg = 2.0 * mesh.CORNERS - 1.0
    K = np.zeros((24, 24))
    for gx in (-1, 1):
        for gy in (-1, 1):
            for gz in (-1, 1):
                p = np.array([gx, gy, gz]) / math.sqrt(3.0)
                t = 1 + sg * p
                dN = 0.125 * np.stack([sg[:, 0] * t[:, 1] * t[:, 2], t[:, 0] * sg[:, 1] * t[:, 2],
                                       t[:, 0] * t[:, 1] * sg[:, 2]], 1)
                B = np.zeros((6, 24))
                B[0, 0::3], B[1, 1::3], B[2, 2::3] = dN[:, 0], dN[:, 1], dN[:, 2]
                B[3, 0::3], B[3, 1::3] = dN[:, 1], dN[:, 0]
                B[4, 1::3], B[4, 2::3] = dN[:, 2], dN[:, 1]
                B[5, 0::3], B[5, 2::3] = dN[:, 2], dN[:, 0]
                K += B.T @ C @ B
    return torch.from_numpy(K).cuda()


class _Plain:
    """K u = sum over active elements of E_e Ke u_e by gather, matrix product and index_add."""

    def __init__(self, dims, Ke, edofs, ndof, spring=None):
        self.Ke, self.ed, self.ndof, self.spring = Ke, edofs, ndof, spring
        self.nel, self.es = edofs.shape

    @classmethod
    def hex(cls, dims, spring=None):
        nx, ny, nz = dims
        d = {"device": "cuda", "dtype": torch.int64}
        ex = torch.arange(nx, **d).reshape(1, 1, -1, 1)
        ey = torch.arange(ny, **d).reshape(1, -1, 1, 1)
        ez = torch.arange(nz, **d).reshape(-1, 1, 1, 1)
        c = torch.from_numpy(mesh.CORNERS).cuda()
        nodes = ((ex + c[:, 0]) * (ny + 1) + ey + c[:, 1]) * (nz + 1) + ez + c[:, 2]
        ed = (3 * nodes.reshape(-1, 8, 1) + torch.arange(3, **d)).reshape(-1, 24)
        return cls(dims, _hex_ke(), ed, 3 * (nx + 1) * (ny + 1) * (nz + 1), spring)

    @classmethod
    def quad(cls, dims):
        nx, ny = dims
        k = [0.5 - NU / 6, 0.125 + NU / 8, -0.25 - NU / 12, -0.125 + 3 * NU / 8, -0.25 + NU / 12, -0.125 - NU / 8,
             NU / 6, 0.125 - 3 * NU / 8]
        o = [[0, 1, 2, 3, 4, 5, 6, 7], [1, 0, 7, 6, 5, 4, 3, 2], [2, 7, 0, 5, 6, 3, 4, 1], [3, 6, 5, 0, 7, 2, 1, 4],
             [4, 5, 6, 7, 0, 1, 2, 3], [5, 4, 3, 2, 1, 0, 7, 6], [6, 3, 4, 1, 2, 7, 0, 5], [7, 2, 1, 4, 3, 6, 5, 0]]
        Ke = torch.tensor([[k[j] for j in r] for r in o], dtype=torch.float64, device="cuda") / (1 - NU * NU)
        d = {"device": "cuda", "dtype": torch.int64}
        n1 = ((ny + 1) * torch.arange(nx, **d).reshape(-1, 1) + torch.arange(ny, **d)).reshape(-1)
        n2 = n1 + ny + 1
        ed = torch.stack([2 * n1, 2 * n1 + 1, 2 * n2, 2 * n2 + 1, 2 * n2 + 2, 2 * n2 + 3, 2 * n1 + 2, 2 * n1 + 3], 1)
        return cls(dims, Ke, ed, 2 * (nx + 1) * (ny + 1))

    def moduli(self, x, penal):
        E = EMIN + x.double() ** penal * (E0 - EMIN)
        return torch.where(E > 1000 * EMIN, E, torch.zeros_like(E))

    def apply(self, E, u):
        out = torch.zeros(self.ndof, dtype=torch.float64, device="cuda")
        for a in range(0, self.nel, 1 << 20):
            ed = self.ed[a:a + (1 << 20)]
            out.index_add_(0, ed.reshape(-1), ((u[ed] @ self.Ke) * E[a:a + (1 << 20), None]).reshape(-1))
        if self.spring:
            out[self.spring[0]] += self.spring[1] * u[self.spring[0]]
        return out

    def inv_diagonal(self, E, free):
        dg = torch.zeros(self.ndof, dtype=torch.float64, device="cuda")
        dg.index_add_(0, self.ed.reshape(-1), (E[:, None] * torch.diagonal(self.Ke)).reshape(-1))
        if self.spring:
            dg[self.spring[0]] += self.spring[1]
        return torch.where(free & (dg > 1e-30), 1.0 / dg, torch.zeros_like(dg))

    def energy(self, u, v):
        out = torch.empty(self.nel, dtype=torch.float64, device="cuda")
        for a in range(0, self.nel, 1 << 20):
            ed = self.ed[a:a + (1 << 20)]
            out[a:a + (1 << 20)] = ((u[ed] @ self.Ke) * v[ed]).sum(1)
        return out

    def solve(self, E, F, free, tol=1e-13, cap=40000, absolute=None, eps=0.0):
        """Jacobi-PCG from zero; `absolute` and `eps`: the 2D worker's stop and shifts."""
        D = self.inv_diagonal(E, free)
        m = free.double()
        U, r = torch.zeros_like(F), F * m
        z = D * r
        p, rz, stop = z.clone(), r @ z, (tol ** 2) * (r @ r) if absolute is None else torch.tensor(absolute ** 2).cuda()
        every = 50 if absolute is None else 1
        for i in range(cap):
            if i % every == 0 and bool((r @ r) < stop):
                break
            Ap = self.apply(E, p) * m
            a = rz / (p @ Ap + eps)
            U += a * p
            r -= a * Ap
            z = D * r
            new = r @ z
            p = z + (new / (rz + eps)) * p
            rz = new
        return U


def _free(mask):
    return torch.from_numpy(np.asarray(mask) == 0).cuda()


def _shifted(a, off):
    """a moved by off along each axis, zero outside."""
    out = torch.zeros_like(a)
    src = tuple(slice(max(0, o), a.shape[i] + min(0, o)) for i, o in enumerate(off))
    dst = tuple(slice(max(0, -o), a.shape[i] + min(0, -o)) for i, o in enumerate(off))
    out[dst] = a[src]
    return out


def _offsets(R, nd):
    r = range(-R, R + 1)
    return [(i, j) for i in r for j in r] if nd == 2 else [(i, j, k) for i in r for j in r for k in r]


def _stencil(a, radius, R):
    """(sum of (radius - dist) a_j, sum of (radius - dist)) over dist <= radius."""
    one, num, den = torch.ones_like(a), torch.zeros_like(a), torch.zeros_like(a)
    for off in _offsets(R, a.dim()):
        d = math.sqrt(sum(o * o for o in off))
        if d <= radius:
            num += (radius - d) * _shifted(a, off)
            den += (radius - d) * _shifted(one, off)
    return num, den


def _filter_sens(x, dc, rmin):
    num, den = _stencil(x * dc, rmin, int(math.floor(rmin)))
    return num / (den * torch.clamp(x, min=1e-3))


def _project(x, beta):
    t = math.tanh(beta * 0.5)
    th = torch.tanh(beta * (x - 0.5))
    return (t + th) / (2 * t), beta * (1 - th * th) / (2 * t)


def _oc(x, dc, volfrac, pres=None, move=0.2):
    l1, l2, new = 0.0, 1e9, x
    while (l2 - l1) / (l2 + l1) > 1e-3:
        lmid = 0.5 * (l2 + l1)
        new = torch.minimum(torch.clamp(x + move, max=1.0), x * torch.sqrt(-dc / lmid))
        new = torch.clamp(torch.maximum(x - move, new), min=0.0)
        if pres is not None:
            new = torch.where(pres == 1, torch.ones_like(new), new)
        if float(new.sum()) > volfrac * x.numel():
            l1 = lmid
        else:
            l2 = lmid
    return new


def _step(plain, x, E_of, U, penal, rmin, beta, proj, guard, shape, volfrac, pres):
    """Sensitivities, filter, OC and change of a design step with the displacements U."""
    x = x.double()
    xp, dp = _project(x, beta) if proj else (x, torch.ones_like(x))
    en = plain.energy(U, U)
    if guard:
        en = torch.clamp(en, min=0.0)
    dc = -penal * xp ** (penal - 1) * E0 * en * dp
    dcn = _filter_sens(x.reshape(shape), dc.reshape(shape), rmin).reshape(-1)
    new = _oc(x, dcn, volfrac, pres)
    return new, float((new - x).abs().max())


def exact(case, seed):
    kind = case["kind"]
    if kind == "simp2d":
        nx, ny = case["nx"], case["ny"]
        x, pres = _inputs_2d(case, seed)
        plain, beta = _Plain.quad((nx, ny)), _beta_2d(case)
        F = torch.from_numpy(mesh.load_vector2d(nx, ny, "down").astype(np.float64)).cuda()
        E = plain.moduli(_project(x.double(), beta)[0], 2.0)
        free = _free(mesh.fixed_mask2d(nx, ny, "left"))
        U = plain.solve(E, F, free, cap=min(worker2d.MAX_CG_ITERATIONS, int(free.sum())), absolute=2e-3, eps=1e-12)
        new, change = _step(plain, x, E, U, 2.0, 1.5, beta, True, False, (nx, ny), _volfrac(x), pres)
        return {"x": new, "compliance": float(F @ U), "change": change}
    nx, ny, nz = _dims(case)
    nel, shape = nx * ny * nz, (nz, ny, nx)
    if kind == "apply":
        x, u = _apply_inputs(case, seed)
        plain = _Plain.hex(_dims(case))
        return plain.apply(plain.moduli(x, 3.0), u.double())
    if kind == "update":
        x, U = _density(_dims(case), seed, "late"), _bending(case, seed)
        plain = _Plain.hex(_dims(case))
        en = plain.energy(U, U)
        dc = -3.0 * x.double() ** 2 * E0 * en
        dcn = _filter_sens(x.double().reshape(shape), dc.reshape(shape), case["rmin"]).reshape(-1)
        new = _oc(x.double(), dcn, _volfrac(x))
        return {"energy": en, "dc": dc, "dcn": dcn, "x": new, "change": float((new - x.double()).abs().max())}
    if kind == "batch" or nel > 3e5:
        return None  # a plain solve of this size takes too long
    free = _free(mesh.fixed_mask(nx, ny, nz, "left"))
    if kind == "adjoint":
        out = _output_dof(case)
        plain = _Plain.hex(_dims(case), spring=(out, 0.1))
        x, _ = _design(case, seed, "early", "line")
        num, den = _stencil(x.double().reshape(shape), 2.0, 2)
        xp = (num / den).reshape(-1)
        E = plain.moduli(xp, 3.0)
        U = plain.solve(E, torch.from_numpy(_load(case, "line")).cuda(), free)
        l = torch.zeros(plain.ndof, dtype=torch.float64, device="cuda")
        l[out] = 1.0
        lam = plain.solve(E, l, free)
        g = -3.0 * xp ** 2 * (E0 - EMIN) * plain.energy(lam, U)
        return {"J": U[out].clone(), "grad": _stencil(g.reshape(shape) / den, 2.0, 2)[0].reshape(-1)}
    stage, load, penal, _ = _setting(case)
    plain = _Plain.hex(_dims(case))
    x, pres = _design(case, seed, stage, load)
    proj = kind == "simp" and case["solver"] != "mixed"
    xp = _project(x.double(), 2.0)[0] if proj else x.double()
    E, F = plain.moduli(xp, penal), torch.from_numpy(_load(case, load)).cuda()
    U = plain.solve(E, F, free)
    if kind == "solve":
        return U
    new, change = _step(plain, x, E, U, penal, 1.5, 2.0, proj, not proj, shape, _volfrac(x), pres)
    return {"x": new, "compliance": float(F @ U), "change": change}
