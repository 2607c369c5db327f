"""Performance cases: what a user of the library has it do, through its public entry points.

One case is a dict of plain values: ``kind`` names the work, ``mesh`` (a named workload of
``fixtures``) or ``target`` and ``mesh_seed`` (a mesh of the batched workload, between 5k and 500k
vertices) its size, ``precision`` the preconditioners' precision. The kinds:

  step       the solves of one time step on a kept hierarchy (SolveStep.run): assembly, ILU,
             BiCGSTAB for u and v, pressure system, AMG-PCG, both to 1e-10 relative
  timestep   one step of the whole time loop at the application's tolerances (TimeStepper.step):
             the solves, the projection, drag and lift, the hierarchy rebuilt every 50 steps
  amg_setup  the pressure hierarchy built again (every 50 steps and after each remesh)
  remesh     what follows a remesh: pattern and assembly plan of the new mesh, ILU colouring, and
             the re-projection of both velocity levels with a new hierarchy
  assembly   the momentum and pressure systems of one step (both matrices, right-hand sides)
  postsolve  what follows the solves: projection, forces, and the error indicators of a remesh
  momentum   ILU(0) factor and BiCGSTAB of one momentum system (forward or transposed)
  vcycle     one V-cycle of the pressure hierarchy on a residual
  adjoint    drag and its gradient over a few differentiated steps (forward and backward)
  batch      several independent systems of uneven sizes on concurrent streams, set-up included
"""
import functools
import math
import os
import random
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
for _p in (ROOT, os.path.join(ROOT, "cylinder-fem-amr_b200")):
    if _p not in sys.path:
        sys.path.insert(0, _p)

import adjoint as ADJ  # noqa: E402
import batch as B  # noqa: E402
import cfa_b200 as cfa  # noqa: E402
import fixtures as F  # noqa: E402
import step as S  # noqa: E402

DT, NU, RHO, STAB, U_MAX, TAU = 1e-3, 1e-3, 1.0, 0.3, 1.5, 1e-3
DT_PROJ = (2.0 / 3.0) * DT
N_MIN, N_MAX = 5_000, 500_000     # the batched workload's range of vertex counts


def listed():
    return [
        # the smallest system of the batched workload: launches and latency
        {"name": "step_5k_fp64", "kind": "step", "target": 5_000, "mesh_seed": 11, "precision": "fp64"},
        # the everyday run of the application: a uniform mesh, its default tolerances
        {"name": "timestep_22k_mixed", "kind": "timestep", "mesh": "c0", "precision": "mixed"},
        # the benchmark's step, in both precisions
        {"name": "step_402k_mixed", "kind": "step", "mesh": "c1", "precision": "mixed"},
        {"name": "step_402k_fp64", "kind": "step", "mesh": "c1", "precision": "fp64"},
        # the largest mesh: the step where bandwidth counts
        {"name": "step_4m_mixed", "kind": "step", "mesh": "c2", "precision": "mixed"},
        # the hierarchy of the benchmark's pressure system, every 50 steps
        {"name": "amg_setup_402k_mixed", "kind": "amg_setup", "mesh": "c1", "precision": "mixed"},
        # an adaptive run remeshes every 10 steps
        {"name": "remesh_43k_fp64", "kind": "remesh", "mesh": "medium", "precision": "fp64"},
        # assembly of one step at the benchmark's size
        {"name": "assembly_402k", "kind": "assembly", "mesh": "c1", "precision": "fp64"},
        # the kernels after the solves, on an adaptive mesh of ordinary size
        {"name": "postsolve_120k", "kind": "postsolve", "target": 120_001, "mesh_seed": 5, "precision": "fp64"},
        # the preconditioner alone, as another Krylov solver would call it
        {"name": "vcycle_60k_fp64", "kind": "vcycle", "target": 60_000, "mesh_seed": 3, "precision": "fp64"},
        # the gradient of the drag: forward and backward sweeps with recomputation
        {"name": "adjoint_22k_mixed", "kind": "adjoint", "mesh": "c0", "precision": "mixed", "steps": 4,
         "checkpoint": 2},
        # a batch of uneven systems, each set up and solved once
        {"name": "batch_8_mixed", "kind": "batch", "count": 8, "target": 100_000, "mesh_seed": 1,
         "precision": "mixed"},
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))))) | 1

    kind = rng.choice(["step", "step", "step", "timestep", "amg_setup", "remesh", "assembly", "postsolve", "momentum",
                       "momentum", "vcycle", "adjoint", "batch"])
    hi = {"remesh": 150_000, "adjoint": 40_000, "batch": 100_000}.get(kind, N_MAX)
    case = {"kind": kind, "target": size(N_MIN, hi), "mesh_seed": rng.randrange(1, 1000),
            "precision": rng.choice(["fp64", "mixed", "mixed"])}
    if kind == "momentum":
        case["transposed"] = rng.random() < 0.33
    if kind == "adjoint":
        case["steps"], case["checkpoint"] = rng.randint(2, 4), rng.randint(1, 3)
    if kind == "batch":
        case["count"] = rng.randint(3, 8)
    return case


# ----------------------------------------------------------------------------------------------
# inputs
# ----------------------------------------------------------------------------------------------
@functools.lru_cache(maxsize=4)
def _mesh(name, target, mesh_seed):
    """The mesh a run keeps for many steps (made once; only the fields are new inputs)."""
    if name:
        return F.make_mesh(name)
    return B.batch_system(mesh_seed, target, target).mesh


def mesh_of(case):
    return _mesh(case.get("mesh"), case.get("target"), case.get("mesh_seed"))


@functools.lru_cache(maxsize=2)
def _batch_meshes(case_key):
    case = dict(case_key)
    rng = random.Random(case["mesh_seed"])
    top = float(case["target"])
    sizes = [top] + [math.exp(rng.uniform(math.log(N_MIN), math.log(top))) for _ in range(case["count"] - 1)]
    return [B.batch_system(case["mesh_seed"] + k, s, s) for k, s in enumerate(sizes)]


def batch_meshes(case):
    return _batch_meshes(tuple(sorted((k, v) for k, v in case.items() if k != "name")))


def fields(m, seed):
    """Velocity of unit amplitude and a pressure: 8 random Fourier modes each."""
    return (F.fourier_field(m.x, m.y, 3 * seed + 1), F.fourier_field(m.x, m.y, 3 * seed + 2),
            0.3 * F.fourier_field(m.x, m.y, 3 * seed + 3))


def precision_of(case):
    return cfa.MIXED if case["precision"] == "mixed" else cfa.FP64


class State:
    pass


def _zeros(k):
    return torch.zeros(k, dtype=torch.float64, device="cuda")


def _up(a):
    return torch.from_numpy(np.ascontiguousarray(a, dtype=np.float64)).to("cuda")


def prepare(case, seed):
    s = State()
    s.case, kind, prec = case, case["kind"], precision_of(case)
    if kind == "batch":
        s.systems = []
        for k, base in enumerate(batch_meshes(case)):
            u, v, p = fields(base.mesh, 100 * seed + k)
            s.systems.append(B.BatchSystem(k, base.mesh, base.nu, u, v, p))
        s.solver = B.BatchSolver(prec, streams=4, keep=True)
        return s
    m = mesh_of(case)
    u, v, p = fields(m, seed)
    s.ctx = cfa.default_context()
    if kind == "adjoint":
        s.nu_node = NU * (1.0 + 0.1 * F.fourier_field(m.x, m.y, 3 * seed + 4))
        s.adj = ADJ.DragAdjoint(m, u, v, p, s.nu_node, steps=case["steps"], checkpoint=case["checkpoint"],
                                precision=prec, tol=1e-11, stab=STAB)
        return s
    if kind == "timestep":
        s.ts = S.TimeStepper(m, u, v, p, precision=prec, dt=DT, nu=NU, stab=STAB, u_max=U_MAX)
        return s
    if kind == "remesh":
        s.mesh, s.prec = m, prec
        s.host = (u, v, 0.9 * u, 0.9 * v, p)
        return s
    if kind == "postsolve":
        s.dm = cfa.DeviceMesh(s.ctx, m)
        s.mass = _zeros(m.n)
        cfa.lumped_mass(s.ctx, s.dm, s.mass)
        s.old = [_up(a) for a in (u, v, 0.9 * u, 0.9 * v, p)]
        s.dp = _up(0.01 * F.fourier_field(m.x, m.y, 3 * seed + 4))
        s.u, s.v, s.p = (a.clone() for a in (s.old[0], s.old[1], s.old[4]))
        s.div, s.gx, s.gy, s.wn, s.vort = (_zeros(m.n) for _ in range(5))
        s.forces, s.rec, s.err = _zeros(2), _zeros(4 * m.n), _zeros(2 * m.ne)
        return s
    s.st = S.SolveStep(m, u, v, p, precision=prec, dt=DT, nu=NU, stab=STAB, u_max=U_MAX)
    st = s.st
    if kind in ("step", "amg_setup", "vcycle"):
        st.amg_setup()
    if kind in ("amg_setup", "vcycle"):
        s.r, s.z = st.rhs_p.clone(), _zeros(m.n)
    if kind == "momentum":
        st.assemble_momentum()
        s.b = (st.rhs_u.clone(), st.rhs_v.clone())
        s.A = st.A.clone()
        if case["transposed"]:
            cfa.transpose_values(st.ctx, st.ilu, st.A, s.A)
        s.xu, s.xv = _zeros(m.n), _zeros(m.n)
    return s


# ----------------------------------------------------------------------------------------------
# one pass
# ----------------------------------------------------------------------------------------------
def run(s):
    kind = s.case["kind"]
    if kind == "step":
        st = s.st
        st.run()
        return {"u": st.u, "v": st.v, "dp": st.dp}
    if kind == "timestep":
        ts = s.ts
        cd, cl = ts.step()
        return {"u": ts.u, "v": ts.v, "p": ts.p, "dp": ts.dp, "vort": ts.vort, "forces": np.array([cd, cl])}
    if kind == "amg_setup":
        st = s.st
        st.amg.setup(st.n, st.nnz, st.dm.rp, st.dm.ci, st.Kp)
        st.amg.apply(st.rhs_p, s.z)          # the new hierarchy at work: its number and sizes of levels vary with u
        d = st.amg.level(0)
        return {"z": s.z, "agg": d["agg"], "omega": d["omega"]}
    if kind == "remesh":
        ctx, m = s.ctx, s.mesh
        dm = cfa.DeviceMesh(ctx, m)
        rp, ci = dm.host_pattern()
        ilu = cfa.MulticolourIlu0(ctx, s.prec)
        ilu.set_pattern(dm.n, rp, ci, dm.rp, dm.ci)
        u, v, uo, vo, p = (_up(a) for a in s.host)
        it = S.project_scheme_consistent(ctx, dm, DT_PROJ, STAB, NU, uo, vo, u, v, p,
                                         amg=cfa.AmgPreconditioner(ctx, s.prec))
        assert it > 0
        s.keep = (dm, ilu)
        return {"rp": dm.rp, "ci": dm.ci, "colour_start": ilu.colour_start, "u": u, "v": v, "u_old": uo, "v_old": vo}
    if kind == "assembly":
        st = s.st
        st.reset()
        st.assemble_momentum()
        st.assemble_pressure()
        return {"A": st.A, "rhs_u": st.rhs_u, "rhs_v": st.rhs_v, "mass": st.mass, "Kp": st.Kp, "rhs_p": st.rhs_p,
                "div": st.div, "oss": st.oss_val, "inv_m": st.inv_m, "elem_s": st.elem_s}
    if kind == "postsolve":
        s.u.copy_(s.old[0])
        s.v.copy_(s.old[1])
        s.p.copy_(s.old[4])
        cfa.project_step(s.ctx, s.dm, DT_PROJ, RHO, RHO * NU, True, s.mass, s.dp, s.div, s.gx, s.gy, s.wn, s.u, s.v,
                         s.p, s.vort)
        cfa.volume_forces(s.ctx, s.dm, s.u, s.v, s.old[0], s.old[1], s.old[2], s.old[3], s.p, 1.5 / DT, -2.0 / DT,
                          0.5 / DT, NU, RHO, s.forces)
        cfa.amr_indicators(s.ctx, s.dm, s.u, s.v, U_MAX, 1.0, s.mass, s.rec, s.err)
        return {"u": s.u, "v": s.v, "p": s.p, "vort": s.vort, "div": s.div, "forces": s.forces, "rec": s.rec,
                "err": s.err}
    if kind == "momentum":
        st = s.st
        s.xu.zero_()
        s.xv.zero_()
        if s.case["transposed"]:
            st.ilu.factor_transposed(st.A)
        else:
            st.ilu.factor(st.A)
        st.mom.solve(st.n, st.dm.rp, st.dm.ci, s.A, s.b[0], s.b[1], s.xu, s.xv, 1000, 1e-10, st.ilu)
        return {"u": s.xu, "v": s.xv}
    if kind == "vcycle":
        s.st.amg.apply(s.r, s.z)
        return s.z
    if kind == "adjoint":
        J, g_nu, g_u = s.adj.gradient()
        return {"J": J, "g_nu": g_nu, "g_u": g_u}
    rep = s.solver.solve(s.systems)
    assert all(r.converged for r in rep.systems)
    return {f"{k}_{q}": s.solver.results[k][i] for k in range(len(s.systems)) for i, q in enumerate(("u", "v", "dp"))}


# ----------------------------------------------------------------------------------------------
# what a pass cannot do without
# ----------------------------------------------------------------------------------------------
def _system(n, ne):
    """Bytes and operations of one step's solve path: the mesh and the fields read, the assembled
    systems written once and read once by their solves, the solution written."""
    nnz = 3 * n + 2 * ne          # a triangulation with one hole: edges = n + ne
    mesh = 12 * ne + 20 * n + 4 * (n + nnz)
    nbytes = mesh + 8 * 3 * n + 2 * 8 * 6 * nnz + 8 * 6 * n + 8 * 3 * n
    return nbytes, 30 * 2 * nnz


def work(case):
    kind = case["kind"]
    if kind == "batch":
        got = [_system(b.mesh.n, b.mesh.ne) for b in batch_meshes(case)]
        return {"bytes": sum(g[0] for g in got), "flops": sum(g[1] for g in got)}
    m = mesh_of(case)
    n, ne = m.n, m.ne
    nnz = 3 * n + 2 * ne
    mesh = 12 * ne + 20 * n
    if kind in ("step", "timestep"):
        b, f = _system(n, ne)
        return {"bytes": b, "flops": f}
    if kind == "amg_setup":        # the matrix in; operators of all levels and their transfers out
        return {"bytes": 12 * nnz + 4 * n + int(1.25 * 12 * nnz) + 2 * 12 * 3 * n, "flops": 12 * 3 * nnz}
    if kind == "remesh":
        b, f = _system(n, ne)
        return {"bytes": b + 8 * nnz, "flops": f}
    if kind == "assembly":
        return {"bytes": mesh + 4 * (n + nnz) + 8 * 5 * n + 8 * 6 * nnz + 8 * 6 * n + 8 * ne, "flops": 300 * ne}
    if kind == "postsolve":
        return {"bytes": mesh + 8 * 7 * n + 8 * 9 * n + 8 * 2 * ne, "flops": 150 * ne}
    if kind == "momentum":
        return {"bytes": 12 * nnz + 4 * n + 8 * 4 * n, "flops": 10 * 2 * nnz}
    if kind == "vcycle":
        vb = 4 if case["precision"] == "mixed" else 8
        return {"bytes": int(1.25 * ((4 + vb) * nnz + 4 * n)) + 16 * n, "flops": 10 * nnz}
    b, f = _system(n, ne)
    return {"bytes": 3 * case["steps"] * b, "flops": 3 * case["steps"] * f}


def tolerance(case):
    kind = case["kind"]
    if kind in ("amg_setup", "vcycle"):
        # FP32 smoothing against FP64: 8e-8 measured; two FP64 orders: 2e-16
        return {"rel": 4e-7, "max": 2e-6} if case["precision"] == "mixed" else {"rel": 1e-14, "max": 1e-12}
    return TOLERANCE[kind]


# Solves stop at their residual tolerance (1e-10 relative; the time loop and the re-projection at
# the application's 1e-7 and 1e-8; the adjoint at 1e-11). What that leaves open in the solution was
# measured as the difference to the exact solution (to a tolerance of 1e-13 for the adjoint) and
# between the two precisions; the limits are about four times the largest. The assembled values and
# the projection are sums in another order.
TOLERANCE = {
    "step": {"rel": 4e-9, "max": 2e-7},
    "timestep": {"rel": 5e-8, "max": 2e-6},
    "remesh": {"rel": 1e-8, "max": 4e-7},
    "assembly": {"rel": 1e-14, "max": 1e-12},
    "postsolve": {"rel": 5e-14, "max": 1e-11},
    "momentum": {"rel": 4e-9, "max": 2e-7},
    "adjoint": {"rel": 3e-9, "max": 5e-8},
    "batch": {"rel": 4e-9, "max": 2e-7},
}


# ----------------------------------------------------------------------------------------------
# the same results from the formulas, in 64 bits, with torch alone
# ----------------------------------------------------------------------------------------------
class _Exact:
    """P1 element formulas and unpreconditioned-quality solves on one mesh."""

    def __init__(self, m):
        self.n, self.ne = m.n, m.ne
        self.t = torch.from_numpy(m.tri.astype(np.int64)).to("cuda")
        self.x, self.y = _up(m.x), _up(m.y)
        self.tag = torch.from_numpy(np.asarray(m.tag).astype(np.int64)).to("cuda")
        X, Y = self.x[self.t], self.y[self.t]
        det = (X[:, 1] - X[:, 0]) * (Y[:, 2] - Y[:, 0]) - (X[:, 2] - X[:, 0]) * (Y[:, 1] - Y[:, 0])
        self.area = 0.5 * det.abs()
        d = (2.0 * self.area)[:, None]
        self.gx = torch.stack([Y[:, 1] - Y[:, 2], Y[:, 2] - Y[:, 0], Y[:, 0] - Y[:, 1]], 1) / d
        self.gy = torch.stack([X[:, 2] - X[:, 1], X[:, 0] - X[:, 2], X[:, 1] - X[:, 0]], 1) / d
        key = (self.t[:, :, None] * self.n + self.t[:, None, :]).reshape(-1)
        uniq, self.pos = torch.unique(key, return_inverse=True)
        self.row, self.col = uniq // self.n, uniq % self.n
        self.nnz = uniq.numel()
        counts = torch.bincount(self.row, minlength=self.n)
        self.rp = torch.cat([counts.new_zeros(1), counts.cumsum(0)])
        self.diag = self.row == self.col
        self.mass = self.nodes((self.area / 3.0)[:, None].expand(-1, 3))
        self.fixed = (self.tag == F.BC_INLET) | (self.tag == F.BC_WALL) | (self.tag == F.BC_CYLINDER)
        self.outlet = self.tag == F.BC_OUTLET

    def nodes(self, e):
        return torch.zeros(self.n, dtype=torch.float64, device="cuda").index_add_(0, self.t.reshape(-1), e.reshape(-1))

    def entries(self, e):
        return torch.zeros(self.nnz, dtype=torch.float64, device="cuda").index_add_(0, self.pos, e.reshape(-1))

    def grad(self, f):
        return (f[self.t] * self.gx).sum(1), (f[self.t] * self.gy).sum(1)

    def matrix(self, val):
        return torch.sparse_csr_tensor(self.rp, self.col, val, (self.n, self.n))

    def momentum(self, u, v, um, vm, p, a0, a1, a2, c1, c2, nu=NU):
        t, area = self.t, self.area[:, None]
        uh, vh = (a1 * u + a2 * um)[t], (a1 * v + a2 * vm)[t]
        w, z = (c1 * u + c2 * um)[t], (c1 * v + c2 * vm)[t]
        wu, wv = w.mean(1), z.mean(1)
        div = (w * self.gx + z * self.gy).sum(1)
        h = torch.sqrt(2.0 * self.area)
        tt, tc, td = 2.0 / TAU, 2.0 * (torch.sqrt(wu * wu + wv * wv) + 1e-12) / h, 4.0 * nu / (h * h)
        tau = (1.0 / torch.sqrt(tt * tt + tc * tc + 9.0 * td * td))[:, None, None]
        dpx, dpy = self.grad(p)
        ug = wu[:, None] * self.gx + wv[:, None] * self.gy
        a3 = self.area[:, None, None]
        M = a3 / 12.0 * (1.0 + torch.eye(3, dtype=torch.float64, device="cuda"))[None]
        K = a3 * (self.gx[:, :, None] * self.gx[:, None, :] + self.gy[:, :, None] * self.gy[:, None, :])
        Ms = (a3 / 3.0 * tau * ug[:, :, None]).expand(-1, 3, 3)
        A = (a0 * (M + Ms) + nu * K + a3 / 3.0 * ug[:, None, :] + 0.5 * div[:, None, None] * M
             + a3 * tau * ug[:, :, None] * ug[:, None, :])
        tw = area / 3.0 + area * tau[:, :, 0] * ug
        fu = ((M + Ms) * uh[:, None, :]).sum(2) - tw * dpx[:, None] / RHO
        fv = ((M + Ms) * vh[:, None, :]).sum(2) - tw * dpy[:, None] / RHO
        val = self.entries(A)
        val = torch.where(self.fixed[self.row], self.diag.double(), val)
        ub = torch.where(self.tag == F.BC_INLET, 4.0 * U_MAX * self.y * (1.0 - self.y), torch.zeros_like(self.y))
        return (val, torch.where(self.fixed, ub, self.nodes(fu)),
                torch.where(self.fixed, torch.zeros_like(ub), self.nodes(fv)))

    def weights(self, u, v, dt, nu=NU):
        h = torch.sqrt(2.0 * self.area)
        ub, vb = u[self.t].mean(1), v[self.t].mean(1)
        return RHO * STAB / (RHO * (4.0 * nu / (h * h) + 2.0 * torch.sqrt(ub * ub + vb * vb) / h)) / dt

    def pressure(self, u, v, p, s, dt):
        third = self.area / 3.0
        gpx, gpy = self.grad(p)
        rs = torch.sqrt(s)
        Gx = self.nodes((rs * third * gpx)[:, None].expand(-1, 3)) / self.mass
        Gy = self.nodes((rs * third * gpy)[:, None].expand(-1, 3)) / self.mass
        sx, sy = rs * Gx[self.t].mean(1), rs * Gy[self.t].mean(1)
        div = (u[self.t] * self.gx + v[self.t] * self.gy).sum(1)
        K = self.area[:, None, None] * (self.gx[:, :, None] * self.gx[:, None, :]
                                        + self.gy[:, :, None] * self.gy[:, None, :])
        val = self.entries((1.0 + s)[:, None, None] * K)
        e = (-(RHO / dt) * third * div)[:, None] - self.area[:, None] * (
            self.gx * (s * gpx - sx)[:, None] + self.gy * (s * gpy - sy)[:, None])
        rhs = torch.where(self.outlet, torch.zeros_like(self.x), self.nodes(e))
        cut = self.outlet[self.row] | self.outlet[self.col]
        val = torch.where(cut, (self.diag & self.outlet[self.row]).double(), val)
        w = (rs * third)[:, None, None]
        oss = [self.entries(w * g) for g in (self.gx[:, None, :].expand(-1, 3, 3), self.gy[:, None, :].expand(-1, 3, 3),
                                             self.gx[:, :, None].expand(-1, 3, 3), self.gy[:, :, None].expand(-1, 3, 3))]
        return val, rhs, self.nodes((third * div)[:, None].expand(-1, 3)), oss

    def solve_pressure(self, val, oss, b):
        """Jacobi-preconditioned CG on K - [not Dirichlet] B^T M^-1 B."""
        K, (Bx, By, Tx, Ty) = self.matrix(val), (self.matrix(o) for o in oss)
        keep = (~self.outlet).double()
        im = 1.0 / self.mass

        def op(q):
            return K @ q - keep * (Tx @ (im * (Bx @ q)) + Ty @ (im * (By @ q)))

        dinv = 1.0 / val[self.diag]
        x, r = torch.zeros_like(b), b.clone()
        z = dinv * r
        p, rz, bn = z.clone(), r @ z, b.norm()
        for it in range(40_000):
            q = op(p)
            a = rz / (p @ q)
            x += a * p
            r -= a * q
            if it % 50 == 49 and float(r.norm()) < 1e-13 * float(bn):
                break
            z = dinv * r
            new = r @ z
            p.mul_(new / rz).add_(z)
            rz = new
        return x

    def solve_momentum(self, val, b, x):
        """Jacobi-preconditioned BiCGSTAB, restarted from its true residual."""
        A = self.matrix(val)
        dinv = 1.0 / val[self.diag]
        bn = b.norm()
        for _ in range(4):
            r = b - A @ x
            if float(r.norm()) <= 1e-14 * float(bn):
                break
            r0, p, goal = r.clone(), r.clone(), max(1e-14 * float(bn), 1e-12 * float(r.norm()))
            rho = r0 @ r
            for it in range(2000):
                y = dinv * p
                v = A @ y
                al = rho / (r0 @ v)
                q = r - al * v
                z = dinv * q
                t = A @ z
                om = (t @ q) / (t @ t)
                x = x + al * y + om * z
                r = q - om * t
                if it % 5 == 4 and float(r.norm()) < goal:
                    break
                new = r0 @ r
                p = r + (new / rho) * (al / om) * (p - om * v)
                rho = new
        return x

    def start(self, u, v):
        ub = torch.where(self.tag == F.BC_INLET, 4.0 * U_MAX * self.y * (1.0 - self.y), torch.zeros_like(self.y))
        return torch.where(self.fixed, ub, u), torch.where(self.fixed, torch.zeros_like(v), v)

    def step(self, u, v, p, coef, dt, nu=NU):
        A, bu, bv = self.momentum(u, v, u, v, p, *coef, nu=nu)
        xu, xv = self.start(u, v)
        xu, xv = self.solve_momentum(A, bu, xu), self.solve_momentum(A, bv, xv)
        val, rhs, _, oss = self.pressure(xu, xv, p, self.weights(xu, xv, dt, nu), dt)
        return xu, xv, self.solve_pressure(val, oss, rhs)

    def correct(self, u, v, p, dp, dt, update, rot):
        """(u, v, p, vorticity, div_num) after the projection with the increment dp."""
        third = (self.area / 3.0)[:, None].expand(-1, 3)
        dx, dy = self.grad(dp)
        om = self.grad(v)[0] - self.grad(u)[1]
        div = self.nodes(-(dt / RHO) * self.area[:, None] * (self.gx * dx[:, None] + self.gy * dy[:, None]))
        free = ~self.fixed
        un = torch.where(free, u - dt / RHO * self.nodes(third * dx[:, None]) / self.mass, u)
        vn = torch.where(free, v - dt / RHO * self.nodes(third * dy[:, None]) / self.mass, v)
        return un, vn, p + update * (dp - rot * div / self.mass), self.nodes(third * om[:, None]) / self.mass, div

    def forces(self, u, v, u1, v1, u2, v2, p, b0, b1, b2):
        phi = (self.tag == F.BC_CYLINDER).double()[self.t]
        ue, ve, pb = u[self.t], v[self.t], p[self.t].mean(1)
        ut, vt = (b0 * u + b1 * u1 + b2 * u2)[self.t], (b0 * v + b1 * v1 + b2 * v2)[self.t]
        (ux, uy), (vx, vy) = self.grad(u), self.grad(v)
        px, py = (phi * self.gx).sum(1), (phi * self.gy).sum(1)
        fx, fy = torch.zeros_like(pb), torch.zeros_like(pb)
        for a in range(3):
            b = (a + 1) % 3
            pm, uu, vv = (0.5 * (q[:, a] + q[:, b]) for q in (phi, ue, ve))
            fx = fx + (0.5 * (ut[:, a] + ut[:, b]) + uu * ux + vv * uy) * pm
            fy = fy + (0.5 * (vt[:, a] + vt[:, b]) + uu * vx + vv * vy) * pm
        fx = self.area / 3.0 * fx + self.area * (NU * (ux * px + uy * py) - pb / RHO * px)
        fy = self.area / 3.0 * fy + self.area * (NU * (vx * px + vy * py) - pb / RHO * py)
        return torch.stack([fx.sum(), fy.sum()])


BDF2 = (1.5 / DT, 2.0 / DT, -0.5 / DT, 2.0, -1.0)
EULER = (1.0 / DT, 1.0 / DT, 0.0, 1.0, 0.0)


def exact(case, seed):
    kind = case["kind"]
    if kind == "adjoint":     # an iterated derivative: no short formula
        return None
    if kind == "batch":
        out = {}
        for k, base in enumerate(batch_meshes(case)):
            u, v, p = (_up(a) for a in fields(base.mesh, 100 * seed + k))
            got = _Exact(base.mesh).step(u, v, p, BDF2, DT_PROJ, nu=base.nu)
            out.update({f"{k}_{q}": got[i].cpu().numpy() for i, q in enumerate(("u", "v", "dp"))})
        return out
    m = mesh_of(case)
    if m.n > 1_000_000:
        return None
    e = _Exact(m)
    u, v, p = (_up(a) for a in fields(m, seed))
    if kind == "step":
        xu, xv, dp = e.step(u, v, p, BDF2, DT_PROJ)
        return {"u": xu, "v": xv, "dp": dp}
    if kind == "timestep":                   # the first step of a new run: backward Euler
        xu, xv, dp = e.step(u, v, p, EULER, DT)
        un, vn, pn, vort, _ = e.correct(xu, xv, p, dp, DT, 1.0, RHO * NU)
        f = -10.0 * e.forces(un, vn, u, v, u, v, pn, 1.0 / DT, -1.0 / DT, 0.0)
        return {"u": un, "v": vn, "p": pn, "dp": dp, "vort": vort, "forces": f}
    if kind == "remesh":
        s, out = e.weights(u, v, DT_PROJ), {"rp": e.rp.int(), "ci": e.col.int(), "colour_start": None}
        for q, fu, fv in (("_old", 0.9 * u, 0.9 * v), ("", u, v)):
            val, rhs, _, oss = e.pressure(fu, fv, p, s, DT_PROJ)
            dp = e.solve_pressure(val, oss, rhs)
            out["u" + q], out["v" + q] = e.correct(fu, fv, p, dp, DT_PROJ, 0.0, 0.0)[:2]
        return out
    if kind == "assembly":
        A, bu, bv = e.momentum(u, v, u, v, p, *BDF2)
        xu, xv = e.start(u, v)
        s = e.weights(xu, xv, DT_PROJ)
        val, rhs, div, oss = e.pressure(xu, xv, p, s, DT_PROJ)
        return {"A": A, "rhs_u": bu, "rhs_v": bv, "mass": e.mass, "Kp": val, "rhs_p": rhs, "div": div,
                "oss": torch.cat(oss), "inv_m": 1.0 / e.mass, "elem_s": s}
    if kind == "postsolve":
        dp = _up(0.01 * F.fourier_field(m.x, m.y, 3 * seed + 4))
        un, vn, pn, vort, div = e.correct(u, v, p, dp, DT_PROJ, 1.0, RHO * NU)
        f = e.forces(un, vn, u, v, 0.9 * u, 0.9 * v, pn, 1.5 / DT, -2.0 / DT, 0.5 / DT)
        third = (e.area / 3.0)[:, None].expand(-1, 3)
        du = un - 4.0 * U_MAX * e.y * (1.0 - e.y)
        rec = [e.nodes(third * g[:, None]) for g in (*e.grad(du), *e.grad(vn))]
        G = torch.stack([r / e.mass for r in rec], 1)[e.t]
        om = (G[:, :, 2] - G[:, :, 1]).abs().amax(1)
        eta = torch.zeros_like(om)
        for a in range(3):
            b = (a + 1) % 3
            ex, ey = (q[e.t[:, b]] - q[e.t[:, a]] for q in (e.x, e.y))
            d = G[:, b] - G[:, a]
            eta = torch.maximum(eta, 0.125 * torch.sqrt((d[:, 0] * ex + d[:, 1] * ey) ** 2
                                                        + (d[:, 2] * ex + d[:, 3] * ey) ** 2))
        return {"u": un, "v": vn, "p": pn, "vort": vort, "div": div, "forces": f, "rec": torch.cat(rec),
                "err": torch.cat([torch.sqrt(2.0 * e.area) * om, eta])}
    if kind == "momentum":
        A, bu, bv = e.momentum(u, v, u, v, p, *BDF2)
        if case["transposed"]:
            order = torch.argsort(e.col * e.n + e.row)
            A = A[order]
        return {"u": e.solve_momentum(A, bu, torch.zeros_like(bu)), "v": e.solve_momentum(A, bv, torch.zeros_like(bv))}
    z = _vcycle_exact(case, seed)
    return z if kind == "vcycle" else {"z": z, "agg": None, "omega": None}


def _vcycle_exact(case, seed):
    """The V(2,2) cycle written out over the hierarchy that the program holds."""
    s = prepare(case, seed)
    amg = s.st.amg
    levels, inv = [amg.level(k) for k in range(amg.num_levels() - 1)], amg.coarse_inverse()

    def csr(d, rows, cols):
        return torch.sparse_csr_tensor(d[0].long(), d[1].long(), d[2], (rows, cols))

    def cycle(k, b):
        if k == len(levels):
            return inv @ b
        d = levels[k]
        n, nc = d["rows"], d["pcols"]
        A, P, R = csr(d["A"], n, n), csr(d["P"], n, nc), csr(d["R"], nc, n)
        rows = torch.repeat_interleave(torch.arange(n, device="cuda"), d["A"][0].long().diff())
        w = d["omega"] / d["A"][2][rows == d["A"][1].long()]
        x = w * b
        x = x + w * (b - A @ x)
        x = x + P @ cycle(k + 1, R @ (b - A @ x))
        for _ in range(2):
            x = x + w * (b - A @ x)
        return x

    return cycle(0, s.r)
