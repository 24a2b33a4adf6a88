"""What a user of this framework has it do, as cases that can be timed and whose results can be compared.

The path is the Newton-Raphson / LoadControl solve of Q1 hexahedral Neo-Hookean solids: residual and tangent
assembly, the linear solve of a tangent, single load steps and whole load paths, with and without enhanced strains,
one system or many independent ones.  A case is a dict of plain values with an ``op``:

  residual   SparseFlatAssembler.vector at a deformed state
  tangent    SparseFlatAssembler.matrix at a deformed state, exported as scipy CSC
  solve      LinearSolver.factorize + solve of a block's assembled FP64 tangent with the reference's default solver tag
  path       LoadControl.run from the undeformed state, FP64 or mixed (FP32 tangent and CG, FP64 residual)
  eas_path   the reference's EAS cantilever test (golden cantilever, point loads)
  eas_block  a load step of the nearly incompressible EAS block: FP64 outer Krylov solve around the FP32 CG
  batched    one load step of independent cantilevers of uneven size

Sizes, materials and loads are those of problems.py, the tests and bench.py.
"""
from __future__ import annotations

import math
import warnings

import numpy as np
import torch

import ikarus_gb300 as ikr
from ikarus_gb300 import problems
from ikarus_gb300.mesh import jitter_interior

# Load factor after one of the load steps of a path (20 steps of the large cantilevers, 10 of the batched ones).
STEP = {"cantilever": 0.05, "eas_block": 0.04, "batched": 0.1}


def listed():
    return [
        # the smallest call: a residual of the 256-element cantilever (convergence checks, observers, small meshes)
        {"name": "residual_16x4x4", "op": "residual", "nx": 16, "ny": 4, "nz": 4},
        # the same call on the headline mesh
        {"name": "residual_128x32x32", "op": "residual", "nx": 128, "ny": 32, "nz": 32},
        # the assembled tangent handed to other code as Eigen's CSC arrays
        {"name": "tangent_24x12x12", "op": "tangent", "nx": 24, "ny": 12, "nz": 12},
        # a linear solve with the reference's default solver tag on a block, odd mesh
        {"name": "solve_61x57x15", "op": "solve", "nx": 61, "ny": 57, "nz": 15},
        # the whole 10-step load path of the small cantilever in FP64: many short solves
        {"name": "path_16x4x4_fp64", "op": "path", "nx": 16, "ny": 4, "nz": 4, "form": "fp64", "steps": 10,
         "end": 1.0, "load": "tip", "slabs": 0},
        # the reference's EAS cantilever test: 20 load steps of ten elements, pure latency
        {"name": "eas_path_10x1x1", "op": "eas_path", "nx": 10, "ny": 1, "nz": 1, "steps": 20},
        # a load step of the learned-predictor workload (pressure on the top face), mixed precision
        {"name": "step_64x16x16_mixed", "op": "path", "nx": 64, "ny": 16, "nz": 16, "form": "mixed", "steps": 1,
         "end": STEP["cantilever"], "load": "pressure", "slabs": 0},
        # a load step of the headline workload, mixed precision
        {"name": "step_128x32x32_mixed", "op": "path", "nx": 128, "ny": 32, "nz": 32, "form": "mixed", "steps": 1,
         "end": STEP["cantilever"], "load": "tip", "slabs": 0},
        # the same with the optional coarse correction of the CG
        {"name": "step_128x32x32_slabs", "op": "path", "nx": 128, "ny": 32, "nz": 32, "form": "mixed", "steps": 1,
         "end": STEP["cantilever"], "load": "tip", "slabs": 16},
        # a load step in plain FP64 (the reference's precision) on a mesh whose FP64 tangent is larger than L2's share
        {"name": "step_80x20x20_fp64", "op": "path", "nx": 80, "ny": 20, "nz": 20, "form": "fp64", "steps": 1,
         "end": STEP["cantilever"], "load": "tip", "slabs": 0},
        # a load step of the nearly incompressible block
        {"name": "eas_block_32x32x8", "op": "eas_block", "nx": 32, "ny": 32, "nz": 8},
        # a load step of many independent cantilevers
        {"name": "batched_128_mixed", "op": "batched", "n": 128, "layout": 7, "form": "mixed"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["residual", "tangent", "solve", "path", "path", "path", "path", "eas_path", "eas_block",
                     "batched"])
    if op == "residual":
        nx = _log_int(rng, 8, 128)
        return {"op": op, "nx": nx, "ny": max(2, nx // rng.randint(4, 8)), "nz": max(2, nx // rng.randint(4, 8))}
    if op == "tangent":
        return {"op": op, "nx": _log_int(rng, 4, 24), "ny": rng.randint(2, 12), "nz": rng.randint(2, 12)}
    if op == "solve":
        nx = _log_int(rng, 12, 64)
        return {"op": op, "nx": nx, "ny": max(2, nx - rng.randint(0, 5)), "nz": max(2, nx // 4 + rng.randint(-1, 1))}
    if op == "eas_path":
        return {"op": op, "nx": rng.randint(4, 12), "ny": rng.randint(1, 2), "nz": rng.randint(1, 2),
                "steps": rng.randint(5, 20)}
    if op == "eas_block":
        n = rng.randint(8, 32)
        return {"op": op, "nx": n, "ny": n, "nz": max(2, n // 4)}
    if op == "batched":
        return {"op": op, "n": _log_int(rng, 8, 128), "layout": rng.randint(1, 999),
                "form": rng.choice(["mixed", "mixed", "fp64"])}
    form = rng.choice(["mixed", "mixed", "fp64"])
    nx = _log_int(rng, 8, 120 if form == "mixed" else 72)
    small = nx <= 24
    return {"op": op, "nx": nx, "ny": max(2, nx // 4 + rng.randint(-1, 1)), "nz": max(2, nx // 4 + rng.randint(-1, 1)),
            "form": form, "steps": rng.randint(2, 5) if small else 1,
            "end": STEP["cantilever"] * (5 if small else 1), "load": rng.choice(["tip", "pressure"]),
            "slabs": rng.choice([0, 0, 0, 8, 16]) if nx >= 48 else 0}


# ---- inputs --------------------------------------------------------------------------------------------------
def _cantilever(case, seed):
    """The cantilever [0,10]x[0,1]x[0,1]: jittered interior nodes, material and loads from the seed."""
    rng = np.random.default_rng(seed)
    p = problems.cantilever(case["nx"], case["ny"], case["nz"], E=1000.0 * rng.uniform(0.8, 1.25),
                            nu=rng.uniform(0.25, 0.35), tol=1e-8, relative=True)
    p.mesh = jitter_interior(p.mesh, 0.1, int(rng.integers(1 << 30)))
    if case.get("load", "tip") == "tip":
        ang = rng.uniform(0.0, 2.0 * math.pi)
        t = rng.uniform(0.6, 1.0) * np.array([0.1 * rng.standard_normal(), math.cos(ang), math.sin(ang)])
        p.face_traction = np.tile(t, (len(p.face_elem), 1))
    else:
        p.face_elem, p.face_local, p.face_traction = problems.learned_loads(p, problems.sample_load_parameters(rng))
    return p


def _displacement(p, seed):
    """A smooth bent state with element-sized noise, zero on the clamped face."""
    rng = np.random.default_rng(seed + 77)
    x = p.mesh.coords
    u = np.zeros_like(x)
    for k in range(1, 4):
        u += (rng.standard_normal(3) * 0.1 / k) * np.sin(0.5 * k * math.pi * x[:, :1] / 10.0) ** 2
    h = 1.0 / max(p.mesh.shape[1:])
    u += 0.02 * h * rng.standard_normal(x.shape)
    u[x[:, 0] < 1e-8] = 0.0
    return u.reshape(-1)


def _settings(form, tol):
    if form == "mixed":
        return ikr.NRSettings(tol=tol, maxIter=30, relative=True, eisenstat_walker=True, linear_rtol=2e-2,
                              linear_rtol_min=1e-5, linear_max_iter=200000)
    return ikr.NRSettings(tol=tol, maxIter=30, relative=True, linear_rtol=1e-10, linear_max_iter=400000)


def _load_control(fes, asm, settings, ls, steps, end, batched=False):
    """The objects a program keeps for its load paths; the linear solver has analysed the undeformed tangent."""
    req = ikr.FERequirements(fes)
    asm.vector(req, dbc=ikr.DBCOption.Full, export=False)
    asm.matrix(req, dbc=ikr.DBCOption.Full, export=False)
    if not batched:
        ls.compute(asm)
    nr = ikr.NewtonRaphson(asm, ikr.NewtonRaphsonConfig(settings, ls))
    lc = ikr.LoadControl(nr, steps, (0.0, end))
    return {"fes": fes, "asm": asm, "ls": ls, "req": req, "lc": lc, "u0": np.zeros(fes.n_dofs)}


def _batch(case, seed):
    """Grids, lengths and the spread of materials and loads from the case; every instance's stiffness and load vary
    with the seed."""
    bp = problems.batched_cantilevers(n=case["n"], seed=case["layout"], E=(5e2, 1e4), t=(0.1, 1.0))
    rng = np.random.default_rng(seed)
    stiff, load = rng.uniform(0.8, 1.25, case["n"]), rng.uniform(0.7, 1.0, case["n"])
    per_elem = np.repeat(stiff, np.diff(bp.elem_offsets))
    bp.lam_e, bp.mu_e = bp.lam_e * per_elem, bp.mu_e * per_elem
    bp.face_traction = bp.face_traction * np.repeat(load, [len(p.face_elem) for p in bp.parts])[:, None]
    return bp


def _solid(case, seed):
    """The compressible block with jittered interior nodes, for linear solves."""
    rng = np.random.default_rng(seed)
    p = problems.eas_block(case["nx"], case["ny"], case["nz"], nu=rng.uniform(0.25, 0.35), eas=0, n_eas=0)
    p.mesh = jitter_interior(p.mesh, 0.1, int(rng.integers(1 << 30)))
    return p


def _solid_displacement(p, seed):
    """A smooth squeezed state, zero on the clamped bottom face."""
    rng = np.random.default_rng(seed + 77)
    x = p.mesh.coords
    u = 0.05 * x[:, 2:] * np.cos(math.pi * (x @ rng.uniform(0.5, 1.5, (3, 3))))
    return u.reshape(-1)


def _state(case, seed):
    if case["op"] == "solve":
        p = _solid(case, seed)
        return p, _solid_displacement(p, seed)
    p = _cantilever(case, seed)
    return p, _displacement(p, seed)


def prepare(case, seed):
    op = case["op"]
    if op in ("residual", "tangent", "solve"):
        p, u = _state(case, seed)
        fes, asm = problems.build_gpu(p, precision=0)
        req = ikr.FERequirements(fes, u, 1.0)
        s = {"op": op, "fes": fes, "asm": asm, "req": req}
        if op == "residual":
            asm.vector(req, dbc=ikr.DBCOption.Full, export=False)
        else:
            asm.matrix(req, dbc=ikr.DBCOption.Full, export=False)
        if op == "solve":
            s["ls"] = ikr.LinearSolver(ikr.SolverTypeTag.sd_SimplicialLDLT)
            s["ls"].compute(asm)
            s["b"] = _rhs(p, seed)
        return s
    if op == "path":
        p = _cantilever(case, seed)
        fes, asm = problems.build_gpu(p, precision=1 if case["form"] == "mixed" else 0)
        ls = ikr.LinearSolver(rtol=1e-10)
        if case["slabs"]:
            ls.set_coarse_space(case["slabs"])
        # the pressure's residual is spread over the whole top face: a smaller tolerance for the same displacement
        st = _settings(case["form"], tol=1e-9 if case["load"] == "tip" else 3e-10)
        return {"op": op, **_load_control(fes, asm, st, ls, case["steps"], case["end"])}
    if op == "eas_path":
        p = _golden(case, seed)
        fes, asm = problems.build_gpu(p, precision=0)
        st = ikr.NRSettings(tol=p.tol, linear_rtol=1e-13)
        s = _load_control(fes, asm, st, ikr.LinearSolver(rtol=1e-13), case["steps"], 1.0)
        return {"op": op, "alpha0": np.zeros((fes.n_elems, fes.n_eas)), **s}
    if op == "eas_block":
        p = _block(case, seed)
        fes, asm = problems.build_gpu(p, precision=1)
        st = ikr.NRSettings(tol=1e-8, maxIter=80, relative=True, eisenstat_walker=True, linear_rtol=1e-2,
                            linear_rtol_min=1e-5, linear_max_iter=5000)
        ls = ikr.LinearSolver(rtol=1e-10)
        ls.set_fp64_outer(restart=20, inner_rtol=1e-2, inner_max_iter=5000)
        s = _load_control(fes, asm, st, ls, 1, STEP["eas_block"])
        return {"op": op, "alpha0": np.zeros((fes.n_elems, fes.n_eas)), **s}
    if op == "batched":
        bp = _batch(case, seed)
        mixed = case["form"] == "mixed"
        fes, asm = problems.build_gpu_batched(bp, precision=1 if mixed else 0)
        st = ikr.NRSettings(tol=1e-9, maxIter=40, relative=True, eisenstat_walker=mixed,
                            linear_rtol=1e-2 if mixed else 1e-10, linear_rtol_min=1e-6, linear_max_iter=20000,
                            backtracks=4)
        ls = ikr.LinearSolver(ikr.SolverTypeTag.gpu_PCG_Batched)
        return {"op": op, **_load_control(fes, asm, st, ls, 1, STEP["batched"], batched=True)}
    raise ValueError(op)


def run(s):
    op = s["op"]
    if op == "residual":
        return s["asm"].vector(s["req"], dbc=ikr.DBCOption.Full)
    if op == "tangent":
        K = s["asm"].matrix(s["req"], dbc=ikr.DBCOption.Full)
        return {"data": K.data, "indices": K.indices, "indptr": K.indptr}
    if op == "solve":
        s["ls"].factorize(s["asm"])
        return s["ls"].solve(s["asm"], s["b"])
    # load paths start from the undeformed state
    req = s["req"]
    if "alpha0" in s:
        s["fes"].alpha = s["alpha0"]
    req.insertGlobalSolution(s["u0"])
    req.insertParameter(0.0)
    info = s["lc"].run(req)
    if not info.success:
        raise RuntimeError("the load path did not converge")
    return req.globalSolution()


def work(case):
    """Bytes: inputs once, outputs once.  Flops: per Newton iteration one residual, one tangent and one product with
    the tangent (the iterations of a linear solve depend on the method)."""
    op = case["op"]
    if op == "batched":
        ne, nn = case["n"] * 18 * 25, case["n"] * 19 * 36
    else:
        ne = case["nx"] * case["ny"] * case["nz"]
        nn = (case["nx"] + 1) * (case["ny"] + 1) * (case["nz"] + 1)
    geometry = 8 * 3 * nn + 4 * 8 * ne
    vec, nnz = 8 * 3 * nn, 9 * 27 * nn
    f_res, f_tan = 8 * 700 * ne, 2 * 9200 * ne
    if op == "residual":
        return {"bytes": geometry + 2 * vec, "flops": f_res}
    if op == "tangent":
        return {"bytes": geometry + vec + 12 * nnz, "flops": f_tan}
    if op == "solve":
        return {"bytes": 8 * nnz + 2 * vec, "flops": 2 * nnz}
    newton = 4 * case.get("steps", 1)
    if op.startswith("eas"):
        f_tan *= 3
    return {"bytes": geometry + 2 * vec, "flops": newton * (f_res + f_tan + 2 * nnz)}


# ---- the same in 64 bits, plain torch --------------------------------------------------------------------------
def _golden(case, seed):
    p = problems.cantilever_golden(2, 9, case["nx"], case["ny"], case["nz"])
    f = np.random.default_rng(seed).uniform(0.8, 1.0)
    p.pl_values = p.pl_values * f
    return p


def _block(case, seed):
    rng = np.random.default_rng(seed)
    return problems.eas_block(case["nx"], case["ny"], case["nz"], pressure=50.0 * rng.uniform(0.8, 1.0))


def _rhs(p, seed):
    b = np.random.default_rng(seed + 5).standard_normal(p.n_dofs)
    b[p.fixed != 0] = 0.0
    return b


_G = 0.5 / math.sqrt(3.0)


def _gradients():
    """Reference gradients of the eight shape functions at the eight Gauss points: (8 points, 8 nodes, 3)."""
    out = np.zeros((8, 8, 3))
    for q in range(8):
        xi = [0.5 + (_G if (q >> d) & 1 else -_G) for d in range(3)]
        for v in range(8):
            n = [xi[d] if (v >> d) & 1 else 1.0 - xi[d] for d in range(3)]
            for d in range(3):
                out[q, v, d] = (1.0 if (v >> d) & 1 else -1.0) * n[(d + 1) % 3] * n[(d + 2) % 3]
    return out


class _Exact:
    """The mesh's forces, tangents and Newton solve in FP64 torch, element by element."""

    def __init__(self, mesh, lam, mu, fixed, faces=None, point=None):
        d = "cuda" if torch.cuda.is_available() else "cpu"
        self.dev = d
        self.X = torch.as_tensor(mesh.coords, device=d)
        self.conn = torch.as_tensor(mesh.conn.astype(np.int64), device=d)
        self.dof = (3 * self.conn[:, :, None] + torch.arange(3, device=d)).reshape(-1, 24)
        self.n = mesh.n_dofs
        ne = mesh.n_elems
        self.lam = torch.as_tensor(lam, dtype=torch.float64, device=d).expand(ne)
        self.mu = torch.as_tensor(mu, dtype=torch.float64, device=d).expand(ne)
        self.free = torch.as_tensor(fixed == 0, device=d).double()
        G = torch.as_tensor(_gradients(), device=d)
        Xe = self.X[self.conn]
        self.dN, self.w = [], []
        for q in range(8):
            J = torch.einsum("evi,vj->eij", Xe, G[q])
            self.dN.append(torch.einsum("vj,ejk->evk", G[q], torch.linalg.inv(J)))
            self.w.append(0.125 * torch.linalg.det(J))
        self.F = torch.zeros(self.n, dtype=torch.float64, device=d)
        if faces is not None:
            self._tractions(mesh, *faces)
        if point is not None:
            self.F.index_add_(0, torch.as_tensor(np.asarray(point[0], dtype=np.int64), device=d),
                              -torch.as_tensor(point[1], device=d))
        self.F *= self.free

    def _tractions(self, mesh, elem, local, t):
        """Dead tractions, one quadrature point at each face's centre."""
        nodes = np.zeros((len(elem), 4), dtype=np.int64)
        for f in range(6):
            v = [k for k in range(8) if ((k >> (f // 2)) & 1) == f % 2]
            sel = local == f
            nodes[sel] = mesh.conn[elem[sel]][:, v]
        x = mesh.coords[nodes]
        a = 0.5 * (x[:, 1] + x[:, 3] - x[:, 0] - x[:, 2])
        b = 0.5 * (x[:, 2] + x[:, 3] - x[:, 0] - x[:, 1])
        area = np.linalg.norm(np.cross(a, b), axis=1)
        val = 0.25 * area[:, None] * t
        F = np.zeros((mesh.n_nodes, 3))
        for k in range(4):
            np.add.at(F, nodes[:, k], val)
        self.F += torch.as_tensor(F.reshape(-1), device=self.dev)

    def scatter(self, fe):
        out = torch.zeros(self.n, dtype=torch.float64, device=self.dev)
        out.index_add_(0, self.dof.reshape(-1), fe.reshape(-1))
        return out

    def forces(self, u):
        ue = u[self.dof].reshape(-1, 8, 3)
        f = torch.zeros_like(ue)
        for dN, w in zip(self.dN, self.w):
            Fm = torch.einsum("evi,evj->eij", ue, dN) + torch.eye(3, dtype=torch.float64, device=self.dev)
            FiT = torch.linalg.inv(Fm).transpose(1, 2)
            lnJ = torch.log(torch.linalg.det(Fm))
            P = self.mu[:, None, None] * (Fm - FiT) + (self.lam * lnJ)[:, None, None] * FiT
            f += torch.einsum("e,eij,evj->evi", w, P, dN)
        return self.scatter(f) * self.free

    def tangents(self, u):
        ue = u[self.dof].reshape(-1, 8, 3)
        ne = len(ue)
        K = torch.zeros(ne, 8, 3, 8, 3, dtype=torch.float64, device=self.dev)
        eye = torch.eye(3, dtype=torch.float64, device=self.dev)
        for dN, w in zip(self.dN, self.w):
            Fm = torch.einsum("evi,evj->eij", ue, dN) + eye
            g = torch.einsum("eji,evj->evi", torch.linalg.inv(Fm), dN)
            lnJ = torch.log(torch.linalg.det(Fm))
            gg = torch.einsum("eai,ebj->eaibj", g, g)
            K += (w * self.lam)[:, None, None, None, None] * gg
            K += (w * (self.mu - self.lam * lnJ))[:, None, None, None, None] * gg.transpose(2, 4)
            m = torch.einsum("e,eak,ebk->eab", w * self.mu, dN, dN)
            for c in range(3):
                K[:, :, c, :, c] += m
        K = K.reshape(ne, 24, 24)
        fe = self.free[self.dof]
        return K * fe[:, :, None] * fe[:, None, :]

    def solve(self, K, b, rtol=1e-13, max_iter=20000):
        """Block-Jacobi CG with the element matrices; the constrained dofs of b are zero."""
        nn = self.n // 3
        D = torch.zeros(nn, 3, 3, dtype=torch.float64, device=self.dev)
        K8 = K.reshape(-1, 8, 3, 8, 3)
        for v in range(8):
            D.index_add_(0, self.conn[:, v], K8[:, v, :, v, :])
        D += torch.diag_embed(1.0 - self.free.reshape(nn, 3))
        Di = torch.linalg.inv(D)

        def mul(x):
            return self.scatter(torch.bmm(K, x[self.dof][:, :, None])[:, :, 0])

        def pre(r):
            return torch.bmm(Di, r.reshape(nn, 3, 1)).reshape(-1)

        x = torch.zeros_like(b)
        for _ in range(2):  # the second sweep on the true residual
            r = b - mul(x)
            z = pre(r)
            p, rz = z.clone(), torch.dot(r, z)
            stop = rtol * float(b.norm())
            for k in range(max_iter):
                q = mul(p)
                a = rz / torch.dot(p, q)
                x = x + a * p
                r = r - a * q
                if k % 50 == 49 and float(r.norm()) <= stop:
                    break
                z = pre(r)
                rz, old = torch.dot(r, z), rz
                p = z + (rz / old) * p
        return x

    def forcing(self, nr, lf):
        """A loose solve is enough far from the solution: every correction adds its own digits."""
        return min(1e-3, max(1e-10, 1e-3 * nr / (abs(lf) * float(self.F.norm()))))

    def newton(self, factors, max_iter=25):
        u = torch.zeros(self.n, dtype=torch.float64, device=self.dev)
        for lf in factors:
            last = math.inf
            for _ in range(max_iter):
                r = lf * self.F - self.forces(u)
                nr = float(r.norm())
                if nr < 1e-7 * lf * float(self.F.norm()) and nr > 0.25 * last:
                    break  # rounding is reached
                last = nr
                u = u + self.solve(self.tangents(u), r, rtol=self.forcing(nr, lf))
        return u


class _ExactEAS(_Exact):
    """Elements with nine enhanced modes: energies differentiated by torch, modes condensed per element."""

    def __init__(self, *a, displacement_gradient, **k):
        super().__init__(*a, **k)
        self.dg = displacement_gradient
        ne = len(self.conn)
        self.alpha = torch.zeros(ne, 9, dtype=torch.float64, device=self.dev)
        G0 = torch.zeros(8, 3, dtype=torch.float64, device=self.dev)
        for v in range(8):
            for d in range(3):
                G0[v, d] = 0.25 if (v >> d) & 1 else -0.25
        J0 = torch.einsum("evi,vj->eij", self.X[self.conn], G0)
        self.J0i, detJ0 = torch.linalg.inv(J0), torch.linalg.det(J0)
        self.scale = torch.stack([detJ0 / (8.0 * w) for w in self.w])
        self.dNs, self.ws = torch.stack(self.dN, 1), torch.stack(self.w, 1)
        xi = torch.tensor([[(_G if (q >> d) & 1 else -_G) for d in range(3)] for q in range(8)], dtype=torch.float64,
                          device=self.dev)
        self.xi = xi

    def _energy(self, v, dN, w, J0i, sc, lam, mu):
        ue, al = v[:24].reshape(8, 3), v[24:].reshape(3, 3)
        H = torch.einsum("vi,qvj->qij", ue, dN)
        eye = torch.eye(3, dtype=torch.float64, device=self.dev)
        M = al[None] * self.xi[:, None, :]  # entry (i, j) linear in xi_j
        if self.dg:
            Fm = eye + H + sc[:, None, None] * (J0i.T @ M @ J0i)
            C = Fm.transpose(1, 2) @ Fm
        else:
            M = 0.5 * (M + M.transpose(1, 2))
            Fm = eye + H
            C = Fm.transpose(1, 2) @ Fm + 2.0 * sc[:, None, None] * (J0i.T @ M @ J0i)
        lnJ = 0.5 * torch.log(self._det(C))
        tr = C[:, 0, 0] + C[:, 1, 1] + C[:, 2, 2]
        return torch.sum(w * (0.5 * mu * (tr - 3.0 - 2.0 * lnJ) + 0.5 * lam * lnJ * lnJ))

    @staticmethod
    def _det(m):
        return (m[:, 0, 0] * (m[:, 1, 1] * m[:, 2, 2] - m[:, 1, 2] * m[:, 2, 1])
                - m[:, 0, 1] * (m[:, 1, 0] * m[:, 2, 2] - m[:, 1, 2] * m[:, 2, 0])
                + m[:, 0, 2] * (m[:, 1, 0] * m[:, 2, 1] - m[:, 1, 1] * m[:, 2, 0]))

    def _condensed(self, u):
        v = torch.cat([u[self.dof], self.alpha], 1)
        arg = (v, self.dNs, self.ws, self.J0i, self.scale.T, self.lam, self.mu)
        g, H = [], []
        grad = torch.func.grad(self._energy)
        both = torch.func.vmap(lambda *a: (grad(*a), torch.func.jacfwd(grad)(*a)))
        with warnings.catch_warnings():
            warnings.simplefilter("ignore")
            for part in zip(*[t.split(1024) for t in arg]):
                a, b = both(*part)
                g.append(a)
                H.append(b)
        g, H = torch.cat(g), torch.cat(H)
        self.D, self.L, self.rt = H[:, 24:, 24:], H[:, 24:, :24], g[:, 24:]
        Y = torch.linalg.solve(self.D, torch.cat([self.L, self.rt[:, :, None]], 2))
        f = g[:, :24] - torch.bmm(self.L.transpose(1, 2), Y[:, :, 24:])[:, :, 0]
        K = H[:, :24, :24] - torch.bmm(self.L.transpose(1, 2), Y[:, :, :24])
        fe = self.free[self.dof]
        return self.scatter(f) * self.free, K * fe[:, :, None] * fe[:, None, :]

    def newton(self, factors, max_iter=25):
        u = torch.zeros(self.n, dtype=torch.float64, device=self.dev)
        for lf in factors:
            last = math.inf
            for _ in range(max_iter):
                f, K = self._condensed(u)
                r = lf * self.F - f
                nr = float(r.norm())
                if nr < 1e-7 * lf * float(self.F.norm()) and nr > 0.25 * last:
                    break  # rounding is reached
                last = nr
                du = self.solve(K, r, rtol=self.forcing(nr, lf))
                rhs = self.rt + torch.bmm(self.L, du[self.dof][:, :, None])[:, :, 0]
                self.alpha = self.alpha - torch.linalg.solve(self.D, rhs)
                u = u + du
        return u


def exact(case, seed):
    op = case["op"]
    if op in ("residual", "tangent", "solve"):
        p, u = _state(case, seed)
        ex = _Exact(p.mesh, p.lam, p.mu, p.fixed, (p.face_elem, p.face_local, p.face_traction))
        u = torch.as_tensor(u, device=ex.dev)
        if op == "residual":
            return (ex.forces(u) - ex.F).cpu().numpy()
        K = ex.tangents(u)
        if op == "solve":
            return ex.solve(K, torch.as_tensor(_rhs(p, seed), device=ex.dev)).cpu().numpy()
        rows = ex.dof[:, :, None].expand(-1, 24, 24).reshape(-1)
        cols = ex.dof[:, None, :].expand(-1, 24, 24).reshape(-1)
        # column-major: sorted by column, then row; the constrained diagonal is one
        T = torch.sparse_coo_tensor(torch.stack([cols, rows]), K.reshape(-1), (ex.n, ex.n)).coalesce()
        v, i = T.values(), T.indices()
        fixed = (ex.free[i[0]] == 0) & (i[0] == i[1])
        return {"data": torch.where(fixed, torch.ones_like(v), v).cpu().numpy(), "indices": None, "indptr": None}
    if op == "path":
        p = _cantilever(case, seed)
        ex = _Exact(p.mesh, p.lam, p.mu, p.fixed, (p.face_elem, p.face_local, p.face_traction))
        return ex.newton([case["end"] * (k + 1) / case["steps"] for k in range(case["steps"])]).cpu().numpy()
    if op == "eas_path":
        p = _golden(case, seed)
        ex = _ExactEAS(p.mesh, p.lam, p.mu, p.fixed, point=(p.pl_dofs, p.pl_values), displacement_gradient=True)
        return ex.newton([(k + 1) / 5 for k in range(5)]).cpu().numpy()
    if op == "eas_block":
        p = _block(case, seed)
        ex = _ExactEAS(p.mesh, p.lam, p.mu, p.fixed, (p.face_elem, p.face_local, p.face_traction),
                       displacement_gradient=False)
        return ex.newton([STEP["eas_block"]]).cpu().numpy()
    if case["n"] > 40:
        return None  # minutes: the hardest instances need thousands of iterations
    bp = _batch(case, seed)
    ex = _Exact(bp.mesh, bp.lam_e, bp.mu_e, bp.fixed, (bp.face_elem, bp.face_local, bp.face_traction))
    return ex.newton([STEP["batched"]]).cpu().numpy()
