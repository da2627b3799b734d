"""Performance cases: the calls a user of this solver spends time in, with inputs, one pass and a
64-bit answer for each.

* ``residual``  -- ``FVMEquation.forward``, the drop-in residual (2D and 3D, boundaries or periodic,
                   the reference's gradient stencil or a widened one).
* ``steps``     -- time stepping of one mesh: CUDA-graph replay with a CFL time step (how the
                   benchmark runs it) or eager steps with the error-adaptive integrator.
* ``ensemble``  -- ``BatchedFVM``: many 2D meshes of 2 000 to 60 000 cells per launch, Adams-Bashforth 3.
* ``operators`` -- the sparse-operator seam: the residual's own operators through ``SPM.spMM / spMV``.
* ``host``      -- ``step_host``: independent states that live in pinned host memory.
* ``propose``   -- the learned corrector's proposal (residual, network inference, conservation shift).
* ``train``     -- one training iteration of the corrector (residual, inputs, forward, backward, Adam).

Meshes are built once per process and shared by all seeds of a case, as a user's program keeps its
mesh; the flow on it comes from the seed.
"""
from __future__ import annotations

import functools
import math
import os

import torch

from fvm_solver_b200 import batched, corrector, workloads
from fvm_solver_b200.equation import FVMEquation, FluidConstitution2D, FluidConstitution3D
from fvm_solver_b200.sparse import SPMB200

CHECKPOINT = os.path.join(os.path.dirname(os.path.abspath(workloads.__file__)), "checkpoints", "corrector_2d_k8.pt")
DEV = "cuda"
ENSEMBLE_SEED = 1234
ENSEMBLE_CFL = 0.3          # the benchmark's ensemble: AB3 needs a smaller step than Runge-Kutta


# ---------------------------------------------------------------------------------------------
# The cases
# ---------------------------------------------------------------------------------------------
def listed():
    return [
        # a small 2D mesh, the reference's default problem size: launches and latency
        dict(name="residual_channel_2k", path="residual", mesh="channel", cells=2000, stencil=0),
        # the widened gradient stencil on an ordinary 2D mesh
        dict(name="residual_channel_wide", path="residual", mesh="channel", cells=30011, stencil=16),
        # 3D flow around a body, a boundary on every side
        dict(name="residual_sphere_120k", path="residual", mesh="sphere", cells=120001, stencil=0),
        # the benchmark's 2D channel case: a trajectory of SSP-RK3 steps as one graph
        dict(name="steps_channel_11k", path="steps", mesh="channel", cells=11300, solver="Butcher/SSP_RK3", steps=10,
             graph=True),
        # the benchmark's periodic box at a size past the L2 cache: RK4
        dict(name="steps_box_855k", path="steps", mesh="box", cells=50, solver="Butcher/RK4", steps=2, graph=True),
        # the reference's default integrator (error-adaptive, FP64 norms) on a 3D mesh, eager
        dict(name="steps_sphere_adaptive", path="steps", mesh="sphere", cells=60013, solver="RK3_SSP4/", steps=4,
             graph=False),
        # the batched ensemble
        dict(name="ensemble_16", path="ensemble", cases=16, steps=9),
        # the operator seam on a small 2D and a large 3D mesh
        dict(name="operators_channel_11k", path="operators", mesh="channel", cells=11300),
        dict(name="operators_box_438k", path="operators", mesh="box", cells=40),
        # snapshots on the host advanced one step each, copies included
        dict(name="host_box_225k", path="host", mesh="box", cells=32, solver="Butcher/RK4", steps=1, states=6),
        # the learned corrector on a batch: one proposal, and one training iteration
        dict(name="corrector_propose_16", path="propose", cases=16),
        dict(name="corrector_train_16", path="train", cases=16),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choice(["residual", "residual", "steps", "steps", "ensemble", "operators", "operators", "host",
                       "propose", "train"])
    mesh = rng.choice(["channel", "sphere", "box"])
    cells = {"channel": _log_int(rng, 1500, 120000), "sphere": _log_int(rng, 20000, 200000),
             "box": _log_int(rng, 8, 42)}[mesh]
    if path == "residual":
        wide = rng.choice([0, 0, 9, 16]) if mesh == "channel" else 0
        return dict(path=path, mesh=mesh, cells=cells, stencil=wide)
    if path == "steps":
        if rng.random() < 0.35:
            solver, graph = rng.choice(["RK3_SSP4/", "Butcher_adapt/RK3_SSP5"]), False
        else:
            solver, graph = rng.choice(["Butcher/RK4", "Butcher/SSP_RK3", "Butcher/RK4_SSP5"]), True
        return dict(path=path, mesh=mesh, cells=cells, solver=solver, steps=rng.randint(1, 6), graph=graph)
    if path == "ensemble":
        return dict(path=path, cases=rng.randint(2, 20), steps=3 * rng.randint(1, 4))
    if path == "operators":
        return dict(path=path, mesh=mesh, cells=cells)
    if path == "host":
        return dict(path=path, mesh="box", cells=_log_int(rng, 8, 32), solver=rng.choice(["Butcher/RK4", "Butcher/SSP_RK3"]),
                    steps=rng.randint(1, 3), states=rng.randint(2, 6))
    return dict(path=path, cases=rng.randint(2, 20))


# ---------------------------------------------------------------------------------------------
# Meshes (built once per process) and flows (from the seed)
# ---------------------------------------------------------------------------------------------
@functools.lru_cache(maxsize=None)
def _mesh(mesh, cells, stencil=0):
    """(workload case, host tables) of one mesh; ``cells`` is the point count per axis of the box."""
    kw = dict(grad_stencil=stencil) if stencil else {}
    if mesh == "channel":
        c = workloads.channel_cylinder(n_cells=cells, **kw)
    elif mesh == "sphere":
        c = workloads.sphere(cells, **kw)
    else:
        c = workloads.taylor_green(cells, **kw)
    return c, c.tables()


@functools.lru_cache(maxsize=None)
def _parts(cases):
    return batched.build_ensemble_tables(cases, base_seed=ENSEMBLE_SEED)


def _case_params(cases):
    p = [workloads.ensemble_params(i, ENSEMBLE_SEED) for i in range(cases)]
    return torch.tensor([[q["mach"], math.log10(q["reynolds"])] for q in p], dtype=torch.float32)


def _flow(state0, centroids, C_v, seed, shift=0.0):
    """A conserved state [N][C] (float32, on the GPU): ``state0`` with seeded smooth velocity (10 %),
    density (2 %) and temperature (1 %) waves; ``shift`` moves the waves' phase (a later instant)."""
    g = torch.Generator().manual_seed(1000003 + int(seed))
    dim = centroids.shape[1]
    C = dim + 2
    s = state0.to(DEV).double()
    x = centroids.to(DEV).double()
    x = x / x.abs().max()
    V, rho = s[:, :dim] / s[:, dim:dim + 1], s[:, dim]
    T = (s[:, dim + 1] / rho - 0.5 * V.square().sum(1)) / C_v
    speed = V.norm(dim=1, keepdim=True)
    wave = torch.zeros((s.shape[0], C), device=DEV, dtype=torch.float64)
    for _ in range(3):
        k = torch.randn(C, dim, generator=g, dtype=torch.float64).to(DEV) * 8.0
        ph = (torch.rand(C, generator=g, dtype=torch.float64) * 2 * math.pi).to(DEV)
        wave += torch.sin(x @ k.t() + ph + shift) / 3
    V = V + 0.1 * speed * wave[:, :dim]
    rho = rho * (1 + 0.02 * wave[:, dim])
    T = T * (1 + 0.01 * wave[:, dim + 1])
    e = rho * (C_v * T + 0.5 * V.square().sum(1))
    return torch.cat([V * rho.unsqueeze(1), rho.unsqueeze(1), e.unsqueeze(1)], 1).float()


def _prims64(s, dim, C_v):
    V = s[:, :dim] / s[:, dim:dim + 1]
    T = (s[:, dim + 1:] / s[:, dim:dim + 1] - 0.5 * V.square().sum(1, keepdim=True)) / C_v
    return torch.cat([V, s[:, dim:dim + 1], T], 1)


def _equation(case, seed):
    c, T = _mesh(case["mesh"], case["cells"], case.get("stencil", 0))
    phy = (FluidConstitution2D if c.dim == 2 else FluidConstitution3D)(c.cfg)
    if "solver" in case:
        c.cfg.solver_name, c.cfg.solver_extra = case["solver"].split("/")
    s = _flow(c.state0, T.kernel.centroids, c.cfg.C_v, seed)
    return FVMEquation.from_kernel_tables(c.cfg, phy, T.kernel, s, build_solver="solver" in case), s


def _batch(case):
    parts = _parts(case["cases"])
    cfg = workloads.ensemble_case(0, device=DEV, base_seed=ENSEMBLE_SEED, cfl=ENSEMBLE_CFL).cfg
    if case["path"] in ("propose", "train"):      # the corrector's fallback integrator
        cfg.solver_name, cfg.solver_extra, cfg.cfl = "Butcher", "SSP_RK3", None
    return batched.BatchedFVM(parts, cfg, device=DEV), cfg


# ---------------------------------------------------------------------------------------------
# One pass of each path
# ---------------------------------------------------------------------------------------------
def prepare(case, seed):
    path = case["path"]
    if path == "residual":
        eq, s = _equation(case, seed)
        prims = _prims64(s.double(), eq.mesh.dim, eq.cfg.C_v).float().contiguous()
        return dict(path=path, eq=eq, prims=prims)
    if path == "steps":
        eq, _ = _equation(case, seed)
        replay = eq.t_solver.graph_steps(case["steps"]) if case["graph"] else None
        return dict(path=path, eq=eq, replay=replay, steps=case["steps"])
    if path == "host":
        eq, s = _equation(case, seed)
        n = case["states"]
        c, T = _mesh(case["mesh"], case["cells"])
        ins = [_flow(c.state0, T.kernel.centroids, c.cfg.C_v, seed, 0.1 * i).cpu().pin_memory() for i in range(n)]
        outs = [torch.empty_like(ins[0]).pin_memory() for _ in range(n)]
        return dict(path=path, eq=eq, ins=ins, outs=outs, steps=case["steps"])
    if path == "operators":
        ops, x = _operators(case["mesh"], case["cells"]), _operands(case, seed)
        return dict(path=path, ops=ops, x=x)
    b, cfg = _batch(case)
    s = _flow(torch.cat([p.state0 for p in b.parts]), b.kt.centroids, cfg.C_v, seed)
    b.cells.state = s
    if path == "ensemble":
        b.t_solver.update_cfl_dt(ENSEMBLE_CFL)
        return dict(path=path, eq=b, steps=case["steps"])
    b.t_solver.update_cfl_dt(0.5)
    m = corrector.CorrectorModel.load(CHECKPOINT, b, _case_params(case["cases"]))
    r0 = torch.empty_like(s)
    if path == "propose":
        m.inputs(s, r0)                               # the network's buffers, kept by the model
        return dict(path=path, m=m, s=s, r0=r0, prop=torch.empty_like(s), out=m.net.forward(m.nbr, store_pre=False))
    m.net.lr = 1e-5                                   # a late, decayed learning rate
    later = _flow(torch.cat([p.state0 for p in b.parts]), b.kt.centroids, cfg.C_v, seed, 0.02)
    m.net._alloc(s.shape[0])
    return dict(path=path, m=m, s=s, later=later, r0=r0, target=torch.empty_like(s))


def run(state):
    path = state["path"]
    if path == "residual":
        return {"dudt": state["eq"].forward(state["prims"])}
    if path == "steps":
        eq = state["eq"]
        if state["replay"] is not None:
            state["replay"]()
        else:
            eq.t_solver.step(state["steps"])
        return {"state": eq.cells.state, "dt": eq.t_solver.dt}
    if path == "ensemble":
        eq = state["eq"]
        eq.t_solver.step(state["steps"])
        return {"state": eq.cells.state, "dt": eq.t_solver.dt}
    if path == "host":
        return {"outs": state["eq"].t_solver.step_host(state["ins"], state["outs"], steps=state["steps"])}
    if path == "operators":
        ops, x = state["ops"], state["x"]
        return {"grad": ops["G"].spMM(x["cells"]), "div": ops["F"].spMM(x["flux"]),
                "face_grad": ops["A"].spMV(x["flat"], x["bias"]), "rho_grad": ops["G"].spMV(x["cells"][:, -2])}
    m, s, r0 = state["m"], state["s"], state["r0"]
    m.res(s, r0)
    if path == "propose":
        m.predict(s, state["prop"], r0)
        return {"residual": r0, "out": state["out"], "proposal": state["prop"]}
    m.inputs(s, r0)
    torch.sub(state["later"], s, out=state["target"])
    state["target"].sub_(m.base).div_(m.scale)
    m.net.train_step(m.nbr, state["target"])
    return {"out": m.net._bufs["out"], "moments": m.net.m, "weights": m.net.params}


@functools.lru_cache(maxsize=4)
def _operators(mesh, cells):
    _, T = _mesh(mesh, cells)
    return {"G": SPMB200(T.ops.G_mats, DEV), "F": SPMB200(T.ops.flux_mat, DEV), "A": SPMB200(T.ops.A_face_grad, DEV)}


def _operands(case, seed):
    c, T = _mesh(case["mesh"], case["cells"])
    p = _prims64(_flow(c.state0, T.kernel.centroids, c.cfg.C_v, seed).double(), c.dim, c.cfg.C_v).float()
    cells = torch.cat([p, p[T.kernel.bc_cell.long().to(DEV)] * 1.01]).contiguous() if T.n_bc else p.contiguous()
    g = torch.Generator(device=DEV).manual_seed(int(seed))
    flux = torch.randn((T.n_facets, T.n_comp), device=DEV, generator=g)
    return {"cells": cells, "flux": flux, "flat": p.reshape(-1).contiguous(), "bias": T.ops.b_face_grad.to(DEV)}


# ---------------------------------------------------------------------------------------------
# Bytes and operations that a pass cannot do without
# ---------------------------------------------------------------------------------------------
def _stage_bytes(N, F, dim):
    """One residual evaluation or stage in one pass: every mesh array and the state read once, the
    result written once (4-byte values)."""
    C, K, KG = dim + 2, dim + 1, dim + 2
    cell = 2 * C + dim * KG + KG + K + K * dim + 2 + 2 * K + 2 * K
    return 4 * (N * cell + F * (2 * dim + 3))


def work(case):
    path = case["path"]
    if path in ("residual", "steps", "operators", "host"):
        c, T = _mesh(case["mesh"], case["cells"], case.get("stencil", 0))
        N, F, dim, C = T.n_cells, T.n_facets, T.dim, T.n_comp
        if path == "operators":
            def ell(A, cols, B, bias=0):
                M = A.shape[0]
                return 8 * A._nnz() + 4 * (cols + M) * B + 4 * M * bias
            ops = T.ops
            by = ell(ops.G_mats, N + T.n_bc, C) + ell(ops.flux_mat, F, C) + ell(ops.A_face_grad, N * C, 1, 1) + \
                ell(ops.G_mats, N + T.n_bc, 1)
            return {"bytes": by, "flops": 2 * (ops.G_mats._nnz() * (C + 1) + ops.flux_mat._nnz() * C + ops.A_face_grad._nnz())}
        kg = T.kernel.kg
        stage = _stage_bytes(N, F, dim) + 4 * N * (kg - dim - 2) * (dim + 1)
        flops = N * (700 if dim == 3 else 350) + F * (420 if dim == 3 else 250)
        if path == "residual":
            return {"bytes": stage, "flops": flops}
        stages = {"RK4": 4, "SSP_RK3": 3, "RK4_SSP5": 5, "RK3_SSP5": 5}.get(case["solver"].split("/")[1], 4)
        n = case["steps"] * stages * case.get("states", 1)
        return {"bytes": stage * n + 8 * N * C * case.get("states", 0), "flops": flops * n}
    parts = _parts(case["cases"])
    N, F = sum(p.kt.n_cells for p in parts), sum(p.kt.n_facets for p in parts)
    stage, flops = _stage_bytes(N, F, 2), N * 350 + F * 250
    if path == "ensemble":
        return {"bytes": stage * case["steps"], "flops": flops * case["steps"]}
    W, L = 64, 4
    net = N * (4 * 8 + 4 * 9 + L * (2 * 4 * W + 12) + 4 * 4)           # features, h in and out per layer, outputs
    gemm = 2 * N * W * (W + L * 2 * W)
    if path == "propose":
        return {"bytes": stage + net + N * 4 * 4 * 3, "flops": flops + gemm}
    return {"bytes": stage + net + N * L * 4 * W * 5, "flops": flops + 3 * gemm}


# ---------------------------------------------------------------------------------------------
# 64-bit answers (plain torch)
# ---------------------------------------------------------------------------------------------
class _Residual64:
    """dU/dt of the finite-volume residual in FP64 from the mesh arrays, single mesh or batch."""

    def __init__(self, kt, gas, mu, mu_b, kappa, lim_p, case=None):
        T_0, S, C_v, gamma, v_factor = gas
        up = lambda t: t.to(DEV)
        self.kt, self.dim, self.C = kt, kt.dim, kt.n_comp
        self.T_0, self.S, self.C_v, self.gamma, self.R, self.vf = T_0, S, C_v, gamma, C_v * (gamma - 1), v_factor
        self.lim_p = lim_p
        self.case = None if case is None else {k: up(v) for k, v in case.items()}
        f64 = lambda v: torch.as_tensor(v, device=DEV, dtype=torch.float64)
        if self.case is None:
            self.mu, self.mu_b, self.kappa = f64(mu), f64(mu_b), f64(kappa)
        else:
            fc = self.case["face_case"].long()
            self.mu, self.mu_b, self.kappa = (f64(v)[fc] for v in (mu, mu_b, kappa))
        self.t = {k: (up(v).double() if v.is_floating_point() else up(v).long())
                  for k, v in vars(kt).items() if isinstance(v, torch.Tensor)}

    def boundary(self, P, prev):
        t, d, C = self.t, self.dim, self.C
        kind, cell = t["bc_kind"], t["bc_cell"]
        neu = (kind == 2).double()
        out = neu * P[cell] + t["bc_b"]
        if prev is not None:
            out = out + neu * torch.einsum("bd,bdc->bc", t["bc_l"], prev[cell])
        if self.kt.n_char:
            b = torch.nonzero(t["bc_char"] >= 0)[:, 0]
            j = t["bc_char"][b]
            U, n = P[t["ch_cell"][j]], t["ch_normal"][j]
            V, rho, T = U[:, :d], U[:, d], U[:, d + 1]
            vn = (V * n).sum(1)
            vt = V - vn[:, None] * n
            p, c = self.R * rho * T, (self.gamma * self.R * T).sqrt()
            if self.case is None:
                scale = 10.0 / c.mean()
            else:
                k = self.case["bc_case"].long()[b]
                nc = int(self.case["bc_case"].max()) + 1
                s = torch.zeros(nc, device=DEV, dtype=torch.float64).index_add_(0, k, c)
                scale = (10.0 * torch.bincount(k, minlength=nc) / s)[k]
            drho, dvn, dp = t["ch_rho"][j] - rho, t["ch_vn"][j] - vn, t["ch_p"][j] - p
            h_dp, h_dvn = 0.5 * dp / c ** 2, 0.5 * rho * dvn / c
            g = [0.5 * (1 - torch.tanh(scale * (vn + q * c))) for q in (-1, 0, 1)]
            x = [(-h_dvn + h_dp) * g[0], (drho - dp / c ** 2) * g[1], (h_dvn + h_dp) * g[2]]
            rho_b = rho + x[0] + x[1] + x[2]
            vn_b = vn + c / rho * (x[2] - x[0])
            p_b = p + c * c * (x[0] + x[2])
            vtb = g[1][:, None] * vt + (1 - g[1][:, None]) * t["ch_vt"][j]
            out[b] = torch.cat([vn_b[:, None] * n + vtb, rho_b[:, None], (p_b / (self.R * rho_b))[:, None]], 1)
        return out

    def limiter(self, delta, dU, eps):
        if self.lim_p != 4:
            raise NotImplementedError
        a, b = delta.abs(), dU.abs()
        S = 2 * b * (a * a + 2 * b * (2 * b - a))
        phi = (a ** 4 + eps + a * S) / (a ** 4 + eps + b * (delta ** 3 + S))
        return torch.where(a < 2 * b, phi, torch.ones_like(phi))

    def __call__(self, P, prev=None):
        t, d, C, K = self.t, self.dim, self.C, self.dim + 1
        N = self.kt.n_cells
        Ub = self.boundary(P, prev) if self.kt.n_bc else P[:0]
        Uc = torch.cat([P, Ub])
        g = torch.zeros((N, d, C), device=DEV, dtype=torch.float64)
        for k in range(self.kt.kg):
            g += t["g_vals"][:, k].t()[:, :, None] * Uc[t["g_cols"][k]][:, None, :]
        up, lo = P.clone(), P.clone()
        for j in range(K):
            slot = (t["nb_slot"] >> (4 * j)) & 15
            X = Uc[t["g_cols"].gather(0, slot[None])[0]]
            up, lo = torch.maximum(up, X), torch.minimum(lo, X)
        phi = None
        for j in range(K):
            dU = torch.einsum("ndc,nd->nc", g, t["disp"][j].t())
            ph = self.limiter(torch.where(dU > 0, up - P, lo - P), dU, t["eps"][:, None])
            phi = ph if phi is None else torch.minimum(phi, ph)
        g = g * phi[:, None, :]
        F = self.kt.n_facets
        U = torch.empty((F, 2, C), device=DEV, dtype=torch.float64)
        gf = torch.empty((F, 2, d, C), device=DEV, dtype=torch.float64)
        for j in range(K):
            side = (t["side"] >> j) & 1
            U[t["c2f"][j], side] = P + torch.einsum("ndc,nd->nc", g, t["disp"][j].t())
            gf[t["c2f"][j], side] = g
        bc = None
        if self.kt.n_bc:
            bc = (t["bc_face"], t["bc_side"])
            U[bc] = Ub
            gf[bc] = g[t["bc_cell"]]
        comp = list(range(d)) + [d + 1]
        gl = gf.mean(1)[:, :, comp]
        nhat = t["normals"] / t["fsize"][:, None]
        dn = t["inv_d"][:, None] * (P[t["fcell"][:, 1]] - P[t["fcell"][:, 0]])
        if bc:
            dn[bc[0]] = t["bc_ga"] * P[t["bc_cell"]] + t["bc_gb"]
        dFdn = dn[:, comp] - torch.einsum("fdk,fd->fk", gl, t["xorth"])
        gF = gl + (dFdn - torch.einsum("fdk,fd->fk", gl, nhat))[:, None, :] * nhat[:, :, None]
        V, rho, T = U[:, :, :d], U[:, :, d], U[:, :, d + 1]
        n = t["normals"]
        mom, v2 = V * rho[:, :, None], V.square().sum(2)
        phin = torch.einsum("fsd,fd->fs", V, n)
        Q, Pr = rho * (self.C_v * T + 0.5 * v2), self.R * rho * T
        Tm = T.mean(1)
        gv = gF[:, :, :d]
        D = 0.5 * (gv + gv.transpose(1, 2))
        mu = self.mu * (Tm / self.T_0) ** 1.5 * (self.T_0 + self.S) / (Tm + self.S)
        mub = self.mu_b * (Tm / self.T_0) ** 2
        I1 = D[:, 0, 0] + D[:, 1, 1]
        tau = (-mub * I1)[:, None, None] * torch.eye(d, device=DEV, dtype=torch.float64) - 2 * mu[:, None, None] * D
        fl = torch.cat([(mom * phin[:, :, None]).mean(1) + Pr.mean(1)[:, None] * n + torch.einsum("fac,fa->fc", tau, n),
                        (rho * phin).mean(1)[:, None],
                        (((Q + Pr) * phin).mean(1) + torch.einsum("fac,fc,fa->f", tau, V.mean(1), n) -
                         self.kappa * dFdn[:, d] * t["fsize"])[:, None]], 1)
        vmax, cmax = v2.amax(1).sqrt(), (self.gamma * self.R * T).amax(1).sqrt()
        vf = torch.clamp(vmax / (cmax + 1e-8), self.vf, 1.0)
        jump = lambda q: (q[:, 0] - q[:, 1])
        fl += 0.5 * t["fsize"][:, None] * torch.cat([(vf * cmax + vmax)[:, None] * jump(mom),
                                                      ((cmax + vmax) * jump(rho))[:, None],
                                                      ((cmax + vmax) * jump(Q))[:, None]], 1)
        out = torch.zeros((N, C), device=DEV, dtype=torch.float64)
        for k in range(self.kt.kf):
            out += t["f_vals"][k][:, None] * fl[t["f_cols"][k]]
        return out, g

    def dt(self, s, cfl):
        """The CFL time step of each case (float32, as the solver keeps it)."""
        P = _prims64(s, self.dim, self.C_v)
        sp = self.t["inv_h"] * (P[:, :self.dim].norm(dim=1) + (self.gamma * self.R * P[:, -1]).sqrt())
        if self.case is None:
            return (cfl / sp.max()).float().double().reshape(1)
        cc = self.case["cell_case"].long()
        top = torch.zeros(int(cc.max()) + 1, device=DEV, dtype=torch.float64).scatter_reduce(0, cc, sp, "amax")
        return (cfl / top).float().double()


_TABLEAU = {
    "RK4": ([[], [0.5], [0, 0.5], [0, 0, 1.0]], [1 / 6, 1 / 3, 1 / 3, 1 / 6], None),
    "SSP_RK3": ([[], [1.0], [0.25, 0.25]], [1 / 6, 1 / 6, 2 / 3], None),
    "RK3_SSP4": ([[], [0.5], [0.5, 0.5], [1 / 6] * 3], [1 / 6, 1 / 6, 1 / 6, 1 / 2], [0.5, 0.5, 0, 0]),
}


def _rk_step(f, s, dt, name, prev):
    """One Runge-Kutta step: (state, increments, embedded difference, last limited gradients)."""
    A, b, lo = _TABLEAU[name]
    k = []
    for row in A:
        r, prev = f(s + sum(a * q for a, q in zip(row, k)) if k else s, prev)
        k.append(dt * r)
    hi = sum(w * q for w, q in zip(b, k))
    return s + hi, k, hi, (None if lo is None else sum(w * q for w, q in zip(lo, k))), prev


def _single64(case):
    c, T = _mesh(case["mesh"], case["cells"], case.get("stencil", 0))
    g = c.cfg
    return c, T, _Residual64(T.kernel, (g.T_0, g.S_const, g.C_v, g.gamma, g.v_factor), g.viscosity, g.visc_bulk,
                             g.thermal_cond, g.lim_p)


def _steps64(R, s, name, steps, adaptive, cfl):
    f = lambda u, prev: R(_prims64(u, R.dim, R.C_v), prev)
    dt, prev = R.dt(s, cfl), None
    for _ in range(steps):
        s0 = s
        s, _, hi, lo, prev = _rk_step(f, s, dt, name, prev)
        if adaptive:
            nrm = lambda q: q.square().sum(0).sqrt()
            E = float((nrm(hi - lo) / (2e-3 + 2e-3 * nrm(hi) + 1e-6 * nrm(s0))).mean())
            a = 0.8 if E > 1 else 0.995
            dt = (dt * (a + (1 - a) * 0.9 * E ** -0.25)).float().double()
        else:
            dt = R.dt(s, cfl)
    return s, dt


def exact(case, seed):
    path = case["path"]
    if path == "operators":
        c, T = _mesh(case["mesh"], case["cells"])
        x = {k: v.double() for k, v in _operands(case, seed).items()}

        def apply(A, X):
            A = A.coalesce()
            i, v = A.indices().to(DEV), A.values().to(DEV).double()
            return torch.zeros((A.shape[0], X.shape[1]), device=DEV, dtype=torch.float64).index_add_(
                0, i[0], v[:, None] * X[i[1]])

        return {"grad": apply(T.ops.G_mats, x["cells"]), "div": apply(T.ops.flux_mat, x["flux"]),
                "face_grad": apply(T.ops.A_face_grad, x["flat"][:, None])[:, 0] + x["bias"],
                "rho_grad": apply(T.ops.G_mats, x["cells"][:, -2:-1])[:, 0]}
    if path in ("residual", "steps", "host"):
        c, T, R = _single64(case)
        start = lambda shift=0.0: _flow(c.state0, T.kernel.centroids, c.cfg.C_v, seed, shift).double()
        if path == "residual":
            return {"dudt": R(_prims64(start(), c.dim, c.cfg.C_v).float().double())[0]}
        name, extra = case["solver"].split("/")
        tab = extra or name
        if tab not in _TABLEAU or (name == "Butcher_adapt"):
            return None
        if path == "steps":
            s, dt = _steps64(R, start(), tab, case["steps"], not extra, c.cfg.cfl)
            return {"state": s, "dt": dt}
        return {"outs": [_steps64(R, start(0.1 * i), tab, case["steps"], False, c.cfg.cfl)[0]
                         for i in range(case["states"])]}
    parts = _parts(case["cases"])
    kt, arrays, _ = batched.concat_tables(parts)
    T_0, S, C_v, gamma, vf, lim_p = parts[0].gas
    R = _Residual64(kt, (T_0, S, C_v, gamma, vf), arrays["case_mu"], arrays["case_mu_b"], arrays["case_kappa"], lim_p,
                    arrays)
    cc = arrays["cell_case"].long().to(DEV)
    s0 = torch.cat([p.state0 for p in parts])
    s = _flow(s0, kt.centroids, C_v, seed).double()
    f = lambda u, prev: R(_prims64(u, 2, C_v), prev)
    if path == "ensemble":
        dt = R.dt(s, ENSEMBLE_CFL)
        h, hist, prev = dt[cc][:, None], [], None
        for _ in range(case["steps"]):
            if len(hist) < 2:
                s, k, _, _, prev = _rk_step(f, s, h, "SSP_RK3", prev)
                hist.insert(0, k[0])
            else:
                r, prev = f(s, prev)
                hist = [h * r] + hist[:2]
                s = s + (23 * hist[0] - 16 * hist[1] + 5 * hist[2]) / 12
        return {"state": s, "dt": dt}
    return _corrector64(case, R, kt, arrays, s, s0, f, seed)


def _corrector64(case, R, kt, arrays, s, s0, f, seed):
    """The corrector's proposal or training iteration in FP64 from the checkpoint's float32 weights."""
    d = torch.load(CHECKPOINT, map_location="cpu", weights_only=True)
    L, k = d["net"]["layers"], int(d["k"])
    p = {n: v.to(DEV).double().requires_grad_(case["path"] == "train") for n, v in d["net"]["params"].items()}
    fmean, finv, scale = (d[n].to(DEV).double() for n in ("fmean", "finv", "scale"))
    cc = arrays["cell_case"].long().to(DEV)
    N = kt.n_cells
    vol = kt.volumes.to(DEV)
    # static features and neighbours
    cen = kt.centroids.to(DEV).double() / torch.tensor([2.0, 1.0], device=DEV, dtype=torch.float64)
    lv = torch.log(vol)
    lv = (lv - lv.mean()) / (lv.std() + 1e-12)
    disp = kt.disp.to(DEV).double().permute(2, 0, 1).reshape(N, -1) / vol.sqrt()[:, None]
    geo = torch.cat([cen, lv[:, None], disp, _case_params(case["cases"]).to(DEV).double()[cc]], 1).float().double()
    cols = kt.g_cols.t().long().to(DEV)
    near = (cols != torch.arange(N, device=DEV)[:, None]) & (cols < N)
    r0, _ = f(s, None)
    base = (k * R.dt(s, 0.5))[cc][:, None] * r0
    X = torch.cat([(torch.cat([s, base], 1) - fmean) * finv, geo], 1)
    silu = torch.nn.functional.silu
    h = silu(X @ p["W_in"][:, :X.shape[1]].t() + p["b_in"])
    count = near.sum(1, keepdim=True).clamp(min=1)
    for l in range(L):
        mean = sum(h[torch.where(near[:, j], cols[:, j], 0)] * near[:, j, None] for j in range(cols.shape[1])) / count
        h = h + silu(torch.cat([h, mean], 1) @ p[f"W{l}"].t() + p[f"b{l}"])
    out = h @ p["W_out"].t() + p["b_out"]
    if case["path"] == "propose":
        S = torch.zeros((case["cases"], 4), device=DEV, dtype=torch.float64).index_add_(0, cc, vol[:, None] * out)
        V = torch.zeros(case["cases"], device=DEV, dtype=torch.float64).index_add_(0, cc, vol)
        shift = S / V[:, None] * scale
        shift[:, :2] = 0
        return {"residual": r0, "out": out, "proposal": s + base + scale * out - shift[cc]}
    later = _flow(s0, kt.centroids, R.C_v, seed, 0.02).double()
    target = (later - s - base) / scale
    (out - target).square().mean().backward()
    g = {n: v.grad for n, v in p.items()}
    return {"out": out.detach(), "moments": {n: 0.1 * v for n, v in g.items()},
            "weights": {n: (v - 1e-5 * g[n] / (g[n].abs() + 1e-8)).detach() for n, v in p.items()}}
