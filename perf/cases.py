"""The work that a user of this package has it do, as cases that can be timed and compared.

Each case goes through the public entry points a driver calls: whole load steps
(``solver``, ``compute_avg_stress``, ``update_int_vars_gp``, with the reference's choices or
with the benchmark settings of ``workloads.bench_stepper``), the Newton system of an iterate
(``newton_update_helper``), its linear solve (``linear_solver``), the constitutive update at
arbitrary Gauss points (``gp_map``), a ragged batch of RVEs (``Batch.step``) and the gradient
of a load history (``LoadHistory``).

``listed()`` gives the cases, ``draw(rng)`` one more of the same ranges, ``prepare(case,
seed)`` what a program has in hand before the call, ``run(state)`` one pass, ``work(case)``
the bytes and operations a pass cannot do without, and ``exact(case, seed)`` the outputs in
plain 64-bit torch where that takes seconds.
"""
from __future__ import annotations

import importlib
import math

import numpy as np
import torch

PKG = "jax-cpfem_gb300"
STRAIN, DT = 1e-3, 0.1            # the load increment of the benchmark workloads


def _mod(name=""):
    return importlib.import_module(PKG + (("." + name) if name else ""))


def listed():
    return [
        # one HEX8 element of copper with per-point parameters: the single-element calibration
        # runs (calibration case 1), where launches and latency are everything
        dict(name="calibration-1-element", kind="steps", path="reference", material="CALIB_CASE1", nx=1, ny=1, nz=1,
             grains=1, steps=4, line_search=False),
        # the 10^3 copper single crystal with the reference driver's own choices (Jacobi
        # BiCGSTAB to 1e-10, guess from the last solution): what a ported driver runs first
        dict(name="copper-10-reference", kind="steps", path="reference", material="COPPER", nx=10, ny=10, nz=10,
             grains=1, steps=2, line_search=False),
        # dual-phase steel on an odd box (ragged groups, no multigrid): the per-phase stiffness
        # and parameters of the DP-steel driver, BCC24
        dict(name="dualphase-13x9x7-reference", kind="steps", path="reference", material="DP_STEEL", nx=13, ny=9, nz=7,
             grains=8, steps=2, line_search=False),
        # the benchmark workload: 32^3 cells, 64 grains, 304 steel, multigrid, FP32 tangent
        dict(name="steel-32-benchmark", kind="steps", path="benchmark", material="BENCH_STEEL", nx=32, ny=32, nz=32,
             grains=64, steps=3, line_search=False),
        # the tantalum workload (24 slip systems) at the size its parity test uses
        dict(name="tantalum-16-benchmark", kind="steps", path="benchmark", material="BENCH_TANTALUM", nx=16, ny=16,
             nz=16, grains=24, steps=3, line_search=False),
        # the Newton system of two successive iterates of a load step: constitutive pass with
        # the consistent tangent, scatter, row elimination
        dict(name="system-steel-32", kind="system", material="BENCH_STEEL", nx=32, ny=32, nz=32, grains=64),
        # the same with 24 slip systems on an odd box
        dict(name="system-tantalum-21x17x11", kind="system", material="BENCH_TANTALUM", nx=21, ny=17, nz=11, grains=24),
        # the linear solve of a Newton iterate to a direct solver's accuracy (the arc-length
        # setting), multigrid with the FP32 V-cycle, on the benchmark mesh
        dict(name="linear-multigrid-32", kind="linear", material="BENCH_STEEL", nx=32, ny=32, nz=32, grains=64,
             precond="mg", precision="fp32", transposed=False),
        # the adjoint's transposed solve with the reference's Jacobi preconditioner
        dict(name="linear-jacobi-transposed-16", kind="linear", material="BENCH_STEEL", nx=16, ny=16, nz=16, grains=24,
             precond="jacobi", precision="fp64", transposed=True),
        # a ragged batch of RVEs (edges and parameters as in the 256-RVE sweep)
        dict(name="batch-24-rves", kind="batch", material="BENCH_STEEL", count=24, edge_min=8, edge_max=16, grains=16,
             steps=2),
        # the gradient of a load history with respect to the Kalidindi parameters and the
        # grains' Euler angles: forward, then the adjoint
        dict(name="gradient-10", kind="gradient", material="BENCH_STEEL", nx=10, ny=10, nz=10, grains=16, steps=2),
        # the constitutive update with its tangent at points of the caller's own (get_tensor_map)
        dict(name="points-steel-60007", kind="points", material="BENCH_STEEL", points=60007, grains=64, tangent=True),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["steps", "steps", "benchmark", "benchmark", "system", "linear", "linear", "batch", "gradient",
                       "points"])
    fcc_or_bcc = rng.choice(["BENCH_STEEL", "COPPER", "BENCH_TANTALUM"])
    if kind == "steps":
        mat = rng.choice(["BENCH_STEEL", "BENCH_TANTALUM", "DP_STEEL", "COPPER", "CALIB_CASE1"])
        n = [_log(rng, 1, 12) for _ in range(3)]
        return dict(kind="steps", path="reference", material=mat, nx=n[0], ny=n[1], nz=n[2],
                    grains=min(n[0] * n[1] * n[2], rng.randint(1, 24)), steps=rng.randint(1, 3),
                    line_search=rng.random() < 0.2)
    if kind == "benchmark":
        # the multigrid hierarchy needs even cell counts
        n = [4 * _log(rng, 2, 8 if fcc_or_bcc != "BENCH_TANTALUM" else 5) for _ in range(3)]
        return dict(kind="steps", path="benchmark", material=fcc_or_bcc, nx=n[0], ny=n[1], nz=n[2],
                    grains=rng.randint(2, 32), steps=rng.randint(1, 3), line_search=False)
    if kind == "system":
        n = [_log(rng, 2, 32) for _ in range(3)]
        return dict(kind="system", material=fcc_or_bcc, nx=n[0], ny=n[1], nz=n[2],
                    grains=min(n[0] * n[1] * n[2], rng.randint(1, 64)))
    if kind == "linear":
        pc = rng.choice(["jacobi", "block3", "mg", "mg"])
        n = [4 * _log(rng, 1, 8) for _ in range(3)] if pc == "mg" else [_log(rng, 3, 24) for _ in range(3)]
        return dict(kind="linear", material="BENCH_STEEL", nx=n[0], ny=n[1], nz=n[2], grains=rng.randint(1, 27),
                    precond=pc, precision=rng.choice(["fp64", "fp32"]), transposed=rng.random() < 0.4)
    if kind == "batch":
        lo = rng.randint(2, 10)
        return dict(kind="batch", material="BENCH_STEEL", count=_log(rng, 2, 32), edge_min=lo,
                    edge_max=lo + rng.randint(0, 6), grains=rng.randint(2, 16), steps=rng.randint(1, 2))
    if kind == "gradient":
        n = [_log(rng, 2, 10) for _ in range(3)]
        return dict(kind="gradient", material=rng.choice(["BENCH_STEEL", "COPPER"]), nx=n[0], ny=n[1], nz=n[2],
                    grains=rng.randint(1, 8), steps=rng.randint(1, 2))
    return dict(kind="points", material=fcc_or_bcc, points=_log(rng, 1, 200000), grains=rng.randint(1, 64),
                tangent=rng.random() < 0.7)


# --------------------------------------------------------------------------- preparation
def _box(case, seed):
    """Mesh, grain of every cell, grain orientations: Voronoi grains from the seed."""
    pkg = _mod()
    mesh = pkg.box_mesh(case["nx"], case["ny"], case["nz"])
    ori, rng = pkg.mesh.voronoi_grains(mesh, case["grains"], seed)
    return mesh, pkg.material.random_quaternions(rng, case["grains"]), ori


def _spec(case):
    return getattr(_mod("material"), case["material"])


def _problem(case, seed, spec):
    mesh, quat, ori = _box(case, seed)
    info = (quat, ori)
    if spec.phases:
        info = (quat, ori, _phases(mesh.cells.shape[0], spec, seed))
    return _mod("problem").CrystalPlasticity(mesh, additional_info=info, material=spec), mesh, quat, ori


def _phases(cells, spec, seed):
    ph = np.zeros(cells, dtype=np.int64)
    ph[:int(cells * spec.phase1_fraction)] = 1
    return np.random.default_rng(seed + 1).permutation(ph)


def _point_inputs(n, spec, seed, grains):
    """Gauss points in the middle of a load history: a tensile increment with noise, a small
    plastic deformation, slip resistances a little above the initial one, random grains.  On
    the GPU, from the seed."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    nrm = lambda *s: torch.randn(*s, generator=gen, dtype=torch.float64, device="cuda")
    uni = lambda *s: torch.rand(*s, generator=gen, dtype=torch.float64, device="cuda")
    eye = torch.eye(3, dtype=torch.float64, device="cuda")
    ug = 2.0 * STRAIN * torch.diag(torch.tensor([-0.3, -0.3, 1.0], dtype=torch.float64, device="cuda"))
    ug = ug + 0.2 * STRAIN * nrm(n, 3, 3)
    fpi = eye + 2e-4 * nrm(n, 3, 3)
    g = spec.gss_initial * (1.0 + 0.2 * uni(n, spec.num_slip))
    slip = 1e-3 * nrm(n, spec.num_slip)
    q = nrm(grains, 4)
    R = torch.from_numpy(_mod("material").rot_mat((q / q.norm(dim=1, keepdim=True)).cpu().numpy())).cuda()
    return ug, fpi, g, slip, R[torch.randint(0, grains, (n,), generator=gen, device="cuda")]


def _iterate(case, seed, spec):
    """A Newton iterate in the middle of a load history, from the seed alone: a displacement
    of 0.3 % tension with a smooth perturbation, and a plastic state that differs from grain to
    grain.  Returns numpy (u, fpi (G, 9), g (G, N))."""
    mesh, quat, ori = _box(case, seed)
    rng = np.random.default_rng(seed + 7)
    P = mesh.points
    u = 3.0 * STRAIN * P * np.array([-0.3, -0.3, 1.0])
    for k in (1, 2):
        a = rng.normal(size=3) * 2e-5
        u = u + a * np.sin(k * math.pi * P[:, [0]]) * np.sin(k * math.pi * P[:, [1]]) * np.sin(k * math.pi * P[:, [2]])
    E, N = mesh.cells.shape[0], spec.num_slip
    dev = rng.normal(size=(case["grains"], 3, 3)) * 5e-4
    dev -= np.trace(dev, axis1=1, axis2=2)[:, None, None] / 3.0 * np.eye(3)
    fpi = np.repeat(np.eye(3) + dev[ori], 8, axis=0).reshape(8 * E, 9)
    g = spec.gss_initial * (1.0 + 0.1 * rng.uniform(size=(case["grains"], N)))
    return u.reshape(-1), fpi, np.repeat(g[ori], 8, axis=0)


def _rollers(mesh, disp):
    return _mod("workloads").roller_lists(mesh, disp)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "points":
        spec = _spec(case)
        # the constitutive map needs a problem of its material; its mesh plays no part
        prob = _mod("problem").CrystalPlasticity(_mod().box_mesh(1, 1, 1), material=spec,
                                                 additional_info=(np.array([[1.0, 0, 0, 0]]), np.zeros(1, int)))
        prob.dt = DT
        return dict(case=case, prob=prob, args=_point_inputs(case["points"], spec, seed, case["grains"]))
    if kind == "batch":
        B = _mod("batch")
        # edges in turn over the range, so that a batch's size is its case's; grains, orientations
        # and parameters (+-20 %) from the seed
        inst = []
        for k in range(case["count"]):
            edge = case["edge_min"] + (5 * k) % (case["edge_max"] - case["edge_min"] + 1)
            inst += B.sample_instances(1, _spec(case), seed=(seed, k), edges=(edge,), grains=(1, case["grains"]))
        b = B.Batch(inst)
        b.predictor = "linear"
        b.problem.fp32_tangent = True
        return dict(case=case, batch=b, params0=b.params)
    if kind == "gradient":
        spec = _spec(case).replace(local_tol=1e-9)
        prob, mesh, quat, ori = _problem(case, seed, spec)
        nodes = _rollers(mesh, 0.0)[0]
        n = case["steps"]
        hist = _mod("adjoint").LoadHistory(
            prob, STRAIN * np.arange(n + 1), DT * np.arange(n + 1),
            lambda i, d: (list(nodes), [0, 1, 2, 2], [0.0, 0.0, 0.0, d]), quat,
            solver_options={"jax_solver": {"tol": 1e-12}, "tol": 1e-10, "rel_tol": 1e-13},
            adjoint_options={"tol": 1e-12})
        rng = np.random.default_rng(seed + 3)
        theta = np.array([spec.h, spec.gss_initial, spec.t_sat, spec.gss_a, spec.xm])
        theta[:3] *= rng.uniform(0.95, 1.05, size=3)
        return dict(case=case, hist=hist, theta=theta, euler=rng.uniform(-20, 20, size=(case["grains"], 3)),
                    bar=rng.normal(size=(n, 3, 3)))
    if kind == "steps":
        spec = _spec(case)
        prob, mesh, quat, ori = _problem(case, seed, spec)
        W = _mod("workloads")
        w = W.Workload("case", mesh, quat, ori, spec, case["steps"], STRAIN, DT)
        return dict(case=case, prob=prob, w=w, params0=prob.internal_vars)
    # "system", "linear": a Newton iterate with its committed state and boundary values
    spec = _spec(case).replace(local_tol=1e-9)
    prob, mesh, quat, ori = _problem(case, seed, spec)
    u, fpi, g = _iterate(case, seed, spec)
    E, N = prob.num_cells, spec.num_slip
    params = prob.internal_vars
    params[0] = torch.from_numpy(fpi).cuda().reshape(E, 8, 3, 3)
    params[1] = torch.from_numpy(g).cuda().reshape(E, 8, N)
    prob.set_params(params)
    prob.dt = DT
    prob.fes[0].set_dirichlet_lists(*_rollers(mesh, 3.0 * STRAIN))
    u = torch.from_numpy(u).cuda()
    if kind == "system":
        return dict(case=case, prob=prob, u=(u, u * (1.0 + 2e-3)))
    S = _mod("solver")
    prob.warm_start_local = prob.fp32_local_jacobian = False
    res, A = S.newton_update_helper(prob, u)
    b, x0 = torch.neg(res), S.initial_increment(prob, u).clone()
    if case["transposed"]:
        gen = torch.Generator(device="cuda").manual_seed(seed)
        b = torch.randn(b.numel(), generator=gen, dtype=torch.float64, device="cuda")
        b[prob.fes[0].bc_dofs.long()] = 0.0
        A, x0 = A.T, torch.zeros_like(b)
    opts = {"tol": 1e-12, "atol": 1e-30, "maxiter": 20000, "precond": case["precond"]}
    if case["precond"] == "mg":
        opts["mg_options"] = {"precision": case["precision"], "coarse_sweeps": 8}
    return dict(case=case, prob=prob, A=A, b=b, x0=x0, opts={"jax_solver": opts})


# --------------------------------------------------------------------------------- passes
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "points":
        P, D, new, _ = state["prob"].gp_map(*state["args"], need_tangent=case["tangent"])
        return [P, D, new] if case["tangent"] else [P, new]
    if kind == "linear":
        return _mod("solver").linear_solver(state["prob"], state["A"], state["b"], state["x0"], state["opts"])
    if kind == "system":
        # the first two iterates of a load history's first step
        S, prob = _mod("solver"), state["prob"]
        prob.reset_local_start()
        for u in state["u"]:
            res, A = S.newton_update_helper(prob, u)
        return [res, A.values]
    if kind == "gradient":
        sig = state["hist"].forward(state["theta"], state["euler"])
        tb, eb = state["hist"].backward(state["bar"])
        return [sig, tb, eb]
    if kind == "batch":
        # a load history of the whole batch from its initial state
        b = state["batch"]
        b.params, b.prev, b.sol = state["params0"], None, torch.zeros_like(b.sol)
        b.problem.reset_local_start()
        szz = [b.step(STRAIN * (i + 1), DT, ktol=1e-6, tol=1e-10, rel_tol=1e-10) for i in range(case["steps"])]
        return [szz, b.sol, list(b.params[:3])]
    S, prob, w = _mod("solver"), state["prob"], state["w"]
    prob.reset_local_start()
    if case["path"] == "benchmark":
        prob.set_params(state["params0"])
        # the benchmark path with its Newton limit tightened, so that the result does not hang
        # on the iterate at which the loop stops
        st = _mod("workloads").bench_stepper(prob, S, w, {"newton": {"tol": 1e-10, "rel_tol": 1e-10}})
        sig = [st.step() for _ in range(case["steps"])]
        return [sig, st.sol, list(st.params[:3])]
    # the reference driver's loop, as written
    sol = torch.zeros(prob.num_total_dofs_all_vars, dtype=torch.float64, device=prob.device)
    params, sig = state["params0"], []
    for i in range(case["steps"]):
        prob.dt = w.dt
        prob.fes[0].set_dirichlet_lists(*w.bc_lists(w.strain_step * (i + 1)))
        prob.set_params(params)
        sol = S.solver(prob, {"jax_solver": {}, "initial_guess": [sol.reshape(-1, 3)],
                              "line_search_flag": case["line_search"]})[0].reshape(-1)
        sig.append(prob.compute_avg_stress(sol.reshape(-1, 3), params))
        params = prob.update_int_vars_gp(sol.reshape(-1, 3), params)
    return [sig, sol, list(params[:3])]


def work(case):
    """Bytes: inputs and state read once, outputs written once.  Operations: one local Newton
    iteration and one tangent per Gauss point and Newton iterate (three iterates a load step,
    two local iterations and a residual evaluation each), the element stiffness, and for the
    linear solves a number of iterations that the preconditioner class needs (a V-cycle counted
    as four operator products)."""
    kind = case["kind"]
    N = 24 if case["material"] in ("BENCH_TANTALUM", "DP_STEEL") else 12
    local, tan = 147.0 * N + 460.0, 231.0 * N + 2730.0
    state = 8.0 * (9 + 2 * N)
    if kind == "points":
        n = case["points"]
        return {"bytes": n * (2 * state + 8.0 * (18 + 9 + (81 if case["tangent"] else 0))),
                "flops": n * (4 * local + (tan if case["tangent"] else 0.0))}
    if kind == "batch":
        e = 0.5 * (case["edge_min"] + case["edge_max"])
        cells, nodes, steps = case["count"] * e ** 3, case["count"] * (e + 1) ** 3, case["steps"]
    else:
        cells = case["nx"] * case["ny"] * case["nz"]
        nodes = (case["nx"] + 1) * (case["ny"] + 1) * (case["nz"] + 1)
        steps = case.get("steps", 1)
    gps, product = 8.0 * cells, 2.0 * 9 * 27 * nodes
    edge = max(case.get("nx", 1), case.get("ny", 1), case.get("nz", 1), case.get("edge_max", 1))
    krylov = 16.0 if case.get("precond") == "mg" or case.get("path") == "benchmark" else 4.0 * edge + 10.0
    solve = krylov * product * (10.0 if krylov == 16.0 else 2.0)
    matrix = 8.0 * 9 * 27 * nodes
    if kind == "linear":
        return {"bytes": matrix + 3 * 24.0 * nodes, "flops": solve}
    iterate = gps * (3 * local + tan + 4 * 2376.0)
    if kind == "system":
        return {"bytes": gps * state + matrix + 48.0 * nodes, "flops": 2 * iterate}
    passes = steps * (2 if kind == "gradient" else 1)
    return {"bytes": passes * (2 * gps * state + matrix + 48.0 * nodes), "flops": passes * 3 * (iterate + solve)}


# ------------------------------------------------------------------------------------ exact
# The same mathematics in plain 64-bit torch: the local solve in the global frame with nine
# unknowns, iterated to rounding, dense linear algebra for the global systems.
def _slip_systems(spec):
    from_table = np.asarray(_mod("material").SLIP_SYSTEMS[spec.slip], dtype=np.float64)
    n = from_table[:, :3] / np.linalg.norm(from_table[:, :3], axis=1)[:, None]
    d = from_table[:, 3:] / np.linalg.norm(from_table[:, 3:], axis=1)[:, None]
    return torch.from_numpy(np.einsum("ai,aj->aij", d, n)).cuda()


def _update_points(spec, F, Fpi, g, R, dt, par, el, tangent):
    """Kalidindi update at a batch of Gauss points: dict with P, D = dP/dF, Fpi, g, dg, sig.
    par (n, 5) = (a, h0, gs, m, r), el (n, 3) = (C11, C12, C44)."""
    n, N = F.shape[0], g.shape[1]
    eye = torch.eye(3, dtype=torch.float64, device=F.device)
    Pa = torch.einsum("nij,ajk,nlk->nail", R, _slip_systems(spec), R)
    a, h0, gs, xm, rq = (par[:, [k]] for k in range(5))
    C = lambda k: el[:, k, None, None]

    def stiff(E):
        e = torch.einsum("nji,nj...k,nkl->ni...l", R, E, R)      # to the lattice frame
        d = torch.diagonal(e, dim1=1, dim2=2)
        t = 2.0 * C(2) * e
        diag = (C(0) - C(1))[..., 0] * d + C(1)[..., 0] * d.sum(1, keepdim=True)
        t = t - torch.diag_embed(torch.diagonal(t, dim1=1, dim2=2)) + torch.diag_embed(diag)
        return R @ t @ R.transpose(1, 2)

    A = F @ Fpi

    def local(S):
        x = torch.einsum("nij,naij->na", S, Pa) / g
        p = spec.ao * dt * x.abs() ** (1.0 / xm - 1.0)
        dg, k = p * x, p / xm / g
        B = eye - torch.einsum("na,naij->nij", dg, Pa)
        Fe = A @ B
        r = S - stiff(0.5 * (Fe.transpose(1, 2) @ Fe - eye))
        return r, dg, k, B, Fe

    def jacobian(k, Fe):
        M = Fe.transpose(1, 2) @ A
        cols = []
        Q = torch.einsum("nij,najk->naik", M, Pa)
        Q = 0.5 * (Q + Q.transpose(2, 3))
        for s in range(N):
            cols.append(stiff(Q[:, s]).reshape(n, 9))
        G = torch.stack(cols, 1)
        return torch.eye(9, dtype=torch.float64, device=F.device) + torch.einsum(
            "nai,na,naj->nij", G, k, Pa.reshape(n, N, 9))

    S = torch.zeros_like(F)
    r, dg, k, B, Fe = local(S)
    rn = r.flatten(1).norm(dim=1)
    for _ in range(60):
        ds = -torch.linalg.solve(jacobian(k, Fe), r.reshape(n, 9)).reshape(n, 3, 3)
        relax = torch.ones_like(rn)
        for sub in range(12):                                    # cut back the points that got worse
            T = S + relax[:, None, None] * ds
            tn = local(T)[0].flatten(1).norm(dim=1)
            worse = ~(tn < rn) & (rn > 1e-9)
            if not bool(worse.any()):
                break
            relax = torch.where(worse, 0.5 * relax, relax)
        S = T
        r, dg, k, B, Fe = local(S)
        rn = r.flatten(1).norm(dim=1)
        if float(rn.max()) < 2e-10 and sub == 0:
            break
    ds = -torch.linalg.solve(jacobian(k, Fe), r.reshape(n, 9)).reshape(n, 3, 3)
    S = S + ds
    r, dg, k, B, Fe = local(S)
    H = Fpi @ B
    det = torch.linalg.det(H)[:, None, None]
    Y = H @ S @ H.transpose(1, 2) / det
    P = F @ Y
    out = {"P": P, "Fpi": H, "dg": dg, "sig": P @ F.transpose(1, 2) / torch.linalg.det(F)[:, None, None]}
    ratio = 1.0 - g / gs
    t = h0 * dg.abs() * ratio.abs() ** a * torch.sign(ratio)
    tot = t.sum(1, keepdim=True)
    if spec.coplanar_q:
        blk = t.reshape(n, N // 3, 3).sum(2).repeat_interleave(3, 1)
        out["g"] = g + rq * (tot - blk) + blk
    else:
        out["g"] = g + (rq * tot).expand_as(g)
    if tangent:
        J = jacobian(k, Fe)
        Hi = torch.linalg.inv(H)
        cols = []
        for c in range(9):
            dF = torch.zeros(3, 3, dtype=torch.float64, device=F.device)
            dF[c // 3, c % 3] = 1.0
            dFe = dF @ H
            dE = Fe.transpose(1, 2) @ dFe
            dS = torch.linalg.solve(J, stiff(0.5 * (dE + dE.transpose(1, 2))).reshape(n, 9)).reshape(n, 3, 3)
            dH = -Fpi @ torch.einsum("na,naij->nij", k * torch.einsum("nij,naij->na", dS, Pa), Pa)
            V = dH @ S @ H.transpose(1, 2)
            dY = (V + V.transpose(1, 2) + H @ dS @ H.transpose(1, 2)) / det
            dY = dY - Y * torch.einsum("nij,nji->n", Hi, dH)[:, None, None]
            cols.append((dF @ Y + F @ dY).reshape(n, 9))
        out["D"] = torch.stack(cols, 2).reshape(n, 3, 3, 3, 3)
    return out


def _tables(case, spec, seed, cells):
    """(par (G, 5), el (G, 3), g0 (G, 1)) of every Gauss point of a box problem."""
    specs = spec.phases or (spec,)
    ph = _phases(cells, spec, seed) if spec.phases else np.zeros(cells, dtype=np.int64)
    rows = np.array([[s.gss_a, s.h, s.t_sat, s.xm, s.r, s.C11, s.C12, s.C44, s.gss_initial] for s in specs])
    t = torch.from_numpy(np.repeat(rows[ph], 8, axis=0)).cuda()
    return t[:, :5], t[:, 5:8], t[:, 8:]


class _ExactBox:
    """HEX8 elements of a uniform box of the unit cube in dense 64-bit torch."""

    def __init__(self, case, seed, spec, mesh, quat, ori):
        self.spec, self.n = spec, mesh.points.shape[0]
        self.cells = torch.from_numpy(mesh.cells).cuda()
        E = mesh.cells.shape[0]
        h = np.array([1.0 / case["nx"], 1.0 / case["ny"], 1.0 / case["nz"]])
        s = np.array([[-1, -1, -1], [1, -1, -1], [1, 1, -1], [-1, 1, -1], [-1, -1, 1], [1, -1, 1], [1, 1, 1], [-1, 1, 1]])
        gr = np.empty((8, 8, 3))
        for q in range(8):
            xi = np.array([q & 1, (q >> 1) & 1, q >> 2]) * 2.0 / math.sqrt(3.0) - 1.0 / math.sqrt(3.0)
            t = 1.0 + s * xi
            gr[q] = 0.25 * s * np.stack([t[:, 1] * t[:, 2], t[:, 0] * t[:, 2], t[:, 0] * t[:, 1]], 1) / h
        self.grad = torch.from_numpy(gr).cuda()
        self.w = float(h.prod()) / 8.0
        R = torch.from_numpy(_mod("material").rot_mat(quat)[ori]).cuda()
        self.R = R.repeat_interleave(8, 0)
        self.par, self.el, self.g0 = _tables(case, spec, seed, E)
        # the last value given to a dof counts
        nodes, comps, _ = _rollers(mesh, 0.0)
        self.bc = [torch.from_numpy(3 * k + c).cuda() for k, c in zip(nodes, comps)]
        self.dofs = (3 * self.cells[:, :, None] + torch.arange(3, device="cuda")).reshape(E, 24)

    def update(self, u, fpi, g, tangent):
        ue = u.reshape(-1, 3)[self.cells]
        F = torch.eye(3, dtype=torch.float64, device="cuda") + torch.einsum("eai,qaj->eqij", ue, self.grad)
        return _update_points(self.spec, F.reshape(-1, 3, 3), fpi, g, self.R, DT, self.par, self.el, tangent)

    def residual(self, o, u, disp):
        P = o["P"].reshape(-1, 8, 3, 3)
        f = torch.einsum("eqij,qaj->eai", P, self.grad) * self.w
        r = torch.zeros(3 * self.n, dtype=torch.float64, device="cuda")
        r.index_add_(0, self.dofs.reshape(-1), f.reshape(-1))
        for k, v in zip(self.bc, (0.0, 0.0, 0.0, disp)):
            r[k] = u[k] - v
        return r

    def matrix(self, o):
        D = o["D"].reshape(-1, 8, 3, 3, 3, 3)
        K = torch.einsum("qaj,eqijkl,qbl->eaibk", self.grad, D, self.grad) * self.w
        A = torch.zeros(9 * self.n * self.n, dtype=torch.float64, device="cuda")
        E = K.shape[0]
        A.index_add_(0, (self.dofs[:, :, None] * (3 * self.n) + self.dofs[:, None, :]).reshape(-1),
                     K.reshape(E, 24, 24).reshape(-1))
        A = A.reshape(3 * self.n, 3 * self.n)
        for k in self.bc:
            A[k] = 0.0
            A[k, k] = 1.0
        return A

    def steps(self, count):
        G, N = self.R.shape[0], self.spec.num_slip
        fpi = torch.eye(3, dtype=torch.float64, device="cuda").repeat(G, 1, 1)
        g, slip = self.g0.expand(G, N).clone(), torch.zeros(G, N, dtype=torch.float64, device="cuda")
        u, sig = torch.zeros(3 * self.n, dtype=torch.float64, device="cuda"), []
        for i in range(count):
            disp, last = STRAIN * (i + 1), math.inf
            for _ in range(40):
                o = self.update(u, fpi, g, True)
                r = self.residual(o, u, disp)
                rn = float(r.norm())
                if rn < 1e-11 or (rn < 1e-9 and rn > 0.5 * last):
                    break
                step, last = torch.linalg.solve(self.matrix(o), -r), rn
                for _ in range(4):                               # back off while the residual grows
                    t = self.update(u + step, fpi, g, False)
                    tn = float(self.residual(t, u + step, disp).norm())
                    if tn < 2.0 * max(rn, 1e-9) or _ == 3:
                        break
                    step = 0.5 * step
                u = u + step
            sig.append(o["sig"].reshape(-1, 8, 3, 3).mean(1))
            fpi, g, slip = o["Fpi"], o["g"], slip + o["dg"]
        E = self.cells.shape[0]
        return [sig, u, [fpi.reshape(E, 8, 3, 3), g.reshape(E, 8, N), slip.reshape(E, 8, N)]]


def exact(case, seed):
    kind = case["kind"]
    if kind == "points":
        spec = _spec(case)
        ug, fpi, g, slip, R = _point_inputs(case["points"], spec, seed, case["grains"])
        rows = [torch.from_numpy(v).cuda()[None].expand(case["points"], -1) for v in
                (spec.param_row(), spec.elastic_row())]
        o = _update_points(spec, torch.eye(3, dtype=torch.float64, device="cuda") + ug, fpi, g, R, DT, *rows,
                           case["tangent"])
        new = [o["Fpi"], o["g"], slip + o["dg"]]
        return [o["P"], o["D"], new] if case["tangent"] else [o["P"], new]
    if kind in ("batch", "gradient"):
        return None
    cells = case["nx"] * case["ny"] * case["nz"]
    if kind == "linear":
        if cells > 16 ** 3:
            return None
        st = prepare(case, seed)
        A = st["A"].to_scipy()
        rows = torch.from_numpy(np.repeat(np.arange(A.shape[0]), np.diff(A.indptr))).cuda()
        M = torch.zeros(A.shape, dtype=torch.float64, device="cuda")
        M[rows, torch.from_numpy(A.indices).cuda().long()] = torch.from_numpy(A.data).cuda()
        lu = torch.linalg.lu_factor(M)
        x = torch.linalg.lu_solve(*lu, st["b"][:, None])
        x = x + torch.linalg.lu_solve(*lu, st["b"][:, None] - M @ x)
        return x[:, 0]
    spec = _spec(case)
    if kind == "system":
        if cells > 20000:
            return None
        spec = spec.replace(local_tol=1e-9)
        mesh, quat, ori = _box(case, seed)
        box = _ExactBox(case, seed, spec, mesh, quat, ori)
        u, fpi, g = (torch.from_numpy(v).cuda() for v in _iterate(case, seed, spec))
        u = u * (1.0 + 2e-3)
        o = box.update(u, fpi.reshape(-1, 3, 3), g, False)
        return [box.residual(o, u, 3.0 * STRAIN), None]
    # whole load steps: the dense solver takes a few seconds up to about a thousand cells
    if cells > 1000:
        return None
    return _ExactBox(case, seed, spec, *_box(case, seed)).steps(case["steps"])
