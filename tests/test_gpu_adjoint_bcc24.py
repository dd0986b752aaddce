"""The backward kernel where its loops and branches differ: 24 slip systems, hardening without
coplanar blocks, a non-integer hardening exponent -- the gradient of a load history against
complex-step derivatives of the oracle's."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("spec_name,changes,n,grains,steps", [
    ("BENCH_TANTALUM", {}, 1, 1, 1), ("BENCH_TANTALUM", {}, 2, 3, 2), ("BENCH_TANTALUM", {"coplanar_q": False}, 2, 3, 2),
    ("BENCH_STEEL", {"coplanar_q": False, "gss_a": 2.5}, 2, 3, 2)])
def test_adjoint_matches_oracle_complex_step(pkg, gpu, spec_name, changes, n, grains, steps):
    from oracle import cpfem_oracle as O
    problem_mod, _ = gpu
    adjoint = importlib.import_module("jax-cpfem_gb300.adjoint")
    spec = getattr(pkg.material, spec_name).replace(local_tol=1e-10, **changes)
    table = O.BCC24 if spec.num_slip == 24 else O.FCC12
    mesh = pkg.box_mesh(n, n, n)
    ori, rng = pkg.mesh.voronoi_grains(mesh, grains, 4)
    quat = pkg.material.random_quaternions(rng, grains)
    prob = problem_mod.CrystalPlasticity(mesh, additional_info=(quat, ori), material=spec)
    p, fn = mesh.points, pkg.mesh.face_nodes
    faces = [fn(p, 0, 0.0), fn(p, 1, 0.0), fn(p, 2, 0.0), fn(p, 2, 1.0)]
    h = adjoint.LoadHistory(prob, np.linspace(0, 2e-3 * steps, steps + 1), np.linspace(0, 0.1 * steps, steps + 1),
                            lambda i, d: (faces, [0, 1, 2, 2], [0.0, 0.0, 0.0, d]), quat,
                            solver_options={"jax_solver": {}, "tol": 1e-10, "rel_tol": 1e-14})
    theta = np.array([spec.h, spec.gss_initial, spec.t_sat, spec.gss_a, spec.xm])
    euler = np.random.default_rng(4).uniform(-20, 20, size=(grains, 3))
    s0 = h.forward(theta, euler).cpu().numpy()[:, 2, 2]
    target = 0.97 * s0 + 1.0
    bar = np.zeros((steps, 3, 3))
    bar[:, 2, 2] = 2.0 * (s0 - target)
    tb, eb = h.backward(bar)

    def f(theta, euler):
        bcs = lambda d: [(nodes, c, v) for nodes, c, v in zip(faces, (0, 1, 2, 2), (0.0, 0.0, 0.0, d))]
        return O.history_stress(p, mesh.cells, table, (spec.C11, spec.C12, spec.C44), quat, ori, theta, euler,
                                h.disps, h.ts, bcs, r=spec.r, coplanar=spec.coplanar_q, ao=spec.ao,
                                local_tol=spec.local_tol, max_sub_step=spec.max_sub_step,
                                solver_options={"tol": 1e-10, "rel_tol": 1e-13, "max_newton": 40})[:, 2, 2]

    s_o = f(theta, euler)
    assert np.abs(s_o - s0).max() < 1e-9 * np.abs(s_o).max()
    w = 2.0 * (s_o - target)
    ct = np.array([w @ O.complex_step(lambda t: f(t, euler), theta, np.eye(5)[k]) for k in range(5)])
    ce = np.array([[w @ O.complex_step(lambda e: f(theta, e), euler, np.eye(3 * grains)[3 * g + k].reshape(grains, 3))
                    for k in range(3)] for g in range(grains)])
    # (hardening parameters do not enter the first step: their derivatives are exact zeros)
    assert (np.abs(tb - ct) <= 1e-6 * np.abs(ct)).all(), (tb, ct)
    assert np.abs(eb - ce).max() < 1e-6 * np.abs(ce).max(), (eb, ce)
