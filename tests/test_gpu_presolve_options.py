"""The FP32 pre-solve of a warm local start is an option of its own."""
import numpy as np
import pytest
import torch

from tests.common import gpu_problem

pytestmark = pytest.mark.gpu


def _problem(pkg, problem_mod, spec):
    """A problem whose warm start (the returned tensor) is the root at the returned u."""
    mesh = pkg.box_mesh(3, 3, 3)
    ori, rng = pkg.mesh.voronoi_grains(mesh, 4, 3)
    prob = gpu_problem(pkg, problem_mod, spec, mesh, pkg.material.random_quaternions(rng, 4), ori)
    prob.dt, prob.timing, prob.predict_local = 0.05, True, False
    P = mesh.points
    u = 2e-3 * np.stack([-0.3 * P[:, 0], -0.3 * P[:, 1] + 0.1 * P[:, 2] ** 2, P[:, 2]], 1)
    u = torch.tensor(u.reshape(-1), device="cuda")
    prob.assemble(u)
    return prob, u, prob._warm().clone()


def _run(prob, u, start):
    """(residual, values, iterations, status word) of a pass from the given warm start"""
    prob._warm().copy_(start)
    res, values, status = prob.assemble(u)
    return res.clone(), values.clone(), prob._bufs["iters"].clone(), int(status.item())


@pytest.mark.parametrize("spec_name", ["BENCH_STEEL", "BENCH_TANTALUM"])
def test_pre_solve_can_be_left_out(pkg, gpu, spec_name):
    """fp32_local_presolve = False (local_flags bit 8 clear) leaves FP32 directions on an FP64
    residual from the start on: other steps, the same root; fp32_local_jacobian = False leaves
    both out."""
    problem_mod, _ = gpu
    prob, u, root = _problem(pkg, problem_mod, getattr(pkg.material, spec_name))
    out = {}
    for jac, pre in ((True, True), (True, False), (False, True), (False, False)):
        prob.fp32_local_jacobian, prob.fp32_local_presolve = jac, pre
        out[jac, pre] = _run(prob, u, 1.5 * root)
        assert out[jac, pre][3] == 0
    r0, v0, i0, _ = out[True, True]
    r1, v1, i1, _ = out[True, False]
    assert not torch.equal(i0, i1)
    assert float((r1 - r0).abs().max() / r0.abs().max()) < 1e-9
    assert float((v1 - v0).abs().max() / v0.abs().max()) < 1e-9
    assert torch.equal(out[False, True][0], out[False, False][0]) and torch.equal(out[False, True][2], out[False, False][2])


@pytest.mark.parametrize("max_iter", [1, 2, 3, 6, 300])
@pytest.mark.parametrize("spec_name", ["BENCH_STEEL", "BENCH_TANTALUM"])
def test_pre_solve_steps_count_toward_max_iter(pkg, gpu, spec_name, max_iter):
    """From a far start: max_iter steps of any kind from the warm start, the step back to S = 0 among
    them, and max_iter more from there; what fails then fails, and what the pass from S = 0 reaches
    in max_iter steps is reached."""
    problem_mod, _ = gpu
    spec = getattr(pkg.material, spec_name)
    prob, u, root = _problem(pkg, problem_mod, spec)
    prob.mat_c.max_iter = max_iter
    prob.warm_start_local = False
    res, _, status = prob.assemble(u)
    cold, cold_status = res.clone(), int(status.item())
    prob.warm_start_local = True
    for start in (3.0 * root, -root, 1e30 * root):
        r, _, its, status = _run(prob, u, start)
        assert int(its.max()) <= 2 * max_iter
        if cold_status == 0:
            assert status == 0 and float((r - cold).abs().max() / cold.abs().max()) < 1e-9
        if max_iter == 1:                 # no pre-solve, the step back to S = 0, one step
            assert torch.equal(r, cold) and status == cold_status
