"""The shared-memory BiCGSTAB of the point preconditioners at the sizes where its layout can
go wrong: one node group, ranges that do not divide over the blocks, fewer nodes than lanes,
rows staged in shared memory and rows streamed (24^3), transposed systems, forced block
counts, restarts; and batches whose teams have one block or many."""
import ctypes
import importlib

import numpy as np
import pytest
import torch

from tests.common import gpu_problem, roller_bcs

pytestmark = pytest.mark.gpu


def _system(pkg, problem_mod, solver_mod, dims):
    mesh = pkg.box_mesh(*dims)
    ori, rng = pkg.mesh.voronoi_grains(mesh, 3, 1)
    quat = pkg.material.random_quaternions(rng, 3)
    prob = gpu_problem(pkg, problem_mod, pkg.material.BENCH_STEEL, mesh, quat, ori,
                       roller_bcs(pkg.mesh, mesh.points, 1e-3))
    prob.dt = 0.1
    u = torch.tensor((1e-3 * mesh.points * [-0.3, -0.3, 1.0]).reshape(-1), device="cuda")
    u = u + 1e-5 * torch.sin(7.0 * torch.arange(u.numel(), dtype=torch.float64, device="cuda"))
    res, A = solver_mod.newton_update_helper(prob, u)
    return prob, A, torch.neg(res), solver_mod.initial_increment(prob, u).clone()


def _residual(A, x, b):
    """||b - A x|| by the host's CSR product in FP64."""
    return float(np.linalg.norm(b.cpu().numpy() - A.to_scipy() @ x.cpu().numpy()))


@pytest.mark.parametrize("dims", [(1, 1, 1), (2, 1, 1), (3, 3, 3), (5, 4, 2), (10, 10, 10), (13, 9, 7), (24, 24, 24)])
@pytest.mark.parametrize("precond", [0, 1, 2])
@pytest.mark.parametrize("transposed", [False, True])
def test_solutions_meet_the_stop_rule(pkg, gpu, dims, precond, transposed):
    """The stop rule holds for the recursive residual; the true one may drift from it by
    rounding: a factor 2 covers it at 1e-10.  The launch's own true residual agrees."""
    problem_mod, solver_mod = gpu
    prob, A, b, x0 = _system(pkg, problem_mod, solver_mod, dims)
    if transposed:
        b = torch.sin(3.0 + torch.arange(b.numel(), dtype=torch.float64, device="cuda"))
        b[prob.fes[0].bc_dofs.long()] = 0.0
        A, x0 = A.T, torch.zeros_like(b)
    x, k, ok = solver_mod.bicgstab(prob, A, b, x0, precond=precond, atol=1e-30)
    bn = float(b.norm())
    true = prob._true_res[2]
    if precond == 0 and not ok:
        return     # the unpreconditioned iteration may break down on the Dirichlet rows (as jax's does)
    assert ok and k > 0
    assert _residual(A, x, b) <= 2e-10 * bn
    assert abs(true - _residual(A, x, b)) <= 1e-12 * bn
    x2, k2, _ = solver_mod.bicgstab(prob, A, b, x0, precond=precond, atol=1e-30)
    assert k2 == k and torch.equal(x2, x)          # fixed summation orders


@pytest.mark.parametrize("blocks", [1, 2, 7, 31, 152])
def test_block_counts(pkg, gpu, blocks):
    problem_mod, solver_mod = gpu
    prob, A, b, x0 = _system(pkg, problem_mod, solver_mod, (5, 4, 3))
    x, k, ok = solver_mod.bicgstab(prob, A, b, x0, atol=1e-30, grid_blocks=blocks)
    assert ok and _residual(A, x, b) <= 2e-10 * float(b.norm())


def test_no_iterations_and_restarts(pkg, gpu):
    """maxiter = 0 returns x0 and its residual; a solve with restarts allowed is the same solve
    where nothing breaks down; deferred reports equal the waited ones."""
    problem_mod, solver_mod = gpu
    prob, A, b, x0 = _system(pkg, problem_mod, solver_mod, (4, 3, 5))
    x, k, ok = solver_mod.bicgstab(prob, A, b, x0, maxiter=0)
    assert k == 0 and not ok and torch.equal(x, x0)
    assert abs(prob._true_res[2] - _residual(A, x0, b)) <= 1e-12 * float(b.norm())
    x1, k1, _ = solver_mod.bicgstab(prob, A, b, x0)
    x2, k2, _ = solver_mod.bicgstab(prob, A, b, x0, restarts=20)
    assert k1 == k2 and torch.equal(x1, x2)
    x3, _, _ = solver_mod.bicgstab(prob, A, b, x0, deferred=True)
    torch.cuda.synchronize()
    capi = importlib.import_module("jax-cpfem_gb300._capi")
    rep = capi.SolveReport.from_address(solver_mod._report_buffer(prob, prob._pending_solve["slot"]).data_ptr())
    assert rep.k == k1 and rep.error == 0 and torch.equal(x3, x1)
    prob._pending_solve = None


def test_nan_in_the_system_stops_at_once(pkg, gpu):
    """A NaN right-hand side: no iteration, not converged (as the comparisons with NaN of the
    reference's loop)."""
    problem_mod, solver_mod = gpu
    prob, A, b, x0 = _system(pkg, problem_mod, solver_mod, (3, 3, 3))
    b[40] = float("nan")
    x, k, ok = solver_mod.bicgstab(prob, A, b, x0)
    assert k == 0 and not ok


@pytest.mark.parametrize("edges", [(1,), (2, 3), (4, 5, 6, 7, 8, 9)])
def test_batches_of_small_teams(pkg, gpu, edges):
    """Teams of one block up to many: every instance agrees with its own solve."""
    batch = importlib.import_module("jax-cpfem_gb300.batch")
    inst = []
    for k, e in enumerate(edges):
        inst += batch.sample_instances(1, pkg.material.BENCH_STEEL, seed=k, edges=(e,), grains=(1, 4))
    b = batch.Batch(inst)
    szz = np.stack([b.step(d, 0.1).cpu().numpy() for d in (1e-3, 2e-3)], axis=1)
    ref = batch.run_serial(inst, [1e-3, 2e-3], 0.1)
    assert np.abs(szz - ref).max() / np.abs(ref).max() < 1e-8
