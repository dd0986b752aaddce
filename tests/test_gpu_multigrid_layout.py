"""The multigrid solve where its layout changes: the dense coarse operator on the first coarse
level (4^3, 8^3), on a later one (16x8x4), none (local_nodes = 1: every level smoothed by the
grid), matrix rows staged or streamed (36^3, whose blocks have a last round of few units), FP64
and FP32 V-cycles, transposed; and a set-up that another hierarchy's has overwritten."""
import numpy as np
import pytest
import torch

from tests.test_gpu_point_solver import _residual, _system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(4, 4, 4), (8, 8, 8), (16, 8, 4), (36, 36, 36)])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("transposed", [False, True])
def test_solutions_meet_the_stop_rule(pkg, gpu, dims, precision, transposed):
    """As for the point preconditioners; and the dense operator is the smoothed levels' own map:
    the Krylov counts agree with those of the grid-wide cycle up to rounding (2 iterations)."""
    problem_mod, solver_mod = gpu
    prob, A, b, x0 = _system(pkg, problem_mod, solver_mod, dims)
    if transposed:
        b = torch.sin(3.0 + torch.arange(b.numel(), dtype=torch.float64, device="cuda"))
        b[prob.fes[0].bc_dofs.long()] = 0.0
        A, x0 = A.T, torch.zeros_like(b)
    counts = []
    for local_nodes in (256, 1):
        opts = {"precision": precision, "local_nodes": local_nodes, "coarse_sweeps": 5, "pre_sweeps": 2,
                "post_sweeps": 2}
        x, k, ok = solver_mod.bicgstab(prob, A, b, x0, precond=3, atol=1e-30, mg_options=opts)
        assert ok and prob._mg.precision == (1 if precision == "fp32" else 0)
        assert _residual(A, x, b) <= 2e-10 * float(b.norm())
        counts.append(k)
    assert abs(counts[0] - counts[1]) <= 2, counts


@pytest.mark.parametrize("post_sweeps", [0, 1, 3])
def test_sweep_counts(pkg, gpu, post_sweeps):
    problem_mod, solver_mod = gpu
    prob, A, b, x0 = _system(pkg, problem_mod, solver_mod, (8, 12, 4))
    for precision in ("fp64", "fp32"):
        x, k, ok = solver_mod.bicgstab(prob, A, b, x0, precond=3, atol=1e-30,
                                       mg_options={"precision": precision, "post_sweeps": post_sweeps})
        assert ok and _residual(A, x, b) <= 2e-10 * float(b.norm())


def test_dense_operator_of_another_hierarchy_is_not_used(pkg, gpu):
    """Two problems whose hierarchies share their scratch arrays: the second set-up overwrites the
    first's dense operator, whose tag then does not match, and the first solve smooths its
    levels itself."""
    problem_mod, solver_mod = gpu
    one = _system(pkg, problem_mod, solver_mod, (8, 8, 8))
    two = _system(pkg, problem_mod, solver_mod, (8, 8, 8))
    p1, A1, b1, x1 = one
    p2, A2, b2, x2 = two
    ref, k, _ = solver_mod.bicgstab(p1, A1, b1, x1, precond=3, atol=1e-30)
    m2 = p2.multigrid()
    m2.scratch[0], m2.scratch[1] = p1._mg.scratch[0], p1._mg.scratch[1]
    p2.mg_setup(A2.values)
    p1.mg_setup = lambda *a, **kw: p1._mg        # keep p1's earlier set-up
    x, k1, ok = solver_mod.bicgstab(p1, A1, b1, x1, precond=3, atol=1e-30)
    assert ok and abs(k1 - k) <= 1 and _residual(A1, x, b1) <= 2e-10 * float(b1.norm())
    assert float((x - ref).abs().max() / ref.abs().max()) < 1e-8
