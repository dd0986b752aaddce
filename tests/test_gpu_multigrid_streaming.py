"""The multigrid solve in the streaming kernel: on one block (12^3 cells' vectors do not fit its shared
memory) and, 44^3 transposed in FP64, by the size rule on all SMs."""
import pytest
import torch

from tests.test_gpu_point_solver import _residual, _system

pytestmark = pytest.mark.gpu


def _transposed(prob, A, b):
    b = torch.sin(3.0 + torch.arange(b.numel(), dtype=torch.float64, device="cuda"))
    b[prob.fes[0].bc_dofs.long()] = 0.0
    return A.T, b, torch.zeros_like(b)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("transposed", [False, True])
@pytest.mark.parametrize("opts", [
    {}, {"local_nodes": 1}, {"pre_sweeps": 2, "coarse_sweeps": 5}, {"post_sweeps": 3}, {"max_levels": 2}])
def test_streamed_solve_is_the_same_method(pkg, gpu, precision, transposed, opts, monkeypatch):
    """The first two iterates are the shared-memory kernel's up to the V-cycle's rounding (FP32: some
    hundred roundings of 6e-8 a cycle, four cycles; FP64 the same of 1e-16), and the stop rule holds."""
    problem_mod, solver_mod = gpu
    prob, A, b, x0 = _system(pkg, problem_mod, solver_mod, (12, 12, 12))
    if transposed:
        A, b, x0 = _transposed(prob, A, b)
    opts = {"precision": precision, **opts}
    solve = lambda blocks, **kw: solver_mod.bicgstab(prob, A, b, x0, precond=3, atol=1e-30, mg_options=opts,
                                                     grid_blocks=blocks, **kw)
    with monkeypatch.context() as m:
        m.setattr(solver_mod, "_fp32_solve_ok", lambda *a: True)      # two iterations are not to converge
        x0s, x1s = solve(0, maxiter=2)[0], solve(1, maxiter=2)[0]
    scale = float((x0s - x0).abs().max())
    assert float((x1s - x0s).abs().max()) <= (1e-4 if precision == "fp32" else 1e-11) * scale
    x, k, ok = solve(1)
    assert ok and prob._mg.precision == (1 if precision == "fp32" else 0)
    assert _residual(A, x, b) <= 2e-10 * float(b.norm())
    assert torch.equal(solve(1)[0], x)


def test_no_post_sweeps_and_restarts(pkg, gpu):
    problem_mod, solver_mod = gpu
    prob, A, b, x0 = _system(pkg, problem_mod, solver_mod, (12, 12, 12))
    for precision in ("fp64", "fp32"):
        x, k, ok = solver_mod.bicgstab(prob, A, b, x0, precond=3, atol=1e-30, restarts=5, grid_blocks=1,
                                       mg_options={"precision": precision, "post_sweeps": 0})
        assert ok and _residual(A, x, b) <= 2e-10 * float(b.norm())


def test_fp32_cycle_that_goes_to_nan_reports_it(pkg, gpu, monkeypatch):
    problem_mod, solver_mod = gpu
    prob, A, b, x0 = _system(pkg, problem_mod, solver_mod, (12, 12, 12))
    prob.mg_setup(A.values, precision="fp32")
    minv, = [t for t in prob._mg_keep if t.data_ptr() == prob._mg.minv32[0]]
    minv.fill_(float("nan"))
    prob.mg_setup = lambda *a, **kw: prob._mg
    monkeypatch.setattr(solver_mod, "_fp32_solve_ok", lambda *a: True)
    x, k, ok = solver_mod.bicgstab(prob, A, b, x0, precond=3, grid_blocks=1)
    assert k == -12 and not ok


def test_large_transposed_system(pkg, gpu):
    problem_mod, solver_mod = gpu
    prob, A, b, x0 = _system(pkg, problem_mod, solver_mod, (44, 44, 44))
    A, b, x0 = _transposed(prob, A, b)
    x, k, ok = solver_mod.bicgstab(prob, A, b, x0, precond=3, atol=1e-30, mg_options={"precision": "fp64"})
    assert ok and _residual(A, x, b) <= 2e-10 * float(b.norm())
