"""What a multigrid set-up leaves for the solves that follow it: whose dense coarse operator lies in
the hierarchy's scratch, and the settings it was formed with."""
import pytest
import torch

from tests.test_gpu_point_solver import _residual, _system

pytestmark = pytest.mark.gpu


def _kept(prob):
    """The problem's next solves use its hierarchy as it stands."""
    prob.mg_setup = lambda *a, **kw: prob._mg


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("local_nodes", [256, 1])
def test_smaller_hierarchy_in_the_same_scratch(pkg, gpu, precision, local_nodes):
    """A 4^3 hierarchy set up in a 16^3 one's scratch writes the front of it only (with a dense
    operator of its own or, local_nodes = 1, without): the 16^3 solve finds that, smooths its
    coarse levels itself, and is bit for bit the solve that was told to (local_nodes = 1)."""
    problem_mod, solver_mod = gpu
    p1, A1, b1, x1 = _system(pkg, problem_mod, solver_mod, (16, 16, 16))
    p2, A2, b2, x2 = _system(pkg, problem_mod, solver_mod, (4, 4, 4))
    p1.mg_setup(A1.values, precision=precision)
    _kept(p1)
    solve = lambda: solver_mod.bicgstab(p1, A1, b1, x1, precond=3, atol=1e-30, maxiter=200)
    dense, k0, ok = solve()
    assert ok
    m2 = p2.multigrid(precision=precision, local_nodes=local_nodes)
    m2.scratch[0], m2.scratch[1] = p1._mg.scratch[0], p1._mg.scratch[1]
    p2.mg_setup(A2.values, precision=precision, local_nodes=local_nodes)
    x, k, ok = solve()
    p1._mg.local_nodes = 1
    ref, kr, _ = solve()
    assert ok and k == kr and torch.equal(x, ref)
    assert abs(k - k0) <= 2 and _residual(A1, x, b1) <= 2e-10 * float(b1.norm())


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("change", [{"coarse_sweeps": 9}, {"pre_sweeps": 2}, {"post_sweeps": 2}, {"omega": 0.3}, {}])
def test_settings_changed_under_a_kept_set_up(pkg, gpu, precision, change):
    """refresh="step" keeps the set-up while the smoother's settings change: the solve is bit for
    bit the one that smooths every level with the new settings (local_nodes = 1).  Unchanged
    settings use the dense operator, whose rounding differs."""
    problem_mod, solver_mod = gpu
    prob, A, b, x0 = _system(pkg, problem_mod, solver_mod, (8, 8, 8))
    prob.mg_setup(A.values, precision=precision, pre_sweeps=1, post_sweeps=1, coarse_sweeps=4, omega=0.45)
    opts = {"precision": precision, "refresh": "step", **change}
    solve = lambda **kw: solver_mod.bicgstab(prob, A, b, x0, precond=3, atol=1e-30, mg_options={**opts, **kw})
    x, k, ok = solve()
    ref, kr, _ = solve(local_nodes=1)
    assert ok and _residual(A, x, b) <= 2e-10 * float(b.norm())
    assert torch.equal(x, ref) == bool(change) and abs(k - kr) <= (0 if change else 2)


def test_other_levels_under_a_kept_set_up(pkg, gpu):
    """max_levels makes a new hierarchy: it is set up although refresh="step" found the step's key."""
    problem_mod, solver_mod = gpu
    prob, A, b, x0 = _system(pkg, problem_mod, solver_mod, (8, 8, 8))
    prob.mg_setup(A.values, refresh="step")
    x, k, ok = solver_mod.bicgstab(prob, A, b, x0, precond=3, atol=1e-30, maxiter=200,
                                   mg_options={"refresh": "step", "max_levels": 2})
    ref, kr, _ = solver_mod.bicgstab(prob, A, b, x0, precond=3, atol=1e-30, mg_options={"max_levels": 2})
    assert ok and k == kr and torch.equal(x, ref)


@pytest.mark.parametrize("bits", [0x7FC00000, -0x400000])       # a NaN without, and with its sign bit
def test_fp32_cycle_that_goes_to_nan_reports_it(pkg, gpu, bits, monkeypatch):
    """Code -12 whatever the NaN's sign (the FP32 diagonal blocks of level 0 are overwritten)."""
    problem_mod, solver_mod = gpu
    prob, A, b, x0 = _system(pkg, problem_mod, solver_mod, (4, 4, 4))
    prob.mg_setup(A.values, precision="fp32")
    minv, = [t for t in prob._mg_keep if t.data_ptr() == prob._mg.minv32[0]]
    minv.view(torch.int32).fill_(bits)
    _kept(prob)
    monkeypatch.setattr(solver_mod, "_fp32_solve_ok", lambda *a: True)      # no FP64 solve after it
    x, k, ok = solver_mod.bicgstab(prob, A, b, x0, precond=3)
    assert k == -12 and not ok
