"""The local Newton's FP32 pre-solve: a warm start, wherever it lies, is first improved in
FP32, and the converged state is the root that the FP64 iteration from S = 0 finds."""
import numpy as np
import pytest
import torch

from tests.common import gpu_problem

pytestmark = pytest.mark.gpu


# 27 cells are 216 Gauss points: one full block of 128 threads and one ragged one.  The local
# stop test leaves ||r|| <= 1e-8 MPa on stresses of tens of MPa and more, so two roots agree to
# 1e-8 / 10 of the stress at worst, and a step taken on the way brings that down further:
# 1e-9 for P's sums and the tangent, as between any two starts.
@pytest.mark.parametrize("start", ["zero", "near", "far", "opposite", "huge", "nan"])
@pytest.mark.parametrize("spec_name", ["BENCH_STEEL", "BENCH_TANTALUM", "COPPER", "DP_MARTENSITE"])
def test_presolved_start_reaches_the_root_of_the_cold_solve(pkg, gpu, spec_name, start):
    problem_mod, _ = gpu
    spec = getattr(pkg.material, spec_name)
    mesh = pkg.box_mesh(3, 3, 3)
    ori, rng = pkg.mesh.voronoi_grains(mesh, 4, 3)
    prob = gpu_problem(pkg, problem_mod, spec, mesh, pkg.material.random_quaternions(rng, 4), ori)
    prob.dt = 0.05
    prob.timing = True
    P = mesh.points
    u = 2e-3 * np.stack([-0.3 * P[:, 0], -0.3 * P[:, 1] + 0.1 * P[:, 2] ** 2, P[:, 2]], 1)
    u = torch.tensor(u.reshape(-1), device="cuda")

    def run():
        res, values, status = prob.assemble(u)
        assert int(status.item()) == 0
        return res.clone(), values.clone(), prob._bufs["iters"].clone()

    prob.warm_start_local = False
    r0, v0, i0 = run()
    prob.warm_start_local = True
    prob.predict_local = False
    w = prob._warm()
    w.zero_()
    run()                                # s_warm is now the root
    root = w.clone()
    w.copy_({"zero": 0.0 * root, "near": root * (1.0 + 1e-6), "far": 1.5 * root, "opposite": -root,
             "huge": 1e30 * root, "nan": root * float("nan")}[start])
    r1, v1, i1 = run()
    assert float((r1 - r0).abs().max() / r0.abs().max()) < 1e-9
    assert float((v1 - v0).abs().max() / v0.abs().max()) < 1e-9
    assert float((w - root).abs().max() / root.abs().max()) < 1e-9
    if start == "nan":                   # no pre-solve: one abandoned step, then the cold solve
        assert torch.equal(i1, i0 + 1) and torch.equal(r1, r0)
