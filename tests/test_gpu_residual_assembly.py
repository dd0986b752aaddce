"""The residual pass of large meshes, which has a kernel of its own."""
import numpy as np
import pytest
import torch

from tests.common import gpu_problem
from tests.test_gpu_node_assembly import fan

pytestmark = pytest.mark.gpu


# above and, (27, 26, 25), below the 20,000 nodes of the rule; a ragged last block of 16 nodes; nodes
# of one to forty cells, an even and an odd number of them
@pytest.mark.parametrize("shape", [(27, 26, 25), (41, 25, 19), (28, 27, 27), ("fan", 20, 500), ("fan", 5, 1900)])
def test_residual_of_a_large_mesh(pkg, gpu, shape):
    problem_mod, _ = gpu
    mesh = fan(pkg, *shape[1:]) if shape[0] == "fan" else pkg.box_mesh(*shape)
    prob = gpu_problem(pkg, problem_mod, pkg.material.BENCH_STEEL, mesh, np.array([[1.0, 0, 0, 0]]),
                       np.zeros(len(mesh.cells), dtype=np.int64))
    assert (prob.num_nodes > 20000) == (shape[0] != 27)
    gen = torch.Generator(device="cuda").manual_seed(3)
    rnd = lambda *s: torch.randn(*s, dtype=torch.float64, device="cuda", generator=gen)
    pw, start = rnd(9, prob.num_gp), rnd(3 * prob.num_nodes)
    res = start.clone()
    prob.scatter(pw, None, res, None)
    again = start.clone()
    prob.scatter(pw, None, again, None)
    assert torch.equal(res, again)
    # the same terms in another order: at most 40 cells x 8 points x 3 products in either sum
    sg = prob.fes[0].shape_grads.reshape(-1, 8, 8, 3)
    dofs = (3 * prob.fes[0].cells.long()[:, :, None] + torch.arange(3, device="cuda")).reshape(-1)
    add = lambda to, P, g: to.index_add_(0, dofs, torch.einsum("ijeq,eqaj->eai", P.reshape(3, 3, -1, 8), g).reshape(-1))
    ref, mag = add(start.clone(), pw, sg), add(start.abs(), pw.abs(), sg.abs())
    assert bool(((res - ref).abs() <= 2 * (40 * 8 * 3 + 2) * 2.0 ** -53 * mag).all())
