"""The assembly gathered by node against the one scattered by cell with atomics: the same sums
of the same terms, on boxes and on meshes whose nodes have more than eight cells."""
import ctypes

import numpy as np
import pytest
import torch

from tests.common import gpu_problem

pytestmark = pytest.mark.gpu


def fan(pkg, sectors, layers):
    """Kite-shaped cells around an axis: its inner nodes have 2 * sectors cells."""
    ang = 2 * np.pi * np.arange(sectors) / sectors
    mid = ang + np.pi / sectors
    ring = np.concatenate([[[0.0, 0.0]], np.stack([np.cos(ang), np.sin(ang)], 1),
                           1.2 / np.cos(np.pi / sectors) * np.stack([np.cos(mid), np.sin(mid)], 1)])
    n = len(ring)
    pts = np.concatenate([np.concatenate([ring, np.full((n, 1), float(z))], 1) for z in range(layers + 1)])
    quads = [[0, 1 + i, 1 + sectors + i, 1 + (i + 1) % sectors] for i in range(sectors)]
    cells = np.array([[z * n + v for v in q] + [(z + 1) * n + v for v in q] for z in range(layers) for q in quads])
    return pkg.mesh.Mesh(pts, cells)


@pytest.mark.parametrize("kp", [None, 0, 1, 2])
@pytest.mark.parametrize("shape", [(1, 1, 1), (2, 1, 1), (5, 4, 3), ("fan", 5, 2), ("fan", 12, 2), ("fan", 20, 3)])
def test_node_assembly_adds_the_terms_of_the_cell_assembly(pkg, gpu, shape, kp):
    problem_mod, _ = gpu
    mesh = fan(pkg, *shape[1:]) if shape[0] == "fan" else pkg.box_mesh(*shape)
    prob = gpu_problem(pkg, problem_mod, pkg.material.BENCH_STEEL, mesh, np.array([[1.0, 0, 0, 0]]),
                       np.zeros(len(mesh.cells), dtype=np.int64))
    lib, G = prob.lib, prob.num_gp
    gen = torch.Generator(device="cuda").manual_seed(3)
    rnd = lambda *s: torch.randn(*s, dtype=torch.float64, device="cuda", generator=gen)
    pw, sg = rnd(9, G), rnd(G * 24)
    dw = None if kp is None else rnd(81, G).to(torch.float32 if kp == 2 else torch.float64)
    res0, vals0 = rnd(3 * prob.num_nodes), None if kp is None else rnd(prob.num_values)
    ptr = lambda x: None if x is None else x.data_ptr()
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)

    def run(by_node, pw, sg, dw, res, vals):
        res, vals = res.clone(), None if vals is None else vals.clone()
        cells = prob.fes[0].cells
        if by_node:
            rc = lib.cpfem_node_assemble(prob.num_cells, prob.num_nodes, ptr(prob._node_ptr), ptr(prob._node_cells),
                                         ptr(sg), prob.sell, ptr(prob.elem_pos), ptr(pw), ptr(dw), ptr(res),
                                         ptr(vals), kp or 0, stream)
        else:
            rc = lib.cpfem_elem_assemble_ex(prob.num_cells, ptr(cells), ptr(sg), prob.sell, ptr(prob.elem_pos), None,
                                            0, ptr(pw), ptr(dw), ptr(res), ptr(vals), kp or 0, stream)
        assert rc == 0
        return res, vals

    r0, v0 = run(False, pw, sg, dw, res0, vals0)
    r1, v1 = run(True, pw, sg, dw, res0, vals0)
    # sums of magnitudes, and per term a rounding of each product and addition on either side:
    # at most 60 cells x 8 x 9 FP64 additions; in FP32 8 x 9 + the three factors' rounding
    ra, va = run(False, pw.abs(), sg.abs(), None if dw is None else dw.abs(), res0.abs(),
                 None if vals0 is None else vals0.abs())
    eps = 2 * (60 * 72 + 4) * 2.0 ** -53
    assert bool(((r1 - r0).abs() <= eps * ra).all())
    if kp is not None:
        bound = (eps + (2 * 80 * 2.0 ** -23 if kp else 0.0)) * va
        assert bool(((v1 - v0).abs() <= bound).all())
        r2, v2 = run(True, pw, sg, dw, res0, vals0)
        assert torch.equal(r1, r2) and torch.equal(v1, v2)
