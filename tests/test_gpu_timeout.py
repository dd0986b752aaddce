"""A solve one of whose blocks never arrives at the grid barriers (a count that starts one short,
every wait short too): it returns an error, and the GPU is as usable as before."""
import ctypes
import importlib

import numpy as np
import pytest
import torch

from tests.test_gpu_point_solver import _system

pytestmark = pytest.mark.gpu
ERR_SOLVE = 4                       # CPFEM_ERR_SOLVE
POLLS = 1 << 16                     # a few hundredths of a second a wait


def _lost(prob, A, b, x0, precond, mg, grid_blocks, deferred=False):
    """(return code, the report's error word)"""
    capi = importlib.import_module("jax-cpfem_gb300._capi")
    problem_mod = importlib.import_module("jax-cpfem_gb300.problem")
    ws = prob._buf("krylov_ws", (int(prob.lib.cpfem_bicgstab_workspace_bytes(prob.num_nodes)) // 8 + 64,))
    opts = capi.KrylovOpts(precond, 0, 50, 0, 0.0, 1e-200, None, grid_blocks, 1 | (2 if deferred else 0))
    if precond == 3:
        opts.mg = ctypes.pointer(prob.mg_setup(A.values, **mg))
    report = torch.zeros(ctypes.sizeof(capi.SolveReport), dtype=torch.uint8).pin_memory()
    opts.report = report.data_ptr()
    info = np.zeros(2, dtype=np.int32)
    x = x0.clone()
    rc = prob.lib.cpfem_probe_lost_block(prob.sell, A.values.data_ptr(), b.data_ptr(), x.data_ptr(), ctypes.byref(opts),
                                         POLLS, ws.data_ptr(), info.ctypes.data, problem_mod._stream())
    torch.cuda.synchronize()
    return rc, capi.SolveReport.from_address(report.data_ptr()).error


# the shared-memory kernel over all SMs, and on seven blocks; the streaming kernel (12^3 nodes' vectors
# do not fit one block's shared memory); both V-cycles
@pytest.mark.parametrize("precond,mg,grid_blocks", [
    (1, {}, 0), (2, {}, 7), (1, {}, 1), (3, {"precision": "fp64"}, 0), (3, {"precision": "fp32"}, 0),
    (3, {"precision": "fp64"}, 1), (3, {"precision": "fp32"}, 1)])
def test_lost_block_ends_the_solve(pkg, gpu, precond, mg, grid_blocks):
    problem_mod, solver_mod = gpu
    prob, A, b, x0 = _system(pkg, problem_mod, solver_mod, (12, 12, 12))
    solve = lambda: solver_mod.bicgstab(prob, A, b, x0, precond=precond, mg_options=dict(mg), grid_blocks=grid_blocks)
    ref, k0, _ = solve()
    rc, _ = _lost(prob, A, b, x0, precond, mg, grid_blocks)
    assert rc == ERR_SOLVE and "timed out" in prob.lib.cpfem_last_error().decode()
    rc, error = _lost(prob, A, b, x0, precond, mg, grid_blocks, deferred=True)
    assert rc == 0 and error != 0
    x, k, _ = solve()
    assert k == k0 and torch.equal(x, ref)
