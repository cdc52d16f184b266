"""A handle's first conjugate-gradient solve may be recorded in a CUDA graph."""

import ctypes as C

import pytest

pytestmark = pytest.mark.gpu

from twophaseflow_b200 import _lib  # noqa: E402
from twophaseflow_b200.workloads import divergence_rhs, droplet_density  # noqa: E402


class _Cfg:
    pseudo_tol = 1e-8
    pseudo_maxiter = 100000
    ppe_iteration_method = "cg"
    ppe_preconditioner = "jacobi"


# the register-resident kernel at its smallest and just below its largest sizes, the marching kernel, and a row too wide
# for it (two kernels an iteration inside a conditional WHILE node)
@pytest.mark.parametrize("N", [(40, 36), (512, 512), (600, 560), (20, 24, 16), (2, 3, 1100)])
def test_first_solve_of_a_handle_under_capture(cuda_device, N):
    """Prepared but never solved: the capture allocates nothing and each replay
    gives the eager solve's bits and counts for the right-hand side of the day."""
    import torch
    from twophaseflow_b200 import PPESolverFVMMatrixFree, UniformGrid
    lib = _lib.load()
    rho = torch.from_numpy(droplet_density(N, n_drops=3, rho_g=1e-1, seed=4)).to(cuda_device)
    fields = [torch.from_numpy(divergence_rhs(N, seed=k)).to(cuda_device) for k in (5, 6)]
    rhs, p = fields[0].clone(), torch.zeros_like(rho)
    s = PPESolverFVMMatrixFree(None, _Cfg(), UniformGrid(N))
    s.prepare_operator(rho)
    torch.cuda.synchronize()
    res = _lib.tpf_ppe_result()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        status = lib.tpf_ppe_solve(s._handle, _lib.dptr(rhs), None, _lib.dptr(p), None, _lib.current_stream_handle(),
                                   C.byref(res))
    assert status == _lib.TPF_OK and res.iterations == -1
    eager = PPESolverFVMMatrixFree(None, _Cfg(), UniformGrid(N))
    for f in fields:
        rhs.copy_(f)
        graph.replay()
        d = s.read_result()
        ref = eager.solve(f, rho)
        assert torch.equal(p, ref)
        for key in ("iterations", "applies", "relative_residual"):
            assert d[f"ppe_low_order_cg_{key}"] == eager.last_diagnostics[f"ppe_low_order_cg_{key}"]
