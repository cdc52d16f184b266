"""The one-launch marching PCG (cg_kernel 3, and the default of 3-D and large
2-D FP64 systems) against the all-global persistent kernel, where its tiles,
segments and copies change shape: planes of one tile, of exactly 512 columns and
one more, odd and even planes, rows wider than half a block's threads, fewer
planes than blocks, a warm start, a pin inside the grid, no preconditioner, and
a row too wide for the kernel (the streaming kernels run instead)."""

import ctypes as C

import pytest

from twophaseflow_b200.workloads import divergence_rhs, droplet_density

pytestmark = pytest.mark.gpu


class _Cfg:
    def __init__(self, **kw):
        self.__dict__.update(kw)


@pytest.mark.parametrize("N,warm,precond", [
    ((1, 1, 1), False, "jacobi"),
    ((2, 3, 1), True, "jacobi"),
    ((9, 31, 15), False, "jacobi"),       # 512 columns: one full tile
    ((9, 26, 18), True, "jacobi"),        # 513: two tiles, an odd plane
    ((40, 36, 44), True, "none"),
    ((3, 4, 299), False, "jacobi"),       # halo wider than a block's threads
    ((2, 3, 1100), False, "jacobi"),      # row too wide: streaming kernels
    ((200, 6, 7), False, "jacobi"),
    ((30, 511), True, "jacobi"),          # 2-D, one tile of 512
    ((300, 600), False, "jacobi"),
])
def test_marching_pcg_matches_persistent_kernel(cuda_device, N, warm, precond):
    """Both reach the 1e-10 relative residual; solutions within 1e-8 of max|p|,
    counts within a tenth (the sums differ in order only)."""
    import torch
    from twophaseflow_b200 import PPESolverFVMMatrixFree, UniformGrid, _lib
    rho = torch.from_numpy(droplet_density(N, seed=51, rho_g=1e-1)).to(cuda_device)
    rhs = torch.from_numpy(divergence_rhs(N, seed=52)).to(cuda_device)
    p0 = torch.from_numpy(divergence_rhs(N, seed=53)).to(cuda_device) if warm else None
    out, its = {}, {}
    for kind in (1, 3):
        s = PPESolverFVMMatrixFree(None, _Cfg(pseudo_tol=1e-10, pseudo_maxiter=100000, ppe_iteration_method="cg",
                                              ppe_preconditioner=precond), UniformGrid(N))
        _lib.check(s.lib.tpf_ppe_set_cg_kernel(s._handle, C.c_int(kind)))
        for _ in range(2):
            out[kind] = s.solve(rhs, rho, 0.0, p0)
        its[kind] = s.last_diagnostics["ppe_low_order_cg_iterations"]
        assert s.last_diagnostics["ppe_low_order_cg_relative_residual"] < 1e-10
    scale = float(torch.max(torch.abs(out[1])))
    assert float(torch.max(torch.abs(out[3] - out[1]))) <= 1e-8 * scale, its
    assert abs(its[1] - its[3]) <= max(1, its[1] // 10), its


def test_marching_pcg_zero_rhs_and_iteration_limit(cuda_device):
    """A zero right-hand side gives zero without iterating, also from a warm
    start; an exhausted limit is reported as such."""
    import torch
    from twophaseflow_b200 import PPESolverFVMMatrixFree, UniformGrid, _lib
    N = (20, 18, 22)
    rho = torch.from_numpy(droplet_density(N, seed=61)).to(cuda_device)
    rhs = torch.from_numpy(divergence_rhs(N, seed=62)).to(cuda_device)
    s = PPESolverFVMMatrixFree(None, _Cfg(pseudo_tol=1e-10, pseudo_maxiter=7, ppe_iteration_method="cg",
                                          ppe_preconditioner="jacobi"), UniformGrid(N))
    _lib.check(s.lib.tpf_ppe_set_cg_kernel(s._handle, C.c_int(3)))
    p = s.solve(torch.zeros_like(rhs), rho, 0.0, rhs)
    assert float(torch.max(torch.abs(p))) == 0.0
    assert s.last_diagnostics["ppe_low_order_cg_iterations"] == 0
    with pytest.raises(RuntimeError):
        s.solve(rhs, rho)
    assert s.last_diagnostics["ppe_low_order_cg_iterations"] == 7
