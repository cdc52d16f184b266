"""Batches of 2-D FP64 systems that fit on chip one by one but not all at once run
as groups: a system that fills a group alone, several that share one, the
smallest last, results in the caller's order; one system that fits nowhere sends
the whole batch to the streaming kernels."""

import pytest

from twophaseflow_b200.workloads import divergence_rhs, droplet_density

pytestmark = pytest.mark.gpu


class _Cfg:
    pseudo_tol = 1e-9
    pseudo_maxiter = 100000
    ppe_iteration_method = "cg"
    ppe_preconditioner = "jacobi"


@pytest.mark.parametrize("shapes", [
    [(96, 200), (512, 512), (300, 280), (40, 36), (400, 390), (330, 300)],
    [(640, 640), (600, 560), (17, 25)],
    [(512, 512), (700, 600), (64, 64)],      # 700 x 600 is too large for the chip
])
def test_grouped_batch_matches_single_solves(cuda_device, shapes):
    """Two solves of relative residual 1e-9: within 1e-7 of max|p| (the systems'
    solutions at that residual are a few 1e-9 apart), counts within one or a
    hundredth (the partial sums differ in order); every residual below the
    tolerance."""
    import torch
    from twophaseflow_b200 import PPESolverFVMMatrixFree, UniformGrid, solve_batched
    solvers = [PPESolverFVMMatrixFree(None, _Cfg(), UniformGrid(N)) for N in shapes]
    rho = [torch.from_numpy(droplet_density(N, seed=70 + k, rho_g=1e-1)).to(cuda_device) for k, N in enumerate(shapes)]
    rhs = [torch.from_numpy(divergence_rhs(N, seed=80 + k)).to(cuda_device) for k, N in enumerate(shapes)]
    pb = solve_batched(solvers, rhs, rho)
    its = [s.last_diagnostics["ppe_low_order_cg_iterations"] for s in solvers]
    for k, s in enumerate(solvers):
        assert s.last_diagnostics["ppe_low_order_cg_relative_residual"] < 1e-9
        p = s.solve(rhs[k], rho[k])
        assert float(torch.max(torch.abs(pb[k] - p))) <= 1e-7 * float(torch.max(torch.abs(p))), shapes[k]
        assert abs(its[k] - s.last_diagnostics["ppe_low_order_cg_iterations"]) <= max(1, its[k] // 100), shapes[k]
