"""The register-resident band PCG at the edges of its nodes-per-thread variants."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from twophaseflow_b200.workloads import divergence_rhs, droplet_density  # noqa: E402

# one block and two; ranges of just under and just over 256 e nodes on 148 blocks for e = 3, 5, 7, 9
# nodes per thread (e = 1 on the first); the longest row; the largest grid
SIZES = [(15, 15), (19, 24), (22, 22), (513, 100), (336, 336), (337, 337), (434, 434), (435, 435), (513, 513), (514, 514),
         (582, 582), (583, 583), (120, 767), (644, 644)]


@pytest.mark.parametrize("N", SIZES)
def test_band_variants_match_the_global_kernel(cuda_device, N):
    """Same system, same recurrences, another order of the partial sums: both
    solves end below the 1e-10 residual and agree to 1e-8 of max|p| (two
    solutions of relative residual 1e-10 of these systems are a few 1e-11
    apart), and the second solve of a handle gives the first one's bits."""
    import torch
    from twophaseflow_b200 import PPESolverFVMMatrixFree, UniformGrid, _lib
    lib = _lib.load()

    class Cfg:
        pseudo_tol = 1e-10
        pseudo_maxiter = 200000
        ppe_iteration_method = "cg"
        ppe_preconditioner = "jacobi"

    rho = torch.from_numpy(droplet_density(N, n_drops=4, rho_g=1e-2, seed=5)).to(cuda_device)
    rhs = torch.from_numpy(divergence_rhs(N, seed=6)).to(cuda_device)
    out, its = {}, {}
    for kind in (1, 2):
        s = PPESolverFVMMatrixFree(None, Cfg(), UniformGrid(N))
        _lib.check(lib.tpf_ppe_set_cg_kernel(s._handle, kind))
        out[kind] = s.solve(rhs, rho)
        its[kind] = s.last_diagnostics["ppe_low_order_cg_iterations"]
        assert s.last_diagnostics["ppe_low_order_cg_relative_residual"] < 1e-10
        if kind == 2:
            assert torch.equal(s.solve(rhs, rho), out[2])
    scale = float(out[1].abs().max())
    assert float((out[2] - out[1]).abs().max()) <= 1e-8 * scale, its
    assert abs(its[1] - its[2]) <= max(1, its[1] // 10), its
    assert np.isfinite(scale)


# one system alone; systems of very different size; more systems than a third of the SMs; rows so long that a
# system cannot have the blocks its nodes ask for
BATCHES = [[(33, 40)], [(16, 16), (90, 70), (260, 250), (17, 300)], [(40 + k % 9, 64 - k % 7) for k in range(64)],
           [(5, 700), (7, 766), (64, 64)]]


@pytest.mark.parametrize("shapes", BATCHES, ids=["one", "unequal", "many", "long_rows"])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_batch_of_any_make_up(cuda_device, shapes, precision):
    """A band-resident batch against each system's own solve: 1e-10 residuals,
    pressures within 1e-8 (mixed 1e-6) of max|p|; a second batch on the
    couplings that are there already (no density given) gives the same bits in
    FP64."""
    import torch
    from twophaseflow_b200 import PPESolverFVMMatrixFree, UniformGrid, solve_batched

    class Cfg:
        pseudo_tol = 1e-10
        pseudo_maxiter = 200000
        ppe_iteration_method = "cg"
        ppe_preconditioner = "jacobi"
        ppe_precision = precision

    solvers = [PPESolverFVMMatrixFree(None, Cfg(), UniformGrid(N)) for N in shapes]
    rho = [torch.from_numpy(droplet_density(N, n_drops=3, rho_g=1e-2, seed=40 + k)).to(cuda_device)
           for k, N in enumerate(shapes)]
    rhs = [torch.from_numpy(divergence_rhs(N, seed=140 + k)).to(cuda_device) for k, N in enumerate(shapes)]
    got = solve_batched(solvers, rhs, rho)
    again = solve_batched(solvers, rhs)
    bar = 1e-8 if precision == "fp64" else 1e-6
    for k, s in enumerate(solvers):
        assert s.last_diagnostics["ppe_low_order_cg_relative_residual"] < 1e-10
        if precision == "fp64":
            assert torch.equal(got[k], again[k])
        one = s.solve(rhs[k], rho[k])
        scale = float(one.abs().max())
        assert float((got[k] - one).abs().max()) <= bar * scale, k
