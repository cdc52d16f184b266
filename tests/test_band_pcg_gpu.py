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


def _exact(grid, rho, rhs, pin):
    """The pinned system's solution beyond 64 bits: factorized in them, residuals of the flux form in extended precision."""
    import scipy.sparse as sp
    import scipy.sparse.linalg as spla
    c = [np.asarray(x, dtype=np.float64) for x in grid.coords]
    d = [np.diff(x) for x in c]
    dv = [np.concatenate([x[:1] / 2, (x[1:] + x[:-1]) / 2, x[-1:] / 2]) for x in d]
    s = [2 / (rho[:-1] + rho[1:]) / d[0][:, None] * dv[1], 2 / (rho[:, :-1] + rho[:, 1:]) / d[1] * dv[0][:, None]]
    idx = np.arange(rho.size).reshape(rho.shape)
    i, j = (np.concatenate(x) for x in ((idx[:-1].ravel(), idx[:, :-1].ravel()), (idx[1:].ravel(), idx[:, 1:].ravel())))
    s = np.concatenate([x.ravel() for x in s])
    b = -(rhs * dv[0][:, None] * dv[1]).ravel()
    b[pin] = 0.0
    diag = np.zeros(rho.size)
    np.add.at(diag, i, s)
    np.add.at(diag, j, s)
    diag[pin] = 1.0
    on = (i != pin) & (j != pin)
    a = sp.coo_matrix((np.concatenate([-s[on], -s[on], diag]),
                       (np.concatenate([i[on], j[on], idx.ravel()]), np.concatenate([j[on], i[on], idx.ravel()]))))
    lu = spla.splu(a.tocsc())
    x = np.zeros(rho.size, np.longdouble)
    for _ in range(5):
        flux = s.astype(np.longdouble) * (x[i] - x[j])
        r = b.astype(np.longdouble)
        np.add.at(r, i, -flux)
        np.add.at(r, j, flux)
        r[pin] = 0.0
        x += lu.solve(r.astype(np.float64))
        x[pin] = 0.0
    return x.reshape(rho.shape)


@pytest.mark.parametrize("trial", [0, 1])
def test_batch_against_the_exact_solution(cuda_device, trial):
    """Sixteen systems to 1e-10, in one launch and one by one, against their
    solutions beyond 64 bits: the error is A^-1 of a residual of 1e-10 of the
    right-hand side, a few 1e-11 of max|p| on these systems, and at most 1e-10."""
    import torch
    from twophaseflow_b200 import PPESolverFVMMatrixFree, UniformGrid, solve_batched

    class Cfg:
        pseudo_tol = 1e-10
        pseudo_maxiter = 200000
        ppe_iteration_method = "cg"
        ppe_preconditioner = "jacobi"

    rng = np.random.default_rng(trial)
    shapes = [tuple(int(n) for n in rng.integers(48, 97, 2)) for _ in range(16)]
    solvers = [PPESolverFVMMatrixFree(None, Cfg(), UniformGrid(N)) for N in shapes]
    rho = [droplet_density(N, n_drops=3, rho_g=1e-2, seed=100 * trial + k) for k, N in enumerate(shapes)]
    rhs = [divergence_rhs(N, seed=1000 + 100 * trial + k) for k, N in enumerate(shapes)]
    rho_d, rhs_d = ([torch.from_numpy(a).to(cuda_device) for a in x] for x in (rho, rhs))
    got = solve_batched(solvers, rhs_d, rho_d)
    for k, s in enumerate(solvers):
        exact = _exact(s.grid, rho[k], rhs[k], s._pin_dof)
        for p in (got[k], s.solve(rhs_d[k], rho_d[k])):
            assert np.abs(p.cpu().numpy() - exact).max() <= 1e-10 * np.abs(exact).max(), shapes[k]
