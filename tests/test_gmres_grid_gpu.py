"""The one-launch GMRES at the edges of its block, line and basis layouts."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from oracle import ppe as oppe  # noqa: E402
from twophaseflow_b200.workloads import bubble_density, divergence_rhs  # noqa: E402


def _solver(N, **kw):
    from twophaseflow_b200 import PPESolverFVMMatrixFree, UniformGrid

    class Cfg:
        pseudo_tol = 1e-10
        pseudo_maxiter = 500
        ppe_iteration_method = "gmres"

    for k, v in kw.items():
        setattr(Cfg, k, v)
    return PPESolverFVMMatrixFree(None, Cfg(), UniformGrid(N))


# one block; two columns per line lane and one node more (64, 65 nodes); 96 / 97, 160 / 161, 288 / 289 nodes (3, 5 and 9
# rows per lane); more columns than rows and the reverse (blocks of one row, blocks of many); the longest lines (544
# nodes); the basis in global memory; beyond the one-launch kernel
SIZES = [(4, 5), (15, 15), (63, 20), (64, 33), (20, 96), (96, 40), (159, 24), (24, 160), (287, 12), (12, 288),
         (300, 6), (6, 300), (543, 20), (20, 543), (200, 180), (20, 544)]


@pytest.mark.parametrize("N", SIZES)
def test_sizes_against_the_direct_solution(cuda_device, N):
    """The true residual (the oracle's operator) is below 1e-9 of ||rhs||, the
    solution within 1e-6 of the direct one, and a second solve of the handle
    gives the same bits."""
    import torch
    rho = bubble_density(N, rho_g=0.1)
    rhs = divergence_rhs(N, seed=3)
    s = _solver(N)
    p = s.solve(torch.from_numpy(rhs).to(cuda_device), torch.from_numpy(rho).to(cuda_device))
    assert s.last_diagnostics["ppe_low_order_gmres_relative_residual"] <= 1e-10
    q = s.solve(torch.from_numpy(rhs).to(cuda_device), torch.from_numpy(rho).to(cuda_device))
    assert torch.equal(p, q)
    o = oppe.FVMMatrixFree(oppe.uniform_coords(N, (1.0, 1.0)), method="gmres", tol=1e-10)
    o.prepare_operator(rho)
    b = rhs.copy()
    b.ravel()[o.pin] = 0.0
    r = b - o.apply(p.cpu().numpy())
    assert np.linalg.norm(r) <= 1e-9 * np.linalg.norm(b)
    pd = oppe.spsolve_fvm(rhs, rho, oppe.uniform_coords(N, (1.0, 1.0)))
    assert np.abs(p.cpu().numpy() - pd).max() <= 1e-6 * np.abs(pd).max()


@pytest.mark.parametrize("kw", [dict(), dict(ppe_restart=7), dict(ppe_restart=1000), dict(ppe_preconditioner="jacobi"),
                                dict(ppe_preconditioner="none", pseudo_tol=1e-6), dict(ppe_restart=200)])
@pytest.mark.parametrize("warm", [False, True])
def test_options_take_the_oracle_s_path(cuda_device, kw, warm):
    """Restart lengths (shorter than, and as long as, the system; a basis or a
    Hessenberg matrix too large for shared memory), preconditioners and an
    initial guess: the oracle's iteration count within 3 % + 2 and its
    solution within 100 tol."""
    N = (18, 23)
    rho = bubble_density(N, rho_g=0.1)
    rhs = divergence_rhs(N, seed=4)
    p0 = divergence_rhs(N, seed=5) * 1e-3 if warm else None
    s = _solver(N, **kw)
    p = s.solve(rhs, rho, 0.0, p0)
    o = oppe.FVMMatrixFree(oppe.uniform_coords(N, (1.0, 1.0)), method="gmres", tol=s.tol, restart=s.restart,
                           preconditioner=s.preconditioner)
    po = o.solve(rhs, rho, p_init=p0)
    it = s.last_diagnostics["ppe_low_order_gmres_iterations"]
    assert abs(it - o.last_iterations) <= 2 + 0.03 * o.last_iterations, (it, o.last_iterations)
    assert np.abs(p - po).max() <= 100 * s.tol * np.abs(po).max()


def test_zero_rhs_and_exhausted_cycles(cuda_device):
    N = (24, 24)
    rho = bubble_density(N, rho_g=0.1)
    s = _solver(N)
    assert not s.solve(np.zeros((25, 25)), rho).any()
    s = _solver(N, pseudo_maxiter=1, ppe_restart=5)
    with pytest.raises(RuntimeError):
        s.solve(divergence_rhs(N, seed=4), rho)


@pytest.mark.parametrize("N", [(24, 20), (700, 600)])
def test_no_cycle_allowed_is_not_converged(cuda_device, N):
    """With no restart cycle allowed the initial guess is not looked at: not
    converged after no iterations and no operator application, even where the
    guess is the solution (one launch, and the column kernels)."""
    import torch
    s = _solver(N, pseudo_tol=1e-3, pseudo_maxiter=0)
    rho = torch.from_numpy(bubble_density(N, rho_g=0.1)).to(cuda_device)
    x = torch.from_numpy(divergence_rhs(N, seed=3)).to(cuda_device)
    x.view(-1)[s._pin_dof] = 0.0
    s.prepare_operator(rho)
    rhs = s.apply(x)
    with pytest.raises(RuntimeError, match="info=0"):
        s.solve(rhs, rho, 0.0, x)
    assert s.last_diagnostics["ppe_low_order_gmres_iterations"] == 0
    assert s.last_diagnostics["ppe_low_order_gmres_applies"] == 0


# just below the sizes where a block's line factors no longer fit beside the Hessenberg matrix: 440^2 at restart 80,
# 512^2 at 60; the longest lines without factors; the basis is in global memory throughout
@pytest.mark.parametrize("N,kw", [((440, 440), dict(ppe_restart=80)), ((512, 512), dict(ppe_restart=30)),
                                  ((512, 512), dict(ppe_restart=60)),
                                  ((540, 540), dict(ppe_restart=80, ppe_preconditioner="jacobi")),
                                  ((543, 530), dict(ppe_restart=30, ppe_preconditioner="none"))])
def test_one_cycle_of_the_largest_systems(cuda_device, N, kw):
    """One restart cycle against the oracle's: the iterate within 1e-8 of its
    largest value (the least-squares problem of a cycle amplifies the round-off
    of two orthogonalizations, some 1e-14, by at most the Hessenberg matrix'
    condition, some 1e4 here), the residual within 1e-8."""
    import torch
    from twophaseflow_b200 import _lib
    s = _solver(N, pseudo_tol=1e-12, pseudo_maxiter=1, **kw)
    rho, rhs = bubble_density(N, rho_g=0.1), divergence_rhs(N, seed=4)
    rho_d, rhs_d = torch.from_numpy(rho).to(cuda_device), torch.from_numpy(rhs).to(cuda_device)
    p, res = torch.empty_like(rhs_d), _lib.tpf_ppe_result()
    assert s.lib.tpf_ppe_solve(s._handle, _lib.dptr(rhs_d), _lib.dptr(rho_d), _lib.dptr(p), None,
                               _lib.current_stream_handle(), res) == _lib.TPF_ENOCONV
    assert res.iterations == s.restart
    o = oppe.FVMMatrixFree(oppe.uniform_coords(N, (1.0, 1.0)), method="gmres", preconditioner=s.preconditioner)
    o.prepare_operator(rho)
    pco = oppe.line_precond_coeffs(o.coeffs, rho, o.c_tau, o.h_min)
    dinv = oppe.jacobi_diag_inv(o.coeffs, o.pin)

    def precondition(r):
        r = r.reshape(o.shape)
        if s.preconditioner == "line_pcr":
            return oppe.line_precond(r, pco, o.pin, None).ravel()
        z = r * dinv if s.preconditioner == "jacobi" else r.copy()
        if s.preconditioner == "jacobi":
            z.ravel()[o.pin] = 0.0
        return z.ravel()
    b = rhs.ravel().copy()
    b[o.pin] = 0.0
    x, _, its = oppe.gmres(lambda v: o.apply(v.reshape(o.shape)).ravel(), precondition, b, np.zeros_like(b), 1e-12,
                           s.restart, 1)
    assert its == s.restart
    rel = np.linalg.norm(b - o.apply(x.reshape(o.shape)).ravel()) / np.linalg.norm(b)
    x[o.pin] = 0.0
    assert np.abs(p.cpu().numpy().ravel() - x).max() <= 1e-8 * np.abs(x).max()
    assert abs(res.rel_residual - rel) <= 1e-8 * rel
