"""The state a pressure-solver handle is left in by batches that are refused or fail.

Called through the C ABI, so that no allocation of the caller's is in the way of
the stream capture that makes the batch's own allocation fail."""

import ctypes as C

import pytest

pytestmark = pytest.mark.gpu

from twophaseflow_b200 import _lib  # noqa: E402
from twophaseflow_b200.workloads import divergence_rhs, droplet_density  # noqa: E402


class _Cfg:
    pseudo_tol = 1e-10
    pseudo_maxiter = 20000
    ppe_iteration_method = "cg"
    ppe_preconditioner = "jacobi"


def _system(N, seed, dev):
    import torch
    from twophaseflow_b200 import PPESolverFVMMatrixFree, UniformGrid
    s = PPESolverFVMMatrixFree(None, _Cfg(), UniformGrid(N))
    rho = torch.from_numpy(droplet_density(N, n_drops=3, rho_g=1e-2, seed=seed)).to(dev)
    rhs = torch.from_numpy(divergence_rhs(N, seed=seed + 1)).to(dev)
    return s, rho, rhs, torch.zeros_like(rhs)


def _batch(lib, systems, rhos, stream):
    n = len(systems)

    def ptrs(values):
        return (C.c_void_p * n)(*[None if v is None else v.data_ptr() for v in values])
    res = (_lib.tpf_ppe_result * n)()
    return lib.tpf_ppe_solve_batched((C.c_void_p * n)(*[s._handle.value for s, *_ in systems]), n,
                                     ptrs([x[2] for x in systems]), ptrs(rhos), ptrs([x[3] for x in systems]),
                                     C.c_void_p(stream.cuda_stream), res)


def _solve(lib, system, rho, stream):
    s, _, rhs, p = system
    res = _lib.tpf_ppe_result()
    return lib.tpf_ppe_solve(s._handle, _lib.dptr(rhs), None if rho is None else _lib.dptr(rho), _lib.dptr(p), None,
                             C.c_void_p(stream.cuda_stream), C.byref(res))


@pytest.mark.parametrize("prepared", [False, True])
def test_failed_batch_leaves_no_system_prepared_for_a_density_it_did_not_see(cuda_device, prepared):
    """A batch whose allocations fail (they are refused while the stream is
    captured) has set up nothing: a solve without a density is refused
    afterwards, whether or not the systems held another density's couplings
    before, and a solve with one is right."""
    import torch
    lib = _lib.load()
    cuda = C.CDLL("libcuda.so.1")
    stream = torch.cuda.Stream()
    old = [_system((30, 30), 3, cuda_device), _system((26, 41), 5, cuda_device)]
    new = [torch.from_numpy(droplet_density(tuple(n - 1 for n in x[1].shape), n_drops=2, rho_g=1e-1, seed=9 + k)).to(cuda_device)
           for k, x in enumerate(old)]
    torch.cuda.synchronize()
    if prepared:
        for x in old:
            assert _solve(lib, x, x[1], stream) == _lib.TPF_OK
    graph = C.c_void_p()
    assert cuda.cuStreamBeginCapture_v2(C.c_void_p(stream.cuda_stream), 0) == 0
    status = _batch(lib, old, new, stream)
    cuda.cuStreamEndCapture(C.c_void_p(stream.cuda_stream), C.byref(graph))
    if graph.value:
        cuda.cuGraphDestroy(graph)
    assert status == _lib.TPF_ECUDA
    for x, rho in zip(old, new):
        assert _solve(lib, x, None, stream) == _lib.TPF_EINVAL
        assert _solve(lib, x, rho, stream) == _lib.TPF_OK
        torch.cuda.synchronize()
        ref = _system(tuple(n - 1 for n in rho.shape), 3, cuda_device)[0].solve(x[2], rho)
        assert torch.equal(x[3], ref)


def test_refused_batch_has_prepared_the_systems_before_the_refused_one(cuda_device):
    """A system without couplings and without a density refuses the batch; the
    systems before it were given their densities and solve for them."""
    import torch
    lib = _lib.load()
    stream = torch.cuda.current_stream()
    a, b = _system((30, 30), 3, cuda_device), _system((26, 41), 5, cuda_device)
    first = torch.full_like(a[1], 1.0)
    assert _solve(lib, a, first, stream) == _lib.TPF_OK
    assert _batch(lib, [a, b], [a[1], None], stream) == _lib.TPF_EINVAL
    assert _solve(lib, a, None, stream) == _lib.TPF_OK
    torch.cuda.synchronize()
    ref = _system((30, 30), 3, cuda_device)
    assert torch.equal(a[3], ref[0].solve(ref[2], ref[1]))
