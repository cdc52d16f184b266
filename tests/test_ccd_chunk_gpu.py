"""The chunk-per-thread CCD kernels at the edges of their chunks, windows and tiles."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from oracle import ccd as occd  # noqa: E402

# nodes of a line: shorter than a chunk of 16 rows, just around one, two and five chunks (the window is four) and
# the 48 head rows; a multiple of 4 (padded pitch); the most rows of 8, 4 and 2 lines per block; beyond them
LENGTHS = [6, 7, 17, 18, 19, 33, 34, 35, 49, 50, 51, 66, 81, 82, 84, 256, 1026, 1027, 2050, 2051, 4098, 4099]


def _tol(f, h, order):
    """1e-12 of the result plus the round-off of the wall closure's own sum,
    8 eps max|f| sum|c| (c_I: 10.7 / h, c_II: 640 / 12 h^2)."""
    c = 10.7 / h if order == 1 else 640.0 / (12.0 * h * h)
    return 8 * np.finfo(np.float64).eps * np.abs(f).max() * c


@pytest.mark.parametrize("n", LENGTHS)
@pytest.mark.parametrize("bc", ["wall", "periodic"])
@pytest.mark.parametrize("axis", [0, 1])
def test_line_lengths_and_ragged_tiles(cuda_device, n, bc, axis):
    """37 lines (no multiple of a tile) of every length, as rows and as
    columns, against the oracle's dense solve; a view that starts off 16 bytes
    gives the same bits."""
    import torch
    from twophaseflow_b200 import CCDSolver, UniformGrid
    shape = (n, 37) if axis == 0 else (37, n)
    N = tuple(s - 1 for s in shape)
    f = np.random.default_rng(n).standard_normal(shape)
    if bc == "periodic":
        f[-1, :] = f[0, :]
        f[:, -1] = f[:, 0]
    ccd = CCDSolver(UniformGrid(N), None, bc_type=bc)
    store = torch.zeros(f.size + 1, dtype=torch.float64, device=cuda_device)
    store[1:] = torch.from_numpy(f.ravel()).to(cuda_device)
    d = ccd.differentiate(torch.from_numpy(f).to(cuda_device), axis)
    u = ccd.differentiate(store[1:].view(shape), axis)
    h = 1.0 / N[axis]
    # the dense 2 n x 2 n solve of the longest lines takes minutes: their middle is compared with the solve of a
    # window of 801 nodes, whose ends are 300 rows away (0.455^300 of them is left)
    for k in range(2):
        assert torch.equal(d[k], u[k])
        got = np.moveaxis(d[k].cpu().numpy(), axis, 0)
        line = np.moveaxis(f, axis, 0)
        if n <= 1027:
            ref = np.moveaxis(occd.differentiate(f, axis, h, bc=bc)[k], axis, 0)
            err = np.abs(got - ref).max()
            tol = 1e-12 * np.abs(ref).max() + (_tol(f, h, k + 1) if bc == "wall" else 0.0)
            assert err <= tol, (k, err, tol)
            continue
        for a in (0, n // 2 - 400, n - 801):
            w = occd.differentiate(np.ascontiguousarray(line[a:a + 801]), 0, h, bc="wall")[k]
            lo = 0 if a == 0 and bc == "wall" else 300
            hi = 801 if a == n - 801 and bc == "wall" else 501
            err = np.abs(got[a + lo:a + hi] - w[lo:hi]).max()
            assert err <= 1e-12 * np.abs(w).max() + _tol(f, h, k + 1), (k, a, err)


@pytest.mark.parametrize("shape,axis", [((300, 200, 160), 0), ((160, 300, 200), 1), ((257, 129, 130), 0),
                                        ((100, 90, 200), 2), ((64, 600, 100), 1)])
@pytest.mark.parametrize("dtype", ["f64", "f32"])
def test_many_lines_match_the_single_line_solve(cuda_device, shape, axis, dtype):
    """The tile width and the staged copies do not enter a line's arithmetic:
    each line of a large field has the bits of its own one-line solve."""
    import torch
    from twophaseflow_b200 import CCDSolver, UniformGrid
    dt = torch.float64 if dtype == "f64" else torch.float32
    f = torch.randn(shape, device=cuda_device, dtype=dt, generator=torch.Generator(device="cuda").manual_seed(3))
    N = tuple(s - 1 for s in shape)
    d = CCDSolver(UniformGrid(N), None, bc_type="wall", dtype=dt).differentiate(f, axis)
    n = shape[axis]
    one = CCDSolver(UniformGrid((n - 1, 6), (1.0, 1.0)), None, bc_type="wall", dtype=dt)
    lines = [t.movedim(axis, 0).reshape(n, -1) for t in (f, *d)]
    m = lines[0].shape[1]
    for c in (0, 1, 15, 16, 31, 32, m // 2 - 3, m - 7):
        cols = slice(c, c + 7)
        e = one.differentiate(lines[0][:, cols].contiguous(), 0)
        for k in range(2):
            assert torch.equal(e[k], lines[1 + k][:, cols]), (c, k)


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
@pytest.mark.parametrize("bc", ["wall", "periodic"])
@pytest.mark.parametrize("axis", [0, 1])
def test_one_bad_value_reaches_its_whole_line(cuda_device, bad, bc, axis):
    """The recurrences carry a value that is not finite from end to end of its
    line, however far the chunks' windows reach, and to no other line."""
    import torch
    from twophaseflow_b200 import CCDSolver, UniformGrid
    f = torch.randn((400, 400), device=cuda_device, dtype=torch.float64)
    if bc == "periodic":
        f[-1], f[:, -1] = f[0].clone(), f[:, 0].clone()
        f[-1, -1] = f[0, 0]
    f[200, 200] = bad
    d = CCDSolver(UniformGrid((399, 399)), None, bc_type=bc).differentiate(f, axis)
    for t in d:
        finite = torch.isfinite(t.movedim(axis, 0))
        assert not bool(finite[:, 200].any())
        finite[:, 200] = True
        assert bool(finite.all())


# many lines of lengths at which a block takes 24, 12, 6 and 3 lines (FP64) and, in FP32 with its blocks of up to 1024
# threads, 28, 24, 32, 28, 24, 16, 12, 8, 6 and 4; longer lines than the chunk kernels take; rows that start off 16 bytes
MANY = [((290, 135, 141), 0), ((135, 330, 141), 1), ((400, 135, 141), 0), ((560, 101, 165), 0), ((99, 660, 145), 1),
        ((1000, 75, 127), 0), ((1340, 75, 97), 0), ((2000, 50, 97), 0), ((37, 2700, 97), 1), ((4097, 25, 97), 0),
        ((4200, 7, 101), 0)]


@pytest.mark.parametrize("shape,axis", MANY)
@pytest.mark.parametrize("bc", ["wall", "periodic"])
@pytest.mark.parametrize("dtype", ["f64", "f32"])
def test_lines_per_block_do_not_enter_a_line(cuda_device, shape, axis, bc, dtype):
    """Each line of a large field has the bits of its own solve among seven
    lines, at the edges of a tile and in the last, ragged one."""
    import torch
    from twophaseflow_b200 import CCDSolver, UniformGrid
    dt = torch.float64 if dtype == "f64" else torch.float32
    f = torch.randn(shape, device=cuda_device, dtype=dt, generator=torch.Generator(device="cuda").manual_seed(4))
    n = shape[axis]
    if bc == "periodic":
        f.select(axis, n - 1).copy_(f.select(axis, 0))
    N = tuple(s - 1 for s in shape)
    d = CCDSolver(UniformGrid(N), None, bc_type=bc, dtype=dt).differentiate(f, axis)
    one = CCDSolver(UniformGrid((n - 1, 6), (1.0, 1.0)), None, bc_type=bc, dtype=dt)
    lines = [t.movedim(axis, 0).reshape(n, -1) for t in (f, *d)]
    m = lines[0].shape[1]
    for c in (0, 9, 25, m // 2 - 3, m - 7):
        cols = slice(c, c + 7)
        e = one.differentiate(lines[0][:, cols].contiguous(), 0)
        for k in range(2):
            assert torch.equal(e[k], lines[1 + k][:, cols]), (c, k)


def _ns_per_node(n, bc, device):
    """FP64 differentiation of n^3 nodes along axis 0, the shortest of seven runs of four."""
    import torch
    from twophaseflow_b200 import CCDSolver, UniformGrid
    f = torch.randn((n, n, n), device=device, dtype=torch.float64)
    ccd = CCDSolver(UniformGrid((n - 1,) * 3), None, bc_type=bc)
    ccd.differentiate(f, 0)
    times = []
    for _ in range(7):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        torch.cuda.synchronize()
        torch.cuda._sleep(200000)   # the calls are queued before the first one runs
        a.record()
        for _ in range(4):
            ccd.differentiate(f, 0)
        b.record()
        torch.cuda.synchronize()
        times.append(a.elapsed_time(b))
    return min(times) / 4 * 1e6 / n**3


def test_time_per_node_has_no_step_beyond_sixteen_chunks(cuda_device):
    """Lines of 17 chunks fill 408 threads of an SM's 512 with 24 lines to a
    block, lines of 16 all of them: at most 512 / 408 times as long a node (it
    was 1.34 with 16 lines, 272 threads)."""
    a, b = (_ns_per_node(n, "wall", cuda_device) for n in (257, 273))
    assert b <= 512 / 408 * a, (a, b)


def test_time_per_node_has_no_step_beyond_two_gigabytes(cuda_device):
    """Field and derivatives of 449^3 nodes are 2.2 GB, of 417^3 1.7; both have
    16 lines to a block, 448 and 416 threads, so the larger field should take no
    longer a node: a tenth is left for the runs' scatter (it was 1.25 to 1.3
    while the SMs took their tiles at a fixed stride and drifted apart)."""
    a, b = (_ns_per_node(n, "periodic", cuda_device) for n in (417, 449))
    assert b <= 1.1 * a, (a, b)


class _Calls:
    """The epilogues of the line solve along one axis, through the C ABI."""

    def __init__(self, shape, axis, bc, dt, device):
        import ctypes as C

        import torch
        from twophaseflow_b200 import _lib
        from twophaseflow_b200.arrays import line_split
        self.lib, self._lib = _lib.load(), _lib
        g = torch.Generator(device="cuda").manual_seed(5)
        self.f, self.u, drho = (torch.randn(shape, device=device, dtype=dt, generator=g) for _ in range(3))
        self.rho, self.drho = torch.rand(shape, device=device, dtype=dt, generator=g) + 1, drho
        n = shape[axis]
        self.plan = C.c_void_p()
        _lib.check(self.lib.tpf_ccd_plan_create(C.byref(self.plan), n, 1.0 / (n - 1),
                                                _lib.TPF_BC_PERIODIC if bc == "periodic" else _lib.TPF_BC_WALL,
                                                _lib.TPF_F64 if dt == torch.float64 else _lib.TPF_F32))
        x = np.arange(n, dtype=np.float64)
        J, dJ = 1.0 + 0.25 * np.sin(x), 0.5 * np.cos(x)
        _lib.check(self.lib.tpf_ccd_plan_set_metric(self.plan, *(a.ctypes.data_as(C.POINTER(C.c_double)) for a in (J, dJ))))
        outer, _, inner = line_split(shape, axis)
        self.split = (outer, inner)

    def __del__(self):
        self.lib.tpf_ccd_plan_destroy(self.plan)

    def run(self, kind, metric, out):
        """out: the fields written (d1, d2), or the one written, which is the
        corrector's u* too and what the variable-density term adds to."""
        p, s = self._lib.dptr, self._lib.current_stream_handle()
        flags = self._lib.TPF_CCD_APPLY_METRIC if metric else 0
        if kind == "plain":
            st = self.lib.tpf_ccd_apply(self.plan, *self.split, p(self.f), p(out[0]), p(out[1]), None, None, flags, s)
        elif kind == "corrector":
            st = self.lib.tpf_ccd_apply_corrector(self.plan, *self.split, p(self.f), p(out[0]), p(self.rho), 0.01,
                                                  p(out[0]), flags, s)
        else:
            st = self.lib.tpf_ccd_apply_vd(self.plan, *self.split, p(self.f), p(self.rho), p(self.drho), p(out[0]), 1,
                                           flags, s)
        self._lib.check(st)


# one warp's elements and less than a batch of them; several batches and a remainder; a ragged last tile; long lines
@pytest.mark.parametrize("shape,axis", [((3, 7), 1), ((5, 33), 1), ((65, 65), 1), ((65, 65), 0), ((41, 130), 1),
                                        ((37, 1500), 1), ((12, 11, 194), 2), ((30, 20, 9), 0), ((9, 50, 21), 1)])
@pytest.mark.parametrize("bc", ["wall", "periodic"])
@pytest.mark.parametrize("dtype", ["f64", "f32"])
@pytest.mark.parametrize("metric", [False, True])
def test_epilogues_against_the_plain_derivatives(cuda_device, shape, axis, bc, dtype, metric):
    """Corrector (in place) and variable-density term (accumulated) equal the
    formulas on the plain call's d1 and d2 to the rounding of the type, some
    operations of 4 eps each; the metric is that of the chain rule."""
    import torch
    dt = torch.float64 if dtype == "f64" else torch.float32
    c = _Calls(shape, axis, bc, dt, cuda_device)
    if bc == "periodic":
        c.f.select(axis, shape[axis] - 1).copy_(c.f.select(axis, 0))
    d = [torch.empty_like(c.f) for _ in range(2)]
    c.run("plain", False, d)
    d1, d2 = (t.double() for t in d)
    if metric:
        x = torch.arange(shape[axis], device=cuda_device, dtype=torch.float64)
        J, dJ = ((1.0 + 0.25 * torch.sin(x)), 0.5 * torch.cos(x))
        J, dJ = (t.view([-1] + [1] * (len(shape) - 1 - axis)) for t in (J, dJ))
        d2 = J * J * d2 + J * dJ * d1
        d1 = J * d1
        m = [torch.empty_like(c.f) for _ in range(2)]
        c.run("plain", True, m)
        for got, want in zip(m, (d1, d2)):
            assert float((got.double() - want).abs().max()) <= 32 * torch.finfo(dt).eps * float(want.abs().max() + d1.abs().max())
    rho, drho, u = c.rho.double(), c.drho.double(), c.u.double()
    eps = 32 * torch.finfo(dt).eps
    step = 0.01 / rho * d1
    if bc == "wall":
        step.select(axis, 0).zero_()
        step.select(axis, shape[axis] - 1).zero_()
    got = c.u.clone()
    c.run("corrector", metric, [got])
    assert float((got.double() - (u - step)).abs().max()) <= eps * float(u.abs().max() + step.abs().max())
    term = d2 / rho - drho / (rho * rho) * d1
    got = c.u.clone()
    c.run("vd", metric, [got])
    size = (d2 / rho).abs().max() + (drho / (rho * rho) * d1).abs().max()
    assert float((got.double() - (u + term)).abs().max()) <= eps * float(u.abs().max() + size)


@pytest.mark.parametrize("dtype", ["f64", "f32"])
def test_epilogues_of_the_contiguous_axis_cost_their_bytes(cuda_device, dtype):
    """The accumulated variable-density term moves 5 values a node where the
    plain call moves 3: at most half as long again as that ratio says (it was
    4.1 instead of 1.7 times as long when each element's operands were waited
    for by themselves)."""
    import torch
    dt = torch.float64 if dtype == "f64" else torch.float32
    c = _Calls((193, 193, 193), 2, "wall", dt, cuda_device)
    out = [torch.zeros_like(c.f) for _ in range(2)]
    times = {}
    for kind in ("plain", "vd"):
        c.run(kind, False, out)
        best = []
        for _ in range(7):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            torch.cuda.synchronize()
            torch.cuda._sleep(200000)
            a.record()
            for _ in range(8):
                c.run(kind, False, out)
            b.record()
            torch.cuda.synchronize()
            best.append(a.elapsed_time(b))
        times[kind] = min(best)
    assert times["vd"] <= 1.5 * 5 / 3 * times["plain"], times


def test_dealt_out_tiles_beside_other_launches(cuda_device):
    """Two streams of calls whose tiles are dealt out, their blocks resident
    beside each other's and taken over as they wait: every call has the bits of
    one that runs by itself."""
    import torch
    from twophaseflow_b200 import CCDSolver, UniformGrid
    shapes = [(1025, 130, 131), (1340, 97, 75)]
    streams = [torch.cuda.Stream() for _ in shapes]
    fields = [torch.randn(s, device=cuda_device, dtype=torch.float64) for s in shapes]
    solvers = [CCDSolver(UniformGrid(tuple(n - 1 for n in s)), None, bc_type="wall") for s in shapes]
    alone = [c.differentiate(f, 0) for c, f in zip(solvers, fields)]
    torch.cuda.synchronize()
    results = [[], []]
    for _ in range(6):
        for k in range(2):
            with torch.cuda.stream(streams[k]):
                results[k].append(solvers[k].differentiate(fields[k], 0))
    torch.cuda.synchronize()
    for k in range(2):
        for d in results[k]:
            assert torch.equal(d[0], alone[k][0]) and torch.equal(d[1], alone[k][1])
