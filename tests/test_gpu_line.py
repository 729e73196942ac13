"""GPU parity of the line kernel (fftb_line.cuh): every radix and stage count, both thread mappings
and the staged sides, forward, inverse, R2C and C2R, with a last tile that is not full.

Reference: numpy's FP64 FFT.  Tolerance (relative L2): an FFT of n points has a root mean square
error of a few eps sqrt(log2 n) (Gentleman and Sande 1966; eps = 6e-8 / 1.1e-16), so 2e-6 (f32)
and 4e-15 (f64) leave a factor of five at n = 4096.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
TOL = {"float32": 2e-6, "float64": 4e-15}

# one length per radix, per pair of stages, and the three- to five-stage plans up to the largest
LENGTHS = [1, 2, 3, 5, 7, 9, 10, 11, 12, 13, 14, 15, 16, 18, 25, 44, 49, 64, 98, 125, 150, 180,
           192, 208, 225, 243, 250, 256, 288, 300, 320, 343, 360, 384, 400, 432,
           480, 500, 512, 600, 625, 640, 768, 900, 960, 675, 1000, 1024, 1250, 2187, 2401, 3125, 4096]
# (points adjacent in memory, lines adjacent) of the input and of the output
SIDES = [("row", "row"), ("col", "col"), ("row", "col"), ("col", "row")]


@pytest.fixture(scope="module")
def F(torch_cuda):
    from fftm_b200 import build
    build.build()
    import fftm_b200
    return fftm_b200


def layout(side, n, lines):
    """(stride, dist) of `lines` lines of n points."""
    return (1, n) if side == "row" else (lines, 1)


def put(a, side):
    return np.ascontiguousarray(a if side == "row" else a.T)


def get(t, side, n, lines):
    a = t.cpu().numpy()
    return a.reshape(lines, n) if side == "row" else a.reshape(n, lines).T


def rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


def lines_for(n):
    # neither a multiple of the lines of a CTA nor a single tile
    return 131 if n <= 64 else (37 if n <= 1024 else 5)


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("sides", SIDES)
@pytest.mark.parametrize("n", LENGTHS)
def test_line_kinds(F, torch_cuda, n, sides, dtype):
    torch = torch_cuda
    rng = np.random.default_rng(n)
    lines = lines_for(n)
    si, so = sides
    real = np.float32 if dtype == "float32" else np.float64
    comp = np.complex64 if dtype == "float32" else np.complex128
    x = (rng.uniform(-1, 1, (lines, n)) + 1j * rng.uniform(-1, 1, (lines, n))).astype(comp)
    for direction, ref in ((F.C2CF, np.fft.fft(x.astype(np.complex128))),
                           (F.C2CB, np.fft.ifft(x.astype(np.complex128)) * n)):
        plan = F.Plan(direction, [n], [n], *layout(si, n, lines), [n], *layout(so, n, lines), lines, dtype=dtype)
        out = torch.empty(lines * n, dtype=torch.complex64 if dtype == "float32" else torch.complex128, device="cuda")
        plan.exec(torch.from_numpy(put(x, si)).cuda(), out)
        assert rel(get(out, so, n, lines), ref) <= TOL[dtype]
    # real lines of 2 n points (the packed half-length line) and of n (odd n: the full line)
    for m in ([2 * n, n] if n % 2 else [2 * n]):
        if m < 2 or m > 4096:
            continue
        h = m // 2 + 1
        u = rng.uniform(-1, 1, (lines, m)).astype(real)
        ref = np.fft.rfft(u.astype(np.float64))
        plan = F.Plan(F.R2C, [m], [m], *layout(si, m, lines), [h], *layout(so, h, lines), lines, dtype=dtype)
        spec = torch.empty(lines * h, dtype=torch.complex64 if dtype == "float32" else torch.complex128, device="cuda")
        plan.exec(torch.from_numpy(put(u, si)).cuda(), spec)
        assert rel(get(spec, so, h, lines), ref) <= TOL[dtype]
        # a spectrum that is not Hermitian in its DC and Nyquist bins: the C2R keeps their real parts
        y = ref.astype(comp)
        y[:, 0] += 0.5j
        if m % 2 == 0:
            y[:, -1] += 0.25j
        plan = F.Plan(F.C2R, [m], [h], *layout(si, h, lines), [m], *layout(so, m, lines), lines, dtype=dtype)
        back = torch.empty(lines * m, dtype=torch.float32 if dtype == "float32" else torch.float64, device="cuda")
        plan.exec(torch.from_numpy(put(y, si)).cuda(), back)
        assert rel(get(back, so, m, lines), u.astype(np.float64) * m) <= TOL[dtype]


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("shape", [(16, 9, 10), (45, 26, 18), (180, 4, 6), (512, 3, 2), (384, 4, 2), (500, 2, 4), (9, 1000, 4)])
def test_sandwich(F, torch_cuda, shape, dtype):
    """The x sandwich of the staged solve at one to three stages (the second transform runs the
    radices in reverse), and the row mapping's sandwich in the 4D pencil order."""
    torch = torch_cuda
    rng = np.random.default_rng(7)
    real = np.float32 if dtype == "float32" else np.float64
    for dims, layout4 in ((shape, None), (shape + (4,), "pencil")):
        f = F.ffts(dtype, strategy_4d=layout4 or "pencil").init(*dims)
        x = rng.uniform(-1, 1, dims).astype(real)
        k2 = 0
        for a, n in enumerate(dims):
            k = np.fft.fftfreq(n, 1.0 / n)
            k2 = k2 + k.reshape([-1 if b == a else 1 for b in range(len(dims))]) ** 2
        spec = np.fft.fftn(x.astype(np.float64))
        ref = np.fft.ifftn(np.where(k2 == 0, 0, -spec / np.where(k2 == 0, 1, k2))).real
        arr = np.ascontiguousarray(x.T) if layout4 else x
        out = torch.empty(arr.shape, dtype=torch.float32 if dtype == "float32" else torch.float64, device="cuda")
        f.poisson(torch.from_numpy(arr).cuda(), out)
        got = out.cpu().numpy()
        assert rel(got.T if layout4 else got, ref) <= TOL[dtype]


def test_strided_points_and_lines(F, torch_cuda):
    """Neither points nor lines adjacent: the side goes through shared memory in its own order."""
    torch = torch_cuda
    n, lines = 60, 33
    rng = np.random.default_rng(3)
    x = (rng.uniform(-1, 1, (lines, n, 2)) + 1j * rng.uniform(-1, 1, (lines, n, 2))).astype(np.complex64)
    plan = F.Plan(F.C2CF, [n], [n], 2, 2 * n, [n], 3, 3 * n, lines, dtype="float32")
    out = torch.zeros(lines * n * 3, dtype=torch.complex64, device="cuda")
    plan.exec(torch.from_numpy(x).cuda(), out)
    got = out.cpu().numpy().reshape(lines, n, 3)
    assert rel(got[..., 0], np.fft.fft(x[..., 0].astype(np.complex128))) <= TOL["float32"]
    assert not got[..., 1:].any()


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("dims,layout4", [((12, 20), None), ((9, 15), None), ((20, 18, 25), None), ((7, 64, 32), None),
                                          ((64, 64, 64), None), ((17, 12, 10), None), ((6, 10, 8, 12), "pencil"),
                                          ((6, 10, 8, 9), "slab"), ((8, 6, 10, 12), "native_xzwy")])
def test_derivatives_of_one_axis(F, torch_cuda, dims, layout4, dtype):
    """derivative() and gradient() (one axis's transform; (17, ...) takes the whole transform, as a
    chirp-z axis does) against i k on numpy's half spectrum: k = index on the half axis and up to
    n/2 on the full axes, the Nyquist bin at +n/2, the C2R keeping the real part of the half
    axis's DC and Nyquist bins.  The multiply raises the rounding of the largest k by n/2 over
    the mean k: four times the transform's tolerance."""
    torch = torch_cuda
    rng = np.random.default_rng(11)
    u = rng.uniform(-1, 1, dims).astype(np.float32 if dtype == "float32" else np.float64)
    d = len(dims)
    spec = np.fft.rfftn(u.astype(np.float64))
    f = F.ffts(dtype, strategy_4d=layout4 or "pencil").init(*dims)
    arr = np.ascontiguousarray(u.T) if layout4 == "pencil" else u
    x = torch.from_numpy(arr).cuda()
    outs = [torch.empty_like(x) for _ in dims]
    f.gradient(x, outs)
    one = torch.empty_like(x)
    for axis, n in enumerate(dims):
        i = np.arange(n // 2 + 1 if axis == d - 1 else n)
        k = np.where(i <= n // 2, i, i - n).reshape([-1 if a == axis else 1 for a in range(d)])
        y = np.fft.ifftn(1j * k * spec, axes=tuple(range(d - 1)))
        ref = np.fft.irfft(y, n=dims[-1], axis=d - 1)
        f.derivative(x, one, axis)
        for got in (outs[axis], one):
            g = got.cpu().numpy()
            assert rel(g.T if layout4 == "pencil" else g, ref) <= 4 * TOL[dtype], axis


def test_short_double_columns_are_as_fast_as_a_copy_allows(F, torch_cuda):
    """Columns of one and two double points in at most twice the time of a copy of the same bytes (1.4
    and 1.0 times it; CTAs of one warp took 5.4 and 2.7 times it)."""
    torch = torch_cuda
    x = torch.randn(1 << 22, dtype=torch.complex128, device="cuda")
    y = torch.empty_like(x)

    def us(fn):
        best = float("inf")
        for _ in range(4):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            for _ in range(10):
                fn()
            b.record()
            b.synchronize()
            best = min(best, a.elapsed_time(b))
        return best

    copy = us(lambda: y.copy_(x))
    for n in (1, 2):
        lines = (1 << 22) // n
        plan = F.Plan(F.C2CF, [n], [n], lines, 1, [n], lines, 1, lines, dtype="float64")
        assert us(lambda: plan.exec(x, y)) <= 2 * copy, n


# from rows to columns, on both sides of the lengths where the mapping changes (double: 4 and more split
# points up to 63, real lines up to 94; float C2R: 3584 points and more), a last tile that is not full
MIXED = [("float64", k, n) for k, ns in (("F", (2, 3, 4, 8, 35, 63, 64)), ("I", (4, 13, 60, 64)),
                                         ("R", (4, 6, 8, 16, 35, 90, 94, 96, 98)),
                                         ("C", (4, 6, 8, 16, 35, 45, 47, 49, 90, 96, 98))) for n in ns]
MIXED += [("float32", "C", n) for n in (3456, 3500, 3584, 3600, 3840, 4096, 8192)]


@pytest.mark.parametrize("dtype,kind,n", MIXED)
def test_rows_to_columns(F, torch_cuda, dtype, kind, n):
    torch = torch_cuda
    rng = np.random.default_rng(n)
    lines, h = (331, n // 2 + 1) if n < 100 else (13, n // 2 + 1)
    real, comp = (np.float32, np.complex64) if dtype == "float32" else (np.float64, np.complex128)
    u = rng.uniform(-1, 1, (lines, n)).astype(real)
    z = (u + 1j * rng.uniform(-1, 1, (lines, n))).astype(comp)
    half = np.fft.rfft(u.astype(np.float64))
    x, ref, d, ni, no = {"F": (z, np.fft.fft(z), F.C2CF, n, n),
                         "I": (z, np.fft.ifft(z) * n, F.C2CB, n, n),
                         "R": (u, half, F.R2C, n, h),
                         "C": (half.astype(comp), u.astype(np.float64) * n, F.C2R, h, n)}[kind]
    out_type = getattr(torch, str(np.dtype(real if kind == "C" else comp)))
    # three points of room behind every line and three lines of room between the rows of the output
    pad = np.full((lines, ni + 3), 1e30, x.dtype)
    pad[:, :ni] = x
    out = torch.full((no, lines + 3), 7.0, dtype=out_type, device="cuda")
    plan = F.Plan(d, [n], [ni], 1, ni + 3, [no], lines + 3, 1, lines, dtype=dtype)
    plan.exec(torch.from_numpy(pad).cuda(), out)
    got = out.cpu().numpy()
    assert rel(got[:, :lines].T, ref) <= TOL[dtype]
    assert (got[:, lines:] == 7.0).all()
