"""Timed cases of the transform path, through the public Python entry points.

A case is one call (or the few calls of one step) that a program makes with a plan it keeps:
the work area and the output arrays are the program's own and are set up once, as the
reference's examples do.  The listed cases stand for:

* roundtrip_64_f32       the small 3D round trip of a solver step on a coarse grid, where the
                         launches and the host path count
* poisson_256_f32        the periodic Poisson solve on the usual single-GPU grid
* roundtrip_256_f64      the same grid in double precision (direct numerical simulation)
* poisson_512_f32        the largest grid: the spectrum is several times the L2 cache
* roundtrip_180_150_125  a box with unequal, non-power-of-two sides, one of them odd
* gradient_192_f32       the velocity gradients of a turbulence step (192 = 3 * 2^6)
* native4d_64_f32        the 4D round trip in the native_xzwy spectrum order
* pencil4d_poisson_f64   a 4D Poisson solve in double precision, uneven sides, pencil order
* forward2d_2048_f32     the spectrum of a 2D field
* lines_1000_f32         one cuFFT-style plan: many contiguous complex lines of 1000 points
* pipeline_128_grad      loss and gradient of a differentiable filter + Poisson pipeline
* batch_512              512 uneven 3D round trips in one call
"""
import math

import numpy as np
import torch

import fftm_b200 as F
import fftm_b200.autograd as A
import fftm_b200.batch as B

DEV = "cuda"
BATCH_AXES = (32, 48, 64, 96, 128)


def _case(kind, op, dims, dtype, **more):
    return dict(kind=kind, op=op, n="x".join(str(d) for d in dims), dtype=dtype, **more)


def listed():
    f32, f64 = "float32", "float64"
    return [
        dict(_case("fft", "roundtrip", (64, 64, 64), f32), name="roundtrip_64_f32"),
        dict(_case("fft", "poisson", (256, 256, 256), f32), name="poisson_256_f32"),
        dict(_case("fft", "roundtrip", (256, 256, 256), f64), name="roundtrip_256_f64"),
        dict(_case("fft", "poisson", (512, 512, 512), f32), name="poisson_512_f32"),
        dict(_case("fft", "roundtrip", (180, 150, 125), f32), name="roundtrip_180_150_125"),
        dict(_case("fft", "gradient", (192, 192, 192), f32), name="gradient_192_f32"),
        dict(_case("fft", "roundtrip", (64, 64, 64, 64), f32, layout="native_xzwy"), name="native4d_64_f32"),
        dict(_case("fft", "poisson", (48, 40, 54, 60), f64, layout="pencil"), name="pencil4d_poisson_f64"),
        dict(_case("fft", "forward", (2048, 2048), f32), name="forward2d_2048_f32"),
        dict(_case("lines", "forward", (1000,), f32, lines=16384), name="lines_1000_f32"),
        dict(_case("pipeline", "gradient", (128, 128, 128), f32), name="pipeline_128_grad"),
        dict(_case("batch", "roundtrip", (512,), f32, shapes_seed=2), name="batch_512"),
    ]


# ---------------------------------------------------------------------- drawn cases
def _spread(rng, lo, hi):
    return lo * (hi / lo) ** rng.random()


def _length(rng, lo, hi, odd=0.15):
    """An axis length in [lo, hi], spread over its logarithm: a power of two, a product of small
    primes (what a program picks when it can choose), or whatever the data has."""
    n = max(lo, min(hi, int(round(_spread(rng, lo, hi)))))
    u = rng.random()
    if u < odd:
        return n
    if u < odd + 0.3:
        return max(lo, min(hi, 2 ** int(round(math.log2(n)))))

    def smooth(m):
        for p in (2, 3, 5, 7):
            while m % p == 0:
                m //= p
        return m == 1

    while not smooth(n):
        n = n - 1 if n > lo else lo
    return n


def draw(rng):
    u = rng.random()
    dtype = "float64" if rng.random() < 0.3 else "float32"
    if u < 0.5:  # 3D objects
        top = 2 ** 27 if dtype == "float32" else 2 ** 26
        while True:
            dims = tuple(_length(rng, 24, 512) for _ in range(3))
            if rng.random() < 0.4:
                dims = (dims[0],) * 3
            plain = all(max(p for p in range(2, d + 1) if d % p == 0) <= 7 for d in dims)
            if math.prod(dims) <= (top if plain else 2 ** 24):
                break
        op = rng.choice(("roundtrip", "poisson", "poisson", "forward", "gradient"))
        if op == "gradient" and math.prod(dims) > 2 ** 24:
            op = "poisson"
        return _case("fft", op, dims, dtype)
    if u < 0.65:  # 4D objects
        while True:
            dims = tuple(_length(rng, 12, 96, odd=0.1) for _ in range(4))
            if 2 ** 16 <= math.prod(dims) <= 2 ** 24:
                break
        return _case("fft", rng.choice(("roundtrip", "poisson")), dims, dtype,
                     layout=rng.choice(("pencil", "slab", "native_xzwy")))
    if u < 0.77:  # 2D objects
        dims = tuple(_length(rng, 128, 4096, odd=0.1) for _ in range(2))
        return _case("fft", rng.choice(("roundtrip", "forward", "poisson")), dims, dtype)
    if u < 0.87:  # plans over contiguous lines
        n = _length(rng, 64, 4096)
        return _case("lines", rng.choice(("forward", "inverse")), (n,), dtype,
                     lines=max(1, int(_spread(rng, 2 ** 18, 2 ** 24) / n)))
    if u < 0.93:
        return _case("pipeline", "gradient", tuple(_length(rng, 32, 192, odd=0.0) for _ in range(3)), "float32")
    return _case("batch", "roundtrip", (int(_spread(rng, 16, 512)),), "float32", shapes_seed=rng.randrange(1 << 20))


# ---------------------------------------------------------------------- inputs
def _dims(case):
    return tuple(int(v) for v in case["n"].split("x"))


def _types(case):
    return (torch.float32, torch.complex64) if case["dtype"] == "float32" else (torch.float64, torch.complex128)


def _work_area(obj, cdtype):
    return torch.empty(max(1, -(-obj.work_size // (8 if cdtype == torch.complex64 else 16))), dtype=cdtype, device=DEV)


def _logical_axes(case):
    """The tensor dimension of each logical axis (x, y, z, w)."""
    d = len(_dims(case))
    return (3, 2, 1, 0) if case.get("layout") == "pencil" else tuple(range(d))


def _real_shape(case):
    dims = _dims(case)
    return dims[::-1] if case.get("layout") == "pencil" else dims


def _field(case, seed):
    """A periodic field: sin x sin 2y cos 3z (cos w) plus 0.1 U[-1, 1], its mean removed for the
    Poisson solves; U[-1, 1] for the plain transforms."""
    real, _ = _types(case)
    gen = torch.Generator(device=DEV).manual_seed(int(seed))
    x = torch.rand(_real_shape(case), dtype=real, device=DEV, generator=gen) * 2 - 1
    if case["op"] not in ("poisson", "gradient"):
        return x
    x *= 0.1
    wave = None
    for a, (n, ax) in enumerate(zip(_dims(case), _logical_axes(case))):
        g = 2 * math.pi * torch.arange(n, dtype=torch.float64, device=DEV) / n
        s = (torch.sin(g), torch.sin(2 * g), torch.cos(3 * g), torch.cos(g))[a]
        shape = [1] * x.dim()
        shape[ax] = n
        s = s.reshape(shape).to(real)
        wave = s if wave is None else wave * s
    x += wave
    return x.sub_(x.mean())


def _line_data(case, seed):
    real, comp = _types(case)
    gen = torch.Generator(device=DEV).manual_seed(int(seed))
    x = torch.randn((case["lines"], _dims(case)[0], 2), dtype=real, device=DEV, generator=gen)
    return torch.view_as_complex(x)


def _pipeline_field(case, seed):
    gen = torch.Generator(device=DEV).manual_seed(int(seed))
    g = [2 * math.pi * torch.arange(n, dtype=torch.float64, device=DEV) / n for n in _dims(case)]
    u = torch.sin(g[0])[:, None, None] * torch.cos(g[1])[None, :, None] * torch.cos(g[2])[None, None, :]
    return (u.float() + 0.05 * torch.randn(_dims(case), device=DEV, generator=gen)).requires_grad_(True)


def _low_pass(case, dtype):
    nx, ny, nz = _dims(case)
    kx = torch.fft.fftfreq(nx, 1.0 / nx, device=DEV, dtype=torch.float64)
    ky = torch.fft.fftfreq(ny, 1.0 / ny, device=DEV, dtype=torch.float64)
    kz = torch.arange(nz // 2 + 1, device=DEV, dtype=torch.float64)
    k2 = kx[:, None, None] ** 2 + ky[None, :, None] ** 2 + kz[None, None, :] ** 2
    return torch.exp(-k2 / (2 * 16.0 ** 2)).to(dtype)


def _batch_shapes(case):
    rng = np.random.default_rng(case["shapes_seed"])
    return [tuple(int(v) for v in rng.choice(BATCH_AXES, size=3)) for _ in range(_dims(case)[0])]


def _batch_data(case, seed):
    # every axis is a multiple of 4, so the packed transforms leave no alignment gaps
    gen = torch.Generator(device=DEV).manual_seed(int(seed))
    return torch.rand(sum(math.prod(s) for s in _batch_shapes(case)), device=DEV, generator=gen) * 2 - 1


def prepare(case, seed):
    real, comp = _types(case)
    kind, op = case["kind"], case["op"]
    state = {"case": case}
    if kind == "lines":
        n, lines = _dims(case)[0], case["lines"]
        plan = F.Plan(F.C2CF if op == "forward" else F.C2CB, [n], batch=lines, dtype=case["dtype"])
        work = torch.empty(max(1, plan.get_work_size() // 8 + 1), dtype=torch.complex64, device=DEV)
        plan.set_work_area(work)
        x = _line_data(case, seed)
        return dict(state, plan=plan, work=work, x=x, out=torch.empty_like(x))
    if kind == "batch":
        bt = B.Batch(_batch_shapes(case))
        x = _batch_data(case, seed)
        work = torch.empty(bt.spectrum_total, dtype=torch.complex64, device=DEV)
        bt.set_work_area(work)
        return dict(state, batch=bt, work=work, x=x, out=torch.empty_like(x))
    obj = F.ffts(case["dtype"], strategy_4d=case.get("layout", "pencil")).init(*_dims(case))
    work = _work_area(obj, comp)
    obj.set_work_area(work)
    state.update(obj=obj, work=work)
    if kind == "pipeline":
        return dict(state, u=_pipeline_field(case, seed), g=_low_pass(case, torch.complex64))
    x = _field(case, seed)
    state["x"] = x
    if op in ("roundtrip", "forward"):
        state["spec"] = torch.empty(obj.spectrum_shape(), dtype=comp, device=DEV)
    if op in ("roundtrip", "poisson"):
        state["out"] = torch.empty_like(x)
    if op == "gradient":
        state["outs"] = [torch.empty_like(x) for _ in _dims(case)]
    return state


def run(state):
    case = state["case"]
    kind, op = case["kind"], case["op"]
    if kind == "lines":
        state["plan"].exec(state["x"], state["out"])
        return state["out"]
    if kind == "batch":
        state["batch"].exec(B.ROUNDTRIP, state["x"], state["out"])
        return state["out"]
    obj = state["obj"]
    if kind == "pipeline":
        u = state["u"]
        u.grad = None
        smooth = A.c2r(A.r2c(u, obj) * state["g"], obj, normalized=True)
        w = A.poisson(smooth, obj, -1.0)
        loss = 0.5 * (w * w).sum()
        loss.backward()
        return [loss, w, u.grad]
    if op == "poisson":
        obj.poisson(state["x"], state["out"])
        return state["out"]
    if op == "gradient":
        obj.gradient(state["x"], state["outs"])
        return state["outs"]
    obj.forward(state["x"], state["spec"])
    if op == "forward":
        return state["spec"]
    obj.backward(state["spec"], state["out"], normalized=True)
    return state["out"]


# ---------------------------------------------------------------------- work and tolerance
def work(case):
    """Bytes: every array of a call read or written once (a round trip is two calls, and so
    reads the spectrum that it wrote); operations: 2.5 N log2 N of a real transform, 5 N log2 N
    of a complex one."""
    rb = 4 if case["dtype"] == "float32" else 8
    dims = _dims(case)
    if case["kind"] == "lines":
        pts = dims[0] * case["lines"]
        return {"bytes": 4.0 * rb * pts, "flops": 5.0 * pts * math.log2(dims[0])}
    if case["kind"] == "batch":
        total, flops = 0.0, 0.0
        for s in _batch_shapes(case):
            total += B.transform_bytes(s, rb)
            flops += 5.0 * math.prod(s) * math.log2(math.prod(s))
        return {"bytes": total, "flops": flops}
    n = math.prod(dims)
    half = 2 if len(dims) == 3 else 3 if len(dims) == 4 else 1
    nc = n // dims[half] * (dims[half] // 2 + 1)
    one = 2.5 * n * math.log2(n)
    if case["kind"] == "pipeline":
        # r2c, multiply by g, c2r and Poisson solve, and their adjoints
        spec = 2 * rb * nc
        return {"bytes": 2.0 * (2 * (rb * n + spec) + 3 * spec + 2 * rb * n), "flops": 8 * one}
    ops = {"forward": (rb * n + 2 * rb * nc, 1), "roundtrip": (2 * (rb * n + 2 * rb * nc), 2),
           "poisson": (2 * rb * n, 2), "gradient": (rb * n * (1 + len(dims)), 1 + len(dims))}
    b, transforms = ops[case["op"]]
    return {"bytes": float(b), "flops": transforms * one}


def tolerance(case):
    """About four times the distance from the exact transform that the path shows: 2e-7 to 3e-7
    (float) and 5e-16 (double) for transforms and solves; a derivative weights the largest
    wavenumbers, whose rounding it multiplies (1e-6), and the pipeline chains four transforms."""
    derived = case["op"] == "gradient"
    if case["dtype"] == "float64":
        return {"rel": 8e-15 if derived else 3e-15}
    return {"rel": 4e-6 if derived else 1.5e-6}


# ---------------------------------------------------------------------- exact values
def _wavenumbers(case, shape, half_axis):
    k2 = 0
    ks = []
    for a, (n, ax) in enumerate(zip(_dims(case), _logical_axes(case))):
        k = (torch.arange(n // 2 + 1, device=DEV, dtype=torch.float64) if a == half_axis
             else torch.fft.fftfreq(n, 1.0 / n, device=DEV, dtype=torch.float64))
        if a != half_axis and n % 2 == 0:
            k[n // 2] = n / 2  # the Nyquist index keeps its positive sign
        s = [1] * len(shape)
        s[ax] = -1
        k = k.reshape(s)
        ks.append(k)
        k2 = k2 + k * k
    return ks, k2


def exact(case, seed):
    dims = _dims(case)
    if case["kind"] == "lines":
        x = _line_data(case, seed).to(torch.complex128)
        return torch.fft.fft(x) if case["op"] == "forward" else torch.fft.ifft(x) * dims[0]
    if case["kind"] == "batch":
        return _batch_data(case, seed).double()  # a round trip gives its input back
    if case["kind"] == "pipeline":
        u = _pipeline_field(case, seed).detach().double().requires_grad_(True)
        _, k2 = _wavenumbers(case, dims, 2)
        inv = torch.where(k2 == 0, torch.zeros_like(k2), -1.0 / torch.where(k2 == 0, torch.ones_like(k2), k2))
        # the multiplier as the program holds it, rounded to its type
        spec = torch.fft.rfftn(u) * _low_pass(case, torch.complex64).to(torch.complex128) * inv
        w = torch.fft.irfftn(spec, s=dims)
        loss = 0.5 * (w * w).sum()
        loss.backward()
        return [loss.detach(), w.detach(), u.grad]
    x = _field(case, seed).double()
    if case["op"] == "roundtrip":
        return x
    half = len(dims) - 1
    spec = torch.fft.rfftn(x, dim=_logical_axes(case))  # the last logical axis is the half axis
    ks, k2 = _wavenumbers(case, spec.shape, half)
    if case["op"] == "forward":
        return spec
    axes = _logical_axes(case)

    def back(s):  # the full axes first, then the half axis, whose DC and Nyquist bins keep the real parts
        return torch.fft.irfft(torch.fft.ifftn(s, dim=axes[:half]), n=dims[half], dim=axes[half])

    if case["op"] == "gradient":
        return [back(1j * k * spec) for k in ks]
    inv = torch.where(k2 == 0, torch.zeros_like(k2), -1.0 / torch.where(k2 == 0, torch.ones_like(k2), k2))
    return back(spec * inv)
