"""Launches that start under their predecessor's tail (programmatic launches): calls queued back to back
with other inputs through the same buffers, replayed from a captured graph, and moved between streams.

Each result is compared with torch's transform in FP64; an FFT of n points has a root mean square error
of a few eps sqrt(log2 n), so 2e-6 (f32) and 4e-15 (f64) leave a factor of five, and the Poisson
solve two transforms' worth.
"""
import pytest

pytestmark = pytest.mark.gpu
TOL = {"float32": 2e-6, "float64": 8e-15}

# fused 4D (both plane shapes), fused 3D with and without clusters, staged passes of line kernels alone,
# line kernels beside chirp-z passes (which are launched without the attribute), 2D
CASES = [((32, 64, 128, 64), "native_xzwy", "float32"), ((64, 64, 64, 64), "native_xzwy", "float32"),
         ((32, 32, 64, 64), "slab", "float32"), ((64, 64, 64), None, "float32"), ((64, 256, 256), None, "float32"),
         ((128, 128, 128), None, "float32"), ((96, 60, 50), None, "float32"), ((48, 40, 63), None, "float64"),
         ((30, 17, 64), None, "float32"), ((512, 300), None, "float32"), ((20, 24, 18, 30), "native_xzwy", "float64")]


@pytest.fixture(scope="module")
def F(torch_cuda):
    from fftm_b200 import build
    build.build()
    import fftm_b200
    return fftm_b200


def _types(torch, dtype):
    return (torch.float32, torch.complex64) if dtype == "float32" else (torch.float64, torch.complex128)


def _object(F, torch, dims, layout, dtype):
    real, comp = _types(torch, dtype)
    f = F.ffts(dtype, strategy_4d=layout or "slab").init(*dims)
    if f.work_size:
        f.set_work_area(torch.empty(f.work_size // (8 if dtype == "float32" else 16) + 1, dtype=comp, device="cuda"))
    return f


def _spectrum(torch, x, layout):
    s = torch.fft.rfftn(x.double())
    return s.permute(1, 2, 3, 0) if layout == "native_xzwy" else s


def _poisson(torch, x):
    k2 = 0
    for a, n in enumerate(x.shape):
        k = torch.fft.fftfreq(n, 1.0 / n, dtype=torch.float64, device=x.device)
        if a == x.dim() - 1:
            k = k[:n // 2 + 1].abs()
        k2 = k2 + (k ** 2).reshape([-1 if b == a else 1 for b in range(x.dim())])
    s = torch.fft.rfftn(x.double())
    s = torch.where(k2 == 0, torch.zeros_like(s), -s / torch.where(k2 == 0, torch.ones_like(k2), k2))
    return torch.fft.irfftn(s, s=x.shape)


def _rel(a, b):
    return float((a - b).norm() / b.norm())


def _check(torch, x, spec, back, sol, layout, dtype):
    assert _rel(spec, _spectrum(torch, x, layout)) <= TOL[dtype]
    assert _rel(back.double(), x.double()) <= 2 * TOL[dtype]
    assert _rel(sol.double(), _poisson(torch, x)) <= 2 * TOL[dtype]


@pytest.mark.parametrize("dims,layout,dtype", CASES)
def test_queued_calls_with_other_inputs(F, torch_cuda, dims, layout, dtype):
    """Eight rounds of calls without a synchronisation, each on an input of its own, all through one work
    area and one spectrum: a kernel that reads or writes before its predecessor is through shows
    in a round's results."""
    torch = torch_cuda
    real, comp = _types(torch, dtype)
    f = _object(F, torch, dims, layout, dtype)
    gen = torch.Generator(device="cuda").manual_seed(5)
    shared = torch.empty(f.spectrum_shape(), dtype=comp, device="cuda")
    rounds = [dict(x=torch.randn(dims, dtype=real, device="cuda", generator=gen) * 10.0 ** (i % 3),
                   spec=torch.empty_like(shared), back=torch.empty(dims, dtype=real, device="cuda"),
                   sol=torch.empty(dims, dtype=real, device="cuda")) for i in range(8)]
    f.poisson(rounds[0]["x"], rounds[0]["sol"])  # first uses are over before the queue starts
    torch.cuda.synchronize()
    for r in rounds:
        f.forward(r["x"], r["spec"])
        f.forward(r["x"], shared)
        f.backward(shared, r["back"], normalized=True)
        f.poisson(r["x"], r["sol"])
    torch.cuda.synchronize()
    for r in rounds:
        _check(torch, r["x"], r["spec"], r["back"], r["sol"], layout, dtype)


@pytest.mark.parametrize("dims,layout,dtype", CASES)
def test_captured_calls(F, torch_cuda, dims, layout, dtype):
    """The same calls captured into a graph (the launches become programmatic edges), replayed back to
    back with other inputs."""
    torch = torch_cuda
    real, comp = _types(torch, dtype)
    f = _object(F, torch, dims, layout, dtype)
    x = torch.zeros(dims, dtype=real, device="cuda")
    spec, shared = (torch.empty(f.spectrum_shape(), dtype=comp, device="cuda") for _ in range(2))
    back, sol = torch.empty_like(x), torch.empty_like(x)

    def calls():
        f.forward(x, spec)
        f.forward(x, shared)
        f.backward(shared, back, normalized=True)
        f.poisson(x, sol)

    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        calls()
    side.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        calls()
    kept = []
    for i in range(4):
        x.copy_(torch.randn(dims, dtype=real, device="cuda"))
        graph.replay()
        graph.replay()  # again, the same input: a replay right behind another
        kept.append([t.clone() for t in (x, spec, back, sol)])
    torch.cuda.synchronize()
    for xs in kept:
        _check(torch, *xs, layout, dtype)


@pytest.mark.parametrize("dims,layout,dtype", [CASES[0], CASES[3], CASES[6], CASES[8]])
def test_captured_among_other_work(F, torch_cuda, dims, layout, dtype):
    """Captured behind and between a kernel, a copy and a memset of torch's, and behind a join of two
    streams (a launch with two predecessors): the edges to those are full ones."""
    torch = torch_cuda
    real, comp = _types(torch, dtype)
    f = _object(F, torch, dims, layout, dtype)
    x = torch.zeros(dims, dtype=real, device="cuda")
    x2, back, sol = (torch.empty_like(x) for _ in range(3))
    spec, kept = (torch.empty(f.spectrum_shape(), dtype=comp, device="cuda") for _ in range(2))
    side = torch.cuda.Stream()

    def calls():
        main = torch.cuda.current_stream()
        side.wait_stream(main)
        with torch.cuda.stream(side):
            sol.mul_(0)              # a kernel beside ...
        torch.mul(x, 2, out=x2)      # ... a kernel
        main.wait_stream(side)
        f.forward(x2, spec)          # two predecessors
        kept.copy_(spec)             # a copy
        f.backward(spec, back, normalized=True)
        spec.zero_()                 # a memset
        f.poisson(x2, sol)
        back.mul_(0.5)

    warm = torch.cuda.Stream()
    warm.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(warm):
        calls()
    warm.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        calls()
    results = []
    for _ in range(4):
        x.copy_(torch.randn(dims, dtype=real, device="cuda"))
        graph.replay()
        graph.replay()
        results.append([t.clone() for t in (x, kept, back, sol)])
    torch.cuda.synchronize()
    for xs, spectrum, b, u in results:
        _check(torch, xs, spectrum / 2, b, u / 2, layout, dtype)


def test_calls_follow_the_stream(F, torch_cuda):
    """One object and one plan used on two streams in turn: each call runs on the stream it is given or
    finds current, also when it is the stream of two calls ago, and when the handle was last used on
    another one."""
    torch = torch_cuda
    f = _object(F, torch, (60, 48, 50), None, "float32")
    plan = F.Plan(F.C2CF, [1000], batch=64)
    x = torch.randn(60, 48, 50, device="cuda")
    z = torch.randn(64, 1000, dtype=torch.complex64, device="cuda")
    s1, s2 = torch.cuda.Stream(), torch.cuda.Stream()
    spec = torch.empty(f.spectrum_shape(), dtype=torch.complex64, device="cuda")
    y = torch.empty_like(z)
    f.forward(x, spec)
    plan.exec(z, y)
    ref, zref = torch.fft.rfftn(x.double()), torch.fft.fft(z.to(torch.complex128))
    torch.cuda.synchronize()

    def on(stream, how):
        """Runs both calls on `stream` while the other one is busy for about 150 ms."""
        other = s2 if stream is s1 else s1
        a, b = torch.zeros_like(spec), torch.zeros_like(y)
        torch.cuda.synchronize()
        with torch.cuda.stream(other):
            torch.cuda._sleep(300_000_000)
        if how == "argument":
            f.forward(x, a, stream=stream)
            plan.exec(z, b, stream=stream)
        else:
            with torch.cuda.stream(stream):
                f.forward(x, a)
                plan.exec(z, b)
        stream.synchronize()
        assert not other.query()  # it did not wait for the other stream
        assert _rel(a, ref) <= TOL["float32"] and _rel(b, zref) <= TOL["float32"]

    for stream, how in ((s1, "argument"), (s2, "argument"), (s1, "current"), (s1, "argument"), (s2, "current"),
                        (s2, "current"), (s1, "argument")):
        on(stream, how)
    a = torch.zeros_like(spec)
    f.forward(x, a)  # back on the default stream
    assert _rel(a, ref) <= TOL["float32"]
