"""Passes may start while the kernel before them in the stream still runs; they
wait for it before they touch shared data.  Chains of calls that read what the
call before wrote, in place and through torch kernels in between, eager and
captured in a CUDA graph, must equal the same calls with a synchronisation
after each, bit for bit."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("shape", [(32, 32, 32), (45, 36, 50), (128, 96, 64)], ids=lambda s: "x".join(map(str, s)))
def test_chained_calls(shape, precision):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import p3dfft_gb300 as pg
    f64 = precision == "f64"
    nx, ny, nz = shape
    rdt, cdt = (torch.float64, torch.complex128) if f64 else (torch.float32, torch.complex64)
    plan = pg.Plan(nx, ny, nz, precision=pg.F64 if f64 else pg.F32)
    other = pg.Plan(nx, ny, nz, precision=pg.F64 if f64 else pg.F32)
    if f64:
        other.set_range(pg.RANGE_AUTO)  # a reduction kernel before the passes
    gen = torch.Generator(device="cuda")
    gen.manual_seed(1)
    x0 = torch.rand((nz, ny, nx), dtype=rdt, device="cuda", generator=gen)
    x, b, r = torch.empty_like(x0), torch.empty(plan.complex_shape, dtype=cdt, device="cuda"), torch.empty_like(x0)

    def chain(wait):
        x.copy_(x0)
        for i in range(6):
            p = (plan, other)[i % 2]
            p.ftran_r2c(x, out=b)
            wait()
            b.mul_(0.5)
            wait()
            p.btran_c2r(b, out=r)
            wait()
            p.ftran_r2c(r, out=b)
            wait()
            plan.btran_c2r(b, out=x)
            wait()
            x.mul_(1.0 / (0.5 * x.numel() ** 2))
            wait()
        return x.clone()

    want = chain(torch.cuda.synchronize)
    assert torch.equal(chain(lambda: None), want)
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        got = chain(lambda: None)
    s.synchronize()
    assert torch.equal(got, want)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = chain(lambda: None)
    for _ in range(2):
        out.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, want)
    plan.check()
    other.check()
    plan.close()
    other.close()
