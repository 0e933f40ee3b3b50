"""Performance cases of the transform path, through the public Python API.

Every case is a dict of plain values with a "kind":

* "fwd", "bwd", "round": one r2c transform, one c2r transform, or both one
  after the other, through ``Plan`` on device arrays, with ``nv`` fields per
  call and optional pruning (``nxc``, ``nyc``, ``nzc``).
* "cheby": the Chebyshev derivative (``ffc`` transform and recurrence).
* "spectrum": a forward transform in the STRIDE1 layout and its shell spectrum.
* "batch": many uneven grids, forward and backward, in one ``Batch`` launch.

``listed`` holds the cases looked at one by one, ``draw`` makes more of the
same ranges, ``prepare`` makes what a caller has in hand (plan, inputs),
``run`` is one pass, ``work`` what a pass cannot do without, and ``exact`` the
result in 64 bits from torch alone.
"""
import math
import random

import torch

import p3dfft_gb300 as pg

DEVICE = "cuda"


def listed():
    return [
        # a single small field: the call's latency (launches, host work) is what a caller waits for
        {"name": "fwd_f64_32", "kind": "fwd", "prec": 64, "nx": 32, "ny": 32, "nz": 32},
        # a small single-precision field with odd and uneven sides, wavenumber to physical space
        {"name": "bwd_f32_45x36x50", "kind": "bwd", "prec": 32, "nx": 45, "ny": 36, "nz": 50},
        # the small cubic grid of the benchmark: both directions of one time step
        {"name": "round_f64_128", "kind": "round", "prec": 64, "nx": 128, "ny": 128, "nz": 128},
        # the headline grid of the benchmark in double precision, each direction by itself
        {"name": "fwd_f64_1024", "kind": "fwd", "prec": 64, "nx": 1024, "ny": 1024, "nz": 1024},
        {"name": "bwd_f64_1024", "kind": "bwd", "prec": 64, "nx": 1024, "ny": 1024, "nz": 1024},
        # the headline grid in single precision
        {"name": "fwd_f32_1024", "kind": "fwd", "prec": 32, "nx": 1024, "ny": 1024, "nz": 1024},
        # the benchmark's non-cubic grid (mixed radix 2, 3 and 5) in single precision
        {"name": "bwd_f32_768x1024x540", "kind": "bwd", "prec": 32, "nx": 768, "ny": 1024, "nz": 540},
        # odd sides with factors 3, 5 and 7, as a caller picks for a domain's aspect ratio
        {"name": "fwd_f64_441x350x405", "kind": "fwd", "prec": 64, "nx": 441, "ny": 350, "nz": 405},
        # three velocity components, dealiased by the 2/3 rule: 384^3 points, 256^3 modes kept
        {"name": "round_f64_384_pruned_256_nv3", "kind": "round", "prec": 64, "nx": 384, "ny": 384, "nz": 384,
         "nxc": 256, "nyc": 256, "nzc": 256, "nv": 3},
        # a channel-flow wall-normal derivative: Chebyshev points along z
        {"name": "cheby_f64_512x512x257", "kind": "cheby", "prec": 64, "nx": 512, "ny": 512, "nz": 257},
        # z-contiguous output of the STRIDE1 layout and the energy spectrum of a diagnostics step
        {"name": "spectrum_f64_256", "kind": "spectrum", "prec": 64, "nx": 256, "ny": 256, "nz": 256},
        # many uneven grids at once (adaptive blocks, serving): one launch for all
        {"name": "batch_f32_24", "kind": "batch", "prec": 32, "grids": 24, "grid_seed": 4},
    ]


def _smooth(limit, b, c, d):
    s = set()
    for i in range(11):
        for j in range(b + 1):
            for k in range(c + 1):
                for m in range(d + 1):
                    n = 2 ** i * 3 ** j * 5 ** k * 7 ** m
                    if 12 <= n <= limit:
                        s.add(n)
    return sorted(s)


# lengths that callers pick: powers of two and three times one most of all, then products of 2, 3 and 5, then of 7 too
SIDES = [_smooth(1536, 1, 0, 0), _smooth(1536, 6, 4, 0), _smooth(1536, 6, 4, 2)]


def _side(rng, target, even=False):
    """One of the few admissible lengths nearest to target."""
    family = rng.choice([0, 0, 1, 1, 2])
    near = sorted((n for n in SIDES[family] if not even or n % 2 == 0), key=lambda n: abs(math.log(n / target)))
    return rng.choice(near[:2 if family == 0 else 6])


def _grid(rng, lo, hi, even=False):
    """Three sides of a grid whose point count is log-uniform in [2^lo, 2^hi]."""
    while True:
        u = rng.uniform(lo, hi)
        e = [rng.uniform(-0.8, 0.8) for _ in range(3)]
        m = sum(e) / 3
        n = [_side(rng, min(1536.0, max(12.0, 2 ** (u / 3 + x - m))), even) for x in e]
        if n[0] * n[1] * n[2] <= 2 ** hi:
            return n


def draw(rng):
    kind = rng.choice(["fwd", "bwd", "round", "fwd", "bwd", "pruned", "cheby", "spectrum", "batch"])
    prec = rng.choice([64, 32])
    if kind == "batch":
        return {"kind": "batch", "prec": prec, "grids": rng.randint(4, 32), "grid_seed": rng.randint(10, 10 ** 6)}
    if kind == "pruned":
        nx, ny, nz = _grid(rng, 14, 26, even=True)
        return {"kind": "round", "prec": prec, "nx": nx, "ny": ny, "nz": nz, "nxc": 2 * (nx // 3), "nyc": 2 * (ny // 3),
                "nzc": 2 * (nz // 3), "nv": rng.randint(1, 4)}
    if kind == "cheby":
        nx, ny, nz = _grid(rng, 14, 26)
        return {"kind": "cheby", "prec": prec, "nx": nx, "ny": ny, "nz": min(nz, 512) + 1}
    nx, ny, nz = _grid(rng, 14, 27.5 if kind in ("round", "spectrum") else 29)
    return {"kind": kind, "prec": prec, "nx": nx, "ny": ny, "nz": nz}


# ------------------------------------------------------------------ inputs
def _real_dtype(case):
    return torch.float64 if case["prec"] == 64 else torch.float32


def _complex_dtype(case):
    return torch.complex128 if case["prec"] == 64 else torch.complex64


def _field(nx, ny, nz, gen, dtype):
    """A few large-scale Fourier modes with random amplitudes and phases, and
    broad-band noise below them."""
    modes = 6
    r = random.Random(gen.initial_seed())

    def wave(n, k):
        return torch.arange(n, dtype=torch.float64, device=DEVICE) * (2 * math.pi * k / n)

    cols, rows = [], []
    for _ in range(modes):
        kx, ky, kz = r.randint(0, max(1, nx // 4)), r.randint(0, max(1, ny // 4)), r.randint(0, max(1, nz // 4))
        amp, phase = r.uniform(0.2, 1.0), r.uniform(0, 2 * math.pi)
        yz = (wave(nz, kz)[:, None] + wave(ny, ky)[None, :] + phase).reshape(-1)
        cols += [amp * torch.cos(yz), -amp * torch.sin(yz)]
        rows += [torch.cos(wave(nx, kx)), torch.sin(wave(nx, kx))]
    x = torch.rand((nz * ny, nx), dtype=dtype, device=DEVICE, generator=gen).sub_(0.5).mul_(0.2)
    x.addmm_(torch.stack(cols, 1).to(dtype), torch.stack(rows, 0).to(dtype))
    return x.reshape(nz, ny, nx)


def _spectrum_field(nx, ny, nz, nxc, nyc, nzc, gen, dtype):
    """Random modes under a decaying envelope, as a turbulent field's."""
    shape = (nzc, nyc, nxc // 2 + 1)

    def freq(n):
        k = torch.arange(n, device=DEVICE, dtype=dtype)
        return torch.minimum(k, n - k)

    c = torch.rand(shape + (2,), dtype=dtype, device=DEVICE, generator=gen).sub_(0.5)
    ez = 1 / (1 + freq(nzc) / 8)
    ey = 1 / (1 + freq(nyc) / 8)
    ex = 1 / (1 + torch.arange(shape[2], device=DEVICE, dtype=dtype) / 8)
    c.mul_((ez[:, None] * ey[None, :])[:, :, None, None]).mul_(ex[None, None, :, None])
    return torch.view_as_complex(c)


def _batch_grids(case):
    r = random.Random(case["grid_seed"])
    sides = [48, 64, 96, 120, 128, 160, 192, 256]
    jobs = []
    for i in range(case["grids"]):
        jobs.append((r.choice(sides), r.choice(sides), r.choice(sides), "fwd" if i % 2 == 0 else "bwd"))
    return jobs


def _pruned(case):
    return case.get("nxc", case["nx"]), case.get("nyc", case["ny"]), case.get("nzc", case["nz"])


def _inputs(case, seed):
    gen = torch.Generator(device=DEVICE)
    gen.manual_seed(seed)
    rdt = _real_dtype(case)
    if case["kind"] == "batch":
        out = []
        for nx, ny, nz, kind in _batch_grids(case):
            if kind == "fwd":
                out.append(torch.rand((nz, ny, nx), dtype=rdt, device=DEVICE, generator=gen).mul_(2).sub_(1))
            else:
                out.append(_spectrum_field(nx, ny, nz, nx, ny, nz, gen, rdt))
        return out
    nx, ny, nz, nv = case["nx"], case["ny"], case["nz"], case.get("nv", 1)
    if case["kind"] in ("bwd", "round"):
        c = [_spectrum_field(nx, ny, nz, *_pruned(case), gen, rdt) for _ in range(nv)]
        return c[0] if nv == 1 else torch.stack(c)
    x = [_field(nx, ny, nz, gen, rdt) for _ in range(nv)]
    return x[0] if nv == 1 else torch.stack(x)


# ------------------------------------------------------------------ a pass
LZ = 2.0


def prepare(case, seed):
    prec = pg.F64 if case["prec"] == 64 else pg.F32
    data = _inputs(case, seed)
    if case["kind"] == "batch":
        jobs = []
        for (nx, ny, nz, kind), x in zip(_batch_grids(case), data):
            plan = pg.Plan(nx, ny, nz, precision=prec)
            if kind == "fwd":
                out = torch.empty(plan.complex_shape, dtype=_complex_dtype(case), device=DEVICE)
            else:
                out = torch.empty(plan.real_shape, dtype=_real_dtype(case), device=DEVICE)
            jobs.append({"plan": plan, "kind": pg.JOB_FORWARD if kind == "fwd" else pg.JOB_BACKWARD, "in": x, "out": out})
        batch = pg.Batch(prec)
        batch.set_jobs(jobs)
        return {"case": case, "batch": batch, "jobs": jobs, "outs": [j["out"] for j in jobs]}
    layout = pg.LAYOUT_STRIDE1 if case["kind"] == "spectrum" else pg.LAYOUT_XYZ
    plan = pg.Plan(case["nx"], case["ny"], case["nz"], *_pruned(case), precision=prec, layout=layout)
    return {"case": case, "plan": plan, "x": data}


def run(state):
    case = state["case"]
    kind, nv = case["kind"], case.get("nv", 1)
    if kind == "batch":
        state["batch"].launch()
        return state["outs"]
    plan, x = state["plan"], state["x"]
    if kind == "fwd":
        return plan.ftran_r2c(x, nv=nv)
    if kind == "bwd":
        return plan.btran_c2r(x, nv=nv)
    if kind == "round":  # modes to points (where a solver forms its products) and back
        r = plan.btran_c2r(x, nv=nv)
        return r, plan.ftran_r2c(r, nv=nv)
    if kind == "cheby":
        return plan.cheby(x, LZ)
    b = plan.ftran_r2c(x)
    return b, plan.spectrum(b, scale=1.0 / (case["nx"] * case["ny"] * case["nz"]))


# ------------------------------------------------------------------ work
def _one_work(nx, ny, nz, nxc, nyc, nzc, prec):
    real = nx * ny * nz * (prec // 8)
    cplx = (nxc // 2 + 1) * nyc * nzc * (prec // 4)
    flops = 2.5 * nx * ny * nz * math.log2(nx * ny * nz)
    return real + cplx, flops


def work(case):
    if case["kind"] == "batch":
        w = [_one_work(nx, ny, nz, nx, ny, nz, case["prec"]) for nx, ny, nz, _ in _batch_grids(case)]
        return {"bytes": sum(b for b, _ in w), "flops": sum(f for _, f in w)}
    times = (2 if case["kind"] == "round" else 1) * case.get("nv", 1)
    b, f = _one_work(case["nx"], case["ny"], case["nz"], *_pruned(case), case["prec"])
    return {"bytes": times * b, "flops": times * f}


# ------------------------------------------------------------------ 64 bits
def _keep(n, nc):
    """Indices of the nc modes kept of n: the low (nc + 1) // 2 and the top rest."""
    h = (nc + 1) // 2
    return torch.tensor(list(range(h)) + list(range(n - (nc - h), n)), device=DEVICE)


def _forward64(x, nx, ny, nz, nxc, nyc, nzc, dct=False):
    b = torch.fft.rfft(x.double(), dim=2)[:, :, : nxc // 2 + 1].contiguous()
    b = torch.fft.fft(b, dim=1)
    if nyc != ny:
        b = b[:, _keep(ny, nyc)]
    if dct:
        b = torch.fft.fft(torch.cat([b, b[1:-1].flip(0)], 0), dim=0)[:nz]
    else:
        b = torch.fft.fft(b, dim=0)
    return b if nzc == nz else b[_keep(nz, nzc)]


def _backward64(c, nx, ny, nz, nxc, nyc, nzc):
    c = c.to(torch.complex128)
    if nzc != nz:
        full = torch.zeros((nz,) + c.shape[1:], dtype=c.dtype, device=DEVICE)
        full[_keep(nz, nzc)] = c
        c = full
    c = torch.fft.ifft(c, dim=0, norm="forward")
    if nyc != ny:
        full = torch.zeros((nz, ny, c.shape[2]), dtype=c.dtype, device=DEVICE)
        full[:, _keep(ny, nyc)] = c
        c = full
    c = torch.fft.ifft(c, dim=1, norm="forward")
    if c.shape[2] < nx // 2 + 1:
        full = torch.zeros((nz, ny, nx // 2 + 1), dtype=c.dtype, device=DEVICE)
        full[:, :, : c.shape[2]] = c
        c = full
    # a real line ignores the imaginary parts of its mean and Nyquist modes
    c[:, :, 0].imag.zero_()
    if nx % 2 == 0:
        c[:, :, nx // 2].imag.zero_()
    return torch.fft.irfft(c, n=nx, dim=2, norm="forward")


def _cheby64(b, nx, ny, nz):
    out = b * (1.0 / (float(nx * ny) * float(nz - 1)))
    lfac = 4.0 / LZ
    old = out[nz - 2].clone()
    out[nz - 2] = lfac * float(nz - 1) * out[nz - 1] * 0.5
    out[nz - 1] = 0
    for k in range(nz - 3, -1, -1):
        new = out[k].clone()
        out[k] = lfac * float(k + 1) * old + out[k + 2]
        old = new
    out[0] *= 0.5
    return out


def _shells64(b, nx, ny, nz):
    """Shell sums of k^2 |b|^2 of b [z][y][x]."""
    def fold(i, n):
        return torch.where(i + 1 > n // 2, n - i, i).double()

    k2 = (fold(torch.arange(nz, device=DEVICE), nz)[:, None, None] ** 2
          + fold(torch.arange(ny, device=DEVICE), ny)[None, :, None] ** 2
          + torch.arange(b.shape[2], device=DEVICE).double()[None, None, :] ** 2)
    kmax = int(math.sqrt(float(nx) ** 2 + float(ny) ** 2 + float(nz) ** 2) * 0.5 + 0.5)
    ik = (torch.sqrt(k2) + 0.5).long()
    w = k2 * (b.real ** 2 + b.imag ** 2)
    keep = ik <= kmax
    return torch.bincount(ik[keep], weights=w[keep], minlength=kmax + 1)[: kmax + 1]


def exact(case, seed):
    data = _inputs(case, seed)
    if case["kind"] == "batch":
        out = []
        for (nx, ny, nz, kind), x in zip(_batch_grids(case), data):
            fn = _forward64 if kind == "fwd" else _backward64
            out.append(fn(x, nx, ny, nz, nx, ny, nz))
        return out
    nx, ny, nz, nv = case["nx"], case["ny"], case["nz"], case.get("nv", 1)
    dims = (nx, ny, nz, *_pruned(case))
    if case["kind"] == "cheby":
        return _cheby64(_forward64(data, *dims, dct=True), nx, ny, nz)
    if case["kind"] == "spectrum":
        b = _forward64(data, *dims)
        return b.permute(2, 1, 0).contiguous(), _shells64(b / (nx * ny * nz), nx, ny, nz)
    fields = [data] if nv == 1 else list(data)

    def many(fn, xs):
        r = [fn(x, *dims) for x in xs]
        return r[0] if nv == 1 else torch.stack(r)

    if case["kind"] == "fwd":
        return many(_forward64, fields)
    r = many(_backward64, fields)
    if case["kind"] == "bwd":
        return r
    return r, many(_forward64, [r] if nv == 1 else list(r))
