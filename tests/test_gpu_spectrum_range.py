"""Shell spectra of small modes, of a wide range of magnitudes and of long rows
against the oracle's restatement of the spectrum sample.

A mode's weight k^2 |B|^2 is formed in double-float, whose low word ends at
binary32's smallest number 2^-149: each of the few products of a mode is off by
at most 2^-150 and its factors by 2^-47 of themselves, so a mode of weight w
adds an error of at most 2^-45 w + 2^-147 (k^2 + 1).  The sums over runs of
modes and over a shell add rounding of binary64 size, under 1e-12 of the shell's
sum with the former.
"""
import numpy as np
import pytest

from oracle import p3dfft_oracle as orc

pytestmark = pytest.mark.gpu

REL = 1e-12


@pytest.fixture(scope="module")
def torch_cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def _modes(shape, precision, seed, amplitude):
    """Random modes [z][y][x] of the given amplitude (a number or an array), as
    the path's format holds them."""
    rng = np.random.default_rng(seed)
    b = (rng.uniform(-1, 1, size=shape) + 1j * rng.uniform(-1, 1, size=shape)) * amplitude
    return b if precision == "f64" else b.astype(np.complex64).astype(np.complex128)


def _decay(nx, ny, nz, last):
    """1 at k = 0 down to 2^-last at the largest |k|."""
    k = [np.minimum(np.arange(m), n - np.arange(m)) for m, n in ((nz, nz), (ny, ny), (nx // 2 + 1, nx))]
    k2 = k[0][:, None, None] ** 2 + k[1][None, :, None] ** 2 + k[2][None, None, :] ** 2
    r = np.sqrt(k2 / k2.max())
    return 2.0 ** (-last * r)


@pytest.mark.parametrize("stride1", [False, True])
@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("k2_weight", [True, False])
@pytest.mark.parametrize("case", ["2^-40", "2^-49", "tail to 2^-64", "zero modes"])
def test_small_modes(torch_cuda, case, k2_weight, precision, stride1):
    import p3dfft_gb300 as pg
    nx, ny, nz = 32, 30, 28
    amp = {"2^-40": 2.0 ** -40, "2^-49": 2.0 ** -49, "tail to 2^-64": _decay(nx, ny, nz, 64),
           "zero modes": np.where(_decay(nx, ny, nz, 1) < 0.7, 0.0, 2.0 ** -45)}[case]
    b = _modes((nz, ny, nx // 2 + 1), precision, 11, amp)
    if stride1:
        b = np.ascontiguousarray(b.transpose(2, 1, 0))
    plan = pg.Plan(nx, ny, nz, precision=pg.F64 if precision == "f64" else pg.F32,
                   layout=pg.LAYOUT_STRIDE1 if stride1 else pg.LAYOUT_XYZ)
    t = torch_cuda.from_numpy(b).to("cuda", torch_cuda.complex128 if precision == "f64" else torch_cuda.complex64)
    got = plan.spectrum(t, flags=pg.SPEC_K2 if k2_weight else 0).cpu().numpy()
    plan.close()
    want = orc.shell_spectrum(b, nx, ny, nz, stride1=stride1, k2_weight=k2_weight)
    ones = np.ones_like(b)
    floor = 2.0 ** -147 * (orc.shell_spectrum(ones, nx, ny, nz, stride1=stride1, k2_weight=False)
                           + (orc.shell_spectrum(ones, nx, ny, nz, stride1=stride1) if k2_weight else 0.0))
    assert np.all(np.abs(got - want) <= REL * want + floor)


@pytest.mark.parametrize("form", ["plan", "batch"])
@pytest.mark.parametrize("amplitude", [2.0 ** -40, 2.0 ** -49])
def test_spectrum_of_a_small_field(torch_cuda, amplitude, form):
    """A white field near the bottom of the binary64 window, through the transform."""
    import p3dfft_gb300 as pg
    n = 32
    a = np.random.default_rng(3).uniform(-1, 1, size=(n, n, n)) * amplitude
    x = torch_cuda.from_numpy(a).cuda()
    plan = pg.Plan(n, n, n, precision=pg.F64)
    b = plan.ftran_r2c(x)
    if form == "plan":
        e = plan.spectrum(b)
    else:
        e = torch_cuda.empty(int(np.sqrt(3.0) * n * 0.5 + 0.5) + 1, dtype=torch_cuda.float64, device="cuda")
        batch = pg.Batch(pg.F64).set_jobs([{"plan": plan, "kind": pg.JOB_SPECTRUM, "in": x, "out": e}])
        batch.launch()
        batch.check()
        batch.close()
    plan.check()
    plan.close()
    want = orc.shell_spectrum(b.cpu().numpy(), n, n, n)
    assert orc.normalised_linf(e.cpu().numpy(), want) <= REL


@pytest.mark.parametrize("stride1", [False, True])
@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("flags", ["0", "K2", "HERMITIAN", "both"])
@pytest.mark.parametrize("grid", [(256, 9, 10), (257, 8, 7), (600, 7, 9), (9, 8, 256), (10, 9, 257), (7, 6, 600), (512, 5, 34),
                                  (34, 512, 6), (2, 40, 30), (2, 3, 2)], ids=lambda s: "x".join(map(str, s)))
def test_long_rows_and_shared_bins(torch_cuda, grid, flags, precision, stride1):
    """Rows of more modes than a warp takes at once, full runs per lane, and rows
    along which the bin hardly changes (all lanes end in it)."""
    import p3dfft_gb300 as pg
    nx, ny, nz = grid
    b = _modes((nz, ny, nx // 2 + 1), precision, 17, 1.0)
    if stride1:
        b = np.ascontiguousarray(b.transpose(2, 1, 0))
    plan = pg.Plan(nx, ny, nz, precision=pg.F64 if precision == "f64" else pg.F32,
                   layout=pg.LAYOUT_STRIDE1 if stride1 else pg.LAYOUT_XYZ)
    t = torch_cuda.from_numpy(b).to("cuda", torch_cuda.complex128 if precision == "f64" else torch_cuda.complex64)
    k2, herm = flags in ("K2", "both"), flags in ("HERMITIAN", "both")
    got = plan.spectrum(t, flags=(pg.SPEC_K2 if k2 else 0) | (pg.SPEC_HERMITIAN if herm else 0)).cpu().numpy()
    plan.close()
    want = orc.shell_spectrum(b, nx, ny, nz, stride1=stride1, k2_weight=k2, hermitian=herm)
    assert np.all(np.abs(got - want) <= REL * want + 2.0 ** -147 * b.size)
