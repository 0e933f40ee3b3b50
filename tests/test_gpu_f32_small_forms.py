"""Binary32 passes with half the points per thread and several tiles per group,
and X c2r passes whose short lines arrive by cp.async.

Lengths whose largest radix fills 16 points on each axis, with enough tiles
that the ring of buffers wraps; the narrowest and the long rows of the strided
tiles; lines of a few modes, pruned ones and an odd number of them.

Tolerances: the transform's bounds, normalised L-inf 1e-12 (binary64) and
relative L2 1e-6 (binary32).
"""
import numpy as np
import pytest

from oracle import p3dfft_oracle as orc

pytestmark = pytest.mark.gpu


def _check(shape, precision, stride1=False):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import p3dfft_gb300 as pg
    f64 = precision == "f64"
    nx, ny, nz = shape[:3]
    pruned = shape[3:] or (nx, ny, nz)
    rng = np.random.default_rng(nx + 7 * ny + 31 * nz)
    a = rng.uniform(-1, 1, size=(nz, ny, nx))
    plan = pg.Plan(nx, ny, nz, *pruned, precision=pg.F64 if f64 else pg.F32,
                   layout=pg.LAYOUT_STRIDE1 if stride1 else pg.LAYOUT_XYZ)
    ref = orc.OraclePlan(nx, ny, nz, *pruned, stride1=stride1)
    x = torch.from_numpy(a).to("cuda", torch.float64 if f64 else torch.float32)
    b = plan.ftran_r2c(x)
    want_b = ref.ftran_r2c(x.double().cpu().numpy())
    c = rng.uniform(-1, 1, size=want_b.shape) + 1j * rng.uniform(-1, 1, size=want_b.shape)
    ct = torch.from_numpy(c).to("cuda", torch.complex128 if f64 else torch.complex64)
    r = plan.btran_c2r(ct)
    want_r = ref.btran_c2r(ct.to(torch.complex128).cpu().numpy())
    plan.check()
    plan.close()
    for got, want in ((b.cpu().numpy(), want_b), (r.cpu().numpy(), want_r)):
        if f64:
            assert orc.normalised_linf(got, want) <= 1e-12
        else:
            assert orc.relative_l2(got, want) <= 1e-6


@pytest.mark.parametrize("stride1", [False, True])
@pytest.mark.parametrize("shape", [
    (30, 80, 640), (30, 640, 80), (66, 96, 512), (14, 240, 700), (14, 700, 240), (10, 1536, 96), (10, 96, 1536),
    (6, 3072, 40), (6, 1500, 64), (48, 98, 441), (4, 4096, 48), (4, 48, 2048),
], ids=lambda s: "x".join(map(str, s)))
def test_strided_small_forms(shape, stride1):
    _check(shape, "f32", stride1)


@pytest.mark.parametrize("shape", [(120, 160, 128), (240, 128, 96), (640, 100, 90), (1536, 64, 60), (96, 211, 131)],
                         ids=lambda s: "x".join(map(str, s)))
def test_x_small_forms(shape):
    _check(shape, "f32")


@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("shape", [(16, 33, 31), (24, 65, 40), (48, 64, 60), (60, 40, 41), (64, 63, 65), (64, 64, 64),
                                   (62, 17, 19), (61, 17, 19), (126, 20, 21), (128, 20, 21),
                                   (96, 30, 31, 30, 30, 31), (192, 20, 22, 90, 14, 16)],
                         ids=lambda s: "x".join(map(str, s)))
def test_short_c2r_lines(shape, precision):
    _check(shape, precision)
