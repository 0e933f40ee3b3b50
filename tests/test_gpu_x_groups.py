"""The X passes' thread groups, padded tiles and bulk copies against the oracle.

Line lengths whose shared-memory padding differs (first radix above, at and
below the spacing of a later stage's points), odd line counts (the last pair
of a field has one line), pruned x modes (the c2r tile's missing modes are
zeroed after its copy), lines whose length forbids bulk copies, one line, and
inputs with zeros and values far below the rest (the long binary64 conversion).

Tolerances: the transform's bounds, normalised L-inf 1e-12 (binary64) and
relative L2 1e-6 (binary32).
"""
import numpy as np
import pytest

from oracle import p3dfft_oracle as orc

pytestmark = pytest.mark.gpu

SHAPES = [
    (1024, 3, 5), (512, 7, 9), (256, 5, 31), (128, 33, 31), (384, 5, 7), (96, 65, 3), (2048, 3, 3), (4096, 3, 1),
    (375, 5, 7), (90, 7, 11), (45, 9, 5), (64, 1, 1), (2, 3, 5), (256, 11, 13, 170, 11, 13), (384, 9, 8, 256, 6, 6),
]


@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_x_groups_match_oracle(shape, precision):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import p3dfft_gb300 as pg
    f64 = precision == "f64"
    nx, ny, nz = shape[:3]
    pruned = shape[3:] or (nx, ny, nz)
    rng = np.random.default_rng(nx + 7 * ny + 31 * nz)
    a = rng.uniform(-1, 1, size=(nz, ny, nx))
    a[rng.uniform(size=a.shape) < 0.1] = 0.0
    a[rng.uniform(size=a.shape) < 0.1] *= 2.0 ** -80
    plan = pg.Plan(nx, ny, nz, *pruned, precision=pg.F64 if f64 else pg.F32)
    ref = orc.OraclePlan(nx, ny, nz, *pruned)
    x = torch.from_numpy(a).to("cuda", torch.float64 if f64 else torch.float32)
    b = plan.ftran_r2c(x)
    want_b = ref.ftran_r2c(x.double().cpu().numpy())
    c = rng.uniform(-1, 1, size=want_b.shape) + 1j * rng.uniform(-1, 1, size=want_b.shape)
    ct = torch.from_numpy(c).to("cuda", torch.complex128 if f64 else torch.complex64)
    r = plan.btran_c2r(ct)
    want_r = ref.btran_c2r(ct.to(torch.complex128).cpu().numpy())
    plan.check()
    for got, want in ((b.cpu().numpy(), want_b), (r.cpu().numpy(), want_r)):
        if f64:
            assert orc.normalised_linf(got, want) <= 1e-12
        else:
            assert orc.relative_l2(got, want) <= 1e-6
    plan.close()


@pytest.mark.parametrize("precision", ["f64", "f32"])
def test_x_long_conversion_values(precision):
    """Lines of zeros, subnormals and values below the field's by 2^-90, alone
    in their line, next to ordinary lines."""
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import p3dfft_gb300 as pg
    f64 = precision == "f64"
    rng = np.random.default_rng(5)
    a = rng.uniform(-1, 1, size=(6, 7, 64))
    a[0] = 0.0
    a[1, 2] *= 2.0 ** -90
    a[2, :, ::2] = 5e-324
    plan = pg.Plan(64, 7, 6, precision=pg.F64 if f64 else pg.F32)
    x = torch.from_numpy(a).to("cuda", torch.float64 if f64 else torch.float32)
    got = plan.ftran_r2c_1d(x).cpu().numpy()
    want = np.fft.rfft(x.double().cpu().numpy(), axis=2)
    plan.check()
    plan.close()
    if f64:
        assert orc.normalised_linf(got, want) <= 1e-12
    else:
        assert orc.relative_l2(got, want) <= 1e-6


@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("shape", [(64, 31, 41), (128, 150, 67, 86, 100, 44)], ids=lambda s: "x".join(map(str, s)))
def test_many_fields_with_partial_last_tile(shape, precision):
    """nv fields whose line count leaves each field's last tile partial: the
    tiles after it, of the next field, must not be affected."""
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import p3dfft_gb300 as pg
    nx, ny, nz = shape[:3]
    pruned = shape[3:] or (nx, ny, nz)
    f64 = precision == "f64"
    plan = pg.Plan(nx, ny, nz, *pruned, precision=pg.F64 if f64 else pg.F32)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(3)
    x = torch.rand((5, nz, ny, nx), dtype=torch.float64 if f64 else torch.float32, device="cuda", generator=gen)
    b = plan.ftran_r2c(x, nv=5)
    r = plan.btran_c2r(b, nv=5)
    plan.check()
    for i in range(5):
        bi = plan.ftran_r2c(x[i].contiguous())
        ri = plan.btran_c2r(bi)
        assert torch.equal(b[i], bi)
        assert torch.equal(r[i], ri)
    plan.check()
    plan.close()
