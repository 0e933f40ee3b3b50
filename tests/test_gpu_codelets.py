"""Every codelet radix, alone and combined, on every axis against the oracle.

Each length runs once as the X, once as the Y and once as the Z axis (forward
and backward, so the c2r first stage sees every first radix too).

Tolerances: the transform's bounds, normalised L-inf 1e-12 (binary64) and
relative L2 1e-6 (binary32).
"""
import numpy as np
import pytest

from oracle import p3dfft_oracle as orc

pytestmark = pytest.mark.gpu

LENGTHS = [3, 5, 6, 7, 9, 10, 12, 14, 15, 18, 21, 24, 27, 28, 30, 35, 36, 40, 45, 48, 49, 60, 63, 72, 75, 77, 81, 90,
           98, 100, 105, 120, 125, 135, 147, 150, 160, 175, 189, 196, 210, 225, 240, 245, 270, 315, 343, 350, 405, 441,
           486, 540, 630, 675, 720, 735, 810, 945, 960, 1050, 1225, 1260, 1323, 1500]


@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("n", LENGTHS)
def test_length_on_each_axis(n, precision):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import p3dfft_gb300 as pg
    f64 = precision == "f64"
    for nx, ny, nz in ((n, 3, 6), (10, n, 3), (10, 3, n)):
        rng = np.random.default_rng(n)
        a = rng.uniform(-1, 1, size=(nz, ny, nx))
        plan = pg.Plan(nx, ny, nz, precision=pg.F64 if f64 else pg.F32)
        ref = orc.OraclePlan(nx, ny, nz)
        x = torch.from_numpy(a).to("cuda", torch.float64 if f64 else torch.float32)
        b = plan.ftran_r2c(x).cpu().numpy()
        want_b = ref.ftran_r2c(x.double().cpu().numpy())
        c = rng.uniform(-1, 1, size=want_b.shape) + 1j * rng.uniform(-1, 1, size=want_b.shape)
        ct = torch.from_numpy(c).to("cuda", torch.complex128 if f64 else torch.complex64)
        r = plan.btran_c2r(ct).cpu().numpy()
        want_r = ref.btran_c2r(ct.to(torch.complex128).cpu().numpy())
        plan.check()
        plan.close()
        for got, want in ((b, want_b), (r, want_r)):
            if f64:
                assert orc.normalised_linf(got, want) <= 1e-12
            else:
                assert orc.relative_l2(got, want) <= 1e-6
