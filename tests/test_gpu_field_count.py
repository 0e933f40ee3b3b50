"""Calls of many fields choose their stage plans for all fields together.

A small grid's single field runs the narrow stage plan (short chains), many of
them at once the wide one, so a field's rounding may depend on how many fields
the call has: the results agree with the oracle's, and with those of single
calls, within the transform's bounds rather than bit for bit.  Grids on both
sides of the change, with every field compared.

Tolerances: normalised L-inf 1e-12 (binary64) and relative L2 1e-6 (binary32).
"""
import numpy as np
import pytest

from oracle import p3dfft_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("shape,nv", [((32, 32, 32), 32), ((80, 80, 80), 16), ((96, 64, 80), 8), ((24, 40, 18), 64)],
                         ids=["32x32x32x32", "80x80x80x16", "96x64x80x8", "24x40x18x64"])
def test_many_fields_match_single_fields_and_oracle(shape, nv, precision):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import p3dfft_gb300 as pg
    f64 = precision == "f64"
    nx, ny, nz = shape
    a = np.random.default_rng(nx + nv).uniform(-1, 1, size=(nv, nz, ny, nx))
    x = torch.from_numpy(a).to("cuda", torch.float64 if f64 else torch.float32)
    plan = pg.Plan(nx, ny, nz, precision=pg.F64 if f64 else pg.F32)
    ref = orc.OraclePlan(nx, ny, nz)
    b = plan.ftran_r2c(x, nv=nv)
    r = plan.btran_c2r(b, nv=nv)
    for i in range(nv):
        bi = plan.ftran_r2c(x[i].contiguous())
        ri = plan.btran_c2r(b[i].contiguous())
        want_b = ref.ftran_r2c(x[i].double().cpu().numpy())
        want_r = ref.btran_c2r(b[i].to(torch.complex128).cpu().numpy())
        for got, want in ((b[i], want_b), (bi, want_b), (r[i], want_r), (ri, want_r)):
            if f64:
                assert orc.normalised_linf(got.cpu().numpy(), want) <= 1e-12
            else:
                assert orc.relative_l2(got.cpu().numpy(), want) <= 1e-6
    plan.check()
    plan.close()
