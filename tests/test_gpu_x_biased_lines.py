"""The long binary64 conversion of the X r2c pass under an exponent bias.

A field of 2^-600, far outside the window the pairs can hold, with the bias that
brings it in: every value takes the long conversion and nothing is lost, so each
line x is off by at most 2^-40 sum |x| (far above double-float's own rounding).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [64, 45])
def test_biased_lines(n):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import p3dfft_gb300 as pg
    a = np.ldexp(np.random.default_rng(7).uniform(-1, 1, size=(3, 5, n)), -600)
    plan = pg.Plan(n, 5, 3, precision=pg.F64)
    plan.set_range(pg.RANGE_FIXED, -600)
    got = plan.ftran_r2c_1d(torch.from_numpy(a).cuda()).cpu().numpy()
    plan.check()
    plan.close()
    want = np.fft.rfft(a, axis=2)
    assert np.all(np.abs(got - want).max(axis=2) <= 2.0 ** -40 * np.abs(a).sum(axis=2))
