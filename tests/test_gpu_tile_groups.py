"""The strided passes' thread groups and buffer ring against the oracle.

Sizes at which the kernel forms differ: one tile per SM and many, lengths
whose stages fill every thread and lengths that leave some idle, one group and
eight, more tiles per group than buffers (the ring wraps) with tiles so short
that groups drift apart, partial last tiles, and rows stored by TMA and by
threads (STRIDE1, pruned, odd binary32 rows).

Tolerances: the transform's bounds, normalised L-inf 1e-12 (binary64) and
relative L2 1e-6 (binary32).
"""
import numpy as np
import pytest

from oracle import p3dfft_oracle as orc

pytestmark = pytest.mark.gpu

SHAPES = [
    (30, 1024, 12),          # two groups of whole-warp stages, one tile column block
    (130, 512, 40),
    (66, 256, 300),          # groups with several tiles each
    (6, 64, 4096),           # thousands of tiny tiles along y: the ring wraps many times
    (10, 8, 2048),
    (34, 375, 48),           # 3 and 5 factors: idle threads in every stage
    (48, 540, 20),
    (28, 2048, 10),
    (16, 32, 32),            # fewer tiles than SMs
    (20, 36, 45, 14, 20, 30),  # pruned: gaps on load and store
]


@pytest.mark.parametrize("stride1", [False, True])
@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_groups_match_oracle(shape, precision, stride1):
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
    for got, want in ((b.cpu().numpy(), want_b), (r.cpu().numpy(), want_r)):
        if f64:
            assert orc.normalised_linf(got, want) <= 1e-12
        else:
            assert orc.relative_l2(got, want) <= 1e-6
    plan.close()
