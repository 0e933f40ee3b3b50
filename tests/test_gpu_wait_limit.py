"""How long a pass whose tile copies never arrive may take.

Every wait of a pass has a limit of one second: a group's wait for its load to
be issued, its wait for the load to land, and, once, the CTA's wait for the
loads that no group waits for any more, however many buffers it has.  The test
hook makes the strided passes' barriers expect more bytes than their copies
deliver (nothing faults); two of the three passes of a forward transform have
them, so a call ends within about six seconds.
"""
import time

import numpy as np
import pytest

from oracle import p3dfft_oracle as orc

pytestmark = pytest.mark.gpu


def test_blocked_passes_end_within_their_limits():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import p3dfft_gb300 as pg
    nx, ny, nz = 256, 64, 256  # ten buffers per CTA, all of them loaded at the start
    a = np.random.default_rng(8).uniform(-1, 1, size=(nz, ny, nx))
    x = torch.from_numpy(a).cuda()
    plan = pg.Plan(nx, ny, nz)
    plan.block_tiles(True)
    torch.cuda.synchronize()
    t = time.perf_counter()
    plan.ftran_r2c(x)
    with pytest.raises(pg.P3DFFTError, match="timed out"):
        plan.check()
    assert time.perf_counter() - t < 10
    plan.block_tiles(False)
    b = plan.ftran_r2c(x)
    plan.check()
    plan.close()
    assert orc.normalised_linf(b.cpu().numpy(), orc.OraclePlan(nx, ny, nz).ftran_r2c(a, "fft")) <= 1e-12
