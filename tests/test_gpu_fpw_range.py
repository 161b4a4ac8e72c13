"""FPW and BLS on trial periods beyond the one-FMA bin's range (2^19 cycles over
the curve): two more FP64 operations an evaluation, no more than that."""

import numpy as np
import pytest

import lightcurves as lc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("make", [("FPW", (10,)), ("BoxLeastSquares", (30, 0.01, 0.2))])
def test_time_beyond_the_one_fma_range(make):
    """30 curves of 2000 points x 2000 periods: 1.1 times the kernel time of
    periods within the range (both forms are bound by their shared memory
    updates); a branch per point took 2.6 times."""
    from periodfind_b200 import _native as nat
    from periodfind_b200 import gpu

    rng = np.random.default_rng(5)
    ts = [lc.uniform_times(rng, 2000, 2000.0) for _ in range(30)]
    ms = [rng.normal(15.0, 0.3, 2000).astype(np.float32) for _ in range(30)]
    es = [rng.uniform(0.02, 0.2, 2000).astype(np.float32) for _ in range(30)]
    obj = getattr(gpu, make[0])(*make[1])
    ms_of = []
    for p_min in (0.1, 0.0005):  # 2e4 and 4e6 cycles
        periods = np.geomspace(p_min, 5.0 * p_min, 2000).astype(np.float32)
        best = np.inf
        for _ in range(6):
            obj.periodograms(ts, ms, periods, np.zeros(1, np.float32), errs=es)
            best = min(best, nat.default_context(0).last_kernel_ms)
        ms_of.append(best)
    assert ms_of[1] <= 1.6 * ms_of[0], ms_of
