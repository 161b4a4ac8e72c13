"""CE and AOV on trial periods beyond the fast bin's range: the range is taken
warp by warp and round by round, so short and long periods may meet in one
launch item, and the exact sequence costs no more than its own operations."""

import numpy as np
import pytest

import lightcurves as lc
from oracle import oracle as O

pytestmark = pytest.mark.gpu

SHAPES = [(b, c, r, 0) for b in (32, 64, 128) for c in (1, 2) for r in (1, 4)]


@pytest.mark.parametrize("order", ["up", "down", "mixed"])
@pytest.mark.parametrize("algo", ["CE", "AOV"])
def test_every_range_in_one_item(monkeypatch, algo, order):
    """Periods from 2e8 cycles over the curve to 1 and below, 0.9 of 512 of them
    live, in every shape: the oracle's values."""
    from periodfind_b200 import _native as nat
    from periodfind_b200 import gpu

    ctx = nat.Context(0)
    monkeypatch.setattr(nat, "default_context", lambda device=0: ctx)
    rng = np.random.default_rng(8)
    ts = [lc.uniform_times(rng, n, 900.0) for n in (17, 300, 700)]
    ms = [rng.uniform(0.01, 0.99, len(t)).astype(np.float32) for t in ts]
    periods = np.geomspace(4e-6, 2000.0, 461).astype(np.float32)
    if order == "down":
        periods = periods[::-1].copy()
    elif order == "mixed":
        periods = rng.permutation(periods)
    pdts = np.array([0.0, 1e-9], np.float32)
    if algo == "CE":
        obj, want = gpu.ConditionalEntropy(semantics="cpu"), O.ce(ts, ms, periods, pdts, 10, 10)
        shapes = SHAPES + [(b, c, r, 1) for b in (32, 64) for c in (1, 2) for r in (1, 4)]
    else:
        obj, want = gpu.AOV(15, semantics="cpu"), O.aov_f64(ts, ms, periods, pdts, 15)
        shapes = SHAPES + [(64, 3, r, 0) for r in (1, 4)]
    for shape in shapes:
        ctx.check(ctx.lib.pf_pin_bin_shape(ctx.handle, *shape))
        # One point in another bin moves a value by 1e-3.
        np.testing.assert_allclose(obj.periodograms(ts, ms, periods, pdts), want, rtol=1e-5,
                                   atol=1e-5, err_msg=str(shape))


@pytest.mark.parametrize("algo", ["CE", "AOV"])
def test_time_beyond_the_range(monkeypatch, algo):
    """2000 curves of 300 points x 1000 periods x 3 derivatives, half of the
    cells beyond the fast range: 1.7 (CE) and 1.5 times (AOV) the time within
    it.  One cell after another, set up again for every run of points, and 512
    periods sharing a range made it 2.5 and 2.4 times."""
    import torch

    from periodfind_b200 import _native as nat
    from periodfind_b200 import gpu

    ctx = nat.Context(0)
    monkeypatch.setattr(nat, "default_context", lambda device=0: ctx)
    rng = np.random.default_rng(3)
    off = np.arange(2001, dtype=np.int64) * 300
    t = torch.from_numpy(rng.uniform(0, 2000, off[-1]).astype(np.float32)).cuda()
    m = torch.from_numpy(rng.uniform(0.01, 0.99, off[-1]).astype(np.float32)).cuda()
    pdts = np.array([0.0, 1e-6, -3e-5], np.float32)
    obj = gpu.ConditionalEntropy() if algo == "CE" else gpu.AOV(15)
    best = []
    for p_min in (0.1, 1e-4):
        periods = np.geomspace(p_min, (1000 if p_min > 0.01 else 100) * p_min, 1000)
        times = []
        for _ in range(8):
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            a.record()
            obj.periodograms_device(t, m, off, periods.astype(np.float32), pdts)
            b.record()
            b.synchronize()
            times.append(a.elapsed_time(b))
        best.append(min(times))
    assert best[1] <= 2.1 * best[0], best
