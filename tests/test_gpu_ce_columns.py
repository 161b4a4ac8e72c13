"""Conditional entropy with many magnitude columns on short curves: the cost of
a cell follows its counters, not the number of columns that a curve meets."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _device_ms(n_phase, n_mag, n_points, n_curves=1000, n_per=2000):
    import torch

    from periodfind_b200 import gpu

    rng = np.random.default_rng(1)
    off = np.arange(n_curves + 1, dtype=np.int64) * n_points
    t = torch.from_numpy(rng.uniform(0, 2000, off[-1]).astype(np.float32)).cuda()
    m = torch.from_numpy(rng.normal(0.5, 0.1, off[-1]).clip(0.01, 0.99).astype(np.float32)).cuda()
    periods = np.geomspace(0.1, 100.0, n_per).astype(np.float32)
    ce, times = gpu.ConditionalEntropy(n_phase, n_mag), []
    for _ in range(8):
        a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        a.record()
        ce.periodograms_device(t, m, off, periods, np.zeros(1, np.float32))
        b.record()
        b.synchronize()
        times.append(a.elapsed_time(b))
    return min(times)


def test_time_of_many_columns():
    """60 points a curve, 40 columns against 10: four times the counters for the
    same points.  Sorted by column alone the call took 4 times as long; with
    the points in their own order it takes 2.2 times."""
    assert _device_ms(10, 40, 60) <= 3.0 * _device_ms(10, 10, 60)


@pytest.mark.parametrize("shared", [False, True])
def test_large_histograms_may_share_them(monkeypatch, shared):
    """Where 64 private histograms fill an SM, the tuner weighs one histogram
    per warp and period as well; with small ones it does
    not.  The values are the same bit for bit."""
    from periodfind_b200 import _native as nat
    from periodfind_b200 import gpu

    ctx = nat.Context(0)
    monkeypatch.setattr(nat, "default_context", lambda device=0: ctx)
    rng = np.random.default_rng(2)
    ts = [np.sort(rng.uniform(0, 900, n)).astype(np.float32) for n in (300, 700) for _ in range(30)]
    ms = [rng.uniform(0.01, 0.99, len(t)).astype(np.float32) for t in ts]
    periods = np.geomspace(0.1, 30.0, 1000).astype(np.float32)
    bins = (50, 20) if shared else (10, 20)
    ce, alone = gpu.ConditionalEntropy(*bins), gpu.ConditionalEntropy(*bins)
    got = ce.periodograms(ts, ms, periods, np.zeros(1, np.float32))
    report = ctx.tuning_report()
    # Private histograms: 3 shapes of 50 x 20 bins fit, all 6 of 10 x 20, in 1
    # or 4 rounds; shared ones: 2 shapes, persistent or not.
    assert f"candidates={3 * 2 + 4 if shared else 6 * 2}" in report, report
    other = nat.Context(0)
    monkeypatch.setattr(nat, "default_context", lambda device=0: other)
    alone._flags |= nat.PF_NO_TUNE
    np.testing.assert_array_equal(
        got, alone.periodograms(ts, ms, periods, np.zeros(1, np.float32)))


@pytest.mark.parametrize("n_points, n_mag", [(50, 10), (120, 20), (200, 64)])
def test_orders_are_weighed_before_the_shapes(monkeypatch, n_points, n_mag):
    """The tuner times both point orders in the base shape's block and the other
    shapes for the faster order alone: at most two samples more than the 12 of
    one order, where both in every shape made 20."""
    import re

    from periodfind_b200 import _native as nat
    from periodfind_b200 import gpu

    ctx = nat.Context(0)
    monkeypatch.setattr(nat, "default_context", lambda device=0: ctx)
    rng = np.random.default_rng(3)
    ts = [np.sort(rng.uniform(0, 900, n_points)).astype(np.float32) for _ in range(40)]
    ms = [rng.uniform(0.01, 0.99, n_points).astype(np.float32) for _ in ts]
    periods = np.geomspace(0.1, 30.0, 1000).astype(np.float32)
    ce, alone = gpu.ConditionalEntropy(10, n_mag), gpu.ConditionalEntropy(10, n_mag)
    got = ce.periodograms(ts, ms, periods, np.zeros(1, np.float32))
    counts = [int(c) for c in re.findall(r"candidates=(\d+)", ctx.tuning_report())]
    assert len(counts) == 1 and counts[0] <= 12 + 2, ctx.tuning_report()
    other = nat.Context(0)
    monkeypatch.setattr(nat, "default_context", lambda device=0: other)
    alone._flags |= nat.PF_NO_TUNE
    np.testing.assert_array_equal(
        got, alone.periodograms(ts, ms, periods, np.zeros(1, np.float32)))
