"""The tuner keeps its choices apart by how much of the chip a call fills and,
on a frequency grid, by the number of frequencies against the transform's
block, so that a call's shape does not depend on which size came first."""

import numpy as np
import pytest

import lightcurves as lc

pytestmark = pytest.mark.gpu


def _keys(monkeypatch, calls):
    """Keys of the tuning report of a fresh context after the calls."""
    from periodfind_b200 import _native as nat

    ctx = nat.Context(0)
    monkeypatch.setattr(nat, "default_context", lambda device=0: ctx)
    for call in calls:
        call()
    return {line.split(": ")[0] for line in ctx.tuning_report().splitlines()}


def _curves(n_curves, n):
    rng = np.random.default_rng(n_curves)
    ts = [lc.uniform_times(rng, n, 900.0) for _ in range(n_curves)]
    return ts, [rng.uniform(0.01, 0.99, n).astype(np.float32) for _ in range(n_curves)]


@pytest.mark.parametrize("algo", ["ConditionalEntropy", "AOV", "LombScargle"])
def test_one_curve_and_many(monkeypatch, algo):
    from periodfind_b200 import gpu

    periods = np.geomspace(0.5, 10.0, 1000).astype(np.float32)
    pdts = np.zeros(1, np.float32)

    def call(n_curves):
        return lambda: getattr(gpu, algo)().periodograms(*_curves(n_curves, 300), periods, pdts)

    few, many = _keys(monkeypatch, [call(1)]), _keys(monkeypatch, [call(600)])
    assert few and many and few.isdisjoint(many)
    for order in ((1, 600), (600, 1)):
        assert _keys(monkeypatch, [call(n) for n in order]) == few | many


def test_short_and_long_frequency_grids(monkeypatch):
    from periodfind_b200 import gpu

    ts, ms = _curves(1, 200)

    def call(n_freq):
        return lambda: gpu.LombScargle().periodograms_frequency_grid(ts, ms, 0.1, 1e-4, n_freq)

    seen = set()
    for n_freq in (600, 1100, 2500, 5000, 15000):
        keys = _keys(monkeypatch, [call(n_freq)])
        assert len(keys) == 1 and keys.isdisjoint(seen)
        seen |= keys
    for order in ((1100, 15000), (15000, 1100)):
        assert len(_keys(monkeypatch, [call(n) for n in order])) == 2


def test_one_launch_with_curves_too_short_for_the_transform(monkeypatch):
    """PF_ONE_LAUNCH with curves under 64 points beside long ones: the short ones
    keep the direct form that they have in a launch of their own."""
    from periodfind_b200 import _native as nat
    from periodfind_b200 import gpu

    ctx = nat.Context(0)
    monkeypatch.setattr(nat, "default_context", lambda device=0: ctx)
    rng = np.random.default_rng(3)
    lengths = [20, 33, 63] + [3000] * 8
    ts = [lc.seasonal_times(rng, n, 3000.0).astype(np.float32) for n in lengths]
    ms = [rng.normal(0, 1, n).astype(np.float32) for n in lengths]
    grid = (0.01, 0.0004, 50000)
    ls, one = gpu.LombScargle(), gpu.LombScargle()
    one._flags |= nat.PF_ONE_LAUNCH
    own = ls.periodograms_frequency_grid(ts, ms, *grid)
    assert "trig=transform" in ctx.tuning_report()
    np.testing.assert_array_equal(one.periodograms_frequency_grid(ts, ms, *grid)[:3], own[:3])
