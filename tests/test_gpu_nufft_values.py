"""The non-uniform FFT of the frequency grid on values that strain its
fixed-point grid: every point in one grid cell."""

import numpy as np
import pytest

import lightcurves as lc

pytestmark = pytest.mark.gpu


def _power(ts, ms, f0, df, n, form):
    from periodfind_b200 import _native as nat
    from periodfind_b200.gpu import LombScargle

    ls = LombScargle()
    if form == "transform":
        ls._flags |= nat.PF_TRIG_TRANSFORM
        form = None
    return ls.periodograms_frequency_grid(ts, ms, f0, df, n, trig=form, center=False)


@pytest.mark.parametrize("n", [64, 100, 510, 511, 512, 513, 1022, 1023, 1024, 1535, 2047])
@pytest.mark.parametrize("value", [None, 0.3, -7.7e3])
def test_every_point_in_one_cell(n, value):
    """Integer times at integer frequencies, and equal times: the normal matrix
    is singular at every frequency, so the power is NaN as in the direct form."""
    y = np.random.default_rng(n).normal(0, 1, n) if value is None else np.full(n, value)
    ms = [y.astype(np.float32)]
    for t, f0, df in ((np.arange(n), 1.0, 1.0), (np.zeros(n), 0.1, 0.01)):
        ts = [t.astype(np.float32)]
        assert np.isnan(_power(ts, ms, f0, df, 2048, "sincos")).all()
        assert np.isnan(_power(ts, ms, f0, df, 2048, "transform")).all()
