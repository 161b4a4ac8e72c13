"""The chosen CE / AOV bin kernels at the sizes where their tiling can go
wrong: curve lengths around the groups of 4, 8 and 16 points and the 256-point
tile, period counts around the CTA's columns, few, many and empty magnitude
columns, and both layouts of the sorted CE times.  Against the oracle."""

import numpy as np
import pytest

import lightcurves as lc
from oracle import oracle as O

pytestmark = pytest.mark.gpu

LENGTHS = (1, 2, 3, 4, 5, 7, 8, 9, 12, 15, 16, 17, 23, 24, 31, 33, 63, 240, 255, 256, 257, 260,
           511, 513, 1000)


def _curves(lengths, seed, spread):
    rng = np.random.default_rng(seed)
    ts = [lc.uniform_times(rng, n, 900.0) for n in lengths]
    # spread 0: every point in one magnitude column; small: most of them.
    ms = [np.clip(0.55 + spread * rng.normal(size=n), 0.001, 0.999).astype(np.float32)
          for n in lengths]
    return ts, ms


@pytest.mark.parametrize("n_per", [1, 63, 128, 129, 513])
@pytest.mark.parametrize("n_phase,n_mag,spread", [(10, 10, 0.2), (7, 3, 0.0), (20, 11, 0.03)])
@pytest.mark.parametrize("pdts", [(0.0,), (0.0, 1e-5)])
def test_ce_lengths_and_columns(n_per, n_phase, n_mag, spread, pdts):
    from periodfind_b200.gpu import ConditionalEntropy

    ts, ms = _curves(LENGTHS, n_per + n_phase, spread)
    periods = np.geomspace(0.07, 40.0, n_per).astype(np.float32)
    pdts = np.array(pdts, np.float32)
    got = ConditionalEntropy(n_phase, n_mag, semantics="cpu").periodograms(ts, ms, periods, pdts)
    want = O.ce(ts, ms, periods, pdts, n_phase, n_mag)
    # One point in another bin moves a value by at least about 1 / n = 1e-3;
    # the statistics agree to ~1e-6 of their largest term, ln(n_mag).
    np.testing.assert_allclose(got, want, rtol=1e-5, atol=1e-5)


@pytest.mark.parametrize("n_per", [1, 63, 128, 129, 513])
@pytest.mark.parametrize("n_phase", [2, 10, 15])
def test_aov_lengths(n_per, n_phase):
    from periodfind_b200.gpu import AOV

    ts, ms = _curves([n for n in LENGTHS if n > n_phase + 1], n_per + n_phase, 0.2)
    periods = np.geomspace(0.07, 40.0, n_per).astype(np.float32)
    pdts = np.array([0.0, 1e-5], np.float32)
    got = AOV(n_phase, semantics="cpu").periodograms(ts, ms, periods, pdts)
    want = O.aov_f64(ts, ms, periods, pdts, n_phase)
    # Fixed-point magnitudes of 22 bits or more at these lengths.
    np.testing.assert_allclose(got, want, rtol=1e-5, atol=1e-5)


def test_ce_many_columns_and_short_curves():
    """Thousands of short curves with far more magnitude columns than points:
    the sorted times and run tables are laid out by curve length."""
    from periodfind_b200.gpu import ConditionalEntropy

    rng = np.random.default_rng(5)
    n_curves = 4000
    lens = rng.integers(0, 16, n_curves)
    ts = [lc.uniform_times(rng, int(n), 90.0) for n in lens]
    ms = [rng.uniform(0.0, 0.999, int(n)).astype(np.float32) for n in lens]
    periods = np.geomspace(0.5, 20.0, 5).astype(np.float32)
    pdts = np.zeros(1, np.float32)
    got = ConditionalEntropy(2, 400, semantics="cpu").periodograms(ts, ms, periods, pdts)
    want = O.ce(ts, ms, periods, pdts, 2, 400)
    np.testing.assert_allclose(got, want, rtol=1e-5, atol=1e-5)


@pytest.mark.parametrize("span,pdt", [(900.0, 1e-3), (900.0, -0.05), (30000.0, 2e-4)])
@pytest.mark.parametrize("n_phase", [2, 15, 40])
def test_aov_bins_with_strong_derivatives(span, pdt, n_phase):
    """Period derivatives whose correction is larger than the time itself or
    nearly cancels it: every bin count equal to the reference's."""
    from periodfind_b200.gpu import AOV

    rng = np.random.default_rng(n_phase)
    ts = [lc.uniform_times(rng, n, span) for n in (7, 257, 1000)]
    ms = [rng.random(len(t)).astype(np.float32) for t in ts]
    periods = np.geomspace(0.07, 40.0, 131).astype(np.float32)
    pdts = np.array([pdt], np.float32)
    _, got = AOV(n_phase, mode="chosen", semantics="cpu").bin_counts(ts, ms, periods, pdts)
    for c, (t, m) in enumerate(zip(ts, ms)):
        for i, P in enumerate(periods):
            _, want = O.aov_counts(t, m, P, pdts[0], n_phase)
            np.testing.assert_array_equal(got[c, i, 0], want)
