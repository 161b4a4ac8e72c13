"""Lomb-Scargle on a uniform frequency grid by the non-uniform FFT
(PF_TRIG_TRANSFORM), against the FP64 oracle at the same frequencies.

Bound: 2e-5 of each curve's largest FP64 power, the sincos form's.  The
transform's own error is about 2e-7 of the largest sums (kernel width 8, FP32
grid and FFT), the FP32 statistic's on near-singular cells larger."""

import numpy as np
import pytest

import lightcurves as lc

pytestmark = pytest.mark.gpu


def _ls():
    from periodfind_b200 import _native as nat
    from periodfind_b200.gpu import LombScargle

    ls = LombScargle()
    ls._flags |= nat.PF_TRIG_TRANSFORM
    return ls


@pytest.mark.parametrize("n_freq", [1, 2047, 4096, 4097, 10000])
@pytest.mark.parametrize("f_min,f_max", [(0.01, 20.0), (0.2, 0.45)])
def test_against_fp64(oracle, n_freq, f_min, f_max):
    lengths = [32, 33, 300, 511, 512, 513, 1025, 5000]
    ts, ms, _, _ = lc.ls_study_curves(len(lengths), seed=n_freq, lengths=lengths)
    df = (f_max - f_min) / max(n_freq - 1, 1)
    freqs = f_min + np.arange(n_freq) * df
    ref = oracle.ls_f64(ts, ms, 1.0 / freqs, [0.0])[:, :, 0]
    got = _ls().periodograms_frequency_grid(ts, ms, f_min, df, n_freq, center=False)
    again = _ls().periodograms_frequency_grid(ts, ms, f_min, df, n_freq, center=False)
    np.testing.assert_array_equal(got, again)
    # Scale: the curve's largest power over the whole range, which a grid of
    # one frequency need not reach; its mean square is a lower bound of that.
    scale = np.maximum(ref.max(axis=1), [float(np.mean(m.astype(np.float64) ** 2)) for m in ms])
    assert (np.abs(got - ref) / scale[:, None]).max() <= 2e-5


def test_singular_cells_as_the_direct_form():
    """f = 0 and frequencies on which evenly spaced times alias have a singular
    normal matrix: the direct form's value (NaN) there, and its values beside."""
    from periodfind_b200.gpu import LombScargle

    rng = np.random.default_rng(8)
    ts = [np.arange(n, dtype=np.float32) for n in (64, 700)]
    ms = [lc.center(rng.normal(0, 1, len(t)).astype(np.float32)) for t in ts]
    n_freq, df = 5000, 1.0 / 2048
    got = _ls().periodograms_frequency_grid(ts, ms, 0.0, df, n_freq, center=False)
    want = LombScargle().periodograms_frequency_grid(ts, ms, 0.0, df, n_freq, trig="sincos",
                                                     center=False)
    sing = np.isnan(want)
    assert sing[:, ::2048].all()
    np.testing.assert_array_equal(np.isnan(got), sing)
    ok = ~sing
    assert np.abs(got[ok] - want[ok]).max() <= 2e-4 * np.abs(want[ok]).max()
