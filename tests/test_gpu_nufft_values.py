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


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
def test_values_that_are_not_finite(bad):
    """One magnitude that is not finite: NaN at every frequency of its curve, as
    in the direct form, in no more time than the transform of a clean curve
    needs (point by point it took 30 times that), and the other curves as before."""
    import torch

    from periodfind_b200 import _native as nat

    rng = np.random.default_rng(4)
    n, n_freq, f0, df = 16384, 20000, 0.01, 1e-3
    ts = [lc.seasonal_times(rng, n, 3000.0).astype(np.float32) for _ in range(8)]
    ms = [rng.normal(0, 1, n).astype(np.float32) for _ in range(8)]
    clean = _power(ts, ms, f0, df, n_freq, "transform")
    spoilt = [m.copy() for m in ms]
    spoilt[3][77] = bad
    want = _power(ts, spoilt, f0, df, n_freq, "sincos")
    got = _power(ts, spoilt, f0, df, n_freq, "transform")
    np.testing.assert_array_equal(np.isnan(got), np.isnan(want))
    assert np.isnan(got[3]).all()
    np.testing.assert_array_equal(np.delete(got, 3, 0), np.delete(clean, 3, 0))

    off = np.arange(9, dtype=np.int64) * n
    t = torch.from_numpy(np.concatenate(ts)).cuda()
    out = torch.empty((8, n_freq), device="cuda")
    ctx = nat.default_context(0)
    flags = nat.PF_MODE_CHOSEN | nat.PF_TRIG_TRANSFORM

    def best(mags):
        m = torch.from_numpy(np.concatenate(mags)).cuda()
        times = []
        for _ in range(6):
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            stream = torch.cuda.current_stream()
            a.record()
            ctx.check(ctx.lib.pf_ls_fgrid_dev(ctx.handle, t.data_ptr(), m.data_ptr(),
                                              off.ctypes.data, 8, f0, df, n_freq, flags,
                                              out.data_ptr(), stream.cuda_stream))
            b.record()
            b.synchronize()
            times.append(a.elapsed_time(b))
        return min(times)

    # (4 times leaves room for clocks and launch gaps; the fault was 34 times.)
    assert best(spoilt) <= 4.0 * best(ms)


def _power64(t, y, freqs):
    import torch

    t, y, f = (torch.from_numpy(np.asarray(x, np.float64)).cuda() for x in (t, y, freqs))
    out = []
    for fb in torch.split(f, max(1, 20_000_000 // len(t))):
        th = t[:, None] * fb[None, :]
        th = 2.0 * np.pi * (th - torch.round(th))
        c, s = torch.cos(th), torch.sin(th)
        C, S, cc, cs = y @ c, y @ s, (c * c).sum(0), (c * s).sum(0)
        ss = len(t) - cc
        out.append(0.5 * (ss * C * C - 2.0 * cs * C * S + cc * S * S) / (cc * ss - cs * cs))
    return torch.cat(out).cpu().numpy()


@pytest.mark.parametrize("n", [300, 511, 1023, 2000, 16384])
@pytest.mark.parametrize("kind", ["one", "huge", "percent", "tails", "eclipses"])
def test_values_far_from_the_rest(kind, n):
    """A sinusoid with one value far off (as a leaked sentinel), one of 10^4,
    one in a hundred far off, heavy tails, and eclipses.  Largest error 2e-5 of
    the curve's peak, the bound of tests/test_gpu_nufft.py, and the error
    (2-norm) no larger than the sincos form's; a quarter is left for the
    spread of the two forms' rounding, of about n values each."""
    rng = np.random.default_rng(n)
    t = lc.seasonal_times(rng, n, 3000.0).astype(np.float32)
    y = 0.3 * np.sin(2 * np.pi * 1.37 * t) + rng.normal(0, 0.05, n)
    if kind == "one":
        y[n // 3] = 85.0
    elif kind == "huge":
        y[n // 3] = -1e4
    elif kind == "percent":
        y[rng.integers(0, n, n // 100)] += 30.0
        y[n // 2] = 85.0
    elif kind == "tails":
        y += 0.3 * rng.standard_t(1.5, n)
    else:
        y = np.where(np.mod(1.37 * t, 1.0) < 0.05, -0.5, 0.0) + rng.normal(0, 0.02, n)
    y = (y - y.mean()).astype(np.float32)
    f0, df, n_freq = 0.01, 0.002, 10000
    want = _power64(t, y, f0 + df * np.arange(n_freq))
    err = {form: _power([t], [y], f0, df, n_freq, form)[0] - want
           for form in ("transform", "sincos")}
    np.testing.assert_array_equal(_power([t], [y], f0, df, n_freq, "transform")[0],
                                  _power([t], [y], f0, df, n_freq, "transform")[0])
    assert np.abs(err["transform"]).max() <= 2e-5 * want.max()
    assert np.linalg.norm(err["transform"]) <= 1.25 * np.linalg.norm(err["sincos"])
