"""Every built launch shape of the chosen CE / AOV bin kernels, pinned one after
the other: the same values bit for bit, and the oracle's, at the curve lengths
and period counts where the tiling can go wrong, on periods in each range of the
fold, and with strong period derivatives."""

import numpy as np
import pytest

import lightcurves as lc
from oracle import oracle as O

pytestmark = pytest.mark.gpu

# Groups of 4, 8 and 16 points, the 256-point tile, the 512-point log table.
LENGTHS = (0, 1, 3, 4, 5, 7, 8, 9, 15, 16, 17, 31, 33, 255, 256, 257, 260, 511, 512, 513, 1000)
SHAPES = [(b, c, r, 0) for b in (32, 64, 128) for c in (1, 2) for r in (1, 4)]
OWN_ORDER = [(b, c, r, 1) for b in (32, 64) for c in (1, 2) for r in (1, 4)]
THREE = [(64, 3, r, 0) for r in (1, 4)]


def _curves(lengths, seed, span=900.0):
    rng = np.random.default_rng(seed)
    ts = [lc.uniform_times(rng, n, span) for n in lengths]
    ms = [np.clip(0.55 + 0.2 * rng.normal(size=n), 0.001, 0.999).astype(np.float32)
          for n in lengths]
    return ts, ms


@pytest.fixture
def pinned(monkeypatch):
    """A fresh context behind the classes, and a call that pins its shape."""
    from periodfind_b200 import _native as nat

    ctx = nat.Context(0)
    monkeypatch.setattr(nat, "default_context", lambda device=0: ctx)
    return lambda shape: ctx.check(ctx.lib.pf_pin_bin_shape(ctx.handle, *shape))


# 0.07: one FMA a point.  0.0004: 2.2e6 cycles, past its range of 2^19.
# 4e-6: 2.2e8 cycles times the phase bins, past 2^30: the exact sequence.
@pytest.mark.parametrize("p_min", [0.07, 4e-4, 4e-6])
@pytest.mark.parametrize("n_per", [1, 65, 513])
@pytest.mark.parametrize("n_phase,n_mag", [(10, 10), (7, 3), (5, 60)])
def test_ce_shapes(pinned, n_phase, n_mag, n_per, p_min):
    from periodfind_b200.gpu import ConditionalEntropy

    ts, ms = _curves(LENGTHS, n_per)
    periods = np.geomspace(p_min, 600.0 * p_min, n_per).astype(np.float32)
    pdts = np.array([0.0, 1e-5 if p_min > 0.01 else 1e-9], np.float32)
    ce = ConditionalEntropy(n_phase, n_mag, semantics="cpu")
    want = O.ce(ts, ms, periods, pdts, n_phase, n_mag)
    first = None
    for shape in SHAPES + OWN_ORDER:
        pinned(shape)
        got = ce.periodograms(ts, ms, periods, pdts)
        # One point in another bin moves a value by 1e-3; see
        # tests/test_gpu_bin_shapes.py.
        np.testing.assert_allclose(got, want, rtol=1e-5, atol=1e-5, err_msg=str(shape))
        first = got if first is None else first
        np.testing.assert_array_equal(got, first, err_msg=str(shape))


@pytest.mark.parametrize("p_min", [0.07, 4e-4, 4e-6])
@pytest.mark.parametrize("n_per", [1, 65, 513])
@pytest.mark.parametrize("n_phase", [2, 15])
def test_aov_shapes(pinned, n_phase, n_per, p_min):
    from periodfind_b200.gpu import AOV

    ts, ms = _curves([n for n in LENGTHS if n > n_phase + 1], n_per)
    periods = np.geomspace(p_min, 600.0 * p_min, n_per).astype(np.float32)
    pdts = np.array([0.0, 1e-5 if p_min > 0.01 else 1e-9], np.float32)
    aov = AOV(n_phase, semantics="cpu")
    want = O.aov_f64(ts, ms, periods, pdts, n_phase)
    first = None
    for shape in SHAPES + THREE:
        pinned(shape)
        got = aov.periodograms(ts, ms, periods, pdts)
        np.testing.assert_allclose(got, want, rtol=1e-5, atol=1e-5, err_msg=str(shape))
        first = got if first is None else first
        np.testing.assert_array_equal(got, first, err_msg=str(shape))


@pytest.mark.parametrize("span,pdt", [(900.0, 1e-3), (900.0, -0.05), (30000.0, 2e-4)])
@pytest.mark.parametrize("algo", ["CE", "AOV"])
def test_strong_derivatives(pinned, algo, span, pdt):
    """Corrections larger than the time itself or nearly cancelling it, in every
    shape that a call may take (the counts of tests/test_gpu_bin_shapes.py come
    from the one-period reference form)."""
    from periodfind_b200 import gpu

    ts, ms = _curves((40, 257, 1000), 3, span)
    periods = np.geomspace(0.07, 40.0, 131).astype(np.float32)
    pdts = np.array([pdt], np.float32)
    if algo == "CE":
        obj, shapes = gpu.ConditionalEntropy(10, 10, semantics="cpu"), SHAPES + OWN_ORDER
        want = O.ce(ts, ms, periods, pdts, 10, 10)
    else:
        obj, shapes = gpu.AOV(15, semantics="cpu"), SHAPES + THREE
        want = O.aov_f64(ts, ms, periods, pdts, 15)
    for shape in shapes:
        pinned(shape)
        np.testing.assert_allclose(obj.periodograms(ts, ms, periods, pdts), want, rtol=1e-5,
                                   atol=1e-5, err_msg=str(shape))


def test_shapes_that_are_not_built(pinned):
    from periodfind_b200 import _native as nat
    from periodfind_b200 import gpu

    for shape in ((16, 1, 1, 0), (256, 1, 1, 0), (64, 4, 1, 0), (32, 3, 1, 0), (64, 1, 2, 0),
                  (128, 1, 1, 1)):
        with pytest.raises(nat.PeriodfindError):
            pinned(shape)
    ts, ms = _curves((100,), 1)
    args = ts, ms, np.ones(4, np.float32), np.zeros(1, np.float32)
    pinned((128, 2, 1, 0))
    with pytest.raises(nat.PeriodfindError):  # 512 KB of counters
        gpu.ConditionalEntropy(50, 20).periodograms(*args)
    pinned((64, 3, 1, 0))
    with pytest.raises(nat.PeriodfindError):  # three periods: AOV only
        gpu.ConditionalEntropy().periodograms(*args)
    pinned((0, 0, 0, 0))
    gpu.ConditionalEntropy().periodograms(*args)


@pytest.mark.parametrize("cpu", [False, True])
def test_count_reciprocals(cpu):
    """1 / c for every count a bin can hold, correctly rounded."""
    import torch

    from periodfind_b200 import _native as nat

    out = torch.empty(65535, dtype=torch.float64, device="cuda")
    ctx = nat.default_context(0)
    ctx.check(ctx.lib.pf_count_rcp_dev(ctx.handle, nat.PF_SEM_CPU if cpu else 0, 65535,
                                       out.data_ptr(), torch.cuda.current_stream().cuda_stream))
    np.testing.assert_array_equal(out.cpu().numpy(), 1.0 / np.arange(1, 65536, dtype=np.float64))
