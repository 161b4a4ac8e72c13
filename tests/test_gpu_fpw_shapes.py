"""The chosen FPW and BLS kernels at the edges of their tiling (groups of four
points, 256-point tiles, the CTA's columns for each block shape, the one-FMA
bin's range and beyond, narrow and wide window ranges): equal to the plain
form bit for bit, as both add the points in curve order."""

import numpy as np
import pytest

import lightcurves as lc

pytestmark = pytest.mark.gpu

LENGTHS = (0, 1, 3, 4, 5, 255, 256, 257, 259, 600)


@pytest.mark.parametrize("n_per", [1, 64, 65, 255, 257, 600])
@pytest.mark.parametrize("make", [("FPW", (10,)), ("FPW", (32,)), ("FPW", (33,)), ("FPW", (128,)),
                                  ("BoxLeastSquares", (20, 0.05, 0.3)),
                                  ("BoxLeastSquares", (50, 0.01, 0.99)),
                                  ("BoxLeastSquares", (7, 0.3, 0.3)),
                                  ("BoxLeastSquares", (100, 0.4, 0.9))])
@pytest.mark.parametrize("p_min", [0.07, 0.0004])
def test_chosen_equals_plain(make, n_per, p_min):
    from periodfind_b200 import gpu

    rng = np.random.default_rng(n_per)
    ts = [lc.uniform_times(rng, n, 900.0) for n in LENGTHS]
    ms = [rng.normal(15.0, 0.3, n).astype(np.float32) for n in LENGTHS]
    es = [rng.uniform(0.02, 0.2, n).astype(np.float32) for n in LENGTHS]
    # p_min 0.0004: up to 2.2e6 cycles, past the one-FMA bin's 2^19.
    periods = np.geomspace(p_min, 40.0, n_per).astype(np.float32)
    pdts = np.array([0.0, 1e-6], np.float32)
    cls, args = getattr(gpu, make[0]), make[1]
    got, want = (cls(*args, mode=m).periodograms(ts, ms, periods, pdts, errs=es)
                 for m in ("chosen", "plain"))
    np.testing.assert_array_equal(got, want)
