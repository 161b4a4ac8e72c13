"""The device statistics over row lengths: the edges of numpy's summation tree,
rows staged in shared memory and rows read from global memory, against numpy
on the same periodogram.
Rows of tiny curves hold many equal values, so the order of ties is checked."""

import numpy as np
import pytest

import lightcurves as lc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_per", [2, 7, 8, 9, 127, 128, 129, 255, 257, 1000, 2049, 8192,
                                   8193, 20000, 20001, 47999, 60001, 300007])
@pytest.mark.parametrize("algo,n_stats", [("ce", 1), ("ce", 7), ("ls", 1), ("ls", 40)])
def test_rows_equal_numpy(algo, n_stats, n_per):
    from periodfind_b200 import gpu

    if n_stats >= n_per:
        pytest.skip("calc() takes numpy there")
    rng = np.random.default_rng(n_per)
    ts = [lc.uniform_times(rng, n, 200.0) for n in (9, 60)]
    ms = [rng.normal(15.0, 0.3, len(t)).astype(np.float32) for t in ts]
    P = np.geomspace(0.3, 90.0, n_per).astype(np.float32)
    D = np.zeros(1, np.float32)
    obj = gpu.ConditionalEntropy() if algo == "ce" else gpu.LombScargle()
    got = obj.calc(ts, ms, P, D, output="stats", n_stats=n_stats)
    for g, pg in zip(got, obj.calc(ts, ms, P, D, output="periodogram")):
        x = pg.data[:, 0]
        best = np.argsort(x if algo == "ce" else -x, kind="stable")[:n_stats]
        med = np.median(x)
        want = (np.mean(pg.data), np.std(pg.data), med, np.median(np.abs(x - med)))
        rows = [g] if n_stats == 1 else g
        assert [r.value for r in rows] == list(x[best])
        assert [r.params[0] for r in rows] == list(P[best])
        for r in rows:
            assert (r.mean, r.std, r.median, r.mad) == want
