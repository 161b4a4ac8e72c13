"""The peak search with one to eight warps per row (few rows, min_distance up
to 1) and by one warp's replay (min_distance 3) against the oracle's
find_top_peaks: row lengths around the steps' and parts' borders, many equal
values, lists that are not filled, NaN and infinities, rising rows (every
extremum enters the list)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("flat", [3, 1023, 1024, 2048, 4095, 4096, 4097, 8191, 8200, 20001])
@pytest.mark.parametrize("rows", [1, 7, 741, 1481, 2961])
@pytest.mark.parametrize("n_peaks,md", [(1, 1), (7, 0), (32, 1), (32, 3)])
def test_against_oracle(oracle, flat, rows, n_peaks, md):
    from periodfind_b200.gpu import find_top_peaks_batched

    if rows * flat > 2e7:
        pytest.skip("large")
    rng = np.random.default_rng(flat + rows)
    d = rng.normal(size=(rows, flat, 1)).astype(np.float32)
    d[::3] = np.round(d[::3])             # many ties
    d[1::5, flat // 2:] = 1.0             # flat halves: short lists
    d[2::7] += np.linspace(0, 50, flat, dtype=np.float32)[:, None]
    if flat > 100:
        d[::2, 50] = np.inf
        d[::2, 77] = np.nan
        d[::2, flat - 9] = -np.inf
    for use_max in (True, False):
        got = find_top_peaks_batched(d, n_peaks, md, use_max)
        want = oracle.find_top_peaks_batched(d, n_peaks, md, use_max)
        np.testing.assert_array_equal(got[0], want[0])
        np.testing.assert_array_equal(got[1], want[1])
