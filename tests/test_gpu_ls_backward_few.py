"""The backward of the Lomb-Scargle power on many short curves: threads without a
second point spend nothing on one."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _ms(n_points, n_curves=1000, n_freq=1000):
    import torch

    from periodfind_b200 import ls_grad
    from periodfind_b200 import _native as nat

    rng = np.random.default_rng(1)
    off = np.arange(n_curves + 1, dtype=np.int64) * n_points
    t = torch.from_numpy(rng.uniform(0, 2000, off[-1]).astype(np.float32)).cuda()
    y = torch.from_numpy(rng.normal(0, 1, off[-1]).astype(np.float32)).cuda()
    w = torch.from_numpy(2 * np.pi / np.geomspace(0.1, 100.0, n_freq)).cuda()
    _, d1, _, coef = ls_grad.ls_derivatives(t, y, w, off, second=False)
    g = torch.ones((n_curves, n_freq), device="cuda")
    grad = torch.empty_like(t)
    ctx = nat.default_context(0)
    stream = torch.cuda.current_stream().cuda_stream
    times = []
    for _ in range(12):
        a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        torch.cuda._sleep(200000)
        a.record()
        ctx.check(ctx.lib.pf_ls_backward_dev(
            ctx.handle, t.data_ptr(), off.ctypes.data, n_curves, w.data_ptr(), 0, n_freq,
            g.data_ptr(), d1.data_ptr(), coef.data_ptr(), None, grad.data_ptr(), stream))
        b.record()
        b.synchronize()
        times.append(a.elapsed_time(b))
    return min(times)


def test_time_follows_the_points():
    """100 points a curve against 512: a fifth of the evaluations, a quarter with
    whole warps; half if every thread summed two points.  The rest is staging."""
    assert _ms(100) <= 0.55 * _ms(512)
