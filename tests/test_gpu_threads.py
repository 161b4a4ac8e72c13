"""Distinct contexts in several host threads at once, on launches of one kernel
that take different amounts of shared memory."""

import threading

import numpy as np
import pytest

import lightcurves as lc

pytestmark = pytest.mark.gpu


def test_contexts_in_threads():
    """CE with 10 and 60 magnitude columns in one launch shape (28 and 156 KB a
    CTA), from device pointers, so that a call is little more than its
    launches: every call succeeds and leaves the values it gives alone."""
    import torch

    from periodfind_b200 import _native as nat

    rng = np.random.default_rng(6)
    t = lc.uniform_times(rng, 40, 200.0)
    m = rng.uniform(0.01, 0.99, 40).astype(np.float32)
    periods = np.geomspace(0.3, 90.0, 200).astype(np.float32)
    off = np.array([0, 40], np.int64)
    d_t, d_m, d_p, d_d = (torch.from_numpy(x).cuda()
                          for x in (t, m, periods, np.zeros(1, np.float32)))

    def make(bins):
        ctx, stream = nat.Context(0), torch.cuda.Stream()
        out = torch.zeros(200, device="cuda")
        args = (ctx.handle, d_t.data_ptr(), d_m.data_ptr(), off.ctypes.data, 1, d_p.data_ptr(),
                200, d_d.data_ptr(), 1, 10, bins, 1, 1, nat.PF_MODE_CHOSEN | nat.PF_NO_TUNE,
                out.data_ptr(), stream.cuda_stream)
        return ctx, stream, out, args

    jobs = [make(bins) for bins in (10, 60, 10, 60)]
    torch.cuda.synchronize()
    want = []
    for ctx, stream, out, args in jobs:
        ctx.check(ctx.lib.pf_ce_dev(*args))
        stream.synchronize()
        want.append(out.clone())
    torch.cuda.synchronize()
    errors = []

    def loop(job):
        ctx, stream, _, args = job
        try:
            for k in range(8000):
                ctx.check(ctx.lib.pf_ce_dev(*args))
                if k % 500 == 499:
                    stream.synchronize()
        except Exception as e:  # reported by the main thread
            errors.append(repr(e))

    threads = [threading.Thread(target=loop, args=(job,)) for job in jobs]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    torch.cuda.synchronize()
    assert not errors, errors
    for (_, _, out, _), w in zip(jobs, want):
        assert torch.equal(out, w)
