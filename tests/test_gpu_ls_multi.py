"""The LS derivative kernels where a warp takes four frequencies at once: the
values equal the warp-per-frequency kernel's bit for bit (calls of under 64
frequencies take that one), on curve lengths and frequency counts around its
sets, one and several staged tiles, and the FP64 phase beyond the
split-precision range.  The backward kernel with one and two points per thread
against FP64."""

import numpy as np
import pytest

import lightcurves as lc

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("n_freq", [64, 65, 127, 130, 1025])
@pytest.mark.parametrize("span", [1.0, 4000.0])
def test_equals_warp_per_frequency(n_freq, span):
    from periodfind_b200 import ls_grad

    lengths = [1, 33, 64, 300, 2048, 2049, 4100]
    ts, ms, _, _ = lc.ls_study_curves(len(lengths), seed=n_freq, lengths=lengths)
    # span 4000: up to 20 cycles / day over 1.2e7 days, beyond 2^21 turns.
    ts = [(t * span).astype(np.float32) for t in ts]
    w = torch.from_numpy(2 * np.pi * np.geomspace(0.01, 20.0, n_freq)).cuda()
    off = np.zeros(len(ts) + 1, np.int64)
    np.cumsum(lengths, out=off[1:])
    t, y = (torch.from_numpy(np.concatenate(xs).astype(np.float32)).cuda() for xs in (ts, ms))
    for second in (False, True):
        whole = ls_grad.ls_derivatives(t, y, w, off, second)
        parts = [ls_grad.ls_derivatives(t, y, w[k:k + 40], off, second)
                 for k in range(0, n_freq, 40)]
        for j, got in enumerate(whole):
            if got is not None:
                assert torch.equal(got, torch.cat([p[j] for p in parts], dim=1)), j


@pytest.mark.parametrize("n_curves,length", [(3, 700), (950, 300)])
def test_backward_both_shapes(n_curves, length):
    """One point per thread (few CTAs) and two: dL/dy against FP64."""
    from periodfind_b200 import ls_grad

    rng = np.random.default_rng(n_curves)
    n_freq = 130
    t = np.sort(rng.uniform(0, 1000.0, (n_curves, length)), axis=1).astype(np.float32)
    y = rng.normal(0, 0.3, t.shape).astype(np.float32)
    w = 2 * np.pi * np.geomspace(0.05, 5.0, n_freq)
    g = rng.normal(size=(n_curves, n_freq)).astype(np.float32)
    off = np.arange(n_curves + 1, dtype=np.int64) * length
    tc, yc = (torch.from_numpy(a.reshape(-1)).cuda() for a in (t, y))
    yc.requires_grad_(True)
    p = ls_grad.ls_power(tc, yc, torch.from_numpy(w).cuda(), off)
    p.backward(torch.from_numpy(g).cuda())
    td = torch.from_numpy(t).cuda().double()
    td = td - 0.5 * (td.min(1, keepdim=True).values + td.max(1, keepdim=True).values)
    th = td[:, :, None] * torch.from_numpy(w).cuda()
    co, si = torch.cos(th), torch.sin(th)
    yd = torch.from_numpy(y).cuda().double()[:, :, None]
    C, S, CC, CS = (yd * co).sum(1), (yd * si).sum(1), (co * co).sum(1), (co * si).sum(1)
    SS = length - CC
    det = CC * SS - CS * CS
    gd = torch.from_numpy(g).cuda().double()
    al, be = gd * (SS * C - CS * S) / det, gd * (CC * S - CS * C) / det
    want = (co * al[:, None] + si * be[:, None]).sum(2)
    err = (yc.grad.view(n_curves, length) - want).abs().max() / want.abs().max()
    assert float(err) <= 2e-6
