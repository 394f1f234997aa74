"""The segment statistics of the peak search select order statistics by histograms of the values'
span: columns where a span has to be divided again (ties, one value, two values, values over many
decades and signs, an infinite one), the smallest and largest segments, and numbers of widths that
take one or several groups, against numpy's percentiles."""
import ctypes

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _columns(rng, n, nw):
    s = np.empty((n, nw), dtype=np.float32)
    for c in range(nw):
        k = c % 8
        x = 2.5 + 0.25 * rng.standard_normal(n)
        if k == 1:
            x = np.round(x, 1)
        elif k == 2:
            x = np.full(n, 3.25)
        elif k == 3:
            x = np.where(rng.random(n) < 0.5, -1e30, 1e-30)
        elif k == 4:
            x = np.sign(rng.standard_normal(n)) * 10.0 ** rng.uniform(-40, 38, n)
        elif k == 5:
            x[:: max(1, n // 3)] = 1e6
        elif k == 6:
            x[0] = np.inf if n > 8 else 1.0
        elif k == 7:
            x = rng.standard_normal(n)
        s[:, c] = x
    return s


@pytest.mark.parametrize("p,nw", [(1, 10), (2, 3), (9, 17), (37, 40), (129, 8), (1174, 10),
                                  (2350, 12), (16384, 9)])
def test_segment_selection(p, nw):
    import torch

    from riptide_b200 import _lib, libcpp

    rng = np.random.default_rng(p * 41 + nw)
    T, m = 100.0, 7
    n = m * p + min(p, 3) - 1
    f = np.linspace(3.0, 3.0 - 5.0 * (m - 0.5) / T, n)
    at = rng.integers(1, n - 2, n // 4) if n > 8 else np.empty(0, dtype=int)
    f[at], f[at + 1] = f[at + 1].copy(), f[at].copy()  # bins of a search overlap a little
    periods = 1.0 / f
    snrs = _columns(rng, n, nw)
    per, snr = torch.from_numpy(periods).cuda(), torch.from_numpy(snrs).cuda()
    rows = np.array([0, n], dtype=np.uint64)
    tobs, off = np.array([T]), np.zeros(2, dtype=np.uint64)
    fc = torch.empty(m, dtype=torch.float64, device="cuda")
    sc = torch.empty((m, nw), dtype=torch.float64, device="cuda")
    dp = ctypes.POINTER(ctypes.c_double)
    _lib.check(_lib.load().rt_peak_segments(
        libcpp._ptr(per), libcpp._ptr(snr), nw, rows.ctypes.data_as(_lib._u64p), 1,
        tobs.ctypes.data_as(dp), 5.0, 6.0, off.ctypes.data_as(_lib._u64p), libcpp._ptr(fc),
        libcpp._ptr(sc), libcpp._stream()))
    assert int(off[1]) == m
    fc, sc = fc.cpu().numpy(), sc.cpu().numpy()
    for iw in range(nw):
        fr, smed, sstd = O.segment_stats(1.0 / periods, snrs[:, iw].astype(float), T)
        assert np.array_equal(fc, fr)
        assert np.array_equal(sc[:, iw], smed + 6.0 * sstd), iw
