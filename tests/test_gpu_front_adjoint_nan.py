"""rt_front_adjoint of series that hold NaN, without normalisation: every window's gradient goes to
the element that the forward selects, a NaN ranking after every number."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _expected(x, g, k, width):
    """float64 restatement: mean-scrunch, the selected element of each edge-padded window, np.interp's
    weights of every sample on the points around it."""
    n, half = x.size, width // 2
    nl = n // k
    lores = x[:nl * k].astype(np.float64).reshape(nl, k).mean(axis=1)
    pos = (np.arange(n) - 0.5 * (k - 1)) / k
    j = np.clip(np.floor(pos), 0, nl - 1).astype(int)
    a = np.where((pos < 0) | (pos >= nl - 1), 0.0, pos - j)
    glo = np.zeros(nl)
    np.add.at(glo, j, g * (1.0 - a))
    np.add.at(glo, np.minimum(j + 1, nl - 1), g * a)
    win = np.lib.stride_tricks.sliding_window_view(np.pad(lores, half, mode="edge"), width)
    sel = np.argsort(win, axis=1, kind="stable")[:, half] + np.arange(nl) - half
    gsel = np.zeros(nl)
    np.add.at(gsel, np.clip(sel, 0, nl - 1), glo)
    out = g.astype(np.float64)
    out[:nl * k] -= np.repeat(gsel / k, k)
    return out


@pytest.mark.parametrize("k,width", [(1, 3), (1, 101), (3, 11), (2, 257)])
@pytest.mark.parametrize("count", [1, 7, 60])
def test_front_adjoint_nan(k, width, count):
    import torch

    from riptide_b200 import _lib, libcpp

    rng = np.random.default_rng(k + width + count)
    lengths = np.array([900, 1500], dtype=np.uint64)
    n = int(lengths.sum())
    x, g = ((3 * rng.standard_normal(n)).astype(np.float32) for _ in range(2))
    x[rng.choice(n, count, replace=False)] = np.nan
    dx, dg = (torch.from_numpy(v).cuda() for v in (x, g))
    want, a = [], 0
    for L in lengths.astype(int):
        want.append(_expected(x[a:a + L], g[a:a + L], k, width))
        a += L
    want = np.concatenate(want)
    # float64 sums rounded to float32 twice
    tol = 4 * 2.0 ** -24 * np.abs(want).max()
    for _ in range(3):
        got = torch.empty_like(dg)
        _lib.check(_lib.load().rt_front_adjoint(
            libcpp._ptr(dx), None, libcpp._ptr(dg), lengths.ctypes.data_as(_lib._u64p), 2, None,
            k * width, width, libcpp._ptr(got), libcpp._stream()))
        assert np.abs(got.cpu().numpy() - want).max() <= tol
