"""Folds against float64 sums of the same windows, within the roundings that the device makes: a
window's sum, the scale and their product to float32, then one rounding per row added (or one for a
column's window). The bound of every output value is summed from the values themselves, so it stays
far below them. With room for the folded blocks (two kernels) and without (one, a scratch allocation
that fails, injected on the host)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -24


def _windows(x, f, n):
    """Sums of n windows of f values along axis 0 and of their magnitudes (downsample.hpp:44-82)."""
    k = np.arange(n, dtype=np.float64)
    start = k * f
    end = start + f
    lo = np.floor(start).astype(np.int64)
    hi = np.minimum(np.floor(end), x.shape[0] - 1.0).astype(np.int64)
    wlo = ((lo + 1) - start).astype(np.float32).astype(np.float64)
    whi = (end - hi).astype(np.float32).astype(np.float64)
    shape = (n,) + (1,) * (x.ndim - 1)
    out = []
    for v in (x, np.abs(x)):
        c = np.concatenate([np.zeros_like(v[:1]), np.cumsum(v, axis=0)])
        out.append(wlo.reshape(shape) * v[lo] + (c[hi] - c[lo + 1]) + whi.reshape(shape) * v[hi])
    return out


def _fold(x, tsamp, period, bins, subints):
    """(values, bound) of a fold, in float64."""
    f = period / bins / tsamp
    n = int(np.floor(x.size / f))
    m = n // bins
    y, mag = _windows(x.astype(np.float64), f, m * bins)
    scale = float(np.float32((m * f) ** -0.5))
    y, mag = (y * scale).reshape(m, bins), (mag * scale).reshape(m, bins)
    # (float64 sums, here by differences of running sums: below 2^-36 of the magnitudes)
    err = 2 * EPS * np.abs(y) * 1.01 + 2.0 ** -36 * mag
    if subints == 1 or m == 1:
        partial = np.abs(np.cumsum(y, axis=0))
        return y.sum(axis=0), err.sum(axis=0) + EPS * 1.01 * partial.sum(axis=0)
    if subints is None or subints == m:
        return y, err
    vf = m / subints
    out, _ = _windows(y, vf, int(np.floor(m / vf)))
    bound, _ = _windows(err, vf, int(np.floor(m / vf)))
    return out, bound + EPS * 1.01 * np.abs(out)


@pytest.fixture(params=[True, False], ids=["room", "no room"])
def room(request):
    from riptide_b200 import _lib

    yield lambda: _lib.check(_lib.load().rt_inject_scratch_fault(0 if request.param else 1))
    _lib.check(_lib.load().rt_inject_scratch_fault(0))


def _check(room, data, tsamp, folds):
    import riptide_b200 as rb
    from riptide_b200.folding import fold_batched

    ts = rb.TimeSeries(data, tsamp)
    room()
    got = fold_batched(ts, [p for p, _, _ in folds], [b for _, b, _ in folds],
                       [s for _, _, s in folds])
    for (p, b, s), y in zip(folds, got):
        ref, bound = _fold(data, tsamp, p, b, s)
        assert y.shape == ref.shape, (p, b, s)
        assert bound.max() < 0.01 * np.abs(ref).max(), (p, b, s)
        assert (np.abs(y - ref) <= bound).all(), (p, b, s)


FACTORS = [1.01, 2.3, 8.99, 9.0, 17.9, 18.1, 35.9, 36.1, 71.9, 72.1, 143.9, 144.1, 700.3]


@pytest.mark.parametrize("bins", [1, 31, 33, 100])
def test_lane_edges(room, bins):
    n, tsamp = 300007, 1e-3
    data = np.random.default_rng(bins).standard_normal(n).astype(np.float32)
    folds = []
    for f in FACTORS:
        m = int(n / f) // bins
        for s in (1, None, max(1, m // 3), max(1, m - 1)):
            folds.append((f * bins * tsamp, bins, s))
    _check(room, data, tsamp, folds)


@pytest.mark.parametrize("rows", [1, 2, 127, 128, 129, 257])
def test_row_counts(room, rows):
    bins, f, tsamp = 64, 3.7, 1e-3
    n = int(rows * bins * f) + 3
    data = np.random.default_rng(rows).standard_normal(n).astype(np.float32)
    _check(room, data, tsamp, [(f * bins * tsamp, bins, s) for s in (1, None)])


@pytest.mark.parametrize("f,injected", [(1.0726, 0), (1.0728, 0), (1.0728, 1)])
def test_large_block(f, injected):
    # 2^25 folded values and two rows more, which take no scratch memory, and exactly that many
    from riptide_b200 import _lib

    n, tsamp, bins = 36000001, 1e-3, 4096
    data = np.random.default_rng(4).standard_normal(n).astype(np.float32)
    _check(lambda: _lib.check(_lib.load().rt_inject_scratch_fault(injected)), data, tsamp,
           [(f * bins * tsamp, bins, 1 if injected else 100)])
