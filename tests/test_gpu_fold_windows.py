"""Folds by lanes per window: factors around each change of the number of lanes (9 times a power
of two) and of the loop unrolled over a lane's samples, phase bins that are no multiple of 32, row
counts around the 128 that are summed at a time, batches that exceed the scratch memory, and a
folded block that alone does."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _check(data, tsamp, folds):
    import riptide_b200 as rb
    from riptide_b200.folding import fold_batched

    ts = rb.TimeSeries(data, tsamp)
    got = fold_batched(ts, [p for p, _, _ in folds], [b for _, b, _ in folds],
                       [s for _, _, s in folds])
    for (p, b, s), y in zip(folds, got):
        ref = O.fold(data, tsamp, p, b, s)
        assert y.shape == ref.shape
        # both sides round sums of f + 2 samples (and of the rows) to float32; the oracle holds
        # the window sums in float32: f + 2 roundings of at most the window's magnitude, scaled by
        # (rows f)^-1/2, and one per row added
        f = p / b / tsamp
        rows = data.size * tsamp / p
        peak = np.abs(data).max() * (f + 2) / np.sqrt(rows * f)
        n = rows if s == 1 else (rows / s if s else 1)
        tol = 2.0 ** -24 * (f + 2 + n) * peak * max(1.0, n)
        np.testing.assert_allclose(y, ref, rtol=0, atol=tol)


FACTORS = [1.01, 2.3, 8.99, 9.0, 17.9, 18.1, 35.9, 36.1, 71.9, 72.1, 143.9, 144.1, 700.3]


@pytest.mark.parametrize("bins", [1, 31, 33, 100])
def test_fold_lane_edges(bins):
    n, tsamp = 300007, 1e-3
    data = np.random.default_rng(bins).standard_normal(n).astype(np.float32)
    folds = []
    for f in FACTORS:
        m = int(n / f) // bins
        for s in (1, None, max(1, m // 3), max(1, m - 1)):
            folds.append((f * bins * tsamp, bins, s))
    _check(data, tsamp, folds)


@pytest.mark.parametrize("rows", [1, 2, 127, 128, 129, 257])
def test_fold_row_counts(rows):
    bins, f, tsamp = 64, 3.7, 1e-3
    n = int(rows * bins * f) + 3
    data = np.random.default_rng(rows).standard_normal(n).astype(np.float32)
    _check(data, tsamp, [(f * bins * tsamp, bins, s) for s in (1, None)])


def test_fold_batches():
    import riptide_b200 as rb
    from riptide_b200.folding import fold, fold_batched

    # 1.9 million values a block: 17 of them fill the scratch memory
    n, tsamp, bins = 2000003, 1e-3, 64
    ts = rb.TimeSeries(np.random.default_rng(3).standard_normal(n).astype(np.float32), tsamp)
    periods = [tsamp * bins * (1.04 + 0.001 * k) for k in range(40)]
    subs = [(1, 7, None)[k % 3] for k in range(40)]
    for k, y in enumerate(fold_batched(ts, periods, bins, subs)):
        if k % 9 == 0 or k in (17, 18, 35):
            assert np.array_equal(y, fold(ts, periods[k], bins, subs[k])), k


def test_fold_large_block():
    n, tsamp, bins = 36000001, 1e-3, 4096
    data = np.random.default_rng(4).standard_normal(n).astype(np.float32)
    # 2^25 folded values and two rows more, and exactly that many
    for f in (1.0726, 1.0728):
        assert (int(n / f) // bins * bins > 1 << 25) == (f == 1.0726)
        _check(data, tsamp, [(f * bins * tsamp, bins, 1), (f * bins * tsamp, bins, 100)])
