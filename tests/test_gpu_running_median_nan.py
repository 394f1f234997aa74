"""Running medians of series that hold NaN: a NaN ranks after every number (as np.sort has it), in
the windows that hold it; every other window's median is exact."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _expected(x, width):
    half = width // 2
    w = np.lib.stride_tricks.sliding_window_view(np.pad(x, half, mode="edge"), width)
    return np.sort(w, axis=1)[:, half]


@pytest.mark.parametrize("width", [1, 3, 101, 129, 131, 257])
def test_running_median_nan(width):
    import riptide_b200 as rb

    rng = np.random.default_rng(width)
    for n in (512, 1000, 6786):
        for count in (1, 5, 200):
            for ties in (False, True):
                x = (rng.integers(-3, 4, n) if ties else rng.standard_normal(n)).astype(np.float32)
                at = rng.choice(n, count, replace=False)
                x[at] = np.nan
                x[at[1::2]] = -np.nan
                want = _expected(x, width)
                for _ in range(3):
                    got = rb.running_median(x, width)
                    assert np.array_equal(got, want, equal_nan=True), (n, count, ties)
    # only infinities around it, and a tile of nothing else
    x = np.full(700, -np.inf, dtype=np.float32)
    x[350:] = np.inf
    x[[3, 340, 360, 699]] = np.nan
    assert np.array_equal(rb.running_median(x, width), _expected(x, width), equal_nan=True)
    x = np.full(700, np.nan, dtype=np.float32)
    assert np.isnan(rb.running_median(x, width)).all()


def test_signed_zeros():
    # equal values: the one that comes first in the window's order of positions
    import riptide_b200 as rb
    from oracle import oracle as O

    rng = np.random.default_rng(0)
    x = rng.choice(np.array([-0.0, 0.0, 1.0, -1.0], dtype=np.float32), 2000)
    got = rb.running_median(x, 101)
    assert np.array_equal(got, O.C().running_median(x, 101))
    w = np.lib.stride_tricks.sliding_window_view(np.pad(x, 50, mode="edge"), 101)
    want = np.take_along_axis(w, np.argsort(w, axis=1, kind="stable"), axis=1)[:, 50]
    assert np.array_equal(np.signbit(got), np.signbit(want))
