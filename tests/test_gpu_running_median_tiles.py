"""The stages before the search at the edges of their tiles: running medians of narrow and wide
tiles with ties and infinities, scrunch factors of one to 32 leaves with few and many points per
warp, interpolation spans. All bit for bit against the C restatement / numpy."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width", [1, 3, 7, 101, 127, 129, 131, 255, 257, 259])
def test_running_median_tile_edges(width):
    import riptide_b200 as rb

    rng = np.random.default_rng(width)
    for n in (width + 1, 128, 129, 256, 257, 511, 1000):
        if n <= width:
            continue
        x = rng.integers(-9, 10, n).astype(np.float32)  # many ties
        assert np.array_equal(rb.running_median(x, width), O.C().running_median(x, width)), n
        x = rng.standard_normal(n).astype(np.float32)
        x[rng.integers(0, n, 5)] = np.inf
        x[rng.integers(0, n, 5)] = -np.inf
        assert np.array_equal(rb.running_median(x, width), O.C().running_median(x, width)), n


@pytest.mark.parametrize("k", [2, 7, 8, 9, 127, 128, 129, 618, 1000, 4095, 4096])
def test_scrunch_and_interpolation(k):
    import riptide_b200 as rb

    rng = np.random.default_rng(k)
    minpts = 11
    for points in (13, 300):
        x = (rng.standard_normal(points * k + k // 2) * 3 + 100).astype(np.float32)
        assert np.array_equal(rb.fast_running_median(x, k * minpts, minpts),
                              O.fast_running_median(x, k * minpts, minpts)), points
