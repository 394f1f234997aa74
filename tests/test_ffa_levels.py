"""The FFA job levels (csrc/ffa_core.cuh): the row-number pattern that the row groups and quads
rely on, and the transforms at the sizes where a level changes its loop -- fewer than 17 bins
(plain loop), 8 / 16 / 32 column chunks of a row (one, two or four groups a warp) and more
(several warp tasks a row), subtrees of 4 to 8 rows, one and several stages."""
import numpy as np
import pytest

from oracle import oracle as O


def _rows(n):
    """h(s), t(s) of a node of n rows, as the kernels round them (transforms.hpp:17-24)."""
    mh = n >> 1
    den = np.float32(n - 1)
    kh = np.float64(np.float32(mh - 1) / den)
    kt = np.float64(np.float32(n - mh - 1) / den)
    s = np.arange(n)
    # one rounding of the exact k * s + 0.5: the product is exact in float64
    return ((kh * s + 0.5).astype(np.float32).astype(np.int64),
            (kt * s + 0.5).astype(np.float32).astype(np.int64))


def test_row_pattern():
    # every node size for which the kernels use it (kRegularRows)
    for n in range(2, 8193):
        h, t = _rows(n)
        s = np.arange(n)
        p = n & 1
        assert np.array_equal(t, (s + p) >> 1), n
        half = (n >> 1) & ~1
        thr = (half if h[half] == half // 2 else half - 2) if p else n
        assert np.array_equal(h, (s >> 1) - ((s > thr) & (s % 2 == 0))), n


EDGE_BINS = [2, 9, 16, 17, 18, 61, 62, 133, 134, 277, 278, 288, 289, 565, 566, 4096]


@pytest.mark.gpu
@pytest.mark.parametrize("b", EDGE_BINS)
def test_ffa2_level_edges(b):
    import riptide_b200 as rb

    rng = np.random.default_rng(b)
    for m in (3, 4, 5, 6, 7, 8, 9, 16, 31, 33, 64, 65, 127, 129, 257, 511):
        if m * b > 600000:
            continue
        x = rng.standard_normal((m, b)).astype(np.float32)
        assert np.array_equal(rb.libcpp.ffa2(x), O.C().ffa2(x)), (m, b)


@pytest.mark.gpu
@pytest.mark.parametrize("bmin,bmax,n,tsamp", [
    (13, 19, 30000, 1e-2),       # plain loops below 17 bins, groups from there
    (60, 64, 150000, 4e-3),      # 8 chunks and more
    (130, 136, 300000, 2e-3),    # 16 chunks and more
    (240, 260, 400000, 1e-3),    # the first cycle folds the series itself
    (262, 268, 400000, 1e-3),    # 8 and 16 S/N threads in one plan
    (274, 292, 400000, 1e-3),    # one and two warp tasks a row
    (556, 570, 700000, 5e-4),    # S/N prefix passes unrolled and looped
])
def test_search_level_edges(bmin, bmax, n, tsamp):
    # the persistent kernel against the C restatement on the same normalised series; the peak is
    # compared by its S/N (equal maxima may tie)
    import riptide_b200 as rb

    rng = np.random.default_rng(n)
    x = rb.generate_signal(n, 2.3 * bmin, ducy=0.05, amplitude=20.0, rng=rng)
    x = O.normalise(x).astype(np.float32)
    w = O.generate_width_trials(bmin)
    args = (x, tsamp, w, bmin * tsamp, min(25.0 * bmin * tsamp, n * tsamp / 9), bmin, bmax)
    p, fb, s = rb.libcpp.periodogram(*args)
    rp, rfb, rs = O.C().periodogram(*args)
    assert np.array_equal(p, rp) and np.array_equal(fb, rfb)
    assert np.allclose(s, rs, rtol=1e-5, atol=2e-5)


def test_head_row_threshold():
    # an odd node's even rows s > (n / 2 rounded down to even) have h(s) = s / 2 - 1, no others
    for n in range(3, 8193, 2):
        h, _ = _rows(n)
        s = np.arange(0, n, 2)
        assert np.array_equal(h[s], (s >> 1) - (s > ((n >> 1) & ~1))), n
