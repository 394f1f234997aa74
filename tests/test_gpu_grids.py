"""How calls are spread over the SMs, at the sizes where the rule changes: the boxcar S/N with
0, 1 and several warps of profiles a CTA; transforms of few jobs, split into jobs of half the rows
while that takes no further stage; series short enough for the small downsampling segments."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bins,per_warp", [(64, 8), (250, 4), (400, 2), (700, 1)])
def test_snr_rows_per_cta(bins, per_warp):
    import riptide_b200 as rb

    widths = np.array([1, 2, 3, 9, 20])
    rng = np.random.default_rng(bins)
    edge = 148 * per_warp
    for rows in (1, per_warp + 1, edge - 1, edge, edge + 1, 2 * edge + 1):
        x = rng.standard_normal((rows, bins)).astype(np.float32)
        # a few float32 roundings of terms below 100 (|sum of a row| < 5 sqrt(bins))
        ref = O.C().snr2(x.astype(np.float64), widths, 1.0, f64=True)
        np.testing.assert_allclose(rb.libcpp.snr2(x, widths, 1.0), ref, rtol=0,
                                   atol=16 * 100 * 2.0 ** -24)


@pytest.mark.parametrize("b", [24, 133, 251, 500])
def test_ffa2_few_jobs(b):
    import riptide_b200 as rb

    rng = np.random.default_rng(b)
    for m in (1000 // (b // 24), 70000 // b, 200000 // b, 1500000 // b, 4000000 // b + 1):
        x = rng.standard_normal((m, b)).astype(np.float32)
        assert np.array_equal(rb.libcpp.ffa2(x), O.C().ffa2(x)), (m, b)


# segments of 1,024 samples for factors up to 254 and at most 128 CTAs of the large shape, each
# 8,192 samples less a halo of the factor + 2 in whole warps
@pytest.mark.parametrize("factor,nsamp", [(1.5, 1000), (4.1, 1044480), (4.1, 1044481),
                                          (253.5, 300001), (254.5, 300001)])
def test_downsample_segments(factor, nsamp):
    import riptide_b200 as rb

    x = np.random.default_rng(nsamp).standard_normal(nsamp).astype(np.float32)
    # sums of factor + 2 terms, in float64 on the device and in float32 in the oracle
    tol = 2.0 ** -24 * (factor + 2) ** 2 * np.abs(x).max()
    np.testing.assert_allclose(rb.libcpp.downsample(x, factor), O.C().downsample(x, factor),
                               rtol=0, atol=tol)
