"""Downsampling by factors whose multiples round up to the first sample of a segment (1.2 does so at
every segment of the kernel): the same bits on every call, whatever device and shared memory held
before, and the float64 window sums."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _poison(value):
    """Leaves `value` in free device memory, in L2 and in the SMs' caches."""
    import torch

    a = torch.full((1 << 26,), value, device="cuda")
    a.clone()
    torch.cuda.synchronize()
    del a
    torch.cuda.empty_cache()


def _windows(x, f):
    n = int(np.floor(x.size / f))
    k = np.arange(n, dtype=np.float64)
    start, end = k * f, k * f + f
    lo = np.floor(start).astype(np.int64)
    hi = np.minimum(np.floor(end), x.size - 1.0).astype(np.int64)
    c = np.concatenate([[0.0], np.cumsum(x.astype(np.float64))])
    return ((lo + 1) - start) * x[lo] + (c[hi] - c[lo + 1]) + (end - hi) * x[hi]


@pytest.mark.parametrize("f", [1.2, 1.44, 1.728, 2.0736, 1.1, 13.02])
@pytest.mark.parametrize("n", [60000, 3600000])
def test_same_bits_every_time(f, n):
    import torch

    import riptide_b200 as rb

    x = np.random.default_rng(n).standard_normal(n).astype(np.float32)
    ref = _windows(x, f)
    d = torch.from_numpy(x).cuda()
    first = rb.libcpp.downsample(d, f)
    # float32 weights and one rounding of a sum of f + 2 terms
    tol = 2.0 ** -24 * (2 + f + 2) * np.abs(x).max()
    assert np.abs(first.cpu().numpy() - ref).max() <= tol
    for value in (float("nan"), 3e30, -3e30, 1.0):
        _poison(value)
        for _ in range(10):
            assert torch.equal(rb.libcpp.downsample(d, f), first), value


def test_first_run_of_a_plan():
    # a search whose first cycles downsample by 1.2 and 1.44, in memory that held NaN
    import torch

    import riptide_b200 as rb

    n, trials = 60000, 60
    d = torch.randn(n * trials, device="cuda", generator=torch.Generator("cuda").manual_seed(3))
    kw = dict(period_min=0.02, period_max=0.16, bins_min=20, bins_max=23, widths=[1, 2, 3],
              deredden=False, already_normalised=True)
    runs = []
    for value in (0.0, float("nan"), 3e30):
        _poison(value)
        bs = rb.BatchedSearch([n] * trials, 1e-3, **kw)
        runs += [[t.clone() for t in bs.run(d)] for _ in range(4)]
        bs.close()
    for run in runs[1:]:
        assert all(torch.equal(a, b) for a, b in zip(run, runs[0]))
