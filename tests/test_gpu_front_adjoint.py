"""rt_front_adjoint (normalise and deredden adjoints of a batch) against the torch restatement
of both steps, at the edges of its tiles: scrunch factors 1 and up, windows of one and more
tiles, end points, uneven lengths. float64 sums in another order, rounded to float32 twice: a
few float32 roundings of the largest gradient."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width,minpts,lengths", [
    (0, 0, [1000, 77]),                    # normalise only
    (21, 21, [400, 129, 257]),             # no scrunching
    (300, 101, [700, 5003]),               # factor 2
    (1010, 101, [1100, 12345, 30001]),     # factor 10, windows nearly as long as the series
    (2 * 257 * 3, 257, [9000, 2400]),      # the widest window
    (3 * 128, 3, [128 * 130, 128 * 4 + 127]),
])
@pytest.mark.parametrize("normalise", [True, False])
def test_front_adjoint(width, minpts, lengths, normalise):
    import torch

    from riptide_b200 import _lib, grad, libcpp

    rng = np.random.default_rng(width + minpts)
    n = int(sum(lengths))
    # distinct scrunched means: which element a tied median selects is not defined
    x, z, g = (torch.from_numpy((3 * rng.standard_normal(n)).astype(np.float32)).cuda() for _ in range(3))
    stds = rng.uniform(0.5, 2.0, len(lengths))
    want, a = torch.empty_like(g), 0
    for L, s in zip(lengths, stds):
        sl = slice(a, a + L)
        gy = g[sl].clone()
        if normalise:
            zd, gd = z[sl].double(), g[sl].double()
            gy = ((gd - gd.mean() - zd * (gd * zd).mean()) / s).float()
        want[sl] = gy - grad._rmed_adjoint(x[sl], gy, width, minpts) if minpts else gy
        a += L
    got = torch.empty_like(g)
    dbl = ctypes.POINTER(ctypes.c_double)
    lens = np.asarray(lengths, dtype=np.uint64)
    if not (normalise or minpts):
        pytest.skip("nothing to do")
    _lib.check(_lib.load().rt_front_adjoint(
        libcpp._ptr(x), libcpp._ptr(z), libcpp._ptr(g), lens.ctypes.data_as(_lib._u64p), len(lengths),
        stds.ctypes.data_as(dbl) if normalise else None, width, minpts, libcpp._ptr(got),
        libcpp._stream()))
    # up to `width` gradients meet in one element, divided by the scrunch factor
    tol = 4 * 2.0 ** -24 * float(want.abs().max())
    assert float((got - want).abs().max()) <= tol
    rc = _lib.load().rt_front_adjoint(
        libcpp._ptr(x), libcpp._ptr(z), libcpp._ptr(g), lens.ctypes.data_as(_lib._u64p), len(lengths),
        None, 259, 259, libcpp._ptr(got), libcpp._stream())
    assert rc == _lib.RT_EINVAL
