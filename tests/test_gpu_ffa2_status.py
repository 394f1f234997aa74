"""ffa2 of large blocks whose bounded wait runs out (a later stage waits for one job more than the
stage before has, injected on the host): the status says so, the result is NaN, and the numpy entry
point raises; the next call is right again."""
import ctypes

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

M, B = 33000, 250  # enough jobs for the persistent kernel


def _status(x, polls, fault):
    import torch

    from riptide_b200 import _lib, libcpp

    out = torch.zeros_like(x)
    status = torch.full((1,), -1, dtype=torch.int32, device="cuda")
    _lib.check(_lib.load().rt_ffa2_status(libcpp._ptr(x), x.shape[0], x.shape[1], libcpp._ptr(out),
                                          libcpp._ptr(status), polls, fault, libcpp._stream()))
    return out, int(status.item())


def test_wait_that_runs_out():
    import torch

    from riptide_b200 import _lib, libcpp

    x = np.random.default_rng(1).standard_normal((M, B)).astype(np.float32)
    d = torch.from_numpy(x).cuda()
    want = O.C().ffa2(x)
    out, status = _status(d, 0, _lib.RT_FAULT_NONE)
    assert status == _lib.RT_OK and np.array_equal(out.cpu().numpy(), want)
    out, status = _status(d, 20000, _lib.RT_FAULT_STAGE_WAIT)
    assert status == _lib.RT_ETIMEOUT and bool(torch.isnan(out).all())
    out, status = _status(d, 0, _lib.RT_FAULT_NONE)
    assert status == _lib.RT_OK and np.array_equal(out.cpu().numpy(), want)
    assert np.array_equal(libcpp.ffa2(d).cpu().numpy(), want)


def test_numpy_entry_point_raises(monkeypatch):
    from riptide_b200 import _lib, libcpp

    x = np.random.default_rng(2).standard_normal((M, B)).astype(np.float32)
    lib = _lib.load()
    real = lib.rt_ffa2_status

    class Faulty(object):
        def __getattr__(self, name):
            return getattr(lib, name)

        @staticmethod
        def rt_ffa2_status(i, r, c, o, s, polls, fault, stream):
            return real(i, r, c, o, s, 20000, _lib.RT_FAULT_STAGE_WAIT, stream)

    with monkeypatch.context() as mp:
        mp.setattr(_lib, "_lib", Faulty())
        with pytest.raises(_lib.RiptideError, match="bounded wait"):
            libcpp.ffa2(x)
    assert np.array_equal(libcpp.ffa2(x), O.C().ffa2(x))


@pytest.mark.parametrize("m,b", [(0, 250), (1, 250), (300, 251), (97, 9)])
def test_status_of_small_blocks(m, b):
    import torch

    from riptide_b200 import _lib

    x = np.random.default_rng(m).standard_normal((m, b)).astype(np.float32)
    out, status = _status(torch.from_numpy(x).cuda(), 0, _lib.RT_FAULT_NONE)
    assert status == _lib.RT_OK
    if m:
        assert np.array_equal(out.cpu().numpy(), O.C().ffa2(x))


def test_bad_arguments():
    import torch

    from riptide_b200 import _lib, libcpp

    x = torch.zeros(4, 8, device="cuda")
    s = torch.zeros(1, dtype=torch.int32, device="cuda")
    f = _lib.load().rt_ffa2_status
    for status, polls, fault in ((None, 0, 0), (libcpp._ptr(s), -1, 0), (libcpp._ptr(s), 0, 2)):
        assert f(libcpp._ptr(x), 4, 8, libcpp._ptr(x), status, polls, fault,
                 ctypes.c_void_p(0)) == _lib.RT_EINVAL
