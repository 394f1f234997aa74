"""ffa2 and benchmark_ffa2 without room for the scratch memory that it would like to have (a scratch allocation that
fails, injected on the host): a launch per stage instead of the persistent kernel, an error where
there is no other way, and the next call as before."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture
def no_room():
    from riptide_b200 import _lib

    def inject(nth):
        _lib.check(_lib.load().rt_inject_scratch_fault(nth))

    yield inject
    inject(0)


@pytest.mark.parametrize("m,b", [(33000, 250), (120000, 9), (9000, 1000)])
def test_ffa2_by_stages(no_room, m, b):
    import torch

    from riptide_b200 import libcpp

    x = np.random.default_rng(m).standard_normal((m, b)).astype(np.float32)
    d = torch.from_numpy(x).cuda()
    want = O.C().ffa2(x)
    for nth in (1, 0):
        no_room(nth)
        assert np.array_equal(libcpp.ffa2(d).cpu().numpy(), want)
        no_room(nth)
        assert np.array_equal(libcpp.ffa2(x), want)


def test_ffa2_without_room(no_room):
    from riptide_b200 import libcpp

    x = np.random.default_rng(0).standard_normal((300, 251)).astype(np.float32)
    no_room(1)
    with pytest.raises(MemoryError):
        libcpp.ffa2(x)
    assert np.array_equal(libcpp.ffa2(x), O.C().ffa2(x))


def test_benchmark_ffa2(no_room):
    # by stages where the persistent kernel's copies find no room; nothing is left allocated
    import torch

    from riptide_b200 import _lib, libcpp

    assert libcpp.benchmark_ffa2(33000, 250, 2) > 0
    torch.cuda.synchronize()
    _lib.check(_lib.load().rt_release_scratch())
    free = torch.cuda.mem_get_info()[0]
    no_room(1)
    assert libcpp.benchmark_ffa2(33000, 250, 2) > 0
    no_room(1)
    with pytest.raises(MemoryError):
        libcpp.benchmark_ffa2(300, 251, 2)
    torch.cuda.synchronize()
    _lib.check(_lib.load().rt_release_scratch())
    assert abs(torch.cuda.mem_get_info()[0] - free) <= 2 << 20
