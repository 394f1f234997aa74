"""ffa2 of blocks of a thousand jobs and more (the persistent kernel): rows of whole 16-byte units
and others, blocks that start off a 16-byte boundary, few and many bins, several streams at once."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,b", [(33000, 250), (33001, 251), (9000, 1000), (8191, 1001),
                                 (300001, 24), (120000, 9)])
def test_ffa2_large(m, b):
    import torch

    import riptide_b200 as rb

    x = np.random.default_rng(m).standard_normal((m + 1, b)).astype(np.float32)
    dev = torch.from_numpy(x).cuda()
    for first in (0, 1):  # the second one starts b floats into the allocation
        ref = O.C().ffa2(x[first:first + m])
        assert np.array_equal(rb.libcpp.ffa2(dev[first:first + m]).cpu().numpy(), ref), first


def test_ffa2_large_streams():
    import torch

    import riptide_b200 as rb

    x = torch.randn(3, 33000, 250, device="cuda")
    want = [rb.libcpp.ffa2(x[i]) for i in range(3)]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(3)]
    got = []
    for rep in range(3):
        for i, st in enumerate(streams):
            with torch.cuda.stream(st):
                got.append((i, rb.libcpp.ffa2(x[i])))
    torch.cuda.synchronize()
    for i, y in got:
        assert torch.equal(y, want[i])
