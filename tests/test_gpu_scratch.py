"""Entry points that take device scratch or pass their descriptors by value, called without a
synchronisation in between: on several streams and threads, on tensors that another stream owns
and that are dropped right after the call."""
import threading

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _work(rb, seed):
    """Calls on one stream, results kept on the device; (got, expected) pairs."""
    import torch

    rng = np.random.default_rng(seed)
    pairs = []
    for m, b in ((300, 251), (1342, 240), (97, 61)):
        x = rng.standard_normal((m, b)).astype(np.float32)
        pairs.append((rb.libcpp.ffa2(torch.from_numpy(x).cuda()), O.C().ffa2(x)))
        w = rb.generate_width_trials(min(b, 100))
        pairs.append((rb.libcpp.snr2(torch.from_numpy(x).cuda(), w, 1.5), O.C().snr2(x, w, 1.5)))
    y = rng.standard_normal(50003 + seed).astype(np.float32)
    pairs.append((rb.libcpp.running_median(torch.from_numpy(y).cuda(), 101),
                  O.C().running_median(y, 101)))
    pairs.append((rb.fast_running_median(torch.from_numpy(y).cuda(), 2001, 101),
                  O.fast_running_median(y, 2001, 101)))
    return pairs


def test_streams_and_threads():
    import torch

    import riptide_b200 as rb

    out = {}

    def run(i):
        with torch.cuda.stream(torch.cuda.Stream()):
            out[i] = [_work(rb, 10 * i + k) for k in range(3)]
            torch.cuda.current_stream().synchronize()

    threads = [threading.Thread(target=run, args=(i,)) for i in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for i in range(3):
        for pairs in out[i]:
            for got, want in pairs:
                assert np.array_equal(got.cpu().numpy(), want)
    rb._lib.check(rb._lib.load().rt_release_scratch())
    for got, want in _work(rb, 99):
        assert np.array_equal(got.cpu().numpy(), want)


def test_input_of_another_stream_dropped_after_the_call():
    # the input belongs to the default stream and is freed as soon as the call returns; what the
    # default stream then allocates must not be written before the side stream has read it
    import torch

    import riptide_b200 as rb

    rng = np.random.default_rng(3)
    x = rng.standard_normal((16001, 251)).astype(np.float32)
    want = O.C().ffa2(x)
    side = torch.cuda.Stream()
    for _ in range(5):
        t = torch.from_numpy(x).cuda()
        torch.cuda.synchronize()
        with torch.cuda.stream(side):
            y = rb.libcpp.ffa2(t)
        shape = t.shape
        del t
        junk = [torch.full(shape, 7.0, device="cuda") for _ in range(4)]
        side.synchronize()
        assert np.array_equal(y.cpu().numpy(), want)
        del junk
