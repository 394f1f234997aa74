"""Bounds of a plan's memory, by arithmetic on the host. Shared memory: the boxcar S/N of the search
kernel reads whole segments of 33 phases, past the end of a row, for whatever number of threads the
plan may give a profile; the last row of a full level buffer is the one that could leave the CTA's
shared memory. Device memory: the ring of stage outputs."""
import numpy as np
import pytest

from oracle import oracle as O


def _stride(b):
    """Floats from one level row to the next: columns and 11 of halo in whole chunks of nine."""
    return (-(-(b + 11) // 9) * 9 + 3) // 4 * 4


def _threads(b, tuned):
    default = 4 if b <= 132 else 8 if b <= 264 else 16 if b <= 528 else 32
    return {default, 16} if tuned and b <= 528 else {default}


def _last_read(mem, b, tpr):
    """Byte after the last one read by the S/N of a level buffer full of rows, the second one."""
    rows = mem["buffer_bytes"] // 4 // _stride(b)
    row = _stride(b) * 4
    return mem["ops_bytes"] + mem["buffer_bytes"] + (rows - 1) * row + max(row, 4 * 33 * tpr)


def _plan(bmin, bmax, n=None, **kw):
    from riptide_b200 import BatchedSearch

    return BatchedSearch([n or 12000 * bmin], 1e-3, period_min=1e-3 * bmin, period_max=8e-3 * bmin,
                         bins_min=bmin, bins_max=bmax, widths=[1], deredden=False, **kw)


TUNED = [({}, False), ({"tuning": {"snr_threads": 16}}, True),
         ({"rules": [{"rows_min": 1, "rows_max": 1 << 20, "bins_min": 1, "bins_max": 4096,
                      "snr_threads": 16}]}, True)]


@pytest.mark.parametrize("kw,tuned", TUNED)
@pytest.mark.parametrize("rows", [200, 12000])
def test_snr_reads_stay_in_shared_memory(rows, kw, tuned):
    for bmin in list(range(2, 100, 5)) + list(range(100, 1057, 21)):
        for bmax in (bmin + max(1, bmin // 12), 2 * bmin):
            bs = _plan(bmin, bmax, n=rows * bmin, **kw)
            mem = bs.memory()
            bs.close()
            assert mem["ops_bytes"] + 2 * mem["buffer_bytes"] <= mem["shared_bytes"]
            for b in range(bmin, min(bmax, 1056) + 1):
                for tpr in _threads(b, tuned):
                    if b <= 33 * tpr:
                        assert _last_read(mem, b, tpr) <= mem["shared_bytes"], (bmin, bmax, b, tpr)


def _transforms(bs):
    import ctypes

    from riptide_b200 import _lib

    arr = (_lib.SearchTransform * bs.stats["num_transforms"])()
    _lib.check(_lib.load().rt_search_plan_transforms(bs._plan, ctypes.cast(arr, ctypes.c_void_p)))
    return arr


# the outputs of the stages take a slot of two copies for each transform of several stages, in a power
# of two up to 256
@pytest.mark.parametrize("bmin,bmax,n,trials", [
    (20, 22, 1 << 26, 1), (20, 23, 1 << 20, 40), (240, 260, 1 << 22, 4), (240, 260, 1 << 16, 1)])
def test_stage_ring_slots(bmin, bmax, n, trials):
    from riptide_b200 import BatchedSearch

    bs = BatchedSearch([n] * trials, 1e-3, period_min=1e-3 * bmin, period_max=4e-3 * bmin,
                       bins_min=bmin, bins_max=bmax, widths=[1], deredden=False)
    try:
        mem, multi = bs.memory(), bs.stats["num_multistage"]
        most = max(4 * t.rows * _stride(t.bins) for t in _transforms(bs))
        assert mem["ring_slots"] == min(256, 1 << max(0, multi - 1).bit_length())
        assert mem["ring_slot_bytes"] <= 2 * most
    finally:
        bs.close()


# no room for all of the ring (injected on the host): fewer slots, the same periodograms
@pytest.mark.gpu
@pytest.mark.parametrize("bmin,bmax,n", [(20, 23, 60000), (2, 4, 9000)])
def test_less_room_for_the_ring(bmin, bmax, n):
    import torch

    import riptide_b200 as rb

    rng = np.random.default_rng(n)
    trials = 60
    x = rng.standard_normal((trials, n)).astype(np.float32)
    w = [1] if bmin < 4 else [1, 2, 3]
    lim = (1e-3 * bmin, 8e-3 * bmin)
    kw = dict(period_min=lim[0], period_max=lim[1], bins_min=bmin, bins_max=bmax, widths=w,
              deredden=False, already_normalised=True)
    bs = rb.BatchedSearch([n] * trials, 1e-3, **kw)
    assert bs.stats["num_multistage"] > 256 == bs.memory()["ring_slots"]
    d = torch.from_numpy(x.ravel()).cuda()
    want = [t.clone() for t in bs.run(d)]
    off = bs.row_offsets
    for t in (0, 17, trials - 1):
        p, fb, s = [v[off[t]:off[t + 1]].cpu().numpy() for v in want]
        rp, rfb, rs = O.C().periodogram(x[t], 1e-3, np.array(w), *lim, bmin, bmax)
        assert np.array_equal(p, rp) and np.array_equal(fb, rfb)
        assert np.allclose(s, rs, rtol=1e-5, atol=2e-5), t
    for room, slots in ((255, 128), (40, 32), (1, 1), (3, 2), (256, 256)):
        bs.inject_fault("ring", room)
        got = bs.run(d)
        assert bs.memory()["ring_slots"] == slots
        assert all(torch.equal(a, b) for a, b in zip(got, want))
    bs.inject_fault("ring", 100)
    bs.inject_fault("alloc", 5)
    with pytest.raises(MemoryError):
        bs.run(d)
    bs.inject_fault(None)
    assert all(torch.equal(a, b) for a, b in zip(bs.run(d), want))
    bs.close()


# bins and threads whose reads leave the smallest room behind the second buffer, with the rows of
# their level buffers filled exactly: transforms of one stage
@pytest.mark.gpu
@pytest.mark.parametrize("bmin,bmax,threads", [(89, 97, 16), (82, 97, 16), (128, 140, 16),
                                               (520, 556, 0), (529, 548, 0), (20, 24, 16)])
def test_full_level_buffers(bmin, bmax, threads):
    import torch

    import riptide_b200 as rb

    kw = {"tuning": {"snr_threads": threads}} if threads else {}
    probe = _plan(bmin, bmax, n=200 * bmin, **kw)
    floats = probe.memory()["buffer_bytes"] // 4
    probe.close()
    for b in sorted({bmin, (bmin + bmax) // 2, bmax}):
        rows = floats // _stride(b)
        n = rows * b  # the first cycle folds the series itself into `rows` rows of b bins
        x = np.random.default_rng(n).standard_normal(n).astype(np.float32)
        w = O.generate_width_trials(bmin)
        args = dict(period_min=1e-3 * bmin, period_max=8e-3 * bmin, bins_min=bmin, bins_max=bmax,
                    widths=w, deredden=False, already_normalised=True)
        bs = rb.BatchedSearch([n], 1e-3, **args, **kw)
        p, fb, s = [t.cpu().numpy() for t in bs.run(torch.from_numpy(x).cuda())]
        bs.close()
        rp, rfb, rs = O.C().periodogram(x, 1e-3, w, 1e-3 * bmin, 8e-3 * bmin, bmin, bmax)
        assert np.array_equal(p, rp) and np.array_equal(fb, rfb)
        assert np.allclose(s, rs, rtol=1e-5, atol=2e-5)
