"""Bounds of a plan's shared memory, by arithmetic on the host: the boxcar S/N of the search kernel
reads whole segments of 33 phases, past the end of a row, for whatever number of threads the plan
may give a profile; the last row of a full level buffer is the one that could leave the CTA's
shared memory."""
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
