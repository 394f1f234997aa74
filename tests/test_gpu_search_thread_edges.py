"""Searches over the bins at which the default number of S/N threads per profile changes (4, 8, 16,
32 threads of 33 phases) and beyond the last (loops instead of unrolled prefix sums), and with 16
threads for fewer bins than they are the default of, against the C restatement."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bmin,bmax,tuning", [
    (130, 135, None), (262, 267, None), (526, 531, None),
    (1050, 1064, None),                       # 1056: unrolled, from 1057 on loops
    (89, 97, {"snr_threads": 16}), (120, 134, {"snr_threads": 16}), (20, 24, {"snr_threads": 16})])
def test_search(bmin, bmax, tuning):
    import torch

    import riptide_b200 as rb

    n = (900 if bmin < 600 else 90) * bmin  # several stages
    rng = np.random.default_rng(bmin)
    x = rb.generate_signal(n, 2.3 * bmin, ducy=0.05, amplitude=20.0, rng=rng)
    x = O.normalise(x).astype(np.float32)
    w = O.generate_width_trials(bmin)
    lim = (1e-3 * bmin, 9e-3 * bmin)
    bs = rb.BatchedSearch([n], 1e-3, period_min=lim[0], period_max=lim[1], bins_min=bmin,
                          bins_max=bmax, widths=w, deredden=False, already_normalised=True,
                          tuning=tuning)
    p, fb, s = [t.cpu().numpy() for t in bs.run(torch.from_numpy(x).cuda())]
    bs.close()
    rp, rfb, rs = O.C().periodogram(x, 1e-3, w, *lim, bmin, bmax)
    assert np.array_equal(p, rp) and np.array_equal(fb, rfb)
    assert np.allclose(s, rs, rtol=1e-5, atol=2e-5)
