"""Searches whose transforms have more rows than the row-number pattern of the FFA levels holds for
(8,192): single levels at the top instead of two at a time, against the C restatement."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bmin,bmax,rows,top", [(240, 242, 9000, 1.12), (48, 50, 20001, 1.2)])
def test_search(bmin, bmax, rows, top):
    import torch

    import riptide_b200 as rb

    n = rows * bmax
    rng = np.random.default_rng(rows)
    x = rb.generate_signal(n, 1.05 * bmin, ducy=0.05, amplitude=20.0, rng=rng)
    x = O.normalise(x).astype(np.float32)
    w = O.generate_width_trials(bmin)
    lim = (1e-3 * bmin, top * 1e-3 * bmin)
    bs = rb.BatchedSearch([n], 1e-3, period_min=lim[0], period_max=lim[1], bins_min=bmin,
                          bins_max=bmax, widths=w, deredden=False, already_normalised=True)
    p, fb, s = [t.cpu().numpy() for t in bs.run(torch.from_numpy(x).cuda())]
    bs.close()
    rp, rfb, rs = O.C().periodogram(x, 1e-3, w, *lim, bmin, bmax)
    assert np.array_equal(p, rp) and np.array_equal(fb, rfb)
    assert np.allclose(s, rs, rtol=1e-5, atol=2e-5)
