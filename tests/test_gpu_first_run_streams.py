"""The first run of a plan, which uploads its tables, on a stream that does not wait for the default
stream: tables of a megabyte, in memory that held other values."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_first_run_on_a_side_stream():
    import torch

    import riptide_b200 as rb

    n, trials = 1 << 18, 40
    kw = dict(period_min=0.03, period_max=1.0, bins_min=100, bins_max=110, rmed_width=0.5)
    d = torch.randn(n * trials, device="cuda", generator=torch.Generator("cuda").manual_seed(5))
    bs = rb.BatchedSearch([n] * trials, 2.56e-4, **kw)
    assert 8 * bs.stats["num_work_items"] > 1 << 20
    want = [t.clone() for t in bs.run(d)]
    bs.close()
    torch.cuda.synchronize()
    for _ in range(5):
        with torch.cuda.stream(torch.cuda.Stream()):
            bs = rb.BatchedSearch([n] * trials, 2.56e-4, **kw)
            got = bs.run(d)
            assert all(torch.equal(a, b) for a, b in zip(got, want))
            bs.close()
