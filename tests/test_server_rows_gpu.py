"""Serving-core requests on both sides of the row counts where the sweep step
changes its loops (32, 64, 128 and 256 rows; more have a function of their own),
alone and together: the plain path's bytes and sweep counts."""
import numpy as np
import pytest

import jsvd
import workloads

pytestmark = pytest.mark.gpu

SHAPES = [(32, 32), (33, 20), (64, 50), (65, 64), (128, 90), (129, 60), (256, 60), (257, 16), (300, 60), (500, 40),
          (513, 33), (2000, 8), (260, 1), (300, 90)]


@pytest.mark.parametrize("together", [False, True])
def test_bytes_of_the_plain_path(cuda_device, together):
    cfg = jsvd.default_config(epsilon=1e-12)
    mats = [workloads.gaussian_splitmix(m, n, seed=m * 3 + n) for m, n in SHAPES]
    with jsvd.Server(cfg, budget_bytes=1 << 30) as server:
        if together:
            tickets = [server.submit(a, want_u=True) for a in mats]
            got = [server.wait(t) for t in tickets]
        else:
            got = [server.wait(server.submit(a, want_u=True)) for a in mats]
    for a, (u, s, v, sweeps, _) in zip(mats, got):
        w = jsvd.plain_svd(a, cfg)
        assert sweeps == w.sweeps
        assert np.array_equal(s, w.sigma) and np.array_equal(u, w.u) and np.array_equal(v, w.v)
