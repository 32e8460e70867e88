"""Grams of the QR stage whose sum over the rows is split in 2, 4 or 8 parts:
heights at and beside the first that split, a remainder in the last part,
widths with a remainder tile, and the widest that still split in two.

sigma against LAPACK, normwise 1e-15 max(n, 100), and U^T U - I, V^T V - I to
1e-12 n: the bounds of the path's other accuracy tests.  The split depends on
the shape alone, so a second solve gives the same bits.
"""
import numpy as np
import pytest

import jsvd
import oracle
import workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n", [(255, 64), (256, 64), (257, 65), (513, 1), (513, 2), (1023, 130), (1024, 130),
                                 (1500, 65), (700, 300), (2100, 640), (1100, 1024)])
def test_split_grams(m, n):
    a = workloads.spectrum_matrix(m, n, workloads.geometric_sigma(n, 1e-4), n + m)
    jsvd.precond_stats_reset()
    r = jsvd.precond_svd(a, jsvd.default_config(epsilon=1e-14))
    assert jsvd.precond_stats().fallbacks == 0
    err = oracle.sigma_errors(r.sigma, np.linalg.svd(a, compute_uv=False))
    assert err["normwise"] <= 1e-15 * max(n, 100)
    for x in (r.u, r.v):
        assert np.linalg.norm(x.T @ x - np.eye(n)) <= 1e-12 * n
    again = jsvd.precond_svd(a, jsvd.default_config(epsilon=1e-14))
    for x, y in ((r.u, again.u), (r.sigma, again.sigma), (r.v, again.v)):
        np.testing.assert_array_equal(x, y)
