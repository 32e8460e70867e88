"""The Cholesky diagonal blocks of the QR stage (64 columns in panels of 8) at
their edges, through the QR-preconditioned solver: widths around the panel
and block sizes, and pivots outside the range of the hardware's reciprocal
approximation.

sigma against LAPACK, normwise 1e-15 max(n, 100), and U^T U - I, V^T V - I to
1e-12 n: the bounds of the path's other accuracy tests.
"""
import numpy as np
import pytest

import jsvd
import oracle
import workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 7, 8, 9, 16, 57, 63, 64, 65, 71, 72, 73, 127, 128, 129])
def test_widths_around_panels_and_blocks(n):
    m = n + 40
    a = workloads.spectrum_matrix(m, n, workloads.geometric_sigma(n, 1e-4), n)
    jsvd.precond_stats_reset()
    r = jsvd.precond_svd(a, jsvd.default_config(epsilon=1e-14))
    assert jsvd.precond_stats().fallbacks == 0
    err = oracle.sigma_errors(r.sigma, np.linalg.svd(a, compute_uv=False))
    assert err["normwise"] <= 1e-15 * max(n, 100)
    for x in (r.u, r.v):
        assert np.linalg.norm(x.T @ x - np.eye(n)) <= 1e-12 * n


@pytest.mark.parametrize("scale", [1e152, 1e-152])
def test_pivots_outside_the_approximation_range(scale):
    """Orthogonal columns: the Grams are diagonal with entries near 1e304 or
    1e-304, and nothing rotates."""
    n = 70
    a = np.zeros((100, n))
    a[np.arange(n), np.arange(n)] = scale
    jsvd.precond_stats_reset()
    r = jsvd.precond_svd(a, jsvd.default_config(epsilon=1e-14))
    assert jsvd.precond_stats().fallbacks == 0
    np.testing.assert_allclose(r.sigma, scale, rtol=1e-14)
    assert np.linalg.norm(r.v.T @ r.v - np.eye(n)) <= 1e-12 * n
    # U's columns are zero where sigma <= epsilon (the reference's rule)
    want = np.eye(n) if scale > 1e-14 else np.zeros((n, n))
    assert np.linalg.norm(r.u.T @ r.u - want) <= 1e-12 * n
