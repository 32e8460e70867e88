"""The block eigen-solve of the mixed path where its bookkeeping can go wrong:
inner sweep counts (the rows of W are unrolled by eight rounds, a sweep has 63,
so every count ends at another phase), padding columns, a single block pair per
round, and inputs whose Grams take the scaled form of the rotation (d^2 + e^2
out of range).

sigma against LAPACK, normwise 1e-15 max(n, 100), and U^T U - I, V^T V - I to
1e-12 n: the bounds of the path's other accuracy tests.
"""
import numpy as np
import pytest

import jsvd
import oracle
import workloads

pytestmark = pytest.mark.gpu


def check(a, r, scale=1.0):
    n = a.shape[1]
    err = oracle.sigma_errors(r.sigma / scale, np.linalg.svd(a / scale, compute_uv=False))
    assert err["normwise"] <= 1e-15 * max(n, 100)
    assert np.linalg.norm(r.v.T @ r.v - np.eye(n)) <= 1e-12 * n
    if scale >= 1.0:  # U's columns are zero where sigma <= epsilon (the reference's rule)
        assert np.linalg.norm(r.u.T @ r.u - np.eye(n)) <= 1e-12 * n


@pytest.mark.parametrize("inner", [1, 2, 3, 4, 8])
@pytest.mark.parametrize("m,n,tc", [(150, 128, 0), (200, 129, 3), (300, 250, 3)])
def test_inner_sweeps(m, n, tc, inner):
    a = workloads.spectrum_matrix(m, n, workloads.geometric_sigma(n, 1e-3), n + inner)
    jsvd.mixed_set_options(inner_sweeps=inner, tc_max_sweeps=tc)
    try:
        r = jsvd.mixed_svd(a, jsvd.default_config(epsilon=1e-14))
    finally:
        jsvd.mixed_set_options(None)
    check(a, r)


def test_scaled_rotations():
    """Gram entries near 1e152: the squares of the threshold test still fit, and
    d^2 + e^2 is taken with both scaled."""
    scale = 1e76
    a = workloads.spectrum_matrix(180, 140, workloads.geometric_sigma(140, 1e-2), 5) * scale
    jsvd.mixed_set_options(tc_max_sweeps=0)
    try:
        r = jsvd.mixed_svd(a, jsvd.default_config(epsilon=1e-14))
    finally:
        jsvd.mixed_set_options(None)
    check(a, r, scale)


def test_small_rotations_keep_unit_columns():
    """Columns orthogonal to about 1e-12: every pair rotates once, by angles below
    1e-8, whose cosine rounds to 1.  V's leading entries are then 1 to within
    2 ulp (products by 1 and sums of terms below 1e-16); a cosine that is one ulp
    off to one side would move them by about n ulp."""
    m, n = 300, 256
    a = np.zeros((m, n))
    a[np.arange(n), np.arange(n)] = np.linspace(2.0, 1.0, n)
    a += 1e-12 * np.random.default_rng(9).standard_normal((m, n))
    jsvd.mixed_set_options(precondition=0, tc_max_sweeps=0)
    try:
        r = jsvd.mixed_svd(a, jsvd.default_config(epsilon=1e-14))
    finally:
        jsvd.mixed_set_options(None)
    lead = np.abs(r.v).max(axis=0)
    assert np.abs(r.v).max() > 0 and np.count_nonzero(r.v) > n  # it rotated
    assert np.abs(lead - 1.0).max() <= 4.5e-16
