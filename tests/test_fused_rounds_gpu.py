"""The plain path's fused launches (several rounds per launch, up to 1024 rows)
against the one-round kernels, bit for bit.

The shapes sit at the edges of the launch rule: the row counts where the kernel
changes (64, 128, 256, 512, 1024 rows, one row either side), the widths where the
slots per CTA change with the SM count (half the columns at 148, 296, 444), odd
widths (a dummy column), the narrowest matrices, and sweep counts of both
parities (an odd number of launches leaves A in the other buffer).
"""
import numpy as np
import pytest

import jsvd
import oracle
import workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n", [(5, 5), (7, 6), (9, 7), (64, 64), (65, 13), (128, 127), (129, 40), (256, 200),
                                 (257, 65), (96, 33)])
def test_small_shapes_match_the_oracle(m, n):
    a = workloads.gaussian_splitmix(m, n, seed=m + n)
    cfg = jsvd.default_config(epsilon=1e-12)
    for _ in range(2):  # direct launches, then the captured graph
        u, s, v, sweeps = jsvd.plain_svd(a, cfg)
        ou, os_, ov, osw = oracle.plain_svd(a, eps=1e-12, variant=jsvd.arith_variant(), threads=4)
        assert sweeps == osw
        assert np.array_equal(s, os_) and np.array_equal(u, ou) and np.array_equal(v, ov)


@pytest.mark.parametrize("m,n,sweeps", [(512, 296, 3), (513, 297, 2), (512, 298, 2), (1024, 592, 2), (1023, 594, 3),
                                        (1024, 889, 2), (1024, 1024, 1), (1000, 295, 3)])
def test_wide_shapes_match_the_one_round_kernel(m, n, sweeps):
    a = workloads.gaussian_splitmix(m, n, seed=m + n)
    cfg = jsvd.default_config(epsilon=1e-12, max_sweeps=sweeps)
    got = [jsvd.plain_svd(a, cfg) for _ in range(2)]
    jsvd.set_sweep_mode(3)
    try:
        want = jsvd.plain_svd(a, cfg)
    finally:
        jsvd.set_sweep_mode(0)
    for r in got:
        assert r.sweeps == want.sweeps
        assert np.array_equal(r.sigma, want.sigma) and np.array_equal(r.u, want.u) and np.array_equal(r.v, want.v)


def test_special_values_do_not_spread():
    """NaN, infinities, zero columns and subnormals through the fused rounds:
    the same bytes as the one-round kernel."""
    a = workloads.gaussian_splitmix(200, 31, seed=3)
    a[:, 4] = 0.0
    a[:, 5] *= 1e-310
    a[:, 6] *= 1e200
    a[3, 7] = np.nan
    a[9, 8] = np.inf
    cfg = jsvd.default_config(epsilon=1e-12, max_sweeps=4)
    got = jsvd.plain_svd(a, cfg)
    jsvd.set_sweep_mode(3)
    try:
        want = jsvd.plain_svd(a, cfg)
    finally:
        jsvd.set_sweep_mode(0)
    assert got.sweeps == want.sweeps
    for x, y in zip(got[:3], want[:3]):
        assert np.array_equal(x, y, equal_nan=True)
