"""The batched solver's row-specialised loops and its cluster kernels against
the plain path, bit for bit: members at the row counts where the loops change
(32, 64, 128, 256 rows, one either side), odd widths, and each kind of cluster
(two CTAs per SM, an SM per CTA, more than 256 rows), alone and in numbers
that change the launch shape.
"""
import numpy as np
import pytest

import jsvd
import workloads

pytestmark = pytest.mark.gpu

ROWS = [(16, 8), (31, 30), (32, 32), (33, 9), (63, 40), (64, 64), (65, 33), (127, 20), (128, 61), (129, 64), (255, 12),
        (256, 41), (257, 16), (600, 9)]
CLUSTERS = [(150, 130), (200, 151), (228, 189), (232, 215), (250, 250), (300, 190), (520, 120)]


def check(mats, f32=False, sweeps=3):
    import torch

    cfg = jsvd.default_config(epsilon=1e-12, max_sweeps=sweeps)
    b = jsvd.DeviceBatch(mats, torch.device("cuda:0"), f32=f32, want_u=True)
    b.solve(cfg)
    seen = {}
    for a, (u, s, v, sw) in zip(mats, b.results()):
        key = a.tobytes()
        if key not in seen:
            seen[key] = jsvd.plain_svd(a.astype(np.float32).astype(np.float64) if f32 else a, cfg)
        w = seen[key]
        assert sw == w.sweeps
        assert np.array_equal(s, w.sigma) and np.array_equal(u, w.u) and np.array_equal(v, w.v)


@pytest.mark.parametrize("f32", [False, True])
def test_row_bounds(f32):
    check([workloads.gaussian_splitmix(m, n, seed=m * 7 + n) for m, n in ROWS], f32, sweeps=20)


@pytest.mark.parametrize("copies", [40, 700])
def test_launch_shapes(copies):
    mats = [workloads.gaussian_splitmix(m, n, seed=m + n) for m, n in [(20, 17), (40, 24), (70, 60)]]
    check(mats * copies, sweeps=4)


@pytest.mark.parametrize("mask", [0, 0b10000, 0b11100])
def test_clusters(mask):
    old = jsvd.batch_set_cluster_classes(mask)
    try:
        check([workloads.gaussian_splitmix(m, n, seed=m + n) for m, n in CLUSTERS], sweeps=2)
    finally:
        jsvd.batch_set_cluster_classes(old)


def test_special_values():
    """Zero columns, subnormals, infinities and NaN: the bytes of the plain path."""
    a = workloads.gaussian_splitmix(200, 171, seed=5)
    a[:, 3] = 0.0
    a[:, 4] *= 1e-310
    a[:, 5] *= 1e160
    a[7, 9] = np.nan
    a[8, 11] = np.inf
    import torch

    cfg = jsvd.default_config(epsilon=1e-12, max_sweeps=2)
    for m in (a, np.ascontiguousarray(a[:90, :40])):
        b = jsvd.DeviceBatch([m], torch.device("cuda:0"), want_u=True)
        b.solve(cfg)
        (u, s, v, sw), = b.results()
        w = jsvd.plain_svd(m, cfg)
        assert sw == w.sweeps
        for x, y in ((s, w.sigma), (u, w.u), (v, w.v)):
            assert np.array_equal(x, y, equal_nan=True)
