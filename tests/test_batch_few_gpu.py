"""Which kernel a member of the two largest size classes gets: by its shape and
by how many members of its class the batch has (csrc/batched.cu:
cluster_choice).  The counts stand on both sides of every line of that rule on
a device of 148 SMs; the results are the plain path's bytes whatever is chosen,
and a few members of class 3 are not left to one CTA each.
"""
import time

import numpy as np
import pytest

import jsvd
import workloads

pytestmark = pytest.mark.gpu

# class 3: with C = 2, without; class 4: two and four CTAs, eight shared, eight
# slots, more than 12 slots, none but eight
SHAPES = [(350, 70), (165, 160), (500, 80), (250, 140), (512, 128), (256, 200), (256, 256)]


@pytest.mark.parametrize("count", [1, 13, 17, 32, 36, 40, 70, 74, 80, 160])
@pytest.mark.parametrize("m,n", SHAPES)
def test_bytes_for_every_choice(cuda_device, m, n, count):
    cfg = jsvd.default_config(epsilon=1e-12, max_sweeps=1)
    a = workloads.gaussian_splitmix(m, n, seed=m + n)
    w = jsvd.plain_svd(a, cfg)
    b = jsvd.DeviceBatch([a] * count, cuda_device, want_u=True)
    b.solve(cfg)
    for u, s, v, sw in b.results():
        assert sw == w.sweeps
        assert np.array_equal(s, w.sigma) and np.array_equal(u, w.u) and np.array_equal(v, w.v)


def _best_ms(b, cfg, reps=5):
    import torch

    best = np.inf
    for _ in range(reps):
        torch.cuda.synchronize()
        t = time.perf_counter()
        b.solve(cfg)
        best = min(best, time.perf_counter() - t)
    return best * 1e3


@pytest.mark.parametrize("m,n", [(350, 70), (200, 130)])
def test_few_members_of_class_3_are_spread_over_the_device(cuda_device, m, n):
    """Eight members on 148 SMs: by clusters 0.25 and 0.35 of the time of one CTA
    each; half is allowed."""
    cfg = jsvd.default_config(epsilon=1e-12)
    b = jsvd.DeviceBatch([workloads.gaussian_splitmix(m, n, seed=i) for i in range(8)], cuda_device)
    chosen = _best_ms(b, cfg)
    old = jsvd.batch_set_cluster_classes(0)
    try:
        alone = _best_ms(b, cfg)
    finally:
        jsvd.batch_set_cluster_classes(old)
    assert chosen <= 0.5 * alone


@pytest.mark.parametrize("shapes", [[(100, 90), (200, 90), (300, 50)], [(200, 130), (350, 70), (165, 160)]])
def test_groups_of_a_class_overlap(cuda_device, shapes):
    """Three members of one class for three kernels (class 2 by rows, class 3 by
    cluster): together they take the longest one's time, and 0.8 of the sum of
    their times is allowed.  One after another they take the sum."""
    cfg = jsvd.default_config(epsilon=1e-12)
    mats = [workloads.gaussian_splitmix(m, n, seed=m + n) for m, n in shapes]
    together = _best_ms(jsvd.DeviceBatch(mats, cuda_device), cfg)
    alone = sum(_best_ms(jsvd.DeviceBatch([a], cuda_device), cfg) for a in mats)
    assert together <= 0.8 * alone


@pytest.mark.parametrize("copies", [1, 12])
def test_bytes_of_overlapping_groups(cuda_device, copies):
    shapes = [(40, 30), (200, 20), (500, 10), (100, 60), (200, 45), (300, 30), (100, 90), (200, 90), (300, 50),
              (200, 130), (350, 70), (165, 160), (500, 80), (250, 140), (512, 128), (256, 200)]
    cfg = jsvd.default_config(epsilon=1e-12, max_sweeps=2)
    mats = [workloads.gaussian_splitmix(m, n, seed=m + n) for m, n in shapes]
    want = [jsvd.plain_svd(a, cfg) for a in mats]
    b = jsvd.DeviceBatch(mats * copies, cuda_device, want_u=True)
    for _ in range(3):
        for x in (b.sigma, b.u, b.v):
            x.fill_(-1.0)
        b.solve(cfg)
        for i, (u, s, v, sw) in enumerate(b.results()):
            w = want[i % len(want)]
            assert sw == w.sweeps
            assert np.array_equal(s, w.sigma) and np.array_equal(u, w.u) and np.array_equal(v, w.v)


@pytest.mark.parametrize("count", [45, 100, 211])
def test_many_ragged_members_of_class_3_keep_its_kernel_where_it_is_faster(cuda_device, count):
    """Ragged members of class 3: with clusters allowed for the class
    at most as long as without (a tenth for the spread of the runs).  A rule by
    whole waves of equal members took 1.8 times as long for 211."""
    rng = np.random.default_rng(count)
    mats = []
    while len(mats) < count:
        m = int(rng.integers(100, 257))
        n = int(rng.integers(8, m + 1))
        if 8 * m * n < 222 * 1024 and 8 * (m * n + n * n) > 227 * 1024:
            mats.append(rng.standard_normal((m, n)))
    cfg = jsvd.default_config(epsilon=1e-12)
    b = jsvd.DeviceBatch(mats, cuda_device)
    chosen = _best_ms(b, cfg, reps=3)
    old = jsvd.batch_set_cluster_classes(1 << 4)
    try:
        kernel = _best_ms(b, cfg, reps=3)
    finally:
        jsvd.batch_set_cluster_classes(old)
    assert chosen <= 1.1 * kernel
