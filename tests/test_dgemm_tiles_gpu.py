"""The FP64 product with two and with three CTAs to an SM (csrc/dgemm.cu:
three_ctas): the same sums either way, at tile counts on both sides of each
line of the rule on 148 SMs, for every op, with and without C's old values and
for lower triangles that are not square.
"""
import time

import numpy as np
import pytest

import jsvd

pytestmark = pytest.mark.gpu


def product(ta, tb, m, n, k, a, b, beta=0.0, c=None, lower=0):
    import torch

    out = torch.zeros((n, m), dtype=torch.float64, device="cuda") if c is None else c.clone()  # column-major
    torch.cuda.synchronize()
    jsvd.dgemm_device("T" if ta else "N", "T" if tb else "N", m, n, k, 0.5, a.data_ptr(), k if ta else m,
                      b.data_ptr(), n if tb else k, beta, out.data_ptr(), m, lower)
    return out


def operands(ta, tb, m, n, k, seed):
    """Column-major op(A) = A (m x k) and op(B) = B (k x n) as the library reads them."""
    import torch

    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    a = torch.randn((m, k), generator=g, dtype=torch.float64, device="cuda")
    b = torch.randn((k, n), generator=g, dtype=torch.float64, device="cuda")
    return a, b, (a if ta else a.T).contiguous(), (b.T if not tb else b).contiguous()


@pytest.mark.parametrize("ta", [False, True])
@pytest.mark.parametrize("tb", [False, True])
@pytest.mark.parametrize("m,n", [(600, 1900), (610, 2300), (1000, 1720), (1000, 3000), (1030, 4610)])
def test_against_exact_bound(cuda_device, ta, tb, m, n):
    """Elementwise |C - exact| <= (k + 4) 2^-53 (|A| |B| / 2 + |C0|): every order of
    k products and sums stays within it (the reference's own error with it: 2x)."""
    import torch

    k = 70
    a, b, da, db = operands(ta, tb, m, n, k, m + n)
    c0 = torch.randn((n, m), dtype=torch.float64, device="cuda")
    for beta in (0.0, -0.75):
        got = product(ta, tb, m, n, k, da, db, beta, c0)
        want = 0.5 * (a @ b) + beta * c0.T
        bound = 2 * (k + 4) * 2.0 ** -53 * (0.5 * a.abs() @ b.abs() + abs(beta) * c0.T.abs())
        assert bool(((got.T - want).abs() <= bound).all())


@pytest.mark.parametrize("ta,tb", [(False, False), (True, False), (False, True), (True, True)])
def test_same_bits_at_every_occupancy(cuda_device, ta, tb):
    """The leading columns of a product do not depend on how many columns follow,
    nor, therefore, on how many CTAs an SM runs (1..9 tiles per SM)."""
    m, k = 512, 200
    _, _, da, _ = operands(ta, tb, m, 64, k, 3)
    a, b, _, _ = operands(ta, tb, m, 64 * 160, k, 3)
    da = (a if ta else a.T).contiguous()
    first = None
    for cols in (64 * 18, 64 * 36, 64 * 40, 64 * 70, 64 * 80, 64 * 100, 64 * 112, 64 * 130, 64 * 160):
        sub = b[:, :cols]
        got = product(ta, tb, m, cols, k, da, (sub.T if not tb else sub).contiguous())
        head = got[:64 * 18]
        first = head if first is None else first
        assert bool((head == first).all())


@pytest.mark.parametrize("m,n", [(1550, 1550), (2048, 2048), (2200, 2200), (3000, 1300), (1300, 3000)])
def test_lower(cuda_device, m, n):
    import torch

    k = 33
    a, b, da, db = operands(True, False, m, n, k, m)
    c0 = torch.full((n, m), 7.0, dtype=torch.float64, device="cuda")
    full = product(True, False, m, n, k, da, db).T
    for beta in (0.0, 1.0):
        got = product(True, False, m, n, k, da, db, beta, c0, lower=1).T
        low = torch.ones((m, n), dtype=torch.bool, device="cuda").tril()
        assert bool((got[~low] == 7.0).all())
        if beta == 0.0:
            assert bool((got[low] == full[low]).all())
        else:
            assert bool(((got - 7.0 - full)[low].abs() <= 2.0 ** -50 * (7.0 + full[low].abs())).all())


def test_three_tiles_per_sm_take_three_ctas(cuda_device):
    """320 tiles (three on the fullest SM) against 288 (two): 1.5 times the time
    with three CTAs to an SM, 1.84 with two."""
    def best(n):
        m, k = 512, 4096
        _, _, da, db = operands(False, False, m, n, k, n)
        ms = np.inf
        for _ in range(8):
            t = time.perf_counter()
            product(False, False, m, n, k, da, db)
            ms = min(ms, time.perf_counter() - t)
        return ms

    assert best(2560) <= 1.68 * best(2304)
