"""Column bookkeeping of the plain path's fused launches (several rounds per
launch, csrc/plain.cu: fused_slot and the level geometry above it), restated in
integer arithmetic and checked on the CPU against the library's round-robin
schedule: every group of every level holds the two columns that the circle
puts in its slot, taken from the group and side the kernel reads; every pair
of every round is recorded exactly once; the last level writes every column
exactly once.
"""
import jsvd
import numpy as np
import pytest


def circle_col_near(n, L, r, pos):
    if pos == 0:
        return 0
    v = pos - 1 - r
    c = 1 + (v + L if v < 0 else v)
    return -1 if c == n else c


def fused_slot(x, half):
    mirrored = x < 0 or x >= half
    return (-x - 1 if x < 0 else (2 * half - 1 - x if x >= half else x)), mirrored


def run_launch(n, r0, R, S):
    """One launch: {(round, pair index): (p, q)} recorded and the columns written."""
    ne = n + (n & 1)
    half, L = ne // 2, ne - 1
    chunks = ((half + 1) // 2 + S - 1) // S
    recorded, written = {}, []
    for b in range(2 * chunks):
        k0 = (b & 1) + 2 * (b >> 1) * S
        own = min(S, (half - k0 + 1) >> 1)
        if own <= 0:
            continue
        held, published = {}, {}  # group -> [top, bottom]; (level, group) -> column
        for lev in range(R):
            w, r = R - 1 - lev, r0 + lev
            for g in range(own + w):
                x = k0 - w + 2 * g
                slot, mir = fused_slot(x, half)
                assert 0 <= slot < half
                p, q = circle_col_near(n, L, r, slot), circle_col_near(n, L, r, ne - 1 - slot)
                pair, real = slot, True
                if n & 1:
                    pos = n - 1 + r
                    pos = 1 + (pos - L if pos >= L else pos)
                    dummy = pos if pos < half else ne - 1 - pos
                    real = slot != dummy
                    pair -= slot > dummy
                assert real == (p >= 0 and q >= 0)
                if lev > 0:
                    top, bottom = held[g]
                    nbr = published[(lev - 1, g + 1)]
                    if not mir:
                        top, bottom = (bottom if slot == 1 else top), nbr
                    else:
                        top, bottom = nbr, (top if slot == half - 1 else bottom)
                    assert (top, bottom) == (p, q)
                held[g] = (p, q)
                writer = real and ((k0 <= x <= k0 + 2 * (own - 1)) if w % 2 == 0 else
                                   ((k0 < x <= k0 + 2 * own - 1 and x < half) or (k0 == 0 and x == -1)))
                if writer:
                    assert (r, pair) not in recorded
                    recorded[(r, pair)] = (p, q)
                if w > 0 and g > 0:
                    pslot, pmir = fused_slot(x - 1, half)
                    want_top = pslot != 1 if pmir else pslot == half - 1
                    published[(lev, g)] = p if want_top else q
                if w == 0:
                    written += [c for c in (p, q) if c >= 0]
    return recorded, written


@pytest.mark.parametrize("n", [5, 6, 7, 8, 17, 18, 31, 48, 65, 100, 101])
@pytest.mark.parametrize("S", [1, 2, 3, 5])
@pytest.mark.parametrize("R", [1, 2, 3, 4, 6, 8])
def test_fused_rounds_follow_the_schedule(n, S, R):
    want = jsvd.round_robin_schedule(n, 0)
    rounds = want.shape[0]
    R = min(R, (n + 1) // 2 - 1)  # the launch rule's bound
    for r0 in range(0, rounds, R):
        live = min(R, rounds - r0)
        recorded, written = run_launch(n, r0, live, S)
        assert sorted(written) == list(range(n))
        for r in range(r0, r0 + live):
            got = np.array([recorded[(r, k)] for k in range(want.shape[1])])
            assert np.array_equal(got, want[r])
