"""What a round of the batched solver's cluster kernel derives from the round
number (csrc/batched.cu: ClusterShare, ClusterRound), restated in integer
arithmetic and checked on the CPU: the buffers a slot reads follow the column
that the circle puts there, and the dummy column of an odd n is found in the
slot and position where the circle has it.
"""
import pytest


@pytest.mark.parametrize("n", [15, 16, 17, 31, 33, 64, 65, 113, 150, 199, 256])
@pytest.mark.parametrize("C", [2, 4, 8])
def test_round_bookkeeping(n, C):
    ne = n + (n & 1)
    half, L = ne // 2, ne - 1
    if half < 2 * C:
        pytest.skip("fewer than two slots per CTA")

    def column(pos, g):  # the circle: position 0 is fixed, the others advance by one per round
        return 0 if pos == 0 else 1 + (pos - 1 - g) % L

    for rank in range(C):
        k0 = rank * half // C
        S = (rank + 1) * half // C - k0
        jt0 = 1 if rank == 0 else 0
        rt, rb = S - jt0 + 1, S + 1
        top, bot = {}, {}  # ring buffer -> column, as the previous round left them
        gt = gb = 0
        dpos = L
        for g in range(2 * L):
            dummy_top = dpos < half
            d = (dpos if dummy_top else L - dpos) - k0
            dummy = d if (n & 1) and 0 <= d < S else -1
            for j in range(S):
                tb, bb = j - jt0 - gt, j + gb
                if tb < 0:
                    tb += rt
                if bb > S:
                    bb -= S + 1
                assert bb == (j + g) % rb
                p, q = column(k0 + j, g), column(ne - 1 - (k0 + j), g)
                if not (jt0 and j == 0):
                    assert tb == (j - jt0 - g) % rt
                    # a column that stays in this CTA stays in its buffer
                    if g > 0 and j > jt0:
                        assert top[tb] == p
                    top[tb] = p
                if g > 0 and j < S - 1:
                    assert bot[bb] == q
                bot[bb] = q
                assert (j == dummy) == (p == n or q == n)
                if j == dummy:
                    assert dummy_top == (p == n)
            gt = 0 if gt == rt - 1 else gt + 1
            gb = 0 if gb == rb - 1 else gb + 1
            dpos = 1 if dpos == L else dpos + 1
