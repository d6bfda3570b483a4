"""CPU checks of the digit scheme with 8-bit leading digits: exact digits, and sums that stay exact integers in FP32."""
import random

import numpy as np
import pytest


def _digits(V, S):
    """The split kernel's closed form: S balanced base-128 digits, the first unbounded."""
    U = V + 64 * ((1 << (7 * (S - 1))) - 1) // 127
    return [U >> (7 * (S - 1))] + [((U >> (7 * (S - 1 - i))) & 127) - 64 for i in range(1, S)]


@pytest.mark.parametrize("S", [5, 6, 7, 8])
def test_wide_digits_are_exact_and_bounded(S):
    rng = random.Random(S)
    lim = 1 << (7 * S)
    cases = [0, 1, -1, lim, -lim, lim - 1, 1 - lim, lim // 2, -lim // 2, lim // 2 + 1]
    for V in cases + [rng.randrange(-lim, lim + 1) for _ in range(20000)]:
        d = _digits(V, S)
        assert sum(x * 128 ** (S - 1 - i) for i, x in enumerate(d)) == V
        assert abs(d[0]) <= 128 and all(abs(x) <= 64 for x in d[1:])


@pytest.mark.parametrize("S", [5, 8])
def test_wide_diagonal_sums_stay_exact(S):
    top = [128] + [64] * (S - 1)
    v = [256 * sum(top[i - 1] * top[g - i - 1] for i in range(1, S + 1) if 1 <= g - i <= S) for g in range(2, S + 2)]
    assert max(v) < 1 << 24  # FP32 accumulators hold exact integers
    assert all(a * 128 + b < 1 << 31 for a, b in zip(v[:-1], v[1:]))  # adjacent diagonals combine in int32
    lo = (v[S - 4] * 128 + v[S - 3]) * 2 ** 14 + v[S - 2] * 128 + v[S - 1]
    hi = sum(x * 128 ** (S - 5 - k) for k, x in enumerate(v[:S - 4]))
    sq = 256 * 64 * 64  # the middle digits' squares, in units of 1 / 128
    assert (lo * 128 + sq < 1 << 53 or S == 5) and hi < 1 << 53  # both halves are exact doubles
    if S == 5:
        assert hi * 2 ** 28 + lo < 1 << 53  # and so is their sum
    for x in (-128, 127, 100):  # digits are exact in bf16: at most 8 significant bits
        assert np.float32(x).view(np.uint32) & 0xFFFF == 0
