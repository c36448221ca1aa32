"""The integer router's arithmetic (csrc/router_i8.cu) modelled on the CPU: digits reproduce their value, the sums of one
level fit int32 and the three partial sums 51 bits at the largest k a CTA can get, and the sum of the levels is the
logit as long as the values are on the grid."""
import re
from fractions import Fraction
from pathlib import Path

import numpy as np

CSRC = Path(__file__).resolve().parents[1] / "ateniaengine_b200" / "csrc"
MAX_K = int(re.search(r"kRouterDigitMaxK = (\d+)", (CSRC / "common.cuh").read_text()).group(1))


def balanced(X, n):
    out = []
    for _ in range(n):
        d = ((X + 128) & 255) - 128
        out.append(d)
        X = (X - d) >> 8
    assert X == 0
    return out[::-1]  # top digit first


def test_digits_reproduce_their_value_and_stay_in_range():
    rng = np.random.default_rng(0)
    for bits, n in ((30, 4), (38, 5)):
        vals = [0, 1, -1, 127, 128, -128, -129, 255, (1 << bits) - 1, -(1 << bits), 1 << (bits - 1), 0x7f7f7f7f & ((1 << bits) - 1)]
        vals += [int(v) for v in rng.integers(-(1 << bits), 1 << bits, 2000)]
        for X in vals:
            d = balanced(X, n)
            assert all(-128 <= v <= 127 for v in d) and -64 <= d[0] <= 64
            assert sum(v * 256 ** (n - 1 - i) for i, v in enumerate(d)) == X
            if n == 4:  # the byte trick of the kernel: X + 0x80808080, each byte xor 0x80
                b = ((X + 0x80808080) & 0xFFFFFFFF) ^ 0x80808080
                assert [((b >> (8 * (3 - i))) & 255) - (256 if (b >> (8 * (3 - i))) & 128 else 0) for i in range(4)] == d


def test_sums_fit_at_the_largest_k():
    top = [64] + [128] * 3, [64] + [128] * 4
    level = [0] * 8
    for i, x in enumerate(top[0]):
        for j, w in enumerate(top[1]):
            level[i + j] += x * w * MAX_K
    assert max(level) < 2 ** 31
    for part in (level[:3], level[3:6], level[6:]):
        assert sum(v << 8 * (len(part) - 1 - n) for n, v in enumerate(part)) < 2 ** 51


def test_levels_add_up_to_the_exact_logit():
    rng = np.random.default_rng(1)
    x = rng.normal(size=96).astype(np.float32)
    x = (x.view(np.uint32) & 0xFFFF0000).view(np.float32)  # bf16 values
    w = (rng.normal(size=96) * 0.02).astype(np.float32)
    x[3], w[5] = 0.0, 0.5
    ex, ew = int(np.floor(np.log2(np.abs(x).max()))) + 1, int(np.floor(np.log2(np.abs(w).max()))) + 1
    X = [int(Fraction(float(v)) * Fraction(2) ** (30 - ex)) for v in x]
    W = [round(Fraction(float(v)) * Fraction(2) ** (38 - ew)) for v in w]
    level = [0] * 8
    for a, b in zip(X, W):
        for i, p in enumerate(balanced(a, 4)):
            for j, q in enumerate(balanced(b, 5)):
                level[i + j] += p * q
    got = Fraction(2) ** (ex + ew - 68) * sum(A * 256 ** (7 - s) for s, A in enumerate(level))
    want = sum(Fraction(float(a)) * Fraction(float(b)) for a, b in zip(x, w))
    # x is on its grid; w within half a step of 2^(ew - 38)
    assert all(Fraction(a) * Fraction(2) ** (ex - 30) == Fraction(float(v)) for a, v in zip(X, x))
    assert abs(got - want) <= sum(abs(Fraction(float(v))) for v in x) * Fraction(2) ** (ew - 39)
    p0, p1, p2 = (level[0] << 16) + (level[1] << 8) + level[2], (level[3] << 16) + (level[4] << 8) + level[5], (level[6] << 8) + level[7]
    assert Fraction(2) ** (ex + ew - 28) * (p0 + Fraction(p1, 2 ** 24) + Fraction(p2, 2 ** 40)) == got
