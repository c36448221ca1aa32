"""The integer router's arithmetic (csrc/router_digits.cuh), compiled for the host: digits reproduce their value, a token is
marked whenever a value of it is off the grid (and only then where a value is small enough to be), the sums of one level fit
int32 and the three partial sums 51 bits at the largest k a CTA can get, and the levels add up to the logit: exactly for values
on the grid, with what is left out added back for the others."""
import ctypes as C
import re
import subprocess
from fractions import Fraction
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parents[1]
MAX_K = int(re.search(r"kRouterDigitMaxK = (\d+)", (ROOT / "ateniaengine_b200/csrc/common.cuh").read_text()).group(1))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = tmp_path_factory.mktemp("digits") / "libdigits.so"
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", str(ROOT / "tests/router_digits_probe.cpp"), "-o", str(so)])
    return C.CDLL(str(so))


def x_digits(lib, X):
    b = lib.digits_x(C.c_int(X)) & 0xFFFFFFFF
    return [((b >> (8 * (3 - i))) & 255) - (256 if (b >> (8 * (3 - i))) & 128 else 0) for i in range(4)]


def w_digits(lib, W):
    out, rest = (C.c_byte * 5)(), C.c_longlong()
    lib.digits_w(C.c_longlong(W), out, C.byref(rest))
    assert rest.value == 0
    return list(out)


def bf16(v):
    """The value of a bf16 pattern (sign off), exactly."""
    field, m = v >> 7, v & 127
    return Fraction(m + (128 if field else 0)) * Fraction(2) ** (max(field, 1) - 134)


def test_digits_reproduce_their_value_and_stay_in_range(lib):
    rng = np.random.default_rng(0)
    for bits, digits in ((30, x_digits), (38, w_digits)):
        vals = [0, 1, -1, 127, 128, -128, -129, 255, (1 << bits) - 1, -(1 << bits), 1 << bits, 1 << (bits - 1), 0x7f7f7f7f & ((1 << bits) - 1)]
        vals += [int(v) for v in rng.integers(-(1 << bits), 1 << bits, 2000)]
        for X in vals:
            d = digits(lib, X)
            assert all(-128 <= v <= 127 for v in d) and -64 <= d[0] <= 64
            assert sum(v * 256 ** (len(d) - 1 - i) for i, v in enumerate(d)) == X


def test_values_off_the_grid_are_marked(lib):
    rng = np.random.default_rng(2)
    for largest in list(range(1, 0x7F80, 97)) + [1, 127, 128, 37 * 128, 0x7F7F]:
        ex = lib.digits_exponent(largest)
        assert bf16(largest) < Fraction(2) ** ex
        unit = Fraction(2) ** (ex - 30)
        edge = max(0, (104 + ex) * 128)
        for v in [1, 2, 127, 128] + list(range(max(1, edge - 140), edge + 3)) + [int(r) for r in rng.integers(1, 0x7F80, 20)]:
            if v > largest:
                continue
            off = bool(lib.digits_off(v, ex))
            on_grid = (bf16(v) / unit).denominator == 1
            assert off or on_grid
            assert not off or v < edge  # a value of eight bits on the grid is not marked
        assert not lib.digits_off(0, ex)  # none but zeros


def test_smallest_value_but_zeros(lib):
    rng = np.random.default_rng(3)
    for _ in range(300):
        h = rng.integers(0, 0x7F80, 16)
        h[rng.random(16) < rng.choice([0.0, 0.5, 0.95])] = 0
        sign = rng.integers(0, 2, 16) << 15
        u = (h | sign).astype(np.uint64)
        pairs = (C.c_uint * 8)(*[int(u[2 * i] | u[2 * i + 1] << np.uint64(16)) for i in range(8)])
        assert lib.digits_smallest(pairs, 8) == (int(h[h > 0].min()) if (h > 0).any() else 0)
    for a, b, want in ((0, 0, 0), (1, 0, 1), (0, 1, 1), (0x8000, 0x8001, 1), (0x7FFF, 0x7F7F, 0x7F7F)):
        assert lib.digits_smallest((C.c_uint * 1)(a | b << 16), 1) == want


def test_sums_fit_at_the_largest_k():
    top = [64] + [128] * 3, [64] + [128] * 4
    level = [0] * 8
    for i, x in enumerate(top[0]):
        for j, w in enumerate(top[1]):
            level[i + j] += x * w * MAX_K
    assert max(level) < 2 ** 31
    for part in (level[:3], level[3:6], level[6:]):
        assert sum(v << 8 * (len(part) - 1 - n) for n, v in enumerate(part)) < 2 ** 51


@pytest.mark.parametrize("outlier", [0, 12, 23, 40, 100])
def test_levels_and_what_they_leave_out_add_up_to_the_exact_logit(lib, outlier):
    rng = np.random.default_rng(1)
    x = rng.normal(size=96).astype(np.float32)
    x[3], x[7] = 0.0, 2.0 ** outlier
    xb = x.view(np.uint32) >> 16  # bf16 values
    w = (rng.normal(size=96) * 0.02).astype(np.float32)
    w[5] = 0.5
    w = (w.view(np.uint32) & 0xFFFF0000).view(np.float32)  # on the grid
    pairs = (C.c_uint * 48)(*[int(xb[2 * i]) | int(xb[2 * i + 1]) << 16 for i in range(48)])
    ex = lib.digits_exponent(int((xb & 0x7FFF).max()))
    off = bool(lib.digits_off(lib.digits_smallest(pairs, 48), ex))
    ew = int(np.floor(np.log2(np.abs(w).max()))) + 1
    xs = [(-1 if v >> 15 else 1) * bf16(int(v) & 0x7FFF) for v in xb]
    X = [round(v * Fraction(2) ** (30 - ex)) for v in xs]
    W = [Fraction(float(v)) * Fraction(2) ** (38 - ew) for v in w]
    assert all(v.denominator == 1 for v in W)
    level = [0] * 8
    for a, b in zip(X, W):
        for i, p in enumerate(x_digits(lib, a)):
            for j, q in enumerate(w_digits(lib, int(b))):
                level[i + j] += p * q
    p3 = (C.c_longlong * 3)()
    lib.digits_levels((C.c_int * 8)(*level), p3)
    got = Fraction(2) ** (ex + ew - 28) * (p3[0] + Fraction(p3[1], 2 ** 24) + Fraction(p3[2], 2 ** 40))
    left = [v - a * Fraction(2) ** (ex - 30) for v, a in zip(xs, X)]
    assert off == (outlier > 12) and (off or not any(left)) and (outlier < 40 or any(left))
    want = sum(a * Fraction(float(b)) for a, b in zip(xs, w))
    assert got + sum(a * Fraction(float(b)) for a, b in zip(left, w)) == want
