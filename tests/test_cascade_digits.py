"""The digit split of the cascade's GEMM steps (via_rs_b200/csrc/cascade_tc.cu ct_pieces and
ct_digit), restated with IEEE doubles and exact-rational FMAs, against the gadget decomposition's
definition (centred lift, round(|c| B^L / Q), balanced base-B digits). No GPU needed.

The kernels never form c in [0, Q): with y_l = c_l (Q / q_l)^-1 mod q_l they take three exact
steps T y_l = p q_l + y_l' per prime (T = B^6) and read 32-bit fractions of the three pieces."""
from fractions import Fraction

import numpy as np
import pytest

from via_rs_b200.params import PAPER_Q1, SECURE_Q1

ROUND = 6755399441055744.0  # 1.5 * 2^52
L, LP = 18, 6


def fma(a, b, c):
    return float(Fraction(a) * Fraction(b) + Fraction(c))


def reference_digits(c, Q, B):
    S = B**L
    cc = c if c <= Q // 2 else c - Q
    v = (abs(cc) * S + Q // 2) // Q
    v = (v if cc >= 0 else -v) % S
    out = []
    for _ in range(L):
        r = v % B
        d = r - B if r > B // 2 else r
        out.append(d)
        v = (v - d) // B
    return out[::-1]  # most significant first: sample order


def centred_by_rounding(a, q):
    """A representative within q / 2 + 1, as the kernels' reductions leave it."""
    r = fma(-((fma(float(a), 1.0 / q, ROUND)) - ROUND), float(q), float(a))
    return r


def kernel_digits(y, q, B):
    T = B**LP
    o = B - 1 - B // 2
    sh = 0
    while (1 << (sh + 1)) < T:
        sh += 1
    M = -(-(1 << (32 + sh)) // T)
    assert 1 << 31 <= M < 1 << 32
    off = o * ((T - 1) // (B - 1)) + 2 * T
    qinv = [1.0 / float(x) for x in q]
    p = []
    for _ in range(3):
        s = 0
        for l in range(2):
            h = float(T) * y[l]
            lo = fma(float(T), y[l], -h)
            u = fma(h, qinv[l], ROUND)
            s += int(u - ROUND)
            y[l] = fma(-(u - ROUND), float(q[l]), h) + lo
            assert abs(y[l]) <= 0.5625 * q[l] and y[l] == int(y[l])
        p.append(s)
    s = fma(y[0], qinv[0], y[1] * qinv[1])
    us = s + ROUND
    rnd = int(us - ROUND)
    if abs(s - (us - ROUND)) > 0.5 - 1e-12:
        num, Q = int(y[0]) * q[1] + int(y[1]) * q[0], q[0] * q[1]
        rnd = 1 if 2 * num > Q else (-1 if 2 * num < -Q else 0)
    carry, f = 2, [0, 0, 0]
    for i in (2, 1, 0):
        x = p[i] + (rnd if i == 2 else 0) + off + carry - 2
        assert 0 <= x < 1 << 29
        carry = (x * M >> 32) >> sh
        assert carry == x // T
        f[i] = ((x - carry * T) * M >> sh) + 1
        assert f[i] < 1 << 32
    out = []
    for i in range(3):
        g = f[i]
        for _ in range(LP):
            g *= B
            out.append((g >> 32) - o)
            g &= (1 << 32) - 1
    return out


@pytest.mark.parametrize("q", [tuple(PAPER_Q1), tuple(SECURE_Q1)])
@pytest.mark.parametrize("B", [18, 20, 3])
def test_digits_equal_the_definition(q, B):
    Q, S = q[0] * q[1], B**L
    rng = np.random.default_rng(B)
    inv = [pow(q[1], -1, q[0]), pow(q[0], -1, q[1])]
    cs = [int(rng.integers(1 << 62)) * int(rng.integers(1 << 20)) % Q for _ in range(400)]
    cs += [0, 1, 2, Q - 1, Q // 2, Q // 2 + 1, Q // 2 - 1]
    # Coefficients whose scaled value lies next to a rounding boundary: c S / Q ~ m + 1/2.
    for _ in range(200):
        m = int(rng.integers(1 << 62)) * int(rng.integers(1 << 20)) % S
        c = (2 * m + 1) * Q // (2 * S)
        cs += [c % Q, (c + 1) % Q]
    for c in cs:
        y = [centred_by_rounding(c % q[l] * inv[l] % q[l], q[l]) for l in range(2)]
        assert kernel_digits(y, q, B) == reference_digits(c, Q, B), c
