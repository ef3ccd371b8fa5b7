"""The FP64 kernels form the source's quotients a/b (a grid-spacing divisor b
with a host-tabulated reciprocal rb = RN(1/b)) by Markstein's correction:
q = RN(a rb), r = RN(a - b q) (one fused multiply-add, exact), RN(q + r rb)
(a second one).  This restates the three roundings exactly with rationals and
checks the claim the kernels rely on, RN(q + r rb) == RN(a/b), on random
operands of the solver's ranges (velocity differences and metric sums over
spacings from 1e-5 to 1e2) and on edge cases of the significands (divisors
and dividends with all-ones or power-of-two significands, and near-ties).
The FP32 strain kernels run the same steps with b and rb rounded separately
from the FP64 spacing, for which the bound on the error is checked."""
import math
import struct
from fractions import Fraction

import numpy as np


def rn(x):
    """round a rational to the nearest double (ties to even)"""
    return float(x)


def markstein(a, b):
    rb = 1.0 / b                                # the host table: RN(1/b)
    q = rn(Fraction(a) * Fraction(rb))          # __dmul_rn(a, rb)
    r = rn(Fraction(a) - Fraction(q) * Fraction(b))    # __fma_rn(-q, b, a)
    return rn(Fraction(r) * Fraction(rb) + Fraction(q))  # __fma_rn(r, rb, q)


def with_mantissa(bits, exp):
    return struct.unpack("<d", struct.pack("<Q", ((exp + 1023) << 52) | (bits & ((1 << 52) - 1))))[0]


def test_random_operands_of_the_solver():
    rng = np.random.default_rng(2024)
    n = 40000
    b = 10.0 ** rng.uniform(-5, 2, n)          # spacings
    a = rng.standard_normal(n) * 10.0 ** rng.uniform(-12, 2, n)  # differences and sums
    bad = [(x, y) for x, y in zip(a.tolist(), b.tolist()) if markstein(x, y) != x / y]
    assert not bad, bad[:5]


def test_significand_edge_cases():
    cases = []
    for eb in (-17, -3, 0, 5):
        for mb in (0, 1, (1 << 52) - 1, (1 << 51), (1 << 52) - 2, 0x5555555555555, 0xAAAAAAAAAAAAA):
            b = with_mantissa(mb, eb)
            for ea in (-40, -9, 0, 3):
                for ma in (0, 1, (1 << 52) - 1, (1 << 51) + 1, 0x123456789ABCD, mb):
                    for s in (1.0, -1.0):
                        cases.append((s * with_mantissa(ma, ea), b))
    # near-ties: a = b * (q + 1/2 ulp) rounded, for quotients of every binade edge
    rng = np.random.default_rng(7)
    for _ in range(2000):
        b = float(10.0 ** rng.uniform(-4, 1))
        q = float(rng.uniform(1, 2)) * 2.0 ** int(rng.integers(-20, 20))
        ulp = math.ulp(q)
        cases.append((rn(Fraction(b) * (Fraction(q) + Fraction(ulp) / 2)), b))
        cases.append((rn(Fraction(b) * (Fraction(q) + Fraction(ulp) / 2)) + math.ulp(b * q), b))
    bad = [(x, y) for x, y in cases if markstein(x, y) != x / y]
    assert not bad, bad[:5]


def test_fp32_quotients_of_separately_rounded_tables():
    """FP32: b = RN(b64) and rb = RN(1/b64), so rb is within 2^-23 of 1/b
    (relative) and not its rounding.  q = RN(a rb) is within 3 ulp of a/b, the
    remainder and the correction carry relative errors of 2^-24 and 2^-22 of
    those 3 ulp, and the result is RN(a/b + e) with |e| below 2^-20 ulp: at most
    (1/2 + 2^-20) ulp from a/b."""
    rng = np.random.default_rng(11)
    n = 20000
    b64 = (10.0 ** rng.uniform(-5, 2, n)).tolist()
    a32 = (rng.standard_normal(n) * 10.0 ** rng.uniform(-6, 2, n)).astype(np.float32)

    def rn32(x):  # of a rational with few more bits than a double holds: no double rounding
        d = float(x)
        f = np.float32(d)
        if Fraction(d) != x:  # decide a midpoint by the rational itself
            lo, hi = sorted((float(np.nextafter(f, np.float32(-np.inf))), float(np.nextafter(f, np.float32(np.inf)))))
            f = min((np.float32(v) for v in (lo, float(f), hi)), key=lambda v: abs(Fraction(float(v)) - x))
        return float(f)

    worst = Fraction(0)
    for a, b64_ in zip(a32.tolist(), b64):
        b, rb = rn32(Fraction(b64_)), rn32(Fraction(1.0 / b64_))
        q = rn32(Fraction(a) * Fraction(rb))
        r = rn32(Fraction(a) - Fraction(q) * Fraction(b))
        z = rn32(Fraction(r) * Fraction(rb) + Fraction(q))
        exact = Fraction(a) / Fraction(b)
        ulp = Fraction(float(np.spacing(np.float32(abs(float(exact))))))
        worst = max(worst, abs(Fraction(z) - exact) / ulp)
    # exact may round up to the next binade, whose spacing is twice: its ulp counts half there
    assert worst <= Fraction(1, 2) + Fraction(1, 1 << 20)
