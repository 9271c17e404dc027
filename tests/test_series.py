"""The series by which the device refines its approximate reciprocal and reciprocal square root
(rcp_pos, rsqrt_pos): with any start of 20 correct bits the result is within 1.5 units in the last
place, every operation rounded to double as the device rounds it (fused multiply-adds once).  This is
the derivation of the bound; test_gpu_reciprocals.py measures the device functions against it."""
import math
import random
from fractions import Fraction as Q


def fma(a, b, c):
    return float(Q(a) * Q(b) + Q(c))


def rcp(b, y):
    e = fma(-b, y, 1.0)
    return fma(y, fma(e, e, e), y)


def rsqrt(x, y):
    e = fma(-(x * y), y, 1.0)
    return fma(y * e, fma(0.375, e, 0.5), y)


def test_refined_reciprocals_are_within_two_ulp():
    rng = random.Random(1)
    for _ in range(3000):
        b = math.ldexp(rng.uniform(1.0, 2.0), rng.randint(-60, 60))
        off = 1.0 + rng.choice([-1.0, 1.0, rng.uniform(-1.0, 1.0)]) * 2.0 ** -20
        r = rcp(b, off / b)
        assert abs(Q(r) * Q(b) - 1) <= Q(3, 2) * Q(2) ** -52
        s = rsqrt(b, off / math.sqrt(b))
        # s^2 b = (1 + d)^2 with d the relative error
        assert abs(Q(s) * Q(s) * Q(b) - 1) <= 2 * Q(3, 2) * Q(2) ** -52
