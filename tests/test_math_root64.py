"""The FP64 reciprocal root's refinement step (CPU only): y + y e (1/2 + 3/8 e) with e = 1 - x y^2, Chebyshev's third-order
method for 1/y^2 = x, on seeds as far off as the hardware approximation.

Tolerance: the result rounds to 2^-53 relative; x y rounds to 2^-53, half of which reaches the result through e / 2; the
method leaves 5/16 e^3 = 3.0e-18 for seeds off by 2^-20 (e = 2^-19), and y e rounds far below: 1.5 x 2^-53 + 3.0e-18 + 1e-21
= 1.70e-16."""
import re
from fractions import Fraction
from pathlib import Path

import numpy as np

HDR = (Path(__file__).resolve().parents[1] / "pawan_b200" / "csrc" / "pair_math.cuh").read_text()


def fma(a, b, c):
    return float(Fraction(a) * Fraction(b) + Fraction(c))


def test_root_step():
    body = re.search(r"double rsqrt_normal\(double x\).*?\n\}", HDR, re.S).group(0)
    assert "fma(-(x * y), y, 1.0)" in body and "fma(y * e, fma(0.375, e, 0.5), y)" in body
    rng = np.random.default_rng(0)
    for k in range(4000):
        x = float(rng.uniform(1.0, 4.0) * 2.0 ** int(rng.integers(-300, 300)))
        off = (-1.0, 1.0, 0.0)[k % 3] * 2.0 ** -20 if k % 4 else rng.uniform(-1, 1) * 2.0 ** -20
        y = float(np.longdouble(1) / np.sqrt(np.longdouble(x)) * (1 + np.longdouble(off)))
        e = fma(-(x * y), y, 1.0)
        r = fma(y * e, fma(0.375, e, 0.5), y)
        # r sqrt(x) - 1 from (r^2 x - 1) / 2, exact
        err = (Fraction(r) * Fraction(r) * Fraction(x) - 1) / 2
        assert abs(err) <= Fraction(1.70e-16)
