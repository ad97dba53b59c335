"""The FP64 closed form's own approximations (CPU only): the degree-20 erfcx fit on 1 <= u <= 100 and the series T on
u < 1, with q from zeta = 3 q + rho^2 F.

Tolerances: erf is formed as 1 - e^{-y^2} z P; SciPy's erfcx and the double arithmetic are good to a few eps, and
e^{-y^2} erfcx <= 0.32 on the interval, so 4e-16 absolute.  The series has no cancellation: 8 eps of q and F."""
import math
import re
from pathlib import Path

import numpy as np
from scipy.special import erfcx

HDR = (Path(__file__).resolve().parents[1] / "pawan_b200" / "csrc" / "pair_math.cuh").read_text()


def array(name):
    return [float(x) for x in re.search(r"%s\[\d+\] = \{[^\n]*?([-+0-9.e,\s]*[-+0-9.e])\s*\};" % name,
                                        re.sub(r"//[^\n]*", "", HDR)).group(1).replace("\n", " ").split(",") if x.strip()]


def scalar(name):
    return float(re.search(r"%s = ([-+0-9.e]+);" % name, HDR).group(1))


def test_erfcx_fit_fp64():
    P = array("kErfcx64")
    assert len(P) == 21
    u = np.exp(np.linspace(0.0, math.log(100.0), 200001))
    y = np.sqrt(u / 2)
    z = 1 / y
    t = scalar("kErfcx64A") * z + scalar("kErfcx64B")
    assert t.min() >= -1 - 1e-12 and t.max() <= 1 + 1e-12
    err = np.exp(-y * y) * (z * np.polyval(P[::-1], t) - erfcx(y))
    assert np.abs(err).max() <= 4e-16


def test_series_fp64():
    T = array("kSeriesT64")
    ref = [(-1) ** m / (2.0 ** m * math.factorial(m) * (2 * m + 5)) for m in range(15)]
    assert np.allclose(T, ref, rtol=4e-16, atol=0)
    # q and F against longer series in extended precision
    u = np.linspace(0.0, 1.0, 2001)
    ul = u.astype(np.longdouble)
    Tl = sum(np.longdouble((-1) ** m) * ul ** m / (np.longdouble(2) ** m * math.factorial(m) * (2 * m + 5)) for m in range(30))
    Sl = sum(np.longdouble((-1) ** m) * ul ** m / (np.longdouble(2) ** m * math.factorial(m) * (2 * m + 3)) for m in range(30))
    Td = np.polyval(T[::-1], u)
    Sd = (np.exp(-0.5 * u) + u * Td) / 3.0
    eps = 8 * np.finfo(np.float64).eps
    assert np.abs(Td / Tl - 1).max() <= eps
    assert np.abs(Sd / Sl - 1).max() <= eps
