"""The octree's near field alone (every cell is near), against the FP64 mode of the direct sum."""
import math

import numpy as np
import pytest
from scipy.special import erf

from pawan_b200 import capi, cases

pytestmark = pytest.mark.gpu
NU = 1e-4


def both(w, leaf):
    """FP64 rates of the direct sum and FP32C rates of the near field."""
    rates = []
    for precision in (capi.FP64, capi.FP32C):
        c = capi.Context(precision=precision, nu=NU)
        k = c.add_wake(w.n)
        c.set_particles(k, w)
        if precision == capi.FP32C:
            c.surrogate_enable(0, leaf_size=leaf, near_widths=1e6, check_targets=0)
        c.solve()
        rates.append(c.rates(k))
    return rates


@pytest.mark.parametrize("radii", [1, 2])
@pytest.mark.parametrize("n,leaf", [(33, 16), (300, 1), (1000, 7), (2000, 256), (2001, 512)])
def test_near_field_rates(gpu, n, leaf, radii):
    """Slices of one radius and of two.  Per target, the pair terms are good to 1e-6 (16 x 2^-24) and a group of 32 sources
    rounds to 32 x 2^-24 of the sum of their magnitudes: q |alpha_s| r for the velocity, at most 4 q |alpha_t| |alpha_s|
    for dalpha (|F| r^2 <= 3 q; the diffusion of nu = 1e-4 is below that)."""
    w = cases.ring_gaussian(stations=max(8, -(-n // 50)), per_section=50, seed=1).subset(n)
    if radii == 2:
        w.sigma[::3] *= 0.8
    d = w.pos[:, None] - w.pos[None]
    r = np.sqrt((d ** 2).sum(-1)) + np.eye(n)
    s = np.sqrt(0.5 * (w.sigma[:, None] ** 2 + w.sigma[None] ** 2))
    q = (erf(r / (math.sqrt(2) * s)) - math.sqrt(2 / math.pi) * r / s * np.exp(-0.5 * (r / s) ** 2)) / (4 * math.pi * r ** 3)
    q = (q * (1 - np.eye(n))) * np.linalg.norm(w.alpha, axis=1)[None]
    scale = ((q * r).sum(1), 4 * q.sum(1) * np.linalg.norm(w.alpha, axis=1))
    for ref, got, m in zip(*both(w, leaf), scale):
        assert (np.linalg.norm(got - ref, axis=1) <= 48 * 2.0 ** -24 * m.max()).all()


def test_near_field_groups(gpu):
    """Compensated every 32 sources.  The rms error of dalpha of this ring is 4.8e-7 of the largest with groups of 32 and
    6.7e-7 with 64 (rounding grows as the square root of the group): the bound lies between."""
    w = cases.ring_gaussian(stations=100, per_section=50, seed=1)
    ref, got = (x[1] for x in both(w, 256))
    assert np.sqrt(((got - ref) ** 2).sum(1).mean() / (ref ** 2).sum(1).max()) <= 5.6e-7
