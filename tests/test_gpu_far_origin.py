"""FP64 sums of wakes far from the origin, where neighbouring cores fall on different FP32 numbers: the box tests that
choose the far limit work in FP32 and must not take such pairs for far ones."""
import numpy as np
import pytest

from oracle import oracle as O
from pawan_b200 import capi, cases

pytestmark = pytest.mark.gpu
NU = 1e-4


def far_ring(n, scale):
    w = cases.ring_stations(stations=n // 25, sigma=0.02, seed=3)
    w.pos = w.pos + scale * np.array([1.0, 0.7, 0.3])
    return w


@pytest.mark.parametrize("shape", [{}, {"block": 128, "tpt": 1}])
@pytest.mark.parametrize("n", [3000, 9000])
@pytest.mark.parametrize("scale", [1e6, 1e7, 3e7])
def test_rates_fp64(gpu, n, scale, shape):
    """1e-12 of the largest rate: the sums' rounding, as for wakes around the origin (differences of positions are
    exact in both sums, so the offset adds nothing)."""
    w = far_ring(n, scale)
    c = capi.Context(precision=capi.FP64, nu=NU, **shape)
    k = c.add_wake(w.n)
    c.set_particles(k, w)
    c.solve()
    rows = np.arange(0, n, 7)
    for got, ref in zip(c.rates(k), O.restate_rates(w, NU, targets=rows)):
        assert np.abs(got[rows] - ref).max() <= 1e-12 * np.abs(ref).max()


@pytest.mark.parametrize("n", [3000, 9000])
@pytest.mark.parametrize("scale", [1e6, 1e7, 3e7])
def test_field(gpu, n, scale):
    """1e-11, as the field tests around the origin."""
    w = far_ring(n, scale)
    c = capi.Context(precision=capi.FP32C, nu=NU)
    k = c.add_wake(w.n)
    c.set_particles(k, w)
    rows = np.arange(0, n, 7)
    ref = O.restate_vorticity_field(w, targets=rows)
    assert np.abs(c.vorticity_field(k)[rows] - ref).max() <= 1e-11 * np.abs(ref).max()
