"""States that are not numbers must show in the results: a NaN that a box test, a vote or a minimum passes over would let
a diverged wake reach its caller as plausible values.  No tolerances: rows are NaN or they are not."""
import numpy as np
import pytest

from pawan_b200 import capi, cases

pytestmark = pytest.mark.gpu
NU = 1e-4


def ring(n, sigma=0.02):
    return cases.ring_stations(stations=max(16, -(-n // 25)), sigma=sigma, seed=3).subset(n)


def context(w, precision=capi.FP32C, **kw):
    c = capi.Context(precision=precision, nu=NU, **kw)
    k = c.add_wake(w.n)
    c.set_particles(k, w)
    return c, k


@pytest.mark.parametrize("n", [40, 300, 3000, 9000])
@pytest.mark.parametrize("what", ["pos", "sigma"])
def test_field_of_a_nan_particle(gpu, n, what):
    """The field sums every particle at every target, so one NaN position or radius makes every row NaN (as PAWAN's sum),
    also where the rest of its slice is beyond the exponential's reach."""
    w = ring(n)
    getattr(w, what)[17] = np.nan
    c, k = context(w)
    assert np.isnan(c.vorticity_field(k)).any(axis=1).all()
