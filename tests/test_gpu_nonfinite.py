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


@pytest.mark.parametrize("n", [40, 300, 3000, 9000])
@pytest.mark.parametrize("kernel", ["gaussian", "highorder"])
def test_rates_of_a_nan_radius(gpu, n, kernel):
    """A NaN radius: the high-order kernel's terms need it for every pair, the Gaussian kernel's for the pairs near the
    particle, itself among them; particles a whole diameter away keep finite rates there."""
    w = ring(n)
    w.sigma[17] = np.nan
    c, k = context(w, kernel=kernel)
    c.solve()
    bad = np.isnan(np.concatenate(c.rates(k), axis=1)).any(axis=1)
    assert bad[17]
    if kernel == "highorder":
        assert bad.all()
    elif n >= 3000:
        assert not bad[n // 2]


def test_surrogate_rates_of_a_nan_radius(gpu):
    w = ring(3000)
    w.sigma[17] = np.nan
    c, k = context(w)
    c.surrogate_enable(0, check_targets=0)
    c.solve()
    v, a = c.rates(k)
    assert np.isnan(v[17]).any() and np.isnan(a[17]).any()


@pytest.mark.parametrize("kernel", ["gaussian", "highorder"])
@pytest.mark.parametrize("what", ["pos", "alpha", "sigma"])
def test_probe_of_a_nan_particle(gpu, what, kernel):
    """Every particle acts on every point, near or far."""
    w = ring(1000)
    getattr(w, what)[17] = np.nan
    c, _ = context(w, kernel=kernel)
    assert np.isnan(c.probe([[1.0, 0.0, 0.01], [30.0, -20.0, 5.0], [0.0, 0.0, 0.0]])).any(axis=1).all()
