"""Which kernel an evaluation takes, seen from the number of kernels it launches: the row list is one launch and the stage
kernel, the CTA-wide tiles of FP32C launch a box kernel before."""
import numpy as np
import pytest

from oracle import oracle as O
from pawan_b200 import capi, cases

pytestmark = pytest.mark.gpu
NU = 1e-4


def rotor(n):
    s = cases.RotorShedder(per_blade=200, omega=10.0)
    parts = [s.shed() for _ in range(n // 800)]
    for age, w in enumerate(reversed(parts)):  # carried down with the inflow since it was shed
        w.pos += age * s.dt * np.array(s.inflow)
    return cases.Wake.concat(parts)


def section_ring(n):
    return cases.ring_gaussian(stations=n // 250, per_section=250, seed=1)


def launches(c):
    c.solve()
    before = c.launch_count()
    c.solve()
    return c.launch_count() - before


@pytest.mark.parametrize("wakes,rows", [((section_ring(40000),), True), ((section_ring(60000),), False),
                                        ((rotor(40000),), True), ((rotor(60000),), True),
                                        ((section_ring(30000), section_ring(30000)), False),
                                        ((rotor(30400), rotor(30400)), True)])
def test_split_positions(gpu, wakes, rows):
    """Beyond 48,000 targets the row list stays for dense filaments only, where its finer boxes save closed-form pairs; the
    rates are the same to the library's gate of 1e-5 either way."""
    c = capi.Context(precision=capi.FP32C, nu=NU, split_positions=True)
    ids = [c.add_wake(w.n, system=s) for s, w in enumerate(wakes)]
    for k, w in zip(ids, wakes):
        c.set_particles(k, w)
    assert launches(c) == (2 if rows else 3)
    for k, w in zip(ids, wakes):
        t = np.linspace(0, w.n - 1, 20).astype(np.int64)
        for got, ref in zip(c.rates(k), O.restate_rates(w, NU, targets=t)):
            assert np.abs(got[t] - ref).max() <= 1e-5 * np.abs(got).max()


@pytest.mark.parametrize("n,most", [(4000, 2), (8192, 2), (8193, 1), (24676, 1), (65536, 1), (65537, 1)])
def test_upload_launches(gpu, n, most):
    """Two halves of the pinned ring at most: uploads that would turn it over (a wait for the stream each time) go through
    the device's staging buffer in one piece."""
    w = section_ring(-(-n // 250) * 250).subset(n)
    c = capi.Context(precision=capi.FP32C, nu=NU)
    k = c.add_wake(n)
    c.set_particles(k, w)
    before = c.launch_count()
    c.set_particles(k, w)
    assert c.launch_count() - before <= most
    for got, ref in zip(c.particles(k), (w.pos, w.alpha, w.sigma, w.vol)):
        assert np.array_equal(got, ref)
