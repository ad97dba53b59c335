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


@pytest.mark.parametrize("kernel,n,npts,by_points", [
    ("gaussian", 1, 30000, True), ("gaussian", 1, 29999, False), ("gaussian", 128, 30001, True),
    ("gaussian", 129, 30000, False), ("gaussian", 257, 100000, True), ("gaussian", 400, 100031, True),
    ("gaussian", 401, 100000, False), ("highorder", 25, 59999, False), ("highorder", 25, 60000, True),
    ("highorder", 3000, 60001, True)])
def test_probe_many_points(gpu, kernel, n, npts, by_points):
    """Calls whose points fill the device sum each point in one thread, one launch instead of two; 1e-11 of the largest
    velocity, as the probe tests of few points."""
    w = cases.ring_stations(stations=max(16, -(-n // 25)), seed=3).subset(n)
    pts = np.random.default_rng(n + npts).normal(0.0, 0.8, (npts, 3))
    c = capi.Context(precision=capi.FP32C, nu=NU, kernel=kernel)
    c.set_particles(c.add_wake(n), w)
    c.probe(pts)
    before = c.launch_count()
    v = c.probe(pts)
    assert c.launch_count() - before == (1 if by_points else 2)
    rows = np.concatenate(([0, 31, 32, 255, 256, npts - 1], np.random.default_rng(1).integers(0, npts, 20)))
    ref = np.array([O.restate_getvi(w, pts[k], kernel) for k in rows])
    assert np.abs(v[rows] - ref).max() <= 1e-11 * np.abs(v).max()


def test_probe_many_points_of_a_nan_particle(gpu):
    for what in ("pos", "sigma", "alpha"):
        w = cases.ring_stations(stations=16, seed=3).subset(100)
        getattr(w, what)[17] = np.nan
        c = capi.Context(precision=capi.FP32C, nu=NU)
        c.set_particles(c.add_wake(100), w)
        v = c.probe(np.random.default_rng(0).normal(0.0, 5.0, (30000, 3)))
        assert np.isnan(v).any(axis=1).all()


@pytest.mark.parametrize("kernel", ["gaussian", "highorder"])
def test_many_small_fp64_systems(gpu, kernel):
    """Four times as many systems of 128 particles take about four times as long (their rows never took slices longer than
    the systems; the first ones also pay for filling the device), and give the rates of the FP64 restatement."""
    ms = []
    for count in (781, 3125):
        wakes = [cases.ring_stations(stations=16, seed=k).subset(128) for k in range(7)]
        c = capi.Context(precision=capi.FP64, nu=NU, kernel=kernel)
        ids = [c.add_wake(128, system=s) for s in range(count)]
        for k in ids:
            c.set_particles(k, wakes[k % 7])
        c.solve()
        c.pair_kernel_time()
        for _ in range(3):
            c.solve()
        t, launches = c.pair_kernel_time()
        ms.append(t / launches)
        for k in (ids[0], ids[-1]):
            for got, ref in zip(c.rates(k), O.restate_rates(wakes[k % 7], NU, kernel=kernel)):
                assert np.abs(got - ref).max() <= 1e-12 * np.abs(ref).max()
    assert ms[1] <= 4.8 * ms[0]


@pytest.mark.parametrize("precision,kernel,split", [(capi.FP32C, "gaussian", False), (capi.FP32C, "gaussian", True),
                                                    (capi.FP32C, "highorder", False)])
def test_class_tuning_keeps_the_row_list(gpu, tmp_path, precision, kernel, split):
    """Three small rings: the row list takes a third of the tiles' time, so tuning by class leaves it (no box kernel before
    the pair launch, one pair launch), from measured and from cached times; results stay within FP32 rounding."""
    wakes = [cases.ring_stations(stations=s, seed=s) for s in (40, 60, 200)]
    cache = str(tmp_path / "tune.jsonl")
    for run in range(2):
        c = capi.Context(precision=precision, nu=NU, kernel=kernel, split_positions=split)
        ids = [c.add_wake(w.n, system=s) for s, w in enumerate(wakes)]
        for k, w in zip(ids, wakes):
            c.set_particles(k, w)
        c.solve()
        before, c0 = [c.rates(k) for k in ids], c.pair_kernel_time()
        for _ in range(3):
            c.solve()
        t0, n0 = c.pair_kernel_time()
        tune = c.autotune_classes(reps=2, cache=cache)
        assert not tune["per_class"] and all(x["from_cache"] == (run == 1) for x in tune["classes"])
        assert launches(c) == 2
        c.pair_kernel_time()
        for _ in range(3):
            c.solve()
        t1, n1 = c.pair_kernel_time()
        assert t1 / n1 <= 1.2 * t0 / n0
        for k, rates in zip(ids, before):
            for got, ref in zip(c.rates(k), rates):
                assert np.array_equal(got, ref)


def test_class_tuning_with_an_older_cache(gpu, tmp_path):
    """Lines without the row list's time: it is timed, and loses to the shapes' recorded times here (1 us)."""
    import json

    import torch
    shapes = capi.kernel_shapes()
    b, t = shapes[1]
    cache = tmp_path / "tune.jsonl"
    cache.write_text("".join(json.dumps({
        "gpu": torch.cuda.get_device_properties(0).name, "precision": "fp32c", "kernel": "gaussian", "class": k, "nmin": 0,
        "nmax": 0, "block": b, "tpt": t, "ms": [0.001 if i == 1 else 9.0 for i in range(len(shapes))]}) + "\n"
        for k in (0, 1)))
    wakes = [cases.ring_stations(stations=s, seed=s) for s in (40, 200)]
    c = capi.Context(precision=capi.FP32C, nu=NU)
    ids = [c.add_wake(w.n, system=s) for s, w in enumerate(wakes)]
    for k, w in zip(ids, wakes):
        c.set_particles(k, w)
    tune = c.autotune_classes(reps=1, cache=str(cache))
    assert all(x["from_cache"] for x in tune["classes"]) and not tune["per_class"]
    assert launches(c) == 3  # the tiles


def test_tuning_under_the_surrogate(gpu):
    """The surrogate's evaluations have no shape: tuning leaves the choice alone, and the row list is back after it."""
    w = cases.ring_stations(stations=40, seed=1)
    c = capi.Context(precision=capi.FP32C, nu=NU)
    k = c.add_wake(w.n)
    c.set_particles(k, w)
    c.solve()
    before = c.rates(k)
    c.surrogate_enable(0)
    (block, tpt), ms = c.autotune(reps=1)
    assert (block, tpt) == (128, 2) and set(ms.values()) == {0.0}
    c.surrogate_disable()
    assert launches(c) == 2  # the row list
    for got, ref in zip(c.rates(k), before):
        assert np.array_equal(got, ref)


def test_tuning_again_at_another_size(gpu):
    """A shape that won at a large size is weighed against the row list when the context is tuned at a small one."""
    big = section_ring(60000)
    small = cases.ring_stations(stations=40, seed=1)
    c = capi.Context(precision=capi.FP32C, nu=NU)
    k = c.add_wake(big.n)
    c.set_particles(k, big)
    c.autotune(reps=1)
    assert launches(c) == 3  # tiles
    c.set_particles(k, small)
    assert launches(c) == 3  # tuned: stays
    c.autotune(reps=2)
    assert launches(c) == 2


@pytest.mark.parametrize("shape", [{}, {"block": 128, "tpt": 1}, {"block": 128, "tpt": 2}, {"block": 64, "tpt": 2},
                                   {"block": 128, "tpt": 4}])
@pytest.mark.parametrize("precision,limit", [(capi.FP32C, 50.0), (capi.FP64, 100.0)])
@pytest.mark.parametrize("n", [33, 1000, 1001, 1024])
def test_pair_counts(gpu, n, precision, limit, shape):
    """Pairs and full-formula pairs as counted on the CPU, in every kernel, also where lanes repeat the last target.  FP32C
    decides u < 50 in FP32, so pairs within 1e-5 of it may go either way."""
    w = cases.ring_stations(stations=-(-n // 25), sigma=0.02, seed=3).subset(n)
    u = ((w.pos[:, None] - w.pos[None]) ** 2).sum(-1) / (0.5 * (w.sigma[:, None] ** 2 + w.sigma[None] ** 2))
    c = capi.Context(precision=precision, nu=NU, **shape)
    c.set_particles(c.add_wake(n), w)
    c.solve()
    pairs, full = c.pair_counts()
    assert pairs == n * (n - 1)
    slack = 1e-5 if precision == capi.FP32C else 1e-12
    assert (u < limit * (1 - slack)).sum() - n <= full <= (u < limit * (1 + slack)).sum() - n


@pytest.mark.parametrize("precision", [capi.FP32C, capi.FP64])
@pytest.mark.parametrize("n", [25, 1000, 5000])
def test_pair_time_of_graph_steps(gpu, n, precision):
    """Pair-kernel times of graph steps against those of the same steps without graphs, which bracket the launch: shorter by
    the launch, about 4 us, and no longer; a few us more either way are allowed."""
    w = cases.ring_stations(stations=-(-n // 25), seed=3).subset(n)
    us = []
    for graphs in (True, False):
        c = capi.Context(precision=precision, nu=NU, use_graphs=graphs)
        c.set_particles(c.add_wake(n), w)
        best = 1e9
        for _ in range(6):
            c.step("rk4", 1e-4, 10)
            t, launches = c.pair_kernel_time()
            assert launches == 40
            best = min(best, 1e3 * t / launches)
        us.append(best)
    assert us[1] - 9.0 <= us[0] <= us[1] + 3.0
    assert us[0] > 0.5 * us[1]
