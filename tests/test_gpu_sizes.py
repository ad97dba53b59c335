"""Kernels whose split of the work depends on the sizes, at the edges of their tiles, chunks and dispatch rules, against
the FP64 restatement.  Tolerances: FP64 paths sum n terms of one sign pattern in another order, n eps = 2e-12 at the
largest n here (2e4), with a margin of five; FP32C paths are held to the library's gate of 1e-5."""
import numpy as np
import pytest

from oracle import oracle as O
from pawan_b200 import capi, cases

pytestmark = pytest.mark.gpu
NU = 1e-4


def ring(n, seed=3, sigma=0.1):
    return cases.ring_stations(stations=max(16, -(-n // 25)), sigma=sigma, seed=seed).subset(n)


def context(wakes, precision, **kw):
    c = capi.Context(precision=precision, nu=NU, **kw)
    ids = [c.add_wake(w.n, system=s) for s, w in enumerate(wakes)]
    for k, w in zip(ids, wakes):
        c.set_particles(k, w)
    return c, ids


@pytest.mark.parametrize("kernel", ["gaussian", "highorder"])
@pytest.mark.parametrize("n,npts", [(1, 1), (1, 2000), (31, 8), (255, 9), (257, 7), (5000, 1), (5001, 17), (20000, 400)])
def test_probe_tiles_and_chunks(gpu, n, npts, kernel):
    """Point tiles of 8, particle chunks of any length, and a scratch need above and below the context's staging."""
    w = ring(n)
    rng = np.random.default_rng(n + npts)
    pts = rng.normal(0.0, 0.8, (npts, 3))
    pts[0] = w.pos[0]  # coincides with a particle, which the restatement (NaN there, as PAWAN) leaves out
    rest = cases.Wake(w.pos[1:], w.alpha[1:], w.sigma[1:], w.vol[1:])
    c, _ = context([w], capi.FP32C, kernel=kernel)
    v = c.probe(pts)
    rows = rng.permutation(npts)[:20]
    rows[0] = 0
    ref = np.array([O.restate_getvi(rest if k == 0 else w, pts[k], kernel) for k in rows])
    assert np.abs(v[rows] - ref).max() <= 1e-11 * np.abs(v).max()


def check_rates(c, k, w, rows, tol=1e-5):
    v, a = c.rates(k)
    rv, ra = O.restate_rates(w, NU, targets=rows)
    scale_v, scale_a = np.abs(v).max(), np.abs(a).max()
    assert np.abs(v[rows] - rv).max() <= tol * scale_v
    assert np.abs(a[rows] - ra).max() <= tol * scale_a


@pytest.mark.parametrize("split", [False, True])
@pytest.mark.parametrize("n", [25, 31, 33, 255, 257, 1000, 6700, 6720, 20011, 48000, 48001])
def test_rates_row_list(gpu, n, split):
    """The row list of small systems: below one row, ragged tiles and slices, and both sides of every rule."""
    w = ring(n)
    w.sigma[: n // 3] = 0.08  # slices of one radius and of two
    c, ids = context([w], capi.FP32C, split_positions=split)
    c.solve()
    rows = np.unique(np.linspace(0, n - 1, 40).astype(np.int64))
    check_rates(c, ids[0], w, rows)


def test_rates_row_list_batch(gpu):
    """Systems of very uneven sizes in one row list, RK3 steps of the batch as of each system alone."""
    wakes = [ring(n, seed=n) for n in (400, 25, 5003, 64, 12000)]
    c, ids = context(wakes, capi.FP32C)
    c.solve()
    for k, w in zip(ids, wakes):
        check_rates(c, k, w, np.unique(np.linspace(0, w.n - 1, 20).astype(np.int64)))
    c.step("rk3", 0.01, 2)
    c.sync()
    for k, w in zip(ids, wakes):
        one, one_id = context([w], capi.FP32C)
        one.step("rk3", 0.01, 2)
        one.sync()
        for x, y in zip(c.state(k), one.state(one_id[0])):
            assert np.abs(x - y).max() <= 1e-6 * np.abs(y).max()


@pytest.mark.parametrize("first,count", [(0, 1), (37, 33), (0, 20000), (19990, 10)])
def test_rates_row_list_target_range(gpu, first, count):
    """Few owned targets of many sources: a tile's rows are split over at most 16 partials."""
    w = ring(20000)
    c, ids = context([w], capi.FP32C)
    c.set_target_range(0, first, count)
    c.solve()
    v, a = c.rates(ids[0])
    rows = np.unique(np.linspace(first, first + count - 1, 20).astype(np.int64))
    rv, ra = O.restate_rates(w, NU, targets=rows)
    assert np.abs(v[rows] - rv).max() <= 1e-5 * np.abs(rv).max()
    assert np.abs(a[rows] - ra).max() <= 1e-5 * np.abs(ra).max()


@pytest.mark.parametrize("n", [25, 33, 257, 1000, 6700, 6720, 20011, 70003])
def test_rates_row_list_highorder(gpu, n):
    w = ring(n)
    w.sigma[: n // 3] = 0.08
    c, ids = context([w], capi.FP32C, kernel="highorder")
    c.solve()
    rows = np.unique(np.linspace(0, n - 1, 40).astype(np.int64))
    v, a = c.rates(ids[0])
    rv, ra = O.restate_rates(w, NU, targets=rows, kernel="highorder")
    assert np.abs(v[rows] - rv).max() <= 1e-5 * np.abs(v).max()
    assert np.abs(a[rows] - ra).max() <= 1e-5 * np.abs(a).max()


def test_autotune_keeps_row_list_or_a_shape(gpu):
    """After tuning, rates are the untuned ones to FP32 rounding, whichever kernel won."""
    w = ring(6000)
    for kernel in ("gaussian", "highorder"):
        c, ids = context([w], capi.FP32C, kernel=kernel)
        c.solve()
        before = c.rates(ids[0])
        (b, t), ms = c.autotune(reps=1)
        assert (b, t) in ms
        for x, y in zip(c.rates(ids[0]), before):
            assert np.abs(x - y).max() <= 1e-5 * np.abs(y).max()


@pytest.mark.parametrize("kernel", ["gaussian", "highorder"])
@pytest.mark.parametrize("n", [25, 31, 33, 255, 257, 1000, 6700, 6720, 20011])
def test_rates_row_list_fp64(gpu, n, kernel):
    """FP64 row list with cores from overlapping to far apart, so that the series, the closed form and the far limit all
    occur; the closed form's F keeps 15 eps at worst (u = 1), so 1e-12 leaves a margin of a few hundred for the sums."""
    w = ring(n)
    w.sigma[: n // 3] = 0.02
    w.sigma[n // 3: n // 2] = 0.3
    c, ids = context([w], capi.FP64, kernel=kernel)
    c.solve()
    rows = np.unique(np.linspace(0, n - 1, 40).astype(np.int64))
    v, a = c.rates(ids[0])
    rv, ra = O.restate_rates(w, NU, targets=rows, kernel=kernel)
    assert np.abs(v[rows] - rv).max() <= 1e-12 * np.abs(v).max()
    assert np.abs(a[rows] - ra).max() <= 1e-12 * np.abs(a).max()


def test_rates_fp64_far_positions(gpu):
    """Positions beyond the range of FP32 boxes: the far limit's unchecked root is not taken."""
    w = ring(400)
    w.pos[7] = [1e30, 2e25, -3e28]
    w.pos[300] = [1e170, 0.0, 0.0]
    c, ids = context([w], capi.FP64)
    c.solve()
    v, a = c.rates(ids[0])
    rows = np.array([0, 8, 100, 399])
    rest = cases.Wake(*(np.delete(x, [7, 300], axis=0) for x in (w.pos, w.alpha, w.sigma, w.vol)))
    rv, ra = O.restate_rates(rest, NU, targets=np.array([0, 7, 99, 397]))
    assert np.abs(v[rows] - rv).max() <= 1e-12 * np.abs(rv).max()
    assert np.abs(a[rows] - ra).max() <= 1e-12 * np.abs(ra).max()


@pytest.mark.parametrize("kernel", ["gaussian", "highorder"])
@pytest.mark.parametrize("n", [25, 33, 255, 257, 3000, 6720, 12011])
def test_field_row_list(gpu, n, kernel):
    """Slices of one and of several radii, some beyond the reach of the exponential."""
    w = ring(n, sigma=0.02)
    w.sigma[: n // 3] = 0.011
    other = ring(40)
    c, ids = context([w, other], capi.FP32C, kernel=kernel)
    for k, x in zip(ids, (w, other)):
        f, ref = c.vorticity_field(k), O.restate_vorticity_field(x, kernel=kernel)
        assert np.abs(f - ref).max() <= 1e-11 * np.abs(ref).max()


def test_field_keeps_non_finite_strengths(gpu):
    """A strength that is not finite reaches every target, also those beyond the exponential's reach (0 x inf)."""
    w = ring(3000, sigma=0.01)
    w.alpha[17, 1] = np.inf
    c, ids = context([w], capi.FP32C)
    assert np.isnan(c.vorticity_field(ids[0])[1600, 1])


@pytest.mark.parametrize("prec", [capi.FP64, capi.FP32C])
@pytest.mark.parametrize("n", [1, 255, 257, 512, 513, 4096, 4097, 8191, 24676, 65536, 65537])
def test_transfers_in_pieces(gpu, n, prec):
    """Uploads and downloads bit for bit, through the pinned ring in pieces and past its largest size; a second upload and
    an append reuse the ring, and the plan follows the sizes."""
    rng = np.random.default_rng(n)
    big = n + 300
    def wake(m):
        return cases.Wake(rng.normal(size=(m, 3)), rng.normal(size=(m, 3)), rng.uniform(0.1, 0.2, m), rng.uniform(1, 2, m))
    c = capi.Context(precision=prec, nu=NU)
    k = c.add_wake(big)
    w = wake(n)
    for _ in range(2):
        c.set_particles(k, w)
        c.set_particles(k, w2 := wake(n))
        more = wake(300)
        c.append_particles(k, more)
        x, a, s, v = c.particles(k)
        for got, ref in ((x, "pos"), (a, "alpha"), (s, "sigma"), (v, "vol")):
            assert np.array_equal(got, np.concatenate([getattr(w2, ref), getattr(more, ref)]))
    c.set_particles(k, w)
    y, b = c.state(k)
    assert np.array_equal(y, w.pos) and np.array_equal(b, w.alpha)
    if n <= 8191:
        c.solve()
        r, d = c.rates(k)
        one, ids = context([w], prec)
        one.solve()
        for got, ref in zip((r, d), one.rates(ids[0])):
            assert np.array_equal(got, ref)


@pytest.mark.parametrize("order", [2, 3])
@pytest.mark.parametrize("n,leaf", [(1, 256), (2, 1), (300, 1), (300, 16), (5000, 7), (5000, 256), (20011, 33)])
def test_surrogate_tree_sizes(gpu, n, leaf, order):
    """Trees of one leaf up to leaves of single particles.  A far cell's particles lie within 0.87 widths of its centroid,
    which is at least five widths off: the quadrupole drops (0.17)^3 = 5e-3 of a far cell's part, which is less than
    half of the field."""
    w = ring(n, sigma=0.02)
    if n > 100:
        w.pos[5] = w.pos[6]  # two particles that no cube separates
    c, ids = context([w], capi.FP32C)
    c.solve()
    ref = c.rates(ids[0])
    c.surrogate_enable(0, leaf_size=leaf, order=order, check_targets=0)
    c.solve()
    t = c.surrogate_tree()
    cells = t["cells"][t["leaves"]]
    order_ = np.argsort(cells[:, 0])
    assert cells[order_][0, 0] == 0 and cells[order_][-1, 1] == n
    assert np.array_equal(cells[order_][1:, 0], cells[order_][:-1, 1])
    for got, want in zip(c.rates(ids[0]), ref):
        assert np.abs(got - want).max() <= 2.5e-3 * np.abs(want).max()


@pytest.mark.parametrize("kernel", ["gaussian", "highorder"])
@pytest.mark.parametrize("npts", [1, 2, 3, 4, 5, 6, 7, 9])
def test_probe_point_tiles(gpu, npts, kernel):
    """Point tiles of four: last tiles of one to four points."""
    w = ring(700)
    pts = np.random.default_rng(npts).normal(0.0, 0.8, (npts, 3))
    c, _ = context([w], capi.FP32C, kernel=kernel)
    v = c.probe(pts)
    ref = np.array([O.restate_getvi(w, p, kernel) for p in pts])
    assert np.abs(v - ref).max() <= 1e-11 * np.abs(v).max()
