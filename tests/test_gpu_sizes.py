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
