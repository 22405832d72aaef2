"""The per-lane queues of the column-density and two-point walks at their edges: walks that queue far more
than a queue holds, walks that queue nothing, warps with idle lanes, and lanes with several targets.

Columns equal the oracle's bit for bit; the two-point sums are within 1e-12 of the per-bin sum of
absolute contributions (the bar of the other two-point tests: only the summation order differs).
"""

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def tg():
    import pytreegrav_gb300 as tg

    return tg


@pytest.mark.parametrize("radius", [0.0, 1e-3, 0.5, 20.0])
@pytest.mark.parametrize("n", [1, 2, 33, 700])
def test_column_queue(tg, n, radius):
    rng = np.random.default_rng(n)
    x = rng.normal(size=(n, 3))
    m = rng.random(n)
    h = np.full(n, radius) * np.where(rng.random(n) < 0.9, 1.0, 0.0)
    rays = rng.normal(size=(5, 3))
    rays /= np.sqrt((rays * rays).sum(1))[:, None]
    ref = O.column_rays(O.OracleTree(x, m, h), x, rays)
    assert np.array_equal(tg.ConstructTree(x, m, h).column_density(x, rays), ref)


@pytest.mark.parametrize("kind", ["density", "velocity", "structure"])
@pytest.mark.parametrize("n,nt", [(1, 1), (40, 3), (3000, 33), (3000, 1)])
@pytest.mark.parametrize("nbins", [1, 60])
def test_corr_queue(tg, kind, n, nt, nbins):
    rng = np.random.default_rng(7 * n + nt)
    x, m, v = rng.normal(size=(n, 3)), rng.random(n) / n, rng.normal(size=(n, 3))
    xt, wt, vt = rng.normal(size=(nt, 3)), rng.random(nt), rng.normal(size=(nt, 3))
    rb = np.geomspace(1e-3, 10.0, nbins + 1)
    t = tg.ConstructTree(x, m, np.zeros(n), vel=v)
    b, w = t.correlation(kind, xt, rb, vel=vt, weight=wt, seed=99)
    ot = O.OracleTree(x, m, np.zeros(n))
    tv = O.tree_velocities(ot, v)
    extra = {} if kind == "density" else dict(vel=vt, weight=wt, tree_vel=tv)
    bo, wo = O.correlation(ot, kind, xt, rb, seed=99, **extra)
    scale, _ = O.correlation(ot, kind, xt, rb, seed=99, absval=True, **extra)
    assert np.all(np.abs(b - bo) <= 1e-12 * np.maximum(scale, 1e-300))
    if kind != "density":
        assert np.all(np.abs(w - wo) <= 1e-12 * np.maximum(wo, 1e-300))


@pytest.mark.parametrize("n", [11, 12, 255, 1024, 1025, 40001])
@pytest.mark.parametrize("kind", ["normal", "lattice", "equal"])
def test_radial_range(tg, n, kind):
    """Ranks of the distances from the median position: numpy's values, bit for bit."""
    from pytreegrav_gb300.tree import radial_range

    rng = np.random.default_rng(n)
    x = rng.normal(size=(n, 3)) * [1e-3, 1.0, 1e4] - [0.0, 3.0, 0.0]
    if kind == "lattice":
        x = np.round(x)  # many equal values, zeros of both signs
    if kind == "equal":
        x = np.full((n, 3), 0.25)
    d = [x[:, k] - np.median(x[:, k]) for k in range(3)]
    r = np.sort(np.sqrt(d[0] * d[0] + d[1] * d[1] + d[2] * d[2]))
    for rank in (0, 10, n // 2, n - 1):
        assert radial_range(x, rank) == (r[rank], r[-1])
