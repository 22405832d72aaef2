"""The per-lane queues of the column-density walk at their edges: walks that queue far more than a queue
holds, walks that queue nothing, and warps with idle lanes. Columns equal the oracle's bit for bit.
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
