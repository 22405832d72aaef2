"""Non-finite input ends a build at its first summary: no more kernels than the same build of finite input launches
(one NaN position makes the bounding cube NaN and all keys equal, which a build that went on would re-key three
times and put in a bucket), and the next build on the library is right."""

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("where", ["position", "mass", "softening"])
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("n", [3, 5000])
def test_build_ends_early(n, bad, where):
    import pytreegrav_gb300 as tg
    from pytreegrav_gb300 import _lib

    L = _lib.load()
    rng = np.random.default_rng(n)
    x, m, h = rng.random((n, 3)), np.full(n, 1.0 / n), np.full(n, 0.01)

    def launches(*a):
        k = L.tg_launch_count()
        try:
            tree = tg.Octree(*a, quadrupole=True)
        except _lib.NonFiniteInput:
            tree = None
        return L.tg_launch_count() - k, tree

    whole, tree = launches(x, m, h)
    assert tree is not None
    args = {"position": x.copy(), "mass": m.copy(), "softening": h.copy()}
    args[where].flat[n // 2] = bad
    count, tree = launches(*args.values())
    assert tree is None and count < whole, (count, whole)
    _, tree = launches(x, m, h)
    assert np.array_equal(tree.TreewalkIndices, O.OracleTree(x, m, h, quadrupole=True).TreewalkIndices)
