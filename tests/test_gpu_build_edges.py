"""Octree builds at the edges of the build's one-pass level scan (tiles of 1024 elements) and of its node slots
(1.5 per particle, grown when chains of close pairs need more): every array bit for bit the oracle's, as in
test_gpu_tree.py."""

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

FIELDS = ["Coordinates", "Masses", "Sizes", "Deltas", "Softenings", "Quadrupoles", "FirstSubnode", "NextBranch",
          "TreewalkIndices"]


def points(kind, n, seed):
    rng = np.random.default_rng(seed)
    if kind == "uniform":
        return rng.random((n, 3))
    if kind == "pairs":  # each two points 1e-5 apart: ~17 nodes of one chain per pair, more than 1.5 per particle
        base = rng.random(((n + 1) // 2, 3))
        return np.repeat(base, 2, axis=0)[:n] + 1e-5 * rng.random((n, 3))
    # radii over eighteen octaves: many levels with a handful of nodes each
    u = rng.normal(size=(n, 3))
    return u / np.linalg.norm(u, axis=1)[:, None] * 2.0 ** (-18 * rng.random((n, 1)))


@pytest.mark.parametrize("kind", ["uniform", "pairs", "octaves"])
@pytest.mark.parametrize("n", [1, 2, 33, 1023, 1024, 1025, 2048, 4097, 20000])
def test_tree_is_the_oracles(kind, n):
    import pytreegrav_gb300 as tg

    x = points(kind, n, n)
    rng = np.random.default_rng(n + 1)
    m, h = rng.random(n) / n, np.full(n, 0.01)
    t = tg.ConstructTree(x, m, h, quadrupole=True)
    ref = O.OracleTree(x, m, h, quadrupole=True)
    assert t.NumNodes == ref.NumNodes
    for f in FIELDS:
        assert np.array_equal(getattr(t, f), getattr(ref, f)), f


@pytest.mark.parametrize("kind", ["uniform", "one digit", "duplicates"])
@pytest.mark.parametrize("n", [2, 31, 511, 513, 4095, 4096, 4097, 8193, 70000, 3 * 2**20 + 1])
def test_morton_order_is_the_oracles(kind, n):
    """The radix sort at the edges of its tiles (4096 pairs; 6144 in long sorts), with digits all alike in most passes and with equal
    keys, whose order must be kept: integers, so equal."""
    import pytreegrav_gb300 as tg

    rng = np.random.default_rng(n)
    x = rng.random((n, 3))
    if kind == "one digit":  # all but the corners of the cube within one cell of level 17
        x = 0.3 + 1e-6 * x
        x[0], x[-1] = 0.0, 1.0
    if kind == "duplicates":
        x = x[rng.integers(0, max(n // 50, 1), n)]
    assert np.array_equal(tg.morton_order(x), O.morton_order(x))
