"""Walks of consecutive targets whose long groups do not stay with one warp.

FP64 walks split them sooner than FP32 ones: fields against the oracle (1e-12, the FP64 walk's bar) at sizes
whose longest groups are split, with softened targets.

FP32: groups walked by a whole block against groups walked by one warp each, bit for bit: the same batches of
list entries, summed apart and added in the same order. The walk of a tree that records per-group
counters keeps one warp per group, so it is the other side; node tests and interactions agree too.

Sizes: one short batch; one node; group counts on both sides of the lines between walking every group by
block, the long ones only, and none (4000 groups, 1400 with every field, 65536), by targets per
group; the accepted sets and fields against the oracle are in test_gpu_walk.py.
"""

import ctypes

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def tg():
    import pytreegrav_gb300 as tg

    return tg


def walk(tree, per_warp, **kw):
    from pytreegrav_gb300 import _lib

    L = _lib.load()
    _lib.check(L.tg_tree_record_group_stats(tree._h, int(per_warp)))
    res = tree.fields(**kw)
    s = tree.last_walk_stats()
    _lib.check(L.tg_tree_record_group_stats(tree._h, 0))
    return res, (s[0], s[1], s[3])


@pytest.mark.parametrize("quadrupole", [False, True])
@pytest.mark.parametrize("fields", [("potential",), ("accel",), ("potential", "accel"), ("tidal",),
                                    ("potential", "accel", "tidal")])
@pytest.mark.parametrize("n,gs", [(1, 8), (5, 4), (33, 8), (1200, 4), (11201, 8), (5599, 4), (32001, 8), (31999, 8),
                                  (30000, 32)])
def test_block_walk(tg, n, gs, fields, quadrupole):
    from pytreegrav_gb300 import synthetic

    x = synthetic.clustered(n, 3) if n > 100 else synthetic.plummer(n, 3)
    rng = np.random.default_rng(n)
    tree = tg.ConstructTree(x, rng.random(n) / n, 0.02 * rng.random(n), quadrupole=True)
    kw = dict({k: True for k in fields}, quadrupole=quadrupole, group_size=gs, theta=0.6)
    # (32000-entry groups would be split when no counters are kept: these systems stay below)
    one, s1 = walk(tree, True, **kw)
    block, s2 = walk(tree, False, **kw)
    for k in one:
        assert np.array_equal(one[k], block[k]), k
    assert s1 == s2
    xt = rng.normal(size=(257, 3)) * 5  # few targets of many sources
    kw.update(pos=xt, soft=np.zeros(257), order="morton")
    one, s1 = walk(tree, True, **kw)
    block, s2 = walk(tree, False, **kw)
    for k in one:
        assert np.array_equal(one[k], block[k]), k
    assert s1 == s2


@pytest.mark.parametrize("quadrupole", [False, True])
@pytest.mark.parametrize("n,gs", [(40, 8), (3001, 8), (12345, 8), (12345, 1), (20011, 16)])
def test_fp64_split(tg, n, gs, quadrupole):
    from pytreegrav_gb300 import synthetic

    x = synthetic.plummer(n, 17)
    rng = np.random.default_rng(n)
    m, h = rng.random(n) / n, np.where(rng.random(n) < 0.2, 0.0, 0.05 * rng.random(n))
    kw = dict(potential=True, accel=True, tidal=True, theta=0.7, quadrupole=quadrupole, group_size=gs)
    ref, _ = O.self_fields(x, m, h, nthreads=O.num_threads(), **kw)
    got = tg.ConstructTree(x, m, h, quadrupole=quadrupole).fields(precision="fp64", **kw)
    alone = tg.ConstructTree(x, m, h, quadrupole=quadrupole).fields(precision="fp64", **dict(kw, potential=False, tidal=False))
    for k in ref:
        a, b = got[k].reshape(n, -1), ref[k].reshape(n, -1)
        assert np.sqrt(np.sum((a - b) ** 2)) < 1e-12 * np.sqrt(np.sum(b**2)), k
    a, b = alone["accel"], ref["accel"]
    assert np.sqrt(np.sum((a - b) ** 2)) < 1e-12 * np.sqrt(np.sum(b**2))


@pytest.mark.parametrize("n", [1, 257, 3001, 100003])
def test_scan_that_does_not_wait(tg, n):
    """The walk arena's one-pass scan of leaf counts when a tile gives up waiting for the tiles before it: the
    prefix then comes from the input itself, so the walk is the same. (Groups of one target: nothing else of
    this walk waits.)"""
    from pytreegrav_gb300 import _lib, synthetic

    L = _lib.load()
    L.tg_set_loop_limits.argtypes = [ctypes.c_int64] * 4
    x = synthetic.plummer(n, 5)
    m, h = np.full(n, 1.0 / n), np.full(n, 0.01)
    kw = dict(accel=True, group_size=1, theta=0.9)
    ref = tg.ConstructTree(x, m, h).fields(**kw)["accel"]
    for _ in range(3):
        tree = tg.ConstructTree(x, m, h)
        L.tg_set_loop_limits(1, 0, 0, 0)
        try:
            got = tree.fields(**kw)["accel"]
        finally:
            L.tg_set_loop_limits(0, 0, 0, 0)
        assert np.array_equal(got, ref)
