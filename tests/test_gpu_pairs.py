"""FP32 walks of the tidal tensor together with other fields, whose sweeps take two sources at a time and add
their terms in order, at short and odd batches and every number of targets per group: against the oracle's FP64
direct sums over nearby particles that no node stands for (theta tiny), and against the fields walked one at a time.

A pair's term takes at most ~20 FP32 operations (2e-6 relative), and a tidal component's terms cancel by up to
a factor of ten in these clouds: 2e-5 of the field's RMS."""

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def rel_rms(a, b):
    a, b = np.asarray(a).reshape(len(a), -1), np.asarray(b).reshape(len(b), -1)
    return np.sqrt(np.mean((a - b) ** 2) / np.mean(b**2))


@pytest.mark.parametrize("gs", [1, 2, 4, 8, 16, 32])
@pytest.mark.parametrize("n", [2, 3, 31, 33, 64, 65, 1500])
@pytest.mark.parametrize("quadrupole", [False, True])
def test_fields_together(n, gs, quadrupole):
    import pytreegrav_gb300 as tg

    rng = np.random.default_rng(n)
    x, m = rng.random((n, 3)), 0.5 + rng.random(n)
    h = np.where(rng.random(n) < 0.3, 0.1, 0.0)  # some pairs softened
    theta = 0.8 if n > 1000 else 1e-3
    kw = dict(quadrupole=quadrupole, group_size=gs, theta=theta)
    tree = tg.ConstructTree(x, m, h, quadrupole=quadrupole)
    got = tree.fields(potential=True, accel=True, tidal=True, **kw)
    one = {k: tree.fields(**{k: True}, **kw)[k] for k in ("potential", "accel", "tidal")}
    ref, _ = O.self_fields(x, m, h, potential=True, accel=True, tidal=True, nthreads=O.num_threads(), **kw)
    for k in one:
        assert rel_rms(got[k], one[k]) < 2e-5, k
        assert rel_rms(got[k], ref[k]) < 2e-5, k


@pytest.mark.parametrize("fields", [("accel",), ("potential",), ("potential", "accel")])
@pytest.mark.parametrize("n,gs", [(16383, 1), (16384, 1), (32768, 2), (40001, 2)])
def test_walks_on_both_sides_of_the_lean_line(n, gs, fields):
    """Monopole walks take the 64-register kernel from 16384 groups on (groups of 1, 2, 16 or 32 targets)."""
    import pytreegrav_gb300 as tg
    from pytreegrav_gb300 import synthetic

    x, m, h = synthetic.plummer(n, 5), np.full(n, 1.0 / n), np.full(n, 0.01)
    kw = dict({k: True for k in fields}, group_size=gs, theta=0.7)
    got = tg.ConstructTree(x, m, h).fields(**kw)
    ref, _ = O.self_fields(x, m, h, nthreads=O.num_threads(), **kw)
    for k in fields:
        assert rel_rms(got[k], ref[k]) < 2e-5, k


@pytest.mark.parametrize("n", [1, 2, 85, 86, 1000])
def test_results_in_arrays_of_their_own(n):
    """Every combination of fields, taken apart on the GPU, against each field asked for alone through the FP64
    direct sum (the same sums) and the FP64 walk with one target per group."""
    import itertools

    import pytreegrav_gb300 as tg
    from pytreegrav_gb300.tree import bruteforce

    rng = np.random.default_rng(n)
    x, m = rng.random((n, 3)), rng.random(n)
    names = ("potential", "accel", "tidal")
    shape = {"potential": (n,), "accel": (n, 3), "tidal": (n, 3, 3)}
    tree = tg.ConstructTree(x, m)
    for k in (1, 2, 3):
        for some in itertools.combinations(names, k):
            kw = {f: True for f in some}
            got = bruteforce(None, None, x, m, None, mutual=True, **kw)
            walked = tree.fields(precision="fp64", group_size=1, theta=1e-3, **kw)
            assert list(got) == list(walked) == list(some)
            for f in some:
                alone = bruteforce(None, None, x, m, None, mutual=True, **{f: True})[f]
                assert got[f].shape == walked[f].shape == shape[f] and got[f].flags.c_contiguous and got[f].base is None
                assert np.allclose(got[f], alone, rtol=1e-12, atol=1e-12 * np.abs(alone).max())
                assert np.allclose(walked[f], alone, rtol=1e-10, atol=1e-10 * np.abs(alone).max())
