"""FP64 walks do not depend on the unit of length.

A system scaled by a power of two has the same tree, and every operation of the FP64 walk scales exactly, so the
walk must accept the same nodes: its node tests and interactions are those of the unscaled system, and its
fields the unscaled ones times the power of the scale. The walk decides in FP32 where that is certain, and
the scales are those at which FP32 squares of distances lose bits (2^-64 to 2^-74: subnormal), vanish (2^-100),
and overflow (2^60 and more: CGS coordinates of a galaxy are ~2^73).

Tolerance on the fields: 1e-12, the FP64 walk's bar (sums are taken in the same order; which sources are swept with
softening depends on an absolute term of 1e-45)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("quadrupole", [False, True])
@pytest.mark.parametrize("power", [-100, -74, -70, -64, 60, 73, 100])
def test_fp64_walk_scales(power, quadrupole):
    import pytreegrav_gb300 as tg
    from pytreegrav_gb300 import synthetic

    n = 20_000
    x = synthetic.plummer(n, 71)
    m = np.full(n, 1.0 / n)
    h = np.random.default_rng(72).uniform(0.0, 0.02, n)
    s = 2.0**power

    def walk(scale):
        tree = tg.ConstructTree(x * scale, m, h * scale, quadrupole=True)
        f = tree.fields(potential=True, accel=True, quadrupole=quadrupole, theta=0.7, precision="fp64")
        stats = tree.last_walk_stats()
        return f, (stats[0], stats[1], stats[3])

    ref, counts = walk(1.0)
    got, counts_s = walk(s)
    assert counts_s == counts
    for k, w in (("potential", 1), ("accel", 2)):
        a, b = got[k] * s**w, ref[k]
        assert np.sqrt(np.sum((a - b) ** 2) / np.sum(b**2)) < 1e-12, k
