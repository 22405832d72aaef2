"""The direct sums at the sizes where their kernels can go wrong.

FP64: bit for bit the oracle's (zero tolerance), in both forms of the kernel -- few targets (targets per
block and tiles of 32 sources with remainders, one source, none in reach) and targets that fill
whole waves of blocks -- for every set of fields, with softened, coincident and self pairs.
"""

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

NAMES = ("potential", "accel", "tidal")


@pytest.fixture(scope="module")
def tg():
    import pytreegrav_gb300 as tg

    return tg


def particles(n, seed):
    rng = np.random.default_rng(seed)
    x = rng.normal(size=(n, 3))
    if n > 3:
        x[n // 2] = x[0]  # coincident
    m = rng.random(n) / n
    h = np.where(rng.random(n) < 0.3, 0.0, 0.4 * rng.random(n))
    return x, m, h


@pytest.mark.parametrize("fields", range(1, 8))
@pytest.mark.parametrize("ns", [1, 31, 32, 33, 225, 700])
def test_fp64_mutual(tg, ns, fields):
    kw = {k: bool(fields >> i & 1) for i, k in enumerate(NAMES)}
    x, m, h = particles(ns, 100 + ns)
    ref = O.bruteforce(x, h, x, m, h, mutual=True, nthreads=O.num_threads(), **kw)
    got = tg.bruteforce(None, None, x, m, h, mutual=True, precision="fp64", **kw)
    for k in got:
        assert np.array_equal(got[k], ref[k]), k


# targets: one; fewer than SMs; several per block; a block's most and one more; most of a wave of blocks
# of 128 targets on 152 SMs; a whole wave (the other kernel); one over it
@pytest.mark.parametrize("nt,ns", [(1, 1), (1, 3000), (151, 33), (153, 64), (1520, 65), (1521, 7), (4865, 40),
                                   (17800, 9), (19456, 9), (19457, 9)])
@pytest.mark.parametrize("fields", [1, 2, 4, 7])
def test_fp64_targets(tg, nt, ns, fields):
    kw = {k: bool(fields >> i & 1) for i, k in enumerate(NAMES)}
    x, m, h = particles(ns, 7 * ns)
    xt, _, ht = particles(nt, 3 * nt)
    xt[-1] = x[-1]  # a target on a source
    ref = O.bruteforce(xt, ht, x, m, h, mutual=False, nthreads=O.num_threads(), **kw)
    got = tg.bruteforce(xt, ht, x, m, h, mutual=False, precision="fp64", **kw)
    for k in got:
        assert np.array_equal(got[k], ref[k]), k
