"""The direct sums at the sizes where their kernels can go wrong.

FP64: bit for bit the oracle's (zero tolerance), in both forms of the kernel -- few targets (targets per
block and tiles of 32 sources with remainders, one source, none in reach) and targets that fill
whole waves of blocks -- for every set of fields, with softened, coincident and self pairs.

FP32: against the FP64 oracle, per target within 2e-5 of the sum of the pairs' magnitudes. The spline's
force near q = 1 is a difference of terms up to 48 times its value, each rounded to 2^-24 about four
times (1.2e-5); a tile's 64 terms per lane are added with at most 64 roundings (4e-6); the rest (the
offset, the square, the reciprocal root's 2 ulp) stays below 4e-6. Positions are float32 exact.
"""

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

FP32_TOL = 2e-5
NAMES = ("potential", "accel", "tidal")


@pytest.fixture(scope="module")
def tg():
    import pytreegrav_gb300 as tg

    return tg


def particles(n, seed, float32=False):
    rng = np.random.default_rng(seed)
    x = rng.normal(size=(n, 3))
    if float32:
        x = x.astype(np.float32).astype(np.float64)
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


@pytest.mark.parametrize("mutual", [True, False])
@pytest.mark.parametrize("ns", [1, 2, 31, 32, 33, 255, 256, 257, 545])
def test_fp32(tg, ns, mutual):
    x, m, h = particles(ns, 11 * ns, float32=True)
    xt, _, ht = (x, m, h) if mutual else particles(130, 5, float32=True)
    got = tg.bruteforce(xt, ht, x, m, h, True, True, False, mutual=mutual, precision="fp32")
    # the FP32 sums drop every pair at r = 0 in either form, as the target form does (a coincident pair's
    # softened potential included)
    ref = O.bruteforce(xt, ht, x, m, h, True, True, False, mutual=False, nthreads=O.num_threads())
    # per pair: the magnitude of its potential and force
    d = x[None] - xt[:, None]
    r = np.sqrt((d * d).sum(-1))
    hh = np.maximum(h[None], ht[:, None])
    if mutual:
        np.fill_diagonal(r, np.inf)
    with np.errstate(divide="ignore", invalid="ignore"):
        phi = np.where(r > 0, m[None] / r, 0.0)
        acc = np.where(r > 0, m[None] / r**2, 0.0)
        near = (r < hh) & (r > 0)
        phi = np.where(near, m[None] * 2.8 / hh, phi)
        acc = np.where(near, m[None] * r * 10.67 / hh**3, acc)
    scale = {"potential": np.nan_to_num(phi).sum(1), "accel": np.nan_to_num(acc).sum(1)[:, None]}
    for k, s in scale.items():
        # one pair's own rounding where the sum is empty
        assert np.all(np.abs(got[k] - ref[k]) <= FP32_TOL * s + 1e-30), (k, np.max(np.abs(got[k] - ref[k]) / (s + 1e-30)))
