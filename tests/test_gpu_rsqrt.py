"""The FP64 walk's reciprocal square root against the exact value, formed in integers.

With e = 1 - x y^2 formed in one rounding (y has 24 bits, so y^2 is exact), what is left of the error before the
last rounding is the series' next term, 5/16 e^3, with |e| < 2^-21 (the FP32 approximation's 2^-22.9 and the
significand's truncation to 24 bits): 2^-64.6 of the value, at most 0.0007 units in the last place, and roundings
of terms below 2^-22 of the value, at most 2^-74 each. The last rounding adds half a unit. Bar: 0.501.
Values: every exponent, odd and even, significands at both ends of the binade and at random. Zeros, subnormals,
infinities, negative values and NaN: what 1/sqrt gives (subnormals: within one unit, the library's bound)."""

import ctypes
from math import isqrt

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def gpu_rsqrt(x):
    import torch

    from pytreegrav_gb300 import _lib

    L = _lib.load()
    L.tg_check_rsqrt64.argtypes = [ctypes.c_void_p, ctypes.c_int64, ctypes.c_void_p, ctypes.c_void_p]
    dx = torch.from_numpy(x).cuda()
    out = torch.empty_like(dx)
    torch.cuda.synchronize()
    assert L.tg_check_rsqrt64(ctypes.c_void_p(dx.data_ptr()), len(x), ctypes.c_void_p(out.data_ptr()), None) == 0
    torch.cuda.synchronize()
    return out.cpu().numpy()


def error_in_ulps(x, y):
    """|y - 1/sqrt(x)| in units in the last place of y's binade, to 2^-60."""
    mx, ex = np.frexp(x)
    m, e = int(mx * 2**53), int(ex) - 53  # x = m 2^e
    if e & 1:
        m, e = 2 * m, e - 1
    # 1/sqrt(x) = 2^(-e/2) / sqrt(m); t = 2^180 / sqrt(m)
    t = isqrt((1 << 360) // m)
    my, ey = np.frexp(y)
    q = int(my * 2**53)  # y = q 2^(ey - 53)
    shift = int(ey) - 53 + e // 2 + 180  # y 2^(e/2) 2^180 = q 2^shift
    return abs((q << shift) - t) / (1 << shift)


def test_rsqrt_of_normal_numbers():
    rng = np.random.default_rng(5)
    exps = np.arange(-1022, 1024)
    frac = np.concatenate([[0, 1, 2**52 - 1, 2**52 - 2, 2**29, 2**29 - 1], rng.integers(0, 2**52, 10)])
    x = np.ldexp(1.0 + frac[None, :] * 2.0**-52, exps[:, None]).ravel()
    x = np.concatenate([x, rng.uniform(0.25, 4.0, 20_000)])
    y = gpu_rsqrt(x)
    worst = max(error_in_ulps(a, b) for a, b in zip(x, y))
    print(f"\nlargest error {worst:.5f} units in the last place of {len(x)} values")
    assert worst < 0.501


def test_rsqrt_of_other_values():
    sub = np.array([5e-324, 1e-310, 2.0**-1023, np.nextafter(2.0**-1022, 0)])
    for a, b in zip(sub, gpu_rsqrt(sub)):
        assert error_in_ulps(a, b) <= 1.0
    x = np.array([0.0, -0.0, np.inf, -np.inf, -1.0, -5e-324, np.nan])
    want = np.array([np.inf, -np.inf, 0.0, np.nan, np.nan, np.nan, np.nan])
    np.testing.assert_array_equal(gpu_rsqrt(x), want)
