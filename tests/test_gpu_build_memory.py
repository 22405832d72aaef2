"""Peak device memory of a build, from inputs already on the device.

A build's temporaries, its node numbering and the tree's own arrays are alive together until the final arrays are
written; the moment pass's child lists and sums come after, in their place. The bound is the sum of those sizes per
particle (N) and node (M):

  N: keys 8, permutation 4, Morton-ordered data 40, levels 1, node starts 4, elements of slots 6, exhausted runs 4,
     particle links 16, node slots 1.5 x 102, walk order 8, the sort's other halves and status words 13 = 257
  M: numbering 20, its sort's halves and status words 13, cells and ranges 32, depth lists 5 = 70
  N + M: the tree's arrays, 80

with 2 % for rounding; the moment pass on top of them (57 bytes per node) would be 8 % above it."""

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("quadrupole", [False, True])
@pytest.mark.parametrize("n", [1_000_000, 2_000_000])
def test_peak_memory_of_a_build(n, quadrupole):
    import torch

    from pytreegrav_gb300 import _lib, synthetic

    L = _lib.load()
    L.tg_memory_use.argtypes = [ctypes.POINTER(ctypes.c_int64)] * 2 + [ctypes.c_int]
    reserved, high = ctypes.c_int64(), ctypes.c_int64()
    x = torch.from_numpy(synthetic.plummer(n, 95)).cuda()
    m = torch.full((n,), 1.0 / n, dtype=torch.float64, device="cuda")
    h = torch.full((n,), 0.01, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()

    def build():
        t = ctypes.c_void_p()
        _lib.check(L.tg_tree_build(x.data_ptr(), m.data_ptr(), h.data_ptr(), n, int(quadrupole), 1, _lib.TG_MEM_DEVICE,
                                   None, ctypes.byref(t)), "build")
        info = _lib.TreeInfo()
        _lib.check(L.tg_tree_info_get(t, ctypes.byref(info)))
        L.tg_tree_free(t)
        torch.cuda.synchronize()
        return int(info.node_hi) - n

    build()
    torch.cuda.synchronize()
    assert L.tg_memory_use(ctypes.byref(reserved), ctypes.byref(high), 1) == 0
    mnode = build()
    assert L.tg_memory_use(ctypes.byref(reserved), ctypes.byref(high), 0) == 0
    bound = 257 * n + 70 * mnode + 80 * (n + mnode)
    print(f"\n{n} particles, {mnode} nodes: {high.value / n:.0f} bytes per particle, bound {bound / n:.0f}")
    assert high.value < 1.02 * bound
