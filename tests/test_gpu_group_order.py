"""The order of a tree's groups comes from a sort; what is no partition of the particles in that order is reported.

The check is run on arrays made here: 1 to 1000 groups, a good order, and each way in which the sort's permutation
or the grouping itself can be wrong. No access is out of range in any of them."""

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def check(perm, groups, n):
    import torch

    from pytreegrav_gb300 import _lib

    L = _lib.load()
    L.tg_check_group_order.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int64, ctypes.c_int64,
                                       ctypes.POINTER(ctypes.c_int), ctypes.c_void_p]
    p = torch.from_numpy(np.asarray(perm, np.uint32).view(np.int32)).cuda()
    g = torch.from_numpy(np.ascontiguousarray(groups, dtype=np.int32)).cuda()
    torch.cuda.synchronize()
    err = ctypes.c_int(-1)
    assert L.tg_check_group_order(p.data_ptr(), g.data_ptr(), len(perm), n, ctypes.byref(err), None) == 0
    return err.value


@pytest.mark.parametrize("ng", [1, 2, 256, 257, 1000])
def test_group_order(ng):
    rng = np.random.default_rng(ng)
    count = rng.integers(1, 33, ng)
    first = np.concatenate([[0], np.cumsum(count)[:-1]])
    n = int(count.sum())
    shuffle = rng.permutation(ng)  # the order in which the groups were emitted
    groups = np.stack([first, count], 1)[shuffle]
    perm = np.argsort(shuffle)
    assert check(perm, groups, n) == 0
    k = ng // 2
    for value in (ng, 2**31, 2**32 - 1):  # no index of a group
        bad = perm.astype(np.int64)
        bad[k] = value
        assert check(bad, groups, n) == 2
    if ng > 1:  # a group twice, another left out; two groups exchanged
        bad = perm.copy()
        bad[k] = bad[k - 1]
        assert check(bad, groups, n) == 2
        bad = perm.copy()
        bad[k], bad[k - 1] = bad[k - 1], bad[k]
        assert check(bad, groups, n) == 2
    for column, step in ((0, 1), (1, 1), (1, -1)):  # a particle left out or taken twice
        bad = groups.copy()
        bad[perm[k], column] += step
        assert check(perm, bad, n) == 2
    assert check(perm, groups, n + 1) == 2  # the last particle left out
