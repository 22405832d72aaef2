"""One tree used from several streams without a synchronisation between the calls: a target set made, and features
computed, on one stream behind a long-running kernel, then evaluated on another. Bit for bit the results of one stream."""

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_calls_on_other_streams_wait_for_queued_work():
    import torch

    from pytreegrav_gb300 import _lib, synthetic

    L = _lib.load()
    n, nt = 200_000, 60_000
    x = torch.from_numpy(synthetic.plummer(n, 61)).cuda()
    m = torch.full((n,), 1.0 / n, dtype=torch.float64, device="cuda")
    h = torch.full((n,), 0.01, dtype=torch.float64, device="cuda")
    xt = torch.from_numpy(np.random.default_rng(62).uniform(-2, 2, (nt, 3))).cuda()
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    big = torch.zeros(1 << 28, device="cuda")
    torch.cuda.synchronize()

    def once(s_make, s_use):
        tree, ts = ctypes.c_void_p(), ctypes.c_void_p()
        make, use = ctypes.c_void_p(s_make.cuda_stream), ctypes.c_void_p(s_use.cuda_stream)
        out = torch.zeros((nt, 3), dtype=torch.float64, device="cuda")
        feat = torch.zeros((n, _lib.TG_THETA_NFEAT), device="cuda")
        own = torch.zeros((n, 3), dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        _lib.check(L.tg_tree_build(x.data_ptr(), m.data_ptr(), h.data_ptr(), n, 1, 1, _lib.TG_MEM_DEVICE, make,
                                   ctypes.byref(tree)), "build")
        _lib.check(L.tg_targets_create(tree, xt.data_ptr(), None, nt, 32, _lib.TG_MEM_DEVICE, make, ctypes.byref(ts)))
        with torch.cuda.stream(s_make):  # the next call's kernels wait behind these
            for _ in range(20):
                big.add_(1.0)
        _lib.check(L.tg_theta_features(tree, 32, 1, feat.data_ptr(), make))
        _lib.check(L.tg_targets_fields(ts, 2, 1, 0.7, 1.0, _lib.TG_FP32, None, _lib.TG_MEM_DEVICE, out.data_ptr(), use))
        _lib.check(L.tg_tree_fields(tree, None, None, n, 2, 1, 0.7, 1.0, 32, _lib.TG_GROUP_TREE, _lib.TG_ORDER_TREE,
                                    _lib.TG_FP32, None, _lib.TG_MEM_DEVICE, own.data_ptr(), use))
        with torch.cuda.stream(s_make):
            for _ in range(20):
                big.add_(1.0)
        _lib.check(L.tg_targets_features(ts, 1, feat.data_ptr(), make))
        L.tg_targets_free(ts)  # the features are still to run
        L.tg_tree_free(tree)
        torch.cuda.synchronize()
        return out.cpu().numpy(), own.cpu().numpy(), feat.cpu().numpy()

    ref = once(a, a)
    for _ in range(3):
        for r, g in zip(ref, once(a, b)):
            assert np.array_equal(r, g)
