"""External targets on the rare branches of their path: sources and targets whose keys run out (pairs closer than the
key lattice, re-keyed within their cells; points that coincide, kept in buckets), and groups whose pending nodes
outgrow the small stack and are walked again with the large one.

Plain walks against the oracle walking the same groups (FP64 1e-12, FP32 1e-5 relative RMS: the walk's bars). The
learned walk against its parts called one by one -- features, inference, tolerances, the walk with those tolerances per
group -- bit for bit (its error budget, which walks groups again, off)."""

import ctypes

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def tg():
    import pytreegrav_gb300 as tg

    return tg


def rel_rms(a, ref):
    a, ref = np.asarray(a).reshape(len(a), -1), np.asarray(ref).reshape(len(ref), -1)
    return np.sqrt(np.sum((a - ref) ** 2) / np.sum(ref**2))


def crowded(n, seed, radius):
    """Points with 2 % close companions at 1e-3 to 1e-13 of the key lattice's 2^-21, and 40 copies of one point."""
    rng = np.random.default_rng(seed)
    d = rng.normal(size=(n, 3))
    x = d / np.linalg.norm(d, axis=1)[:, None] * (radius * rng.random(n) ** (1 / 3))[:, None]
    k = n // 50
    step = 2 * radius * 2.0**-21 * 10.0 ** rng.uniform(-13, -3, k)
    x[:k] = x[k:2 * k] + step[:, None] * rng.normal(size=(k, 3))
    x[2 * k:2 * k + 40] = x[2 * k]
    return np.ascontiguousarray(x[rng.permutation(n)])


def learned_both_ways(ts, quad):
    import torch

    from pytreegrav_gb300 import _lib
    from pytreegrav_gb300 import theta as th

    L, model = _lib.load(), th.ThetaModel.load()
    handle, lam = model.handle(), th.default_lambda(model, quad, True)
    _lib.check(L.tg_theta_model_set_error_budget(handle, 0.0))

    def dev(*shape, dtype=torch.float32):
        t = torch.zeros(shape, dtype=dtype, device="cuda")
        torch.cuda.synchronize()
        return t, ctypes.c_void_p(t.data_ptr())

    ng = ts.ngroups()
    out, p_out = dev(ts.n, 3, dtype=torch.float64)
    _lib.check(L.tg_targets_fields_learned(ts.handle, 2, int(quad), 1.0, handle, lam, 0.7, _lib.TG_MEM_DEVICE, p_out, None))
    whole = out.cpu().numpy()
    feat, p_feat = dev(ng, _lib.TG_THETA_NFEAT)
    u, p_u = dev(ng)
    tol, p_tol = dev(ng)
    _lib.check(L.tg_targets_features(ts.handle, int(quad), p_feat, None))
    _lib.check(L.tg_theta_infer(handle, p_feat, ng, lam, p_u, None))
    _lib.check(L.tg_targets_tolerances(ts.handle, int(quad), p_u, p_tol, None))
    out.zero_()
    torch.cuda.synchronize()
    _lib.check(L.tg_targets_fields(ts.handle, 2, int(quad), float(model.theta_max), 1.0, _lib.TG_FP32, p_tol,
                                   _lib.TG_MEM_DEVICE, p_out, None))
    return whole, out.cpu().numpy()


@pytest.mark.parametrize("quad", [False, True])
@pytest.mark.parametrize("src,tgt", [("crowded", "ball"), ("plummer", "crowded"), ("crowded", "crowded")])
def test_target_sets_with_rekeyed_points(tg, src, tgt, quad):
    from pytreegrav_gb300 import synthetic

    n, nt = 40_000, 12_000
    x = crowded(n, 91, 1.0) if src == "crowded" else synthetic.plummer(n, 91)
    xt = crowded(nt, 92, 0.9) if tgt == "crowded" else \
        np.random.default_rng(92).uniform(-0.5, 0.5, (nt, 3))
    m, h = np.full(n, 1.0 / n), np.full(n, 0.01)
    ht = np.full(nt, 0.002)
    tree = tg.ConstructTree(x, m, h, quadrupole=True)
    if src == "crowded":
        assert tree.HasCoincidentPoints
    ts = tg.TargetSet(tree, xt, ht)
    first, count, _, widx = ts.groups()
    ref = {}
    got_w = O.fields_groups(O.OracleTree(x, m, h, quadrupole=True), xt[widx], ht[widx], first, count, True, True, False,
                            quad, 0.7, nthreads=O.num_threads())
    for k in ("potential", "accel"):
        ref[k] = np.empty_like(got_w[k])
        ref[k][widx] = got_w[k]
    for prec, tol in (("fp64", 1e-12), ("fp32", 1e-5)):
        got = ts.fields(potential=True, accel=True, quadrupole=quad, theta=0.7, precision=prec)
        for k in got:
            assert rel_rms(got[k], ref[k]) < tol, (prec, k)
    whole, parts = learned_both_ways(ts, quad)
    assert np.all(np.isfinite(whole)) and np.array_equal(whole, parts)


@pytest.mark.parametrize("precision,tol", [("fp32", 1e-5), ("fp64", 1e-12)])
def test_target_set_retries_with_the_large_stack(tg, precision, tol):
    """At theta = 0.1 some targets' pending nodes pass the small stack's 1024 entries: the same walk with the large
    stack from the start, and the oracle's."""
    from pytreegrav_gb300 import synthetic

    n, nt = 400_000, 64
    x, m, h = synthetic.plummer(n, 93), np.full(n, 1.0 / n), np.full(n, 0.01)
    xt = np.random.default_rng(94).uniform(-0.3, 0.3, (nt, 3))
    tree = tg.ConstructTree(x, m, h, quadrupole=True)
    ts = tg.TargetSet(tree, xt)
    kw = dict(accel=True, quadrupole=True, theta=0.1, precision=precision)
    small = ts.fields(**kw)["accel"]
    assert tree.last_walk_stats()[2] > 1024
    tree.set_walk_config(4, 4096)
    assert np.array_equal(small, ts.fields(**kw)["accel"])
    first, count, _, widx = ts.groups()
    ref = O.fields_groups(O.OracleTree(x, m, h, quadrupole=True), xt[widx], np.zeros(nt), first, count, False, True, False,
                          True, 0.1, nthreads=O.num_threads())["accel"]
    assert rel_rms(small[widx], ref) < tol
