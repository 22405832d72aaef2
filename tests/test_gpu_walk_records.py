"""Walk records out of range are reported, not followed.

What a walk reads from device memory and then indexes with -- the groups, their roots, the rows of the caller's
order -- is damaged here in memory (through tg_group_arrays and the tree's info), one record at a time. The walk
has to return an error, leave the damaged group out, and write every other target's row as without the
damage; with the record put back, the next walk is the undamaged one. Walks of the tree's own particles and of
a target set, plain and with the learned opening test (whose features are read through the same records)."""

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def view(address, shape, typestr):
    class View:
        __cuda_array_interface__ = {"shape": shape, "typestr": typestr, "data": (address, False), "version": 2}

    return torch.as_tensor(View(), device="cuda")


@pytest.fixture(scope="module")
def env():
    import pytreegrav_gb300 as tg
    from pytreegrav_gb300 import _lib, synthetic
    from pytreegrav_gb300 import theta as th

    L = _lib.load()
    L.tg_group_arrays.argtypes = [ctypes.c_void_p, ctypes.c_void_p] + [ctypes.POINTER(ctypes.c_void_p)] * 2 \
        + [ctypes.POINTER(ctypes.c_int64)]
    model = th.ThetaModel.load()
    n, nt = 20_000, 5_001
    x = synthetic.plummer(n, 81)
    tree = tg.ConstructTree(x, np.full(n, 1.0 / n), np.full(n, 0.01), quadrupole=True)
    xt = np.random.default_rng(82).uniform(-3, 3, (nt, 3))
    return dict(tg=tg, L=L, lib=_lib, model=model, tree=tree, ts=tg.TargetSet(tree, xt), n=n, nt=nt,
                lam=th.default_lambda(model, True))


def run(env, own, learned, out):
    """The walk's status; `out` (device, NaN beforehand) receives the rows written."""
    L, lib, tree, ts = env["L"], env["lib"], env["tree"], env["ts"]
    out.fill_(float("nan"))
    torch.cuda.synchronize()
    o, dev = ctypes.c_void_p(out.data_ptr()), lib.TG_MEM_DEVICE
    if own and learned:
        rc = L.tg_tree_fields_learned(tree._h, 2, 1, 1.0, 32, env["model"].handle(), env["lam"], 0.7, dev, o, None)
    elif own:
        rc = L.tg_tree_fields(tree._h, None, None, env["n"], 2, 1, 0.7, 1.0, 32, lib.TG_GROUP_TREE, lib.TG_ORDER_TREE,
                              lib.TG_FP32, None, dev, o, None)
    elif learned:
        rc = L.tg_targets_fields_learned(ts.handle, 2, 1, 1.0, env["model"].handle(), env["lam"], 0.7, dev, o, None)
    else:
        rc = L.tg_targets_fields(ts.handle, 2, 1, 0.7, 1.0, lib.TG_FP32, None, dev, o, None)
    torch.cuda.synchronize()
    return rc, out.cpu().numpy()


def arrays(env, own):
    g, r, k = ctypes.c_void_p(), ctypes.c_void_p(), ctypes.c_int64()
    assert env["L"].tg_group_arrays(env["tree"]._h, None if own else env["ts"].handle, ctypes.byref(g), ctypes.byref(r),
                                    ctypes.byref(k)) == 0
    return view(g.value, (k.value, 2), "<i4"), view(r.value, (k.value,), "<i4")


@pytest.mark.parametrize("learned", [False, True])
@pytest.mark.parametrize("own", [True, False])
def test_damaged_group_records(env, own, learned):
    nt = env["n"] if own else env["nt"]
    out = torch.empty((nt, 3), dtype=torch.float64, device="cuda")
    rc, ref = run(env, own, learned, out)
    assert rc == 0 and np.all(np.isfinite(ref))
    groups, roots = arrays(env, own)
    mtot = env["tree"].node_hi - env["n"]
    k = len(roots) // 3
    first, count = (int(v) for v in groups[k].cpu())
    cases = [(groups, (k, 0), v) for v in (-1, nt, nt - count + 1, -2**31, 2**31 - 1)]
    cases += [(groups, (k, 1), v) for v in (0, -1, 33, 2**31 - 1)]
    cases += [(roots, k, v) for v in (-1, mtot, 2**31 - 1, -2**31)]
    widx = env["tree"].TreewalkIndices if own else env["ts"].groups()[3]
    rows = widx[first:first + count]
    others = np.setdiff1d(np.arange(nt), rows)
    for arr, at, value in cases:
        was = int(arr[at])
        arr[at] = value
        rc, got = run(env, own, learned, out)
        arr[at] = was
        assert rc == env["lib"].TG_ERR_CUDA, (at, value, rc)
        assert b"out of range" in env["L"].tg_last_error()
        assert np.all(np.isnan(got[rows])), (at, value)
        if not learned:  # (a group's features enter every learned tolerance through the field's mean square)
            assert np.array_equal(got[others], ref[others]), (at, value)
        else:
            assert np.all(np.isfinite(got[others])), (at, value)
    rc, got = run(env, own, learned, out)
    assert rc == 0 and np.array_equal(got, ref)


def test_damaged_rows(env):
    n = env["n"]
    out = torch.empty((n, 3), dtype=torch.float64, device="cuda")
    rc, ref = run(env, True, False, out)
    assert rc == 0
    info = env["lib"].TreeInfo()
    env["lib"].check(env["L"].tg_tree_info_get(env["tree"]._h, ctypes.byref(info)))
    widx = view(info.walk_idx, (n,), "<i8")
    at = n // 2
    for value in (-1, n, 2**40, -2**40):
        was = int(widx[at])
        widx[at] = value
        rc, got = run(env, True, False, out)
        widx[at] = was
        assert rc == env["lib"].TG_ERR_CUDA, value
        assert np.all(np.isnan(got[was]))
        got[was] = ref[was]
        assert np.array_equal(got, ref), value
    rc, got = run(env, True, False, out)
    assert rc == 0 and np.array_equal(got, ref)
