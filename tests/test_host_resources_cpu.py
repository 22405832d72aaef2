"""What the library holds on the host between calls, and what it does when a launch fails, against a stand-in for
the CUDA runtime (fake_cudart.c: several devices, counted resources, launches that can be made to fail; kernels do
nothing). No GPU. Every test runs in a process of its own, in which the stand-in is loaded under the runtime's name."""

import os
import shutil
import subprocess
import sys
import textwrap

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
SONAME = "libcudart.so.13"

PRELUDE = textwrap.dedent("""
    import ctypes, sys
    import numpy as np
    sys.path.insert(0, %r)
    F = ctypes.CDLL(%%r, mode=ctypes.RTLD_GLOBAL)
    F.fake_log.restype = ctypes.c_char_p
    F.fake_host_blocks.restype = F.fake_streams.restype = F.fake_events.restype = ctypes.c_long
    F.fake_device_blocks.restype = ctypes.c_long
    F.fake_patch.argtypes = [ctypes.c_size_t, ctypes.c_void_p, ctypes.c_size_t]
    from pytreegrav_gb300 import _lib
    L = _lib.load()
    n = 64
    x = np.random.default_rng(0).random((n, 3)); m = np.ones(n); h = np.full(n, 0.01)

    def build():
        t = ctypes.c_void_p()
        rc = L.tg_tree_build(_lib.ptr(x), _lib.ptr(m), _lib.ptr(h), n, 1, 1, _lib.TG_MEM_HOST, None, ctypes.byref(t))
        return rc, t
""") % ROOT


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    cc = shutil.which("gcc") or shutil.which("cc")
    if not cc:
        pytest.skip("no C compiler")
    from pytreegrav_gb300 import build

    build.build()
    d = tmp_path_factory.mktemp("fake")
    ver = d / "v.map"
    ver.write_text(SONAME + " { global: *; };\n")
    lib = d / SONAME
    subprocess.check_call([cc, "-O1", "-shared", "-fPIC", "-Wall", "-Werror", "-o", str(lib),
                           os.path.join(HERE, "fake_cudart.c"), "-Wl,-soname," + SONAME,
                           "-Wl,--version-script," + str(ver)])

    def run(code):
        env = dict(os.environ, LD_LIBRARY_PATH=str(d), PYTHONPATH=ROOT)
        r = subprocess.run([sys.executable, "-c", PRELUDE % str(lib) + textwrap.dedent(code)], capture_output=True,
                           text=True, timeout=300, env=env)
        assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-4000:]

    return run


def test_page_locked_words_do_not_grow_with_device_changes(fake):
    """A thread that goes back and forth between two devices: one block per device."""
    fake("""
        perm = np.empty(n, np.int64)
        for i in range(50):
            F.fake_set_device(i % 2)
            assert L.tg_morton_order(_lib.ptr(x), n, _lib.TG_MEM_HOST, _lib.ptr(perm), None) == 0
        assert F.fake_host_blocks() <= 2, F.fake_host_blocks()
        F.fake_new_context(0)  # a device reset: its block died with the old context, another is made
        F.fake_set_device(0)
        for i in range(10):
            assert L.tg_morton_order(_lib.ptr(x), n, _lib.TG_MEM_HOST, _lib.ptr(perm), None) == 0
        assert F.fake_host_blocks() <= 3, F.fake_host_blocks()
    """)


def test_build_streams_do_not_grow_with_device_changes(fake):
    """Builds with node centres on a side stream (the stand-in reports five nodes): each device's streams and events
    are reused, from one thread and from several that end."""
    fake("""
        import threading
        five = (ctypes.c_uint64 * 1)(5)
        F.fake_patch(224, five, 8)  # the round's summary: five nodes made

        def once():
            rc, t = build()
            assert rc == 0, (rc, L.tg_last_error())
            L.tg_tree_free(t)

        for d in (0, 1):
            F.fake_set_device(d)
            once()
        assert b"k_node_centers" in F.fake_log()
        s, e, b = F.fake_streams(), F.fake_events(), F.fake_host_blocks()
        for i in range(50):
            F.fake_set_device(i % 2)
            once()
        for i in range(10):
            t = threading.Thread(target=once)
            t.start()
            t.join()
        assert (F.fake_streams(), F.fake_events(), F.fake_host_blocks()) == (s, e, b)
    """)


def test_side_stream_is_joined_when_a_launch_on_it_fails(fake):
    """A first tree-grouped walk whose targets' preparation fails to launch on the tree's side stream: the caller's
    stream waits for the side stream all the same, and a later walk prepares the targets instead of reading the
    buffer that was never filled."""
    fake("""
        rc, t = build()
        assert rc == 0
        acc = np.empty((n, 3))

        def walk():
            F.fake_clear_log()
            rc = L.tg_tree_fields(t, None, None, n, _lib.TG_FIELD_ACCEL, 1, 0.7, 1.0, 32, _lib.TG_GROUP_TREE,
                                  _lib.TG_ORDER_TREE, _lib.TG_FP32, None, _lib.TG_MEM_HOST, _lib.ptr(acc), None)
            return rc, [l.split() for l in F.fake_log().decode().splitlines()]

        F.fake_fail_launch(b"k_prep_targets")
        rc, log = walk()
        assert rc == _lib.TG_ERR_CUDA, rc
        at = [k for k, l in enumerate(log) if l[0] == "failed-launch"]
        assert len(at) == 1
        side = log[at[0]][2]
        joins = [l[1] for l in log[at[0]:] if l[0] == "record" and l[2] == side]
        assert joins and any(l[0] == "wait" and l[1] in joins and l[2] != side for l in log[at[0]:]), log
        rc, log = walk()
        assert rc == 0, (rc, L.tg_last_error())
        assert any("k_prep_targets" in l[0] for l in log)
    """)


def test_graph_memory_waits_for_the_last_replay(fake):
    """A walk graph replayed on a stream of the caller's and freed: its buffers are given back on a stream that waits for
    that replay first."""
    fake("""
        rc, t = build()
        assert rc == 0
        out, g = np.empty((n, 3)), ctypes.c_void_p()
        assert L.tg_walk_graph_create(t, _lib.TG_FIELD_ACCEL, 0, 0.7, 1.0, 32, _lib.TG_GROUP_TREE, _lib.ptr(out),
                                      ctypes.byref(g)) == 0
        stream = ctypes.c_void_p()
        F.cudaStreamCreateWithFlags(ctypes.byref(stream), 1)
        events = F.fake_events()
        F.fake_clear_log()
        for _ in range(3):
            assert L.tg_walk_graph_launch(g, stream) == 0
        assert L.tg_walk_graph_free(g) == 0
        log = [l.split() for l in F.fake_log().decode().splitlines()]
        replays = [k for k, l in enumerate(log) if l[0] == "graph-launch"]
        assert len(replays) == 3
        frees = [k for k, l in enumerate(log) if l[0] == "free"]
        assert frees
        after = [l[1] for l in log[replays[-1]:] if l[0] == "record" and l[2] == hex(stream.value)]
        waits = [k for k, l in enumerate(log) if l[0] == "wait" and l[1] in after and l[2] == log[frees[0]][2]]
        assert waits and waits[0] < frees[0], log
        assert F.fake_events() <= events + 1  # one event, back in the pool
    """)


def test_work_left_queued_orders_other_streams(fake):
    """What a call leaves queued on its stream -- a target set's groups, features, a grouping, FP64 quadrupoles -- comes
    before the next call's work on another stream, and before the memory is given back on the build's."""
    fake("""
        from pytreegrav_gb300 import theta as th
        A, B = ctypes.c_void_p(), ctypes.c_void_p()
        for s in (A, B):
            F.cudaStreamCreateWithFlags(ctypes.byref(s), 1)
        a, b = hex(A.value), hex(B.value)
        out, feat, ng, quad = np.empty((n, 3)), np.empty((n, 16), np.float32), ctypes.c_int64(), ctypes.c_void_p()

        def log_of(f):
            F.fake_clear_log()
            assert f() == 0, L.tg_last_error()
            return [l.split() for l in F.fake_log().decode().splitlines()]

        def left_behind(log):  # the events recorded on A after its last launch
            last = max(k for k, l in enumerate(log) if l[0].startswith("launch") and l[2] == a)
            events = [l[1] for l in log[last:] if l[0] == "record" and l[2] == a]
            assert events or any(l[0] == "synchronize" and l[2] == a for l in log[last:]), log
            return events

        def waits_first(log, events, stream, what):
            at = [k for k, l in enumerate(log) if l[0].startswith(what) and l[2] == stream]
            assert at, log
            assert not events or any(l[0] == "wait" and l[1] in events and l[2] == stream for l in log[:at[0]]), log

        def fields(stream):
            return L.tg_tree_fields(t, None, None, n, 2, 0, 0.7, 1.0, 32, _lib.TG_GROUP_TREE, _lib.TG_ORDER_TREE, _lib.TG_FP32,
                                    None, _lib.TG_MEM_HOST, _lib.ptr(out), stream)

        first = [lambda: L.tg_tree_groups(t, 32, ctypes.byref(ng), A),
                 lambda: L.tg_theta_features(t, 32, 0, _lib.ptr(feat), A),
                 lambda: L.tg_tree_quadrupoles(t, ctypes.byref(quad), A)]
        for call in first:
            for then in ("other stream", "free"):
                rc, t = build()
                assert rc == 0
                ev = left_behind(log_of(call))
                if then == "free":
                    waits_first(log_of(lambda: L.tg_tree_free(t)), ev, "(nil)", "free")
                else:
                    waits_first(log_of(lambda: fields(B)), ev, b, "launch")
                    L.tg_tree_free(t)
        for then in ("other stream", "features", "free"):
            rc, t = build()
            ts = ctypes.c_void_p()
            ev = left_behind(log_of(lambda: L.tg_targets_create(t, _lib.ptr(x), _lib.ptr(h), n, 32, _lib.TG_MEM_HOST, A,
                                                                ctypes.byref(ts))))
            if then == "other stream":
                log = log_of(lambda: L.tg_targets_fields(ts, 2, 0, 0.7, 1.0, _lib.TG_FP32, None, _lib.TG_MEM_HOST,
                                                         _lib.ptr(out), B))
                waits_first(log, ev, b, "launch")
            elif then == "features":
                ev2 = ev
                log = log_of(lambda: L.tg_targets_features(ts, 0, _lib.ptr(feat), B))
                waits_first(log, ev2, b, "launch")
            L.tg_targets_free(ts)
            waits_first(log_of(lambda: L.tg_tree_free(t)), ev if then == "free" else [], "(nil)", "free")
    """)
