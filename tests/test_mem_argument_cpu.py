"""Where the caller's arrays live (`mem`) is checked before anything is read, by every entry point that takes it:
unknown values, and TG_MEM_HOST_FIELDS (whose `out` is an array of addresses) wherever the header does not list it,
are TG_ERR_BAD_ARG. The handles here are zeroed memory, which no call gets to use."""

import ctypes
import os
import re

import numpy as np
import pytest

from pytreegrav_gb300 import _lib

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
FIELDS_TOO = {"tg_tree_fields", "tg_tree_fields_learned", "tg_targets_fields", "tg_targets_fields_learned",
              "tg_bruteforce"}


def entry_points():
    """(name, parameter names) of every declared function with a `mem` parameter."""
    found = []
    for header in ("pytreegrav_gb300.h", "pytreegrav_gb300_theta.h"):
        src = open(os.path.join(ROOT, "include", header)).read()
        src = re.sub(r"/\*.*?\*/", "", src, flags=re.S)
        for name, params in re.findall(r"tg_status (tg_\w+)\(([^)]*)\);", src):
            names = [re.search(r"(\w+)\s*$", p).group(1) for p in params.split(",")]
            if "mem" in names:
                found.append((name, names))
    return found


def test_header_lists_who_takes_the_fields_form():
    src = open(os.path.join(ROOT, "include", "pytreegrav_gb300.h")).read()
    text = " ".join(src[:src.index("typedef enum")].replace("\n * ", " ").split())
    listed = re.search(r"\. ((?:tg_\w+, )+tg_\w+ and tg_\w+) also take TG_MEM_HOST_FIELDS", text).group(1)
    assert set(re.findall(r"tg_\w+", listed)) == FIELDS_TOO


@pytest.mark.parametrize("name,names", entry_points(), ids=[e[0] for e in entry_points()])
def test_mem_is_checked_first(name, names):
    L = _lib.load()
    data = np.ones(4096)
    handle = ctypes.create_string_buffer(8192)
    out = ctypes.c_void_p()
    small = {"n": 8, "nt": 8, "ns": 8, "n_systems": 1, "group_size": 8, "fields": 2, "theta": 0.7, "theta_fallback": 0.7,
             "G": 1.0, "precision": _lib.TG_FP32, "nrays": 1, "ray_stride": 0, "nbins": 4, "kind": 0, "rank": 1,
             "boxsize": 0.0, "max_bin_size_ratio": 1.0, "out_min": 1.0, "out_max": 2.0, "theta_max": 1.0,
             "log10_lambda": 0.0, "order": _lib.TG_ORDER_TREE, "grouping": _lib.TG_GROUP_BLOCKS}
    offsets = np.array([0, 8], np.int64)
    fn = getattr(L, name)

    def call(mem):
        args = []
        for p, kind in zip(names, fn.argtypes):
            if p == "mem":
                args.append(mem)
            elif p == "stream":
                args.append(None)
            elif p == "offsets":
                args.append(_lib.ptr(offsets))
            elif p in ("tree", "source", "targets", "model", "S", "sources"):
                args.append(ctypes.cast(handle, ctypes.c_void_p))
            elif kind is ctypes.c_void_p:
                args.append(_lib.ptr(data))
            elif kind in (ctypes.c_int, ctypes.c_int64, ctypes.c_int32, ctypes.c_uint64, ctypes.c_double, ctypes.c_float):
                args.append(kind(small.get(p, 0)))
            else:
                args.append(ctypes.byref(out))
        return fn(*args)

    for mem in [-1, 3, 7] + ([] if name in FIELDS_TOO else [_lib.TG_MEM_HOST_FIELDS]):
        assert call(mem) == _lib.TG_ERR_BAD_ARG, mem
