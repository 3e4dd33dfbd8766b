"""Tree builds under more than one CUDA context of a process: what the builder
asks of a context (k_sah_tree's shared memory) is asked of each, so the same
prims give the same tree in the device's primary context and in one that the
process makes for itself, whichever comes first.  In a process of its own: the
contexts are made and made current through the driver API."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CHILD = r"""
import ctypes as C, sys
import numpy as np
import vrg

cu = C.CDLL("libcuda.so.1")
lib = vrg.load_library()
fn = lib.vrg_build_tl_bvh_noalloc
fn.restype = C.c_int32
fn.argtypes = [C.c_void_p] * 3 + [C.c_uint32] + [C.c_void_p] * 3


def ok(e, what):
    assert e == 0, (what, e)


def build(aabbs, power, ids):
    n = len(ids)
    nodes, order = np.zeros((2 * n - 1) * 40, np.uint8), np.zeros(n, np.uint32)
    dev = []
    for a in (aabbs, power, ids, nodes, order):
        p = C.c_uint64()
        ok(cu.cuMemAlloc_v2(C.byref(p), C.c_size_t(a.nbytes)), "alloc")
        ok(cu.cuMemcpyHtoD_v2(p, C.c_void_p(a.ctypes.data), C.c_size_t(a.nbytes)), "in")
        dev.append(p)
    a = [p.value for p in dev]
    st = fn(a[0], a[1], a[2], n, a[3], a[4], None)
    assert st == 0, lib.vrg_last_error()
    for p, a in zip(dev[3:], (nodes, order)):
        ok(cu.cuMemcpyDtoH_v2(C.c_void_p(a.ctypes.data), p, C.c_size_t(a.nbytes)), "out")
    for p in dev:
        ok(cu.cuMemFree_v2(p), "free")
    return nodes.tobytes() + order.tobytes()


rng = np.random.default_rng(3)
sets = []
for n in (2, 40, 2560, 2561):
    lo = (rng.random((n, 3)) * 64).astype(np.float32)
    hi = lo + (rng.random((n, 3)) * 4).astype(np.float32)
    sets.append((np.ascontiguousarray(np.concatenate([lo, hi], 1)), rng.random(n).astype(np.float32),
                 rng.permutation(n).astype(np.uint32)))

primary_first = sys.argv[1] == "primary"
if primary_first:
    ctx = vrg.Context(0)
ok(cu.cuInit(0), "init")
d, own = C.c_int(), C.c_void_p()
ok(cu.cuDeviceGet(C.byref(d), 0), "device")
got = {}
if primary_first:
    got["primary"] = [build(*s) for s in sets]
ok(cu.cuCtxCreate_v2(C.byref(own), 0, d), "create")
got["own"] = [build(*s) for s in sets]
ok(cu.cuCtxSetCurrent(None), "unset")
if not primary_first:
    ctx = vrg.Context(0)
got["again"] = [build(*s) for s in sets]
ctx.close()
first = next(iter(got.values()))
assert all(g == first for g in got.values())
print("same trees", len(got))
"""


@pytest.mark.parametrize("first", ["primary", "own"])
def test_builds_in_two_contexts(vrglib, first):
    env = dict(os.environ)
    env["PYTHONPATH"] = os.path.dirname(vrglib.__file__) + os.pathsep + env.get("PYTHONPATH", "")
    r = subprocess.run([sys.executable, "-c", CHILD, first], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "same trees" in r.stdout, r.stdout + r.stderr
