"""A kernel's bounded wait that runs out (coli_cuda_expire_wait) is reported by the next call that waits for the
device: it returns 0, leaves its outputs alone, and the same call works again behind it. In a process of its own,
because coli_cuda_kernel_status keeps the code."""
import subprocess
import sys
import os

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SCRIPT = r"""
import ctypes as C
import numpy as np
from colibri_b200 import workloads as W
from colibri_b200.backend import Backend, MoeLayer
from tests.util import upload_qt

be = Backend()
assert be.init_devices((0,)) == 1
rng = np.random.default_rng(1)
D, I, E, K = 256, 128, 16, 4
ex = [[upload_qt(be, t) for t in W.expert_weights(D, I, 4, 32, 5 + e)] for e in range(E)]
side = lambda k: [e[k] for e in ex]
lay = MoeLayer(be, D, I, E, K, side(0), side(1), side(2), 0, 0, max_rows=64)
x = rng.standard_normal((64, D)).astype(np.float32)
lg = rng.standard_normal((64, E)).astype(np.float32)
xd, rwd, rbd = (be.pipe_alloc(0, n) for n in (x.nbytes, E * D * 4, E * 4))
rw = rng.standard_normal((E, D)).astype(np.float32)
assert be.pipe_upload(0, xd, x.ctypes.data, x.nbytes) and be.pipe_upload(0, rwd, rw.ctypes.data, rw.nbytes)
assert be.pipe_upload(0, rbd, np.zeros(E, np.float32).ctypes.data, E * 4)

def router(o):
    return be.pipe_router(0, xd, rwd, rbd, D, E, K, C.c_float(0.0), 0, C.c_float(1.0), o[0].ctypes.data, o[1].ctypes.data, o[2].ctypes.data)
def group(o):
    rows = np.array([1, 2], np.int32)
    return be.expert_group(*[Backend.handle_array(side(k)[:2]) for k in range(3)], rows.ctypes.data_as(C.POINTER(C.c_int)), 2,
                           o[0].ctypes.data, x.ctypes.data)
def take(o):
    rows = np.array([1, 2], np.int32)
    if not be.expert_group_issue(*[Backend.handle_array(side(k)[:2]) for k in range(3)], rows.ctypes.data_as(C.POINTER(C.c_int)), 2,
                                 x.ctypes.data):
        return 0
    p = be.expert_group_take(0)
    if not p:
        return 0
    o[0][:] = np.ctypeslib.as_array(C.cast(p, C.POINTER(C.c_float)), shape=o[0].shape)
    return 1
f32 = lambda *s: np.full(s, 77, np.float32)
box = C.c_void_p(ex[0][0])
cases = {
    "pipe_router": (router, [np.full(K, 77, np.int32), f32(K), np.full(1, 77, np.int32)]),
    "pipe_download": (lambda o: be.pipe_download(0, xd, o[0].ctypes.data, o[0].nbytes), [f32(64, D)]),
    "pipe_sync": (lambda o: be.pipe_sync(0), []),
    "matmul": (lambda o: be.matmul(C.byref(box), o[0].ctypes.data, x.ctypes.data, None, None, 4, 8, D, I, 0, 32), [f32(8, I)]),
    "matmul, many rows": (lambda o: be.matmul(C.byref(box), o[0].ctypes.data, x.ctypes.data, None, None, 4, 64, D, I, 0, 32), [f32(64, I)]),
    "expert_mlp": (lambda o: be.expert_mlp(*ex[0], o[0].ctypes.data, x.ctypes.data, 64), [f32(64, D)]),
    "expert_group": (group, [f32(3, D)]),
    "expert_group_take": (take, [f32(3, D)]),
    "moe_layer": (lambda o: be.moe_layer(lay.handle, o[0].ctypes.data, x.ctypes.data, lg.ctypes.data, 4, None, None, None), [f32(4, D)]),
    "moe_layer, many rows": (lambda o: be.moe_layer(lay.handle, o[0].ctypes.data, x.ctypes.data, lg.ctypes.data, 64, o[1].ctypes.data,
                                                    None, None), [f32(64, D), np.full((64, K), 77, np.int32)]),
}
for name, (call, out) in cases.items():
    assert call(out), name                                  # as it is without an expired wait
    want = [o.copy() for o in out]
    for o in out:
        o[...] = 77
    assert be.expire_wait(0)
    assert call(out) == 0, name + ": an expired wait went unnoticed"
    for o in out:
        assert np.all(o == 77), name + ": outputs of a failed call were written"
    assert call(out), name + ": does not work again"
    for o, w in zip(out, want):
        assert np.array_equal(o, w) and not np.all(o == 77), name
    assert be.kernel_status(0) == 1
# seen by a blocking call between issue and take: the issued group may be the one it hit, so its take reports it too
rows = np.array([1, 2], np.int32)
issue = lambda: be.expert_group_issue(*[Backend.handle_array(side(k)[:2]) for k in range(3)],
                                      rows.ctypes.data_as(C.POINTER(C.c_int)), 2, x.ctypes.data)
assert be.expire_wait(0) and issue() and be.pipe_sync(0) == 0 and not be.expert_group_take(0)
assert issue() and be.pipe_sync(0) == 1 and be.expert_group_take(0)
be.shutdown()
print("ok")
"""


def test_expired_wait_is_reported_by_the_call_that_waits():
    r = subprocess.run([sys.executable, "-c", SCRIPT], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stdout + r.stderr
