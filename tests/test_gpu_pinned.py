"""Host-buffer calls whose rows are not staged in a pinned buffer of their size: more rows than such a buffer may hold
(32 MB), and a system that gives no pinned memory at all. Every call against its device-buffer form, bit for bit."""
import os
import shutil
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SCRIPT = r"""
import ctypes as C
import sys
import numpy as np
from colibri_b200 import workloads as W
from colibri_b200.backend import Backend, MoeLayer
from tests.util import upload_qt

be = Backend()
assert be.init_devices((0,)) == 1
rng = np.random.default_rng(1)
D, I, E, K = 512, 256, 8, 2
ex = [[upload_qt(be, t) for t in W.expert_weights(D, I, 4, 32, 5 + e)] for e in range(E)]
side = lambda k: [e[k] for e in ex]
i32p = C.POINTER(C.c_int)

def same(host, dev, what):
    back = np.empty_like(host)
    assert be.pipe_download(0, dev, back.ctypes.data, back.nbytes), what
    assert np.array_equal(host.view(np.uint32), back.view(np.uint32)), what

for M in [int(a) for a in sys.argv[1:]]:
    x = rng.standard_normal((M, D)).astype(np.float32)
    lg = rng.standard_normal((M, E)).astype(np.float32)
    xd, yd, lgd, kd = (be.pipe_alloc(0, n) for n in (x.nbytes, x.nbytes, lg.nbytes, M * (8 * K + 4)))
    assert be.pipe_upload(0, xd, x.ctypes.data, x.nbytes) and be.pipe_upload(0, lgd, lg.ctypes.data, lg.nbytes)
    y = np.full((M, D), np.nan, np.float32)
    # projection
    box = C.c_void_p(ex[0][2])                              # [D, I]
    xi = np.ascontiguousarray(x[:, :I])
    assert be.matmul(C.byref(box), y.ctypes.data, xi.ctypes.data, None, None, 4, M, I, D, 0, 32)
    xid = be.pipe_alloc(0, xi.nbytes)
    assert be.pipe_upload(0, xid, xi.ctypes.data, xi.nbytes) and be.pipe_gemm(ex[0][2], yd, xid, M)
    same(y, yd, "matmul")
    # one expert, then a group of three
    one = np.array([M], np.int32)
    assert be.expert_mlp(*ex[1], y.ctypes.data, x.ctypes.data, M)
    assert be.expert_group_dev(*[Backend.handle_array([h]) for h in ex[1]], one.ctypes.data_as(i32p), 1, yd, xd)
    same(y, yd, "expert_mlp")
    if M >= 3:
        rows = np.array([1, M - 2, 1], np.int32)
        args = [Backend.handle_array(side(k)[:3]) for k in range(3)] + [rows.ctypes.data_as(i32p), 3]
        assert be.expert_group(*args, y.ctypes.data, x.ctypes.data) and be.expert_group_dev(*args, yd, xd)
        same(y, yd, "expert_group")
    # a layer, with its routing
    lay = MoeLayer(be, D, I, E, K, side(0), side(1), side(2), 0, 0, max_rows=M)
    out, idx, w, keff = lay(x, lg)
    n = M * K * 4
    assert be.moe_layer_dev(lay.handle, yd, xd, lgd, M, kd, kd + n, kd + 2 * n)
    same(out, yd, "moe_layer")
    for a, at in ((idx, 0), (w, n), (keff, 2 * n)):
        same(a, kd + at, "routing")
    lay.free()
    for p in (xd, yd, lgd, kd, xid):
        be.pipe_free(0, p)
# the router's answer
rw, b = rng.standard_normal((E, D)).astype(np.float32), np.zeros(E, np.float32)
row = rng.standard_normal(D).astype(np.float32)
xd, rwd, rbd = (be.pipe_alloc(0, a.nbytes) for a in (row, rw, b))
for p, a in ((xd, row), (rwd, rw), (rbd, b)):
    assert be.pipe_upload(0, p, a.ctypes.data, a.nbytes)
idx, w, keff = np.zeros(K, np.int32), np.zeros(K, np.float32), np.zeros(1, np.int32)
assert be.pipe_router(0, xd, rwd, rbd, D, E, K, C.c_float(0.0), 0, C.c_float(1.0), idx.ctypes.data, w.ctypes.data, keff.ctypes.data)
assert list(idx) == list(np.argsort(-(rw.astype(np.float64) @ row))[:K]) and keff[0] == K
assert np.allclose(w, 1 / (1 + np.exp(-(rw[idx].astype(np.float64) @ row))), rtol=1e-5)
assert be.kernel_status(0) == 0
be.shutdown()
print("ok")
"""
SHIM = r"""
#include <stddef.h>
#include <dlfcn.h>
/* only the few words that set-up needs are granted */
int cudaMallocHost(void **p, size_t n) {
    if (n > 64) return 2;
    return ((int (*)(void **, size_t))dlsym(dlopen("libcudart.so.12", RTLD_LAZY | RTLD_NOLOAD), "cudaMallocHost"))(p, n);
}
"""


def run(rows, **env):
    r = subprocess.run([sys.executable, "-c", SCRIPT, *[str(m) for m in rows]], cwd=ROOT, env=dict(os.environ, **env),
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stdout + r.stderr


def test_rows_around_the_pinned_limit():
    run([1, 16384, 16385, 16384 + 4097])                    # 32 MB of rows of 512 floats, and beyond


def test_without_pinned_memory(tmp_path):
    if not shutil.which("gcc"):
        pytest.skip("no host C compiler")
    src, lib = tmp_path / "nopin.c", tmp_path / "nopin.so"
    src.write_text(SHIM)
    subprocess.check_call(["gcc", "-D_GNU_SOURCE", "-shared", "-fPIC", "-o", str(lib), str(src), "-ldl"])
    run([1, 7, 40, 300, 3000], LD_PRELOAD=str(lib))


def test_layers_of_two_threads(be):
    """Host-buffer calls of two layers at once, larger than a layer's own staging: each gets its own rows."""
    import threading
    import numpy as np
    from colibri_b200 import workloads as W
    from colibri_b200.backend import MoeLayer
    from tests.util import upload_qt
    D, I, E, K, M = 4096, 128, 96, 1, 48                     # 0.5 rows an expert: the streaming kernel, with the layer's own workspaces
    ex = [[upload_qt(be, t) for t in W.expert_weights(D, I, 4, 32, 5 + e)] for e in range(8)]
    side = lambda k: [ex[e % 8][k] for e in range(E)]
    lays = [MoeLayer(be, D, I, E, K, side(0), side(1), side(2), 0, 0, max_rows=M) for _ in range(2)]
    rng = np.random.default_rng(0)
    xs = [rng.standard_normal((M, D)).astype(np.float32) for _ in range(2)]
    lgs = [rng.standard_normal((M, E)).astype(np.float32) for _ in range(2)]
    want = [lay(x, lg)[0] for lay, x, lg in zip(lays, xs, lgs)]
    bad = []

    def work(i):
        for _ in range(150):
            if not np.array_equal(lays[i](xs[i], lgs[i])[0], want[i]):
                bad.append(i)
    t = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for a in t:
        a.start()
    for a in t:
        a.join()
    assert not bad and be.kernel_status(0) == 0
    for lay in lays:
        lay.free()
    for e in ex:
        for h in e:
            be.tensor_free(h)
