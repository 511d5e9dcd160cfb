"""Calls of at most 8 rows: the one-launch projection (k_gemv_rows) and grouped calls on the fused
decode kernel with a pass list from the host, at the edges of their ranges, against the CPU oracle."""
import ctypes as C

import numpy as np
import pytest

from colibri_b200.backend import Backend
from tests.test_gpu_grouped import rand_qt
from tests.util import max_rel_err, upload_qt

pytestmark = pytest.mark.gpu
FMTS = [(4, 32, True), (4, 32, False), (4, 128, True), (2, 0, False), (7, 0, False)]


@pytest.mark.parametrize("fmt,gs,half", FMTS)
@pytest.mark.parametrize("I,O", [(128, 32), (1024, 96), (8320, 64)])
def test_projection(be, fmt, gs, half, I, O):
    rng = np.random.default_rng(fmt + gs + I)
    t = rand_qt(rng, O, I, fmt, gs, half=half)
    h = upload_qt(be, t)
    w = t.dequant().astype(np.float64)
    for S in (1, 2, 4, 5, 8):                 # 8 x 8320 is beyond the kernel's activation space: the streaming path
        x = rng.standard_normal((S, I)).astype(np.float32)
        ok, y = be.run_matmul([h], x, None, None, fmt, I, O, gs=gs)
        assert ok
        mag = np.abs(x).astype(np.float64) @ np.abs(w).T
        assert np.all(np.abs(y - x.astype(np.float64) @ w.T) <= 2e-6 * mag + 1e-30), S
    be.tensor_free(h)
    assert be.kernel_status(0) == 0


@pytest.mark.parametrize("fmt,gs,half", FMTS)
@pytest.mark.parametrize("rows", [[1], [8], [5, 3], [1] * 8, [4, 1, 2]])
def test_grouped(be, oracle, fmt, gs, half, rows):
    D, I = 640, 256
    rng = np.random.default_rng(len(rows) + fmt)
    ex = [(rand_qt(rng, I, D, fmt, gs, half=half), rand_qt(rng, I, D, fmt, gs, half=half), rand_qt(rng, D, I, fmt, gs, half=half))
          for _ in rows]
    hs = [[upload_qt(be, t) for t in e] for e in ex]
    x = ((rng.random((sum(rows), D)) - 0.5) * 2).astype(np.float32)
    be.set_tensor_core(0)
    ok, y = be.run_expert_group([h[0] for h in hs], [h[1] for h in hs], [h[2] for h in hs], rows, x, D)
    be.set_tensor_core(1)
    assert ok and be.kernel_status(0) == 0
    off = 0
    for e, r in zip(ex, rows):
        assert max_rel_err(y[off:off + r], oracle.expert_mlp(x[off:off + r], *e)) <= 1e-3
        off += r
    for h in hs:
        for t in h:
            be.tensor_free(t)


@pytest.mark.parametrize("fmt,gs,half", FMTS)
@pytest.mark.parametrize("count", [1, 8, 16, 17])
def test_resident_weighted_sum(be, oracle, fmt, gs, half, count):
    D, I = 512, 256
    rng = np.random.default_rng(count + fmt)
    ex = [(rand_qt(rng, I, D, fmt, gs, half=half), rand_qt(rng, I, D, fmt, gs, half=half), rand_qt(rng, D, I, fmt, gs, half=half))
          for _ in range(count)]
    hs = [[upload_qt(be, t) for t in e] for e in ex]
    x, w = rng.standard_normal((1, D)).astype(np.float32), rng.random(count).astype(np.float32)
    xd, slot, acc = be.pipe_alloc(0, D * 4), be.pipe_alloc(0, D * 4), be.pipe_alloc(0, D * 4)
    assert be.pipe_upload(0, xd, x.ctypes.data, D * 4)
    arr = [Backend.handle_array([h[k] for h in hs]) for k in range(3)]
    assert be.expert_group_resident_issue(*arr, w.ctypes.data, count, 0, xd, slot)
    assert be.expert_group_resident_take(0, (C.c_int * 1)(0), 1, slot, acc, D)
    got = np.empty(D, np.float32)
    assert be.pipe_download(0, acc, got.ctypes.data, D * 4)
    want = sum(wi * oracle.expert_mlp(x, *e)[0] for wi, e in zip(w, ex))
    assert np.all(np.abs(got - want) <= 1e-3 * (np.abs(want) + 1e-3 * np.abs(want).max()))
    for p in (xd, slot, acc):
        be.pipe_free(0, p)
    for h in hs:
        for t in h:
            be.tensor_free(t)
