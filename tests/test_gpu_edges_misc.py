"""Branches chosen by size or alignment: the router GEMV's three forms, the cluster-wide argmax at small and
ragged widths, and transfers of one and several staged pieces."""
import numpy as np
import pytest

import colibri_b200.workloads as W
from colibri_b200.backend import MoeLayer
from tests.test_gpu_router import free_layer, upload_layer

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("E,M", [(8, 1), (33, 9), (64, 74), (64, 75), (200, 40)])      # 64 x 74: the last that fits two waves of 148 x 16
def test_router_forms(be, E, M):
    cfg = dict(W.CONFIGS["c2_small"], E=E, K=2, gating=1, norm_topk=1)
    L = W.HostLayerWeights(cfg, 5 + E)
    g, u, d, sh = upload_layer(be, L)
    rw = np.random.default_rng(E).standard_normal((E, cfg["D"])).astype(np.float32)
    lay = MoeLayer(be, cfg["D"], cfg["I"], E, 2, g, u, d, 1, 1, 1.0, router_w=rw, max_rows=M)
    x = W.activations(M, cfg["D"], M)
    lg = np.zeros((M, E), np.float32)
    for i in range(cfg["D"]):                                   # product and sum rounded separately, in order
        lg += (x[:, i, None] * rw[None, :, i]).astype(np.float32)
    a, b = lay(x), lay(x, lg)
    for p, q in zip(a, b):
        assert np.array_equal(p.view(np.uint32), q.view(np.uint32))
    lay.free()
    free_layer(be, (g, u, d, sh))


@pytest.mark.parametrize("D", [64, 1024, 1028, 1030, 6146])     # D % 4 != 0: the form without bulk copies
def test_pipe_router_widths(be, D):
    import ctypes as C
    E, K = 24, 3
    rng = np.random.default_rng(D)
    x, rw = rng.standard_normal(D).astype(np.float32), (rng.standard_normal((E, D)) / 16).astype(np.float32)
    xd, rwd, rbd = (be.pipe_alloc(0, n * 4) for n in (D, E * D, E))
    zero = np.zeros(E, np.float32)
    for p, h in ((xd, x), (rwd, rw), (rbd, zero)):
        assert be.pipe_upload(0, p, h.ctypes.data, h.nbytes)
    idx, w, keff = np.zeros(K, np.int32), np.zeros(K, np.float32), np.zeros(1, np.int32)
    assert be.pipe_router(0, xd, rwd, rbd, D, E, K, C.c_float(0.0), 0, C.c_float(1.0), idx.ctypes.data, w.ctypes.data, keff.ctypes.data)
    lg = np.zeros(E, np.float32)
    for i in range(D):
        lg += (x[i] * rw[:, i]).astype(np.float32)
    assert list(idx) == list(np.argsort(-lg, kind="stable")[:K]) and keff[0] == K
    assert np.allclose(w, 1 / (1 + np.exp(-lg[idx].astype(np.float64))), rtol=1e-6)
    for p in (xd, rwd, rbd):
        be.pipe_free(0, p)


@pytest.mark.parametrize("S,N", [(1, 1), (3, 7), (2, 8191), (1, 129280), (2, 33333)])
def test_argmax_widths_and_ties(be, S, N):
    x = np.random.default_rng(N).integers(0, max(2, N // 3), (S, N)).astype(np.float32)      # the largest value several times
    xd, od = be.pipe_alloc(0, x.nbytes), be.pipe_alloc(0, S * 4)
    out = np.zeros(S, np.int32)
    assert be.pipe_upload(0, xd, x.ctypes.data, x.nbytes) and be.pipe_argmax(0, od, xd, S, N)
    assert be.pipe_download(0, od, out.ctypes.data, out.nbytes)
    assert np.array_equal(out, x.argmax(1))
    be.pipe_free(0, xd)
    be.pipe_free(0, od)


@pytest.mark.parametrize("nbytes", [4, 65536, 65540, 1 << 20, (2 << 20) + 4, 11 * (1 << 20) + 12])
def test_staged_transfers(be, nbytes):
    a = np.random.default_rng(nbytes).integers(0, 1 << 32, nbytes // 4, dtype=np.uint32)
    b = np.zeros_like(a)
    p = be.pipe_alloc(0, nbytes)
    assert be.pipe_upload(0, p, a.ctypes.data, nbytes) and be.pipe_download(0, p, b.ctypes.data, nbytes)
    assert np.array_equal(a, b)
    be.pipe_free(0, p)


@pytest.mark.parametrize("nbytes", [4, 100000])
def test_transfers_without_an_end_are_refused(be, nbytes):
    p, a = be.pipe_alloc(0, nbytes), np.ones(nbytes // 4, np.float32)
    assert be.pipe_upload(0, p, None, nbytes) == 0 and be.pipe_upload(0, None, a.ctypes.data, nbytes) == 0
    assert be.pipe_download(0, p, None, nbytes) == 0 and be.pipe_download(0, None, a.ctypes.data, nbytes) == 0
    assert be.pipe_upload(0, None, None, 0) == 1 and be.pipe_download(0, None, None, 0) == 1 and np.all(a == 1)
    be.pipe_free(0, p)


@pytest.mark.parametrize("nbytes", [4096, 65536, 3 << 20])
def test_upload_source_may_be_reused(be, nbytes):
    """A pinned source overwritten right behind the call, while the stream is still busy with earlier work."""
    import torch
    want = torch.arange(nbytes // 4, dtype=torch.int32)
    src = want.clone().pin_memory()
    n = 1 << 28
    busy, p = be.pipe_alloc(0, n * 4), be.pipe_alloc(0, nbytes)
    got = np.zeros(nbytes // 4, np.int32)
    for _ in range(8):                                          # about 4 ms of kernels before the copy's turn
        assert be.pipe_add(0, busy, busy, n)
    assert be.pipe_upload(0, p, src.data_ptr(), nbytes)
    src.fill_(-1)
    assert be.pipe_download(0, p, got.ctypes.data, nbytes)
    assert np.array_equal(got, want.numpy())
    be.pipe_free(0, busy)
    be.pipe_free(0, p)


def test_rows_off_their_boundary_are_refused(be):
    """Device rows that kernels read or write 16 bytes at a time: a pointer between the boundaries is an answer of 0 with the
    output left alone, where no kernel needs the boundary the call still runs."""
    import ctypes as C
    from colibri_b200.backend import Backend
    from tests.util import upload_qt
    D, I, E, K, M = 256, 128, 4, 2, 12
    ex = [[upload_qt(be, t) for t in W.expert_weights(D, I, 4, 32, 60 + e)] for e in range(E)]
    side = lambda k: Backend.handle_array([e[k] for e in ex])
    lay = MoeLayer(be, D, I, E, K, [e[0] for e in ex], [e[1] for e in ex], [e[2] for e in ex], 0, 0, max_rows=M)
    rows = np.array([3] * E, np.int32)
    i32 = rows.ctypes.data_as(C.POINTER(C.c_int))
    n = M * D * 4
    x, y, lg = (be.pipe_alloc(0, n + 64) for _ in range(3))
    a = np.random.default_rng(0).standard_normal(n // 4 + 16).astype(np.float32)
    for p in (x, y, lg):
        assert be.pipe_upload(0, p, a.ctypes.data, n + 64)
    calls = {
        "moe_layer_dev": lambda px, py, S: be.moe_layer_dev(lay.handle, py, px, lg + 4, S, None, None, None),
        "expert_group_dev": lambda px, py, S: be.expert_group_dev(side(0), side(1), side(2), i32, E, py, px),
        "ep_expert_group_dev": lambda px, py, S: be.ep_expert_group_dev(side(0), side(1), side(2), E, i32, 1, py, px, 0),
        "pipe_gemm": lambda px, py, S: be.pipe_gemm(ex[0][0], py, px, S),
        "pipe_gemm_noalloc": lambda px, py, S: be.pipe_gemm_noalloc(ex[0][0], py, px, S),
    }
    got = np.empty_like(a)
    for name, call in calls.items():
        for S in (2, M):
            for dx, dy in ((4, 0), (0, 4), (8, 8), (12, 0)):
                if name == "pipe_gemm" and S == 2 and dx == 0:
                    continue
                assert call(x + dx, y + dy, S) == 0, (name, S, dx, dy)
    assert be.pipe_sync(0) and be.pipe_download(0, y, got.ctypes.data, n + 64) and np.array_equal(got, a)
    for name, call in calls.items():
        for S in (2, M):
            assert call(x + 16, y + 32, S) and be.pipe_sync(0), name
    assert be.pipe_gemm(ex[0][0], y + 4, x, 2) and be.pipe_sync(0)                 # few rows: results are stored one by one
    assert be.kernel_status(0) == 0
    lay.free()
    for p in (x, y, lg):
        be.pipe_free(0, p)
    for e in ex:
        for h in e:
            be.tensor_free(h)


@pytest.mark.parametrize("fmt,gs", [(2, 0), (7, 0), (4, 32)])
@pytest.mark.parametrize("bf16", [0, 1])
def test_ep_rows_between_boundaries(be, fmt, gs, bf16):
    """Received rows that start on 8 bytes (bf16: 4) but not on 16 (8): taken whatever the mean of rows per expert, the line
    between the two kernels only says which one is faster. Bit for bit the tensor cores' result of the same rows on a boundary."""
    import ctypes as C
    from colibri_b200.backend import Backend
    from tests.util import upload_qt
    D, I, E = 256, 128, 4
    ex = [[upload_qt(be, t) for t in W.expert_weights(D, I, fmt, gs, 60 + e)] for e in range(E)]
    side = [Backend.handle_array([e[k] for e in ex]) for k in range(3)]
    for counts in ([2, 1, 1, 1], [3, 2, 2, 3], [9, 8, 8, 9]):
        rows = np.array(counts, np.int32)
        n = int(rows.sum())
        x = W.bf16_round(np.random.default_rng(n).standard_normal((n, D)).astype(np.float32))
        raw = (x.view(np.uint32) >> 16).astype(np.uint16) if bf16 else x
        xd, yd = be.pipe_alloc(0, raw.nbytes + 16), be.pipe_alloc(0, x.nbytes)
        out = []
        try:
            for off, mode in ((0, 2), (4 if bf16 else 8, 1)):
                be.set_tensor_core(mode)
                assert be.pipe_upload(0, xd + off, raw.ctypes.data, raw.nbytes)
                assert be.ep_expert_group_dev(*side, E, rows.ctypes.data_as(C.POINTER(C.c_int)), 1, yd, xd + off, bf16), (counts, off)
                y = np.empty((n, D), np.float32)
                assert be.pipe_download(0, yd, y.ctypes.data, y.nbytes)
                out.append(y)
        finally:
            be.set_tensor_core(1)
            be.pipe_free(0, xd)
            be.pipe_free(0, yd)
        assert np.array_equal(*out) and np.any(out[0]), counts
    assert be.kernel_status(0) == 0
    for e in ex:
        for h in e:
            be.tensor_free(h)
