"""Grouped tensor-core GEMM at the edges of its tiles: row counts around the 16-row padding
and the 64-row pass, contractions that fill a partial sum of four 128-column blocks and ones that
end inside it, rows with and without fp16 lo terms in one pass, and a layer whose plan is made on
the device. CPU oracle, max relative error 1e-3."""
import ctypes as C

import numpy as np
import pytest

from colibri_b200 import workloads as W
from colibri_b200.backend import MoeLayer
from tests.test_gpu_grouped import rand_qt
from tests.util import max_rel_err, upload_qt

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fmt,gs", [(4, 32), (2, 0), (7, 0)])
@pytest.mark.parametrize("D,I", [(128, 128), (512, 128), (640, 384), (1152, 256)])
@pytest.mark.parametrize("rows", [[2, 1], [15, 16, 17], [63, 64, 65], [128, 129, 193]])
def test_tile_edges(be, oracle, fmt, gs, D, I, rows):
    rng = np.random.default_rng(D + I + sum(rows) + fmt)
    experts = [(rand_qt(rng, I, D, fmt, gs, half=True), rand_qt(rng, I, D, fmt, gs, half=True),
                rand_qt(rng, D, I, fmt, gs, half=True)) for _ in rows]
    total = sum(rows)
    x = ((rng.random((total, D)) - 0.5) * 2).astype(np.float32)
    x[::3] = W.bf16_round(x[::3])                        # rows without lo terms among rows with them
    hs = [[upload_qt(be, t) for t in e] for e in experts]
    try:
        be.set_tensor_core(2)
        ok, y = be.run_expert_group([h[0] for h in hs], [h[1] for h in hs], [h[2] for h in hs], rows, x, D)
    finally:
        be.set_tensor_core(1)
        for h in hs:
            for t in h:
                be.tensor_free(t)
    assert ok and be.kernel_status(0) == 0
    off = 0
    for e, r in zip(experts, rows):
        assert max_rel_err(y[off:off + r], oracle.expert_mlp(x[off:off + r], *e)) <= 1e-3
        off += r


@pytest.mark.parametrize("E,K,M", [(5, 5, 9), (64, 8, 9), (33, 3, 200), (3, 2, 700)])
def test_device_plan(be, E, K, M):
    """The plan kernel's grouping against the multi-kernel path on the same routing."""
    cfg = dict(D=256, I=128, E=E, K=K, gating=0, norm_topk=0, shared=True, fmt=4, gs=32)
    L = W.HostLayerWeights(cfg, 3)
    up = lambda t: upload_qt(be, t)
    g, u, d = ([up(t) for t in side] for side in (L.gate, L.up, L.down))
    sh = tuple(up(t) for t in L.shared)
    lay = MoeLayer(be, 256, 128, E, K, g, u, d, 0, 0, shared=sh, max_rows=M)
    x, lg = W.activations(M, 256, 1), W.router_logits(M, E, 2, zipf=1.1)
    outs = []
    try:
        for mode in (2, 0):
            be.set_tensor_core(mode)
            outs.append(lay(x, lg))
    finally:
        be.set_tensor_core(1)
        lay.free()
        for t in g + u + d + list(sh):
            be.tensor_free(t)
    assert np.array_equal(outs[0][1], outs[1][1])
    assert max_rel_err(outs[0][0], outs[1][0]) <= 1e-3 and be.kernel_status(0) == 0


@pytest.mark.parametrize("gu,dn,line", [((2, 0), (2, 0), 2.5), ((7, 0), (7, 0), 3), ((2, 0), (7, 0), 3), ((4, 32), (4, 32), 8),
                                        ((2, 0), (4, 32), 4.5), ((7, 0), (4, 64), 4.5), ((4, 32), (2, 0), 5.5), ((4, 128), (7, 0), 5.5)])
def test_rule_looks_at_both_phases(be, oracle, gu, dn, line):
    """On both sides of the line between the streaming kernel (five launches) and the tensor cores (four), for gate and
    up in one format and down in another."""
    import ctypes as C
    D, I, n = 256, 128, 4
    rng = np.random.default_rng(int(line * 10) + gu[0])
    ex = [(rand_qt(rng, I, D, *gu, half=True), rand_qt(rng, I, D, *gu, half=True), rand_qt(rng, D, I, *dn, half=True)) for _ in range(n)]
    hs = [[upload_qt(be, t) for t in e] for e in ex]
    be.set_timing(1)
    try:
        for total, want in ((int(line * n) - 1, 5), (int(line * n), 4)):
            if total <= 8:                                                # (the fused kernel takes these when all formats agree)
                be.set_fused_decode(0)
            rows = [1, total - 4, 2, 1]
            x = ((rng.random((total, D)) - 0.5) * 2).astype(np.float32)
            ok, y = be.run_expert_group([h[0] for h in hs], [h[1] for h in hs], [h[2] for h in hs], rows, x, D)
            ms, launches = C.c_float(), C.c_int()
            assert ok and be.last_timing(0, C.byref(ms), C.byref(launches)) and launches.value == want, total
            off = 0
            for e, r in zip(ex, rows):
                assert max_rel_err(y[off:off + r], oracle.expert_mlp(x[off:off + r], *e)) <= 1e-3
                off += r
    finally:
        be.set_timing(0)
        be.set_fused_decode(3)
        for h in hs:
            for t in h:
                be.tensor_free(t)


@pytest.mark.parametrize("fmt,gs", [(4, 32), (2, 0), (7, 0)])
@pytest.mark.parametrize("nrows", [3, 37, 64])
def test_task_end_over_the_gate_range(be, oracle, fmt, gs, nrows):
    """The SwiGLU's division away from ordinary gates: denominators from 1 to overflow, gates that are zero or tiny. Row by
    row against the oracle (f32 on both sides: 1e-3 with the row's own noise floor)."""
    D, I = 640, 256
    rng = np.random.default_rng(fmt + nrows)
    ex = (rand_qt(rng, I, D, fmt, gs, half=True), rand_qt(rng, I, D, fmt, gs, half=True), rand_qt(rng, D, I, fmt, gs, half=True))
    scale = np.array([1, 40, 1e3, 1e6, 0, 1e-9, 1e-12], np.float32)[np.arange(nrows) % 7]
    x = (((rng.random((nrows, D)) - 0.5) * 2) * scale[:, None]).astype(np.float32)
    hs = [upload_qt(be, t) for t in ex]
    try:
        be.set_tensor_core(2)
        ok, y = be.run_expert_group(hs[:1], hs[1:2], hs[2:], [nrows], x, D)
    finally:
        be.set_tensor_core(1)
        for t in hs:
            be.tensor_free(t)
    assert ok and be.kernel_status(0) == 0
    want = oracle.expert_mlp(x, *ex)
    for s in range(nrows):
        assert np.all(np.isfinite(y[s])) and max_rel_err(y[s], want[s]) <= 1e-3, (s, float(scale[s]))


@pytest.mark.parametrize("E,K,M,topp", [(300, 8, 40, 0.0), (300, 8, 40, 0.6), (1, 1, 33, 0.0), (64, 16, 130, 0.4), (1000, 2, 700, 0.0)])
def test_segment_lists_of_the_streaming_path(be, E, K, M, topp):
    """The streaming path's lists (union, rows of an expert, passes) against the tensor-core plan, which is built by other code:
    more experts than warps, dead entries behind a top-p cut, one expert with all rows, more passes than experts."""
    cfg = dict(D=128, I=128, E=E, K=K, gating=1, norm_topk=1, shared=True, fmt=7, gs=0)
    L = W.HostLayerWeights(cfg, 3)
    up = lambda t: upload_qt(be, t)
    g, u, d = ([up(t) for t in side] for side in (L.gate, L.up, L.down))
    sh = tuple(up(t) for t in L.shared)
    lay = MoeLayer(be, 128, 128, E, K, g, u, d, 1, 1, 2.5, topp, router_bias=L.router_bias, shared=sh, max_rows=M)
    x, lg = W.activations(M, 128, 1), W.router_logits(M, E, 2, zipf=1.1 if E > 1 else 0.0)
    outs = []
    try:
        for mode in (2, 0):
            be.set_tensor_core(mode)
            outs.append(lay(x, lg))
    finally:
        be.set_tensor_core(1)
        lay.free()
        for t in g + u + d + list(sh):
            be.tensor_free(t)
    assert np.array_equal(outs[0][1], outs[1][1]) and np.array_equal(outs[0][3], outs[1][3])
    assert max_rel_err(outs[0][0], outs[1][0]) <= 1e-3 and be.kernel_status(0) == 0


@pytest.mark.parametrize("fmt,gs,D,I", [(7, 0, 6144, 2048), (4, 32, 6144, 2048), (2, 0, 6144, 2048), (4, 32, 5760, 1920)])
def test_repeated_calls_agree(be, fmt, gs, D, I):
    """The same call again and again while every stage of the kernel's rings is in turn the slowest one (passes of 1 to 64 rows),
    also with contractions that end inside a stage of two blocks: bit for bit the same rows, and those of the streaming kernel. A slot that is
    filled again before its last word was read shows here as a few wrong features of one pass, in one call of thirty. Such a
    feature is off by about the results' root mean square; the two kernels differ by 3e-6 of it (2-norm), by the seven deviations of the
    largest of 1e8 values 2e-5."""
    import torch
    n = 256
    rng = np.random.default_rng(fmt)
    ex = [(rand_qt(rng, I, D, fmt, gs, half=True), rand_qt(rng, I, D, fmt, gs, half=True), rand_qt(rng, D, I, fmt, gs, half=True))
          for _ in range(2)]
    lg = W.router_logits(2048, n, 5, zipf=1.1)                     # rows per expert: from 1800 down to one
    rows = np.maximum(1, np.bincount(np.argsort(-lg, axis=1)[:, :8].ravel(), minlength=n)).astype(np.int32)
    x = torch.randn((int(rows.sum()), D), generator=torch.Generator(device="cuda").manual_seed(1), device="cuda").bfloat16().float()
    ys = [torch.empty_like(x) for _ in range(2)]
    hs = [[upload_qt(be, t) for t in ex[e % 2]] for e in range(n)]
    side = [be.handle_array([h[m] for h in hs]) for m in range(3)]
    run = lambda y: be.expert_group_dev(*side, rows.ctypes.data_as(C.POINTER(C.c_int)), n, y.data_ptr(), x.data_ptr())
    torch.cuda.synchronize()
    try:
        be.set_tensor_core(0)
        ok = run(ys[1])
        be.set_tensor_core(2)
        ok, bad = run(ys[0]) and ok, 0
        assert be.kernel_status(0) == 0
        rms = ys[1].double().square().mean().sqrt().item()
        off = (ys[0] - ys[1]).abs().max().item()
        assert 0.0 < off <= 1e-4 * rms, off / rms
        for _ in range(80):
            ok = run(ys[1]) and ok
            assert be.kernel_status(0) == 0
            bad += not torch.equal(*ys)
    finally:
        be.set_tensor_core(1)
        for h in hs:
            for t in h:
                be.tensor_free(t)
    assert ok and be.kernel_status(0) == 0 and bad == 0


@pytest.mark.parametrize("gu,dn,D,I,line", [((2, 0), (2, 0), 1024, 1024, 3), ((7, 0), (7, 0), 1024, 1024, 4), ((4, 32), (4, 32), 1024, 1024, 8),
                                             ((2, 0), (4, 64), 1024, 1024, 4.5), ((4, 32), (7, 0), 1024, 1024, 5.5), ((4, 32), (4, 32), 512, 256, 8),
                                             ((7, 0), (7, 0), 512, 256, 4.5)])
def test_rule_of_layers(be, gu, dn, D, I, line):
    """Layer calls on both sides of their line: the default is bit for bit the streaming kernel's result below it and the
    tensor cores' from it on (the two add in different orders, so their results differ in some bits), and the two agree to 1e-3."""
    E, K = 16, 4
    rng = np.random.default_rng(int(line * 10) + D)
    ex = [(rand_qt(rng, I, D, *gu, half=True), rand_qt(rng, I, D, *gu, half=True), rand_qt(rng, D, I, *dn, half=True)) for _ in range(E)]
    hs = [[upload_qt(be, t) for t in e] for e in ex]
    at = int(line * E / K)
    lay = MoeLayer(be, D, I, E, K, *([h[m] for h in hs] for m in range(3)), 0, 0, max_rows=at)
    try:
        for M, tc in ((at - 1, False), (at, True)):
            be.set_fused_decode(0)
            x, lg = rng.standard_normal((M, D), dtype=np.float32), W.router_logits(M, E, 2)
            out = {}
            for mode in (0, 2, 1):
                be.set_tensor_core(mode)
                out[mode] = lay(x, lg)[0].copy()
            assert max_rel_err(out[0], out[2]) <= 1e-3 and be.kernel_status(0) == 0
            if M >= 9:                                                 # (fewer rows never take the tensor cores)
                assert not np.array_equal(out[0], out[2])
                assert np.array_equal(out[1], out[2] if tc else out[0]), (M, tc)
    finally:
        be.set_tensor_core(1)
        be.set_fused_decode(3)
        lay.free()
        for h in hs:
            for t in h:
                be.tensor_free(t)


@pytest.mark.parametrize("gu,dn,line", [((2, 0), (2, 0), 3), ((7, 0), (7, 0), 3.5), ((4, 32), (4, 32), 8), ((2, 0), (4, 32), 5.5), ((4, 32), (2, 0), 6)])
def test_rule_of_larger_groups(be, gu, dn, line):
    """The line of grouped calls for experts of a million weights and more, by the number of launches (five below, four from it on)."""
    D, I, n = 1024, 1024, 4
    rng = np.random.default_rng(int(line * 10) + gu[0])
    ex = (rand_qt(rng, I, D, *gu, half=True), rand_qt(rng, I, D, *gu, half=True), rand_qt(rng, D, I, *dn, half=True))
    hs = [[upload_qt(be, t) for t in ex] for _ in range(n)]
    be.set_timing(1)
    be.set_fused_decode(0)
    try:
        for total, want in ((int(line * n) - 1, 5), (int(line * n), 4)):
            x = rng.standard_normal((total, D), dtype=np.float32)
            ok, y = be.run_expert_group(*([h[m] for h in hs] for m in range(3)), [1, total - 4, 2, 1], x, D)
            ms, launches = C.c_float(), C.c_int()
            assert ok and be.last_timing(0, C.byref(ms), C.byref(launches)) and launches.value == want, total
    finally:
        be.set_timing(0)
        be.set_fused_decode(3)
        for h in hs:
            for t in h:
                be.tensor_free(t)
    assert be.kernel_status(0) == 0


@pytest.mark.parametrize("gu,dn,line", [((2, 0), (2, 0), 6), ((7, 0), (7, 0), 6), ((4, 32), (4, 32), 8), ((2, 0), (4, 32), 6), ((4, 32), (2, 0), 6)])
@pytest.mark.parametrize("D,I", [(512, 256), (1024, 512), (1024, 896)])
def test_rule_of_small_groups(be, gu, dn, line, D, I):
    """The line of grouped calls for experts of 2^17 weights up to a million, by the number of launches (five below, four from it on)."""
    n = 4
    rng = np.random.default_rng(D + I + gu[0])
    ex = (rand_qt(rng, I, D, *gu, half=True), rand_qt(rng, I, D, *gu, half=True), rand_qt(rng, D, I, *dn, half=True))
    hs = [[upload_qt(be, t) for t in ex] for _ in range(n)]
    be.set_timing(1)
    be.set_fused_decode(0)
    try:
        for total, want in ((line * n - 1, 5), (line * n, 4)):
            x = rng.standard_normal((total, D), dtype=np.float32)
            ok, y = be.run_expert_group(*([h[m] for h in hs] for m in range(3)), [1, total - 4, 2, 1], x, D)
            ms, launches = C.c_float(), C.c_int()
            assert ok and be.last_timing(0, C.byref(ms), C.byref(launches)) and launches.value == want, total
    finally:
        be.set_timing(0)
        be.set_fused_decode(3)
        for h in hs:
            for t in h:
                be.tensor_free(t)
    assert be.kernel_status(0) == 0


@pytest.mark.parametrize("fmt,gs,line", [(2, 0, 3), (7, 0, 4), (4, 32, 8)])
def test_a_layer_says_which_kernel_it_takes(be, fmt, gs, line):
    """coli_cuda_moe_layer_tensor_core against the results of the call itself, around the line and by the setting."""
    D, I, E, K = 1024, 1024, 16, 4
    rng = np.random.default_rng(fmt)
    ex = [upload_qt(be, rand_qt(rng, *s, fmt, gs, half=True)) for s in ((I, D), (I, D), (D, I))]
    at = line * E // K
    lay = MoeLayer(be, D, I, E, K, *([h] * E for h in ex), 0, 0, max_rows=at)
    takes = lambda m: be.moe_layer_tensor_core(lay.handle, m)
    try:
        for M in (at - 1, at):
            x, lg = rng.standard_normal((M, D), dtype=np.float32), W.router_logits(M, E, 2)
            out, says = {}, {}
            for mode in (0, 2, 1):
                be.set_tensor_core(mode)
                out[mode], says[mode] = lay(x, lg)[0].copy(), takes(M)
            assert (says[0], says[2], says[1]) == (0, 1, int(M == at))
            assert np.array_equal(out[1], out[2 if says[1] else 0]) and not np.array_equal(out[0], out[2])
        assert (takes(8), takes(0), takes(at + 1), be.moe_layer_tensor_core(None, 9)) == (0, 0, 0, 0)
    finally:
        be.set_tensor_core(1)
        lay.free()
        for h in ex:
            be.tensor_free(h)
    assert be.kernel_status(0) == 0
