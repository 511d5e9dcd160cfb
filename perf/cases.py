"""Performance cases of the MoE expert-FFN backend: what a user's program has it do.

Every case goes through the public binding (`colibri_b200.backend`, `.stack`, `.ep`) with a
model that is loaded once per process, as an engine loads its weights, and inputs that are
made from a seed. Weights are N(0, 0.02) quantised by the reference converters' rules,
activations N(0, 1) rounded to bf16, router logits N(0, 1): the distributions of the
configurations in `colibri_b200.workloads`. A model holds a few distinct expert matrices on
the host and uploads each of them several times, so every expert has memory of its own on
the GPU while making a model stays quick.

Kinds of case:
  layer   whole MoE layers (route, union, expert FFN, combine) on device or host buffers
  stack   a batched decode step through rmsnorm, MoE layers, the f32 head and the argmax
  ep      one expert-parallel layer of a rank's rows (plan, pack, expert FFN, combine)
  group   the engine's drop-in call: packed rows of some experts in host buffers
  row     the engine's device-resident decode row: rmsnorm, router, resident expert group
  linear  a dense projection with host buffers, in each storage format
  swap    an expert replaced in its device slot by one from host memory, then used once
"""
import collections
import ctypes
import math
import random

import numpy as np
import torch

from colibri_b200.backend import Backend, MoeLayer
from colibri_b200.ep import CudaEpLayer, ExpertMap
from colibri_b200.stack import MoeStack

DEV = 0
SCALE = 2.5           # routed_scale of the sigmoid-gated models
MODEL_BYTES = 60e9    # models kept at a time, oldest out first

OLMOE = dict(D=2048, I=1024, E=64, K=8, gating=0, norm=0, shared=False, fmt=4, gs=32)
DSV3 = dict(D=7168, I=2048, E=256, K=8, gating=1, norm=1, shared=True, fmt=7, gs=0)
DSV3_INT4 = dict(DSV3, fmt=4, gs=32)
GLM = dict(D=6144, I=2048, E=256, K=8, gating=1, norm=1, shared=True, fmt=7, gs=0)


def listed():
    return [
        # One token through the 16 MoE layers of OLMoE-1B-7B, everything resident on the GPU.
        dict(OLMOE, name="olmoe_decode_m1", kind="layer", layers=16, M=1, host=False),
        # Four sequences decoded together by an engine that keeps its activations on the host.
        dict(OLMOE, name="olmoe_decode_host_m4", kind="layer", layers=16, M=4, host=True),
        # A prompt of 251 tokens (an odd count) through the same 16 layers.
        dict(OLMOE, name="olmoe_prefill_m251", kind="layer", layers=16, M=251, host=False),
        # One token through one DeepSeek-V3-sized layer with MXFP4 experts and a shared expert.
        dict(DSV3, name="dsv3_decode_m1", kind="layer", layers=1, M=1, host=False),
        # A serving batch of 64 sequences through that layer: most experts get a row or two.
        dict(DSV3, name="dsv3_batch_m64", kind="layer", layers=1, M=64, host=False),
        # A prompt of 512 tokens through that layer: sixteen rows per expert on average.
        dict(DSV3, name="dsv3_prefill_m512", kind="layer", layers=1, M=512, host=False),
        # Eight candidate tokens verified in one step: four int4 layers, router weights on the
        # device, the f32 head over 129280 entries, logits and picks back on the host.
        dict(DSV3_INT4, name="dsv3_stack_k8", kind="stack", layers=4, M=8, vocab=129280),
        # 2048 rows with a skewed (Zipf) expert load through a GLM-sized expert-parallel layer.
        dict(GLM, name="glm_ep_m2048", kind="ep", M=2048),
        # The engine's grouped call for a small batch: 24 experts share 61 rows unevenly.
        dict(name="engine_group_r61", kind="group", D=6144, I=2048, fmt=4, gs=64, count=24, rows=61),
        # The engine's resident pipeline, one decode row through one layer with per-row int4 experts.
        dict(GLM, name="resident_row", kind="row", fmt=2, gs=0),
        # An attention-sized projection of an FP8 checkpoint for twelve rows.
        dict(name="linear_fp8_s12", kind="linear", fmt=8, gs=0, I=6144, O=8192, S=12),
        # The engine's expert cache takes in an int4 expert (25 MB) and uses it for one row.
        dict(name="expert_swap", kind="swap", D=7168, I=2048, fmt=4, gs=32, S=1),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    """One more case of the same kinds: the layer shapes of the configurations and generic
    ones, row counts over their whole range on a log scale, every storage format."""
    kind = rng.choice(["layer"] * 6 + ["stack", "ep", "group", "group", "row", "linear", "linear", "swap"])
    int4 = lambda: rng.choice([(4, 32), (4, 64), (4, 128), (2, 0), (7, 0)])
    if kind == "layer":
        shape = rng.choice(["olmoe", "dsv3", "other", "other"])
        if shape == "olmoe":
            fmt, gs = int4()
            c = dict(OLMOE, fmt=fmt, gs=gs, layers=rng.choice([4, 8, 16]), M=_log_int(rng, 1, 300))
        elif shape == "dsv3":
            c = dict(DSV3, E=rng.choice([128, 160, 192, 256]), layers=1, M=_log_int(rng, 1, 512))
        else:
            fmt, gs = int4()
            gating = rng.randint(0, 1)
            c = dict(D=128 * rng.randint(8, 40), I=128 * rng.randint(4, 16), E=rng.randint(8, 96), K=rng.randint(2, 8),
                     gating=gating, norm=gating, shared=bool(rng.randint(0, 1)), fmt=fmt, gs=gs, layers=4,
                     M=_log_int(rng, 1, 400))
        return dict(c, kind="layer", host=rng.random() < 0.3)
    if kind == "stack":
        return dict(D=128 * rng.randint(16, 32), I=1024, E=rng.choice([64, 96, 128]), K=8, gating=1, norm=1, shared=True,
                    fmt=4, gs=32, kind="stack", layers=rng.randint(2, 4), M=rng.randint(2, 8),
                    vocab=rng.randint(30000, 60000))
    if kind == "ep":
        return dict(GLM, D=128 * rng.randint(16, 48), E=rng.choice([64, 96, 128]), kind="ep", M=_log_int(rng, 100, 2048))
    if kind == "group":
        fmt, gs = int4()
        count = rng.randint(2, 48)
        return dict(kind="group", D=128 * rng.randint(16, 48), I=128 * rng.randint(8, 16), fmt=fmt, gs=gs, count=count,
                    rows=count + _log_int(rng, 1, 400))
    if kind == "row":
        fmt, gs = int4()
        return dict(GLM, D=128 * rng.randint(16, 48), E=rng.choice([64, 96, 128]), K=rng.randint(4, 8), kind="row",
                    fmt=fmt, gs=gs)
    if kind == "linear":
        fmt, gs = rng.choice([(0, 0), (1, 0), (1, 0), (2, 0), (3, 0), (4, 64), (4, 128), (7, 0), (8, 0), (8, 0)])
        return dict(kind="linear", fmt=fmt, gs=gs, I=128 * rng.randint(8, 56) + rng.choice([0, 0, 0, 16, 6]),
                    O=rng.choice([128 * rng.randint(4, 96), rng.randint(500, 12000)]), S=_log_int(rng, 1, 48))
    fmt, gs = int4()
    return dict(kind="swap", D=128 * rng.randint(16, 56), I=128 * rng.randint(8, 16), fmt=fmt, gs=gs, S=rng.randint(1, 4))


# ---- weights -------------------------------------------------------------------------------
def quantised(w, fmt, gs):
    """f32 [n, O, I] on the GPU -> (codes [n, O, bytes per row], scales [n, ...]) on the host, in
    the container layout that coli_cuda_tensor_upload takes."""
    n, O, I = w.shape
    pad = lambda t, m: torch.nn.functional.pad(t, (0, -t.shape[-1] % m))
    host = lambda t: t.contiguous().cpu().numpy()
    if fmt == 0:
        return host(w), None
    if fmt in (1, 2, 3):
        top = {1: 127.0, 2: 7.0, 3: 1.5}[fmt]
        s = w.abs().amax(-1, keepdim=True).clamp(min=1e-8) / top
        lo, hi = {1: (-127, 127), 2: (-8, 7), 3: (-2, 1)}[fmt]
        q = (w / s).round().clamp(lo, hi).to(torch.int32)
        s = host(s[..., 0].float())
        if fmt == 1:
            return host(q.to(torch.int8)).view(np.uint8), s
        q = q - lo
        if fmt == 2:
            q = pad(q, 2)
            return host((q[..., 0::2] | q[..., 1::2] << 4).to(torch.uint8)), s
        q = pad(q, 4)
        return host((q[..., 0::4] | q[..., 1::4] << 2 | q[..., 2::4] << 4 | q[..., 3::4] << 6).to(torch.uint8)), s
    if fmt == 8:
        wp = torch.nn.functional.pad(w, (0, -I % 128, 0, -O % 128))
        b = wp.reshape(n, wp.shape[1] // 128, 128, wp.shape[2] // 128, 128)
        s = b.abs().amax((2, 4), keepdim=True).clamp(min=1e-8) / 448.0
        q = (b / s).reshape(wp.shape)[:, :O, :I].to(torch.float8_e4m3fn).view(torch.uint8)
        return host(q), host(s[:, :, 0, :, 0].float())
    group = gs if fmt == 4 else 32
    wp = pad(w, group)
    g = wp.reshape(n, O, wp.shape[-1] // group, group)
    top = g.abs().amax(-1, keepdim=True)
    if fmt == 4:
        s = (top / 7.0).clamp(min=1e-6).half().float()     # fp16-valued scales
        q = ((g / s).round().clamp(-8, 7) + 8).to(torch.int32)
        s = host(s[..., 0])
    else:
        e = torch.where(top > 0, torch.ceil(torch.log2(top.double() / 6.0)), torch.full_like(top, -127.0).double()).clamp(-127, 127)
        v = (g / torch.exp2(e).float()).clamp(-6, 6)
        steps = torch.tensor([0.25, 0.75, 1.25, 1.75, 2.5, 3.5, 5.0], device=w.device)     # midpoints of 0 .5 1 1.5 2 3 4 6
        q = torch.bucketize(v.abs(), steps).to(torch.int32) | (v < 0).to(torch.int32) << 3
        s = host((e[..., 0] + 127).to(torch.uint8))
    q = pad(q.reshape(wp.shape)[..., :I], 2)
    return host((q[..., 0::2] | q[..., 1::2] << 4).to(torch.uint8)), s


def random_matrices(n, O, I, fmt, gs, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return quantised(torch.randn((n, O, I), generator=g, device="cuda") * 0.02, fmt, gs)


_backend = None


def backend():
    global _backend
    if _backend is None:
        _backend = Backend()
        if _backend.init_devices((DEV,)) != 1:
            raise RuntimeError("coli_cuda_init failed")
        table = torch.arange(256, dtype=torch.uint8).view(torch.float8_e4m3fn).float().numpy()
        _backend.fp8_set_lut(table.ctypes.data)
    return _backend


class Tensors:
    """Resident tensors, freed with the object."""

    def __init__(self):
        self.handles = []

    def upload(self, w, s, fmt, I, O, gs):
        h = backend().upload(w, s, fmt, I, O, DEV, gs)
        if not h:
            raise RuntimeError("tensor upload refused")
        self.handles.append(h)
        return h

    def experts(self, count, D, I, fmt, gs, seed, distinct=4):
        """-> (gates, ups, downs): `count` handles each."""
        out = []
        for m, (O, K) in enumerate(((I, D), (I, D), (D, I))):
            w, s = random_matrices(min(distinct, count), O, K, fmt, gs, seed * 8 + m)
            out.append([self.upload(w[e % len(w)], s[e % len(w)], fmt, K, O, gs) for e in range(count)])
        return out

    def __del__(self):
        for h in self.handles:
            _backend.tensor_free(h)


# ---- models, loaded once -------------------------------------------------------------------
_models = collections.OrderedDict()


def model(key, nbytes, make):
    """The model of `key`, made on first use; the oldest ones go when MODEL_BYTES are exceeded."""
    if key not in _models:
        while _models and sum(b for _, b in _models.values()) + nbytes > MODEL_BYTES:
            _models.popitem(last=False)
        _models[key] = (make(), nbytes)
    _models.move_to_end(key)
    return _models[key][0]


def bits_per_weight(fmt, gs):
    return {0: 32, 1: 8, 2: 4, 3: 2, 4: 4 + 16 / max(gs, 1), 7: 4.25, 8: 8}[fmt]


def expert_bytes(c):
    return 3 * c["D"] * c["I"] * bits_per_weight(c["fmt"], c["gs"]) / 8


class Layers:
    def __init__(self, c, distinct_layers, max_rows, router):
        D, I, E = c["D"], c["I"], c["E"]
        self.t, self.layers = Tensors(), []
        for li in range(distinct_layers):
            g, u, d = self.t.experts(E, D, I, c["fmt"], c["gs"], 100 + li)
            shared = tuple(h[0] for h in self.t.experts(1, D, I, c["fmt"], c["gs"], 500 + li)) if c["shared"] else None
            rng = np.random.default_rng(7 + li)
            bias = rng.standard_normal(E, dtype=np.float32) * np.float32(0.01) if c["gating"] else None
            rw = rng.standard_normal((E, D), dtype=np.float32) * np.float32(0.02) if router else None
            self.layers.append(MoeLayer(backend(), D, I, E, c["K"], g, u, d, c["gating"], c["norm"],
                                        SCALE if c["gating"] else 1.0, 0.0, router_w=rw, router_bias=bias, shared=shared,
                                        max_rows=max_rows))

    def __del__(self):
        for lay in self.layers:
            lay.free()


class Stack:
    def __init__(self, c):
        D, V = c["D"], c["vocab"]
        self.body = Layers(c, min(2, c["layers"]), 8, True)
        self.t = Tensors()
        g = torch.Generator(device="cuda").manual_seed(3)
        self.head = np.empty((V, D), np.float32)              # tied: the embedding and the head
        for v in range(0, V, 16384):
            n = min(16384, V - v)
            self.head[v:v + n] = (torch.randn((n, D), generator=g, device="cuda") * 0.02).cpu().numpy()
        rng = np.random.default_rng(9)
        ln = [1 + 0.1 * rng.standard_normal(D, dtype=np.float32) for _ in range(c["layers"] + 1)]
        layers = [self.body.layers[i % len(self.body.layers)] for i in range(c["layers"])]
        self.stack = MoeStack(backend(), DEV, D, V, self.head, layers, ln[:-1], ln[-1],
                              self.t.upload(self.head, None, 0, D, V, 0), 1e-6, 8)

    def __del__(self):
        self.stack.free()


class Ep:
    def __init__(self, c):
        self.t = Tensors()
        g, u, d = self.t.experts(c["E"], c["D"], c["I"], c["fmt"], c["gs"], 21)
        sh = tuple(h[0] for h in self.t.experts(1, c["D"], c["I"], c["fmt"], c["gs"], 22))
        bias = torch.randn(c["E"], generator=torch.Generator().manual_seed(23)).cuda() * 0.01
        cfg = dict(D=c["D"], I=c["I"], E=c["E"], K=c["K"], gating=c["gating"], norm_topk=c["norm"])
        self.layer = CudaEpLayer(backend(), DEV, cfg, ExpertMap(c["E"], 1), 0, g, u, d, sh, bias, SCALE, max_rows=2048)


class Row:
    def __init__(self, c):
        D, E = c["D"], c["E"]
        self.t = Tensors()
        self.g, self.u, self.d = self.t.experts(E, D, c["I"], c["fmt"], c["gs"], 31)
        self.sg, self.su, self.sd = (h[0] for h in self.t.experts(1, D, c["I"], c["fmt"], c["gs"], 32))
        g = torch.Generator(device="cuda").manual_seed(33)
        self.rw = torch.randn((E, D), generator=g, device="cuda") * 0.02
        self.rb = torch.randn(E, generator=g, device="cuda") * 0.01
        self.ln = 1 + 0.1 * torch.randn(D, generator=g, device="cuda")
        self.nrm, self.slot, self.acc, self.t1 = (torch.empty(D, device="cuda") for _ in range(4))
        self.hg, self.hu = (torch.empty(c["I"], device="cuda") for _ in range(2))


class Group:
    def __init__(self, c):
        self.t = Tensors()
        self.g, self.u, self.d = self.t.experts(c["count"], c["D"], c["I"], c["fmt"], c["gs"], 41)


class Linear:
    def __init__(self, c):
        self.t = Tensors()
        w, s = random_matrices(1, c["O"], c["I"], c["fmt"], c["gs"], 51)
        self.h = self.t.upload(w[0], None if s is None else s[0], c["fmt"], c["I"], c["O"], c["gs"])


# ---- inputs --------------------------------------------------------------------------------
def activations(rows, D, gen):
    return torch.randn((rows, D), generator=gen, device="cuda").bfloat16().float()


def key_of(c, *names):
    return (c["kind"],) + tuple(c[n] for n in names)


MOE_KEY = ("D", "I", "E", "K", "gating", "norm", "shared", "fmt", "gs")


def group_rows(c):
    """Rows per expert of a grouped call: one each, the rest spread with a skew (the same for every seed)."""
    rng = random.Random(c["rows"] * 1009 + c["count"])
    rows = [1] * c["count"]
    for _ in range(c["rows"] - c["count"]):
        rows[min(int(rng.expovariate(4.0 / c["count"])), c["count"] - 1)] += 1
    rng.shuffle(rows)
    return rows


def prepare(case, seed):
    c, be = case, backend()
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind = c["kind"]
    st = {"case": c, "kind": kind}
    if kind == "layer":
        M, D, E, L = c["M"], c["D"], c["E"], c["layers"]
        st["m"] = m = model(key_of(c, *MOE_KEY, "layers"), E * L * expert_bytes(c), lambda: Layers(c, L, 512, False))
        st["x"] = [activations(M, D, gen) for _ in m.layers]
        st["logits"] = [torch.randn((M, E), generator=gen, device="cuda") for _ in m.layers]
        if c["host"]:
            st["x"], st["logits"] = ([t.cpu().numpy() for t in st[k]] for k in ("x", "logits"))
            st["out"] = [np.empty((M, D), np.float32) for _ in m.layers]
        else:
            st["out"] = [torch.empty((M, D), device="cuda") for _ in m.layers]
    elif kind == "stack":
        nbytes = 2 * c["E"] * expert_bytes(c) + c["vocab"] * c["D"] * 4
        st["m"] = model(key_of(c, *MOE_KEY, "layers", "vocab"), nbytes, lambda: Stack(c))
        st["ids"] = np.random.default_rng(seed).integers(0, c["vocab"], c["M"])
    elif kind == "ep":
        st["m"] = model(key_of(c, *MOE_KEY), c["E"] * expert_bytes(c), lambda: Ep(c))
        st["x"] = activations(c["M"], c["D"], gen)
        rank = torch.randperm(c["E"], generator=torch.Generator().manual_seed(5)).cuda() + 1
        st["logits"] = torch.randn((c["M"], c["E"]), generator=gen, device="cuda") - 1.1 * rank.float().log()
    elif kind == "row":
        st["m"] = model(key_of(c, *MOE_KEY), c["E"] * expert_bytes(c), lambda: Row(c))
        st["x"] = activations(1, c["D"], gen)[0]
        st["h"] = torch.empty(c["D"], device="cuda")
        st["idx"], st["w"], st["keff"] = np.zeros(c["K"], np.int32), np.zeros(c["K"], np.float32), np.zeros(1, np.int32)
    elif kind == "group":
        st["m"] = m = model(key_of(c, "D", "I", "fmt", "gs", "count"), c["count"] * expert_bytes(c), lambda: Group(c))
        st["rows"] = np.array(group_rows(c), np.int32)
        st["args"] = [Backend.handle_array(h) for h in (m.g, m.u, m.d)]
        st["x"] = activations(c["rows"], c["D"], gen).cpu().numpy()
        st["y"] = np.empty_like(st["x"])
    elif kind == "linear":
        st["m"] = model(key_of(c, "I", "O", "fmt", "gs"), c["I"] * c["O"] * 4, lambda: Linear(c))
        st["x"] = activations(c["S"], c["I"], gen).cpu().numpy()
        st["y"] = np.empty((c["S"], c["O"]), np.float32)
    else:
        D, I, fmt, gs = c["D"], c["I"], c["fmt"], c["gs"]
        old = model(key_of(c, "D", "I", "fmt", "gs"), expert_bytes(c),
                    lambda: [random_matrices(1, O, K, fmt, gs, 61 + m) for m, (O, K) in enumerate(((I, D), (I, D), (D, I)))])
        st["t"] = t = Tensors()                              # the device slot, with the expert that leaves it
        st["slot"] = [t.upload(w[0], s[0], fmt, K, O, gs) for (w, s), (O, K) in zip(old, ((I, D), (I, D), (D, I)))]
        st["new"] = [random_matrices(1, O, K, fmt, gs, seed * 8 + m) for m, (O, K) in enumerate(((I, D), (I, D), (D, I)))]
        st["x"] = activations(c["S"], D, gen).cpu().numpy()
        st["y"] = np.empty((c["S"], D), np.float32)
    torch.cuda.synchronize()
    return st


# ---- one pass ------------------------------------------------------------------------------
def _ok(r, what):
    if not r:
        raise RuntimeError(what + " refused")


def run(st):
    c, be, kind = st["case"], backend(), st["kind"]
    if kind == "layer":
        m = st["m"]
        for lay, x, lg, out in zip(m.layers, st["x"], st["logits"], st["out"]):
            if c["host"]:
                lay.run_into(x, lg, out)
            else:
                _ok(be.moe_layer_dev(lay.handle, out.data_ptr(), x.data_ptr(), lg.data_ptr(), c["M"], None, None, None),
                    "coli_cuda_moe_layer_dev")
        return st["out"]
    if kind == "stack":
        return st["m"].stack.step(st["ids"])
    if kind == "ep":
        return st["m"].layer(st["x"], st["logits"])
    if kind == "row":
        return run_row(st)
    if kind == "group":
        rows = st["rows"].ctypes.data_as(ctypes.POINTER(ctypes.c_int))
        _ok(be.expert_group(*st["args"], rows, c["count"], st["y"].ctypes.data, st["x"].ctypes.data), "coli_cuda_expert_group")
        return st["y"]
    if kind == "linear":
        h = ctypes.c_void_p(st["m"].h)
        _ok(be.matmul(ctypes.byref(h), st["y"].ctypes.data, st["x"].ctypes.data, None, None, c["fmt"], c["S"], c["I"], c["O"],
                      DEV, c["gs"]), "coli_cuda_matmul")
        return st["y"]
    for h, (w, s) in zip(st["slot"], st["new"]):
        _ok(be.tensor_update(h, w.ctypes.data, s.ctypes.data), "coli_cuda_tensor_update")
    _ok(be.expert_mlp(*st["slot"], st["y"].ctypes.data, st["x"].ctypes.data, c["S"]), "coli_cuda_expert_mlp")
    return st["y"]


def run_row(st):
    """h = x + shared(norm(x)) + routed(norm(x)) for one row, as the engine's resident pipeline issues it."""
    c, be, m = st["case"], backend(), st["m"]
    D, I, K = c["D"], c["I"], c["K"]
    p = lambda t: t.data_ptr()
    _ok(be.pipe_copy2d(DEV, p(st["h"]), D, p(st["x"]), D, D, 1), "coli_cuda_pipe_copy2d")
    _ok(be.pipe_rmsnorm(DEV, p(m.nrm), p(st["h"]), p(m.ln), 1, D, 1e-6), "coli_cuda_pipe_rmsnorm")
    _ok(be.pipe_router(DEV, p(m.nrm), p(m.rw), p(m.rb), D, c["E"], K, 0.0, 1, SCALE, st["idx"].ctypes.data, st["w"].ctypes.data,
                       st["keff"].ctypes.data), "coli_cuda_pipe_router")
    pick = st["idx"][:int(st["keff"][0])]
    hs = [Backend.handle_array([side[e] for e in pick]) for side in (m.g, m.u, m.d)]
    _ok(be.expert_group_resident_issue(*hs, st["w"].ctypes.data, len(pick), DEV, p(m.nrm), p(m.slot)),
        "coli_cuda_expert_group_resident_issue")
    _ok(be.pipe_gemm(m.sg, p(m.hg), p(m.nrm), 1), "coli_cuda_pipe_gemm")
    _ok(be.pipe_gemm(m.su, p(m.hu), p(m.nrm), 1), "coli_cuda_pipe_gemm")
    _ok(be.pipe_silu_mul(DEV, p(m.hg), p(m.hu), I), "coli_cuda_pipe_silu_mul")
    _ok(be.pipe_gemm(m.sd, p(m.t1), p(m.hg), 1), "coli_cuda_pipe_gemm")
    _ok(be.pipe_add(DEV, p(st["h"]), p(m.t1), D), "coli_cuda_pipe_add")
    devs = (ctypes.c_int * 1)(DEV)
    _ok(be.expert_group_resident_take(DEV, devs, 1, p(m.slot), p(m.acc), D), "coli_cuda_expert_group_resident_take")
    _ok(be.pipe_add(DEV, p(st["h"]), p(m.acc), D), "coli_cuda_pipe_add")
    return st["h"], st["idx"], st["w"]


# ---- what a pass cannot do without -----------------------------------------------------------
def work(case):
    c, kind = case, case["kind"]
    if kind == "linear":
        w, S = c["I"] * c["O"], c["S"]
        return {"bytes": w * bits_per_weight(c["fmt"], c["gs"]) / 8 + 4 * S * (c["I"] + c["O"]), "flops": 2 * w * S}
    D, I = c["D"], c["I"]
    eb, ef = expert_bytes(c), 6 * D * I
    if kind == "group":
        return {"bytes": c["count"] * eb + 8 * c["rows"] * D, "flops": c["rows"] * ef}
    if kind == "swap":
        host = 3 * D * I // 2 + 3 * D * I // (c["gs"] or (32 if c["fmt"] == 7 else D)) * (1 if c["fmt"] == 7 else 4)
        return {"bytes": host + 2 * eb + 8 * c["S"] * D, "flops": c["S"] * ef}
    E, K, M = c["E"], c["K"], 1 if kind == "row" else c["M"]
    hit = E * (1 - (1 - K / E) ** M)                       # experts met by M rows, expected
    if kind == "ep":
        p = [1 / r ** 1.1 for r in range(1, E + 1)]
        hit = sum(1 - (1 - min(1.0, K * q / sum(p))) ** M for q in p)
    shared = 1 if c["shared"] else 0
    layer = {"bytes": (hit + shared) * eb + 4 * M * (2 * D + E), "flops": M * (K + shared) * ef}
    L = c.get("layers", 1)
    total = {k: v * L for k, v in layer.items()}
    if kind in ("stack", "row"):
        total["bytes"] += L * 4 * E * D
        total["flops"] += L * 2 * M * E * D
    if kind == "stack":
        total["bytes"] += 4 * c["vocab"] * (D + M)
        total["flops"] += 2 * M * D * c["vocab"]
    return total


def tolerance(case):
    """f32 activations, exactly decoded weights, f32 accumulation: another order of the sums
    shows about 1e-6 to 1e-5; routing indices and picks are whole numbers."""
    return {"rel": 2e-5, "max": 1e-3, "differ": 0.0}
