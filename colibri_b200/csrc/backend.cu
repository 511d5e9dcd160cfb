// libcoli_cuda_b200: the reference engine's GPU backend interface
// (c/backend_cuda.h) implemented for B200 (sm_100a), plus the additive fused
// MoE-layer entry points. See include/coli_cuda_b200.h for the contract of
// every exported function and the reference declaration it replaces.
//
// There is no CPU fallback anywhere in this file: a call either runs on the
// GPU or returns 0 with its outputs untouched.
#include "../../include/coli_cuda_b200.h"

#include <cstdio>
#include <climits>
#include <cstdlib>
#include <cstring>
#include <cmath>
#include <atomic>
#include <mutex>
#include <utility>
#include <vector>

#include "common.cuh"
#include "host_copy.h"
#include "gemv_stream.cuh"
#include "kernels_misc.cuh"
#include "router.cuh"
#include "moe_decode.cuh"
#include "gemm_tc.cuh"
#include "dense_mma.cuh"
#include "gemv_rows.cuh"
#include "ep_kernels.cuh"

// ---------------------------------------------------------------------------
// Context
// ---------------------------------------------------------------------------
struct Buf {
    void *p = nullptr;
    size_t cap = 0;
};

struct DeviceCtx {
    int device = -1;
    int sms = 0;
    cudaStream_t stream = nullptr;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr, ev_done = nullptr;
    size_t tensor_count = 0, tensor_bytes = 0, physical_bytes = 0;
    // workspaces (grow-only)
    Buf stage_w, stage_s;                     // upload staging
    Buf x, y, bq, bs, pg, pu, hq, hs, pd, segs1, segs2, ctl, gbuf, ubuf, misc;
    Buf pipe[27];
    Buf ep_ws, ep_x, ep_y;                    // expert-parallel layer: plan tables, permuted rows (streaming-kernel path)
    float *host_x = nullptr, *host_y = nullptr;   // pinned rows of the issued group: its alone from issue to the issue after its take
    size_t host_x_cap = 0, host_y_cap = 0;
    float *io_x = nullptr, *io_y = nullptr;       // pinned rows of the blocking host-buffer calls
    size_t io_x_cap = 0, io_y_cap = 0;
    bool tc = false;                          // the grouped GEMM was built as its register split needs it
    bool chain = false;                       // the last thing this call put on the stream is a kernel
    IoPieces io = {};                         // events of the pieces of a call's result
    uint32_t *check = nullptr;                // scale facts of an upload: 4 words on the device, then pinned
    uint32_t *check_host = nullptr;
    int group_pending = 0;                    // a group is issued and not taken; -1: and a wait has expired since
    int *status = nullptr;                    // pinned host int the kernels store into (kstat_set): sticky kernel status
    unsigned int *dec_sync = nullptr;         // fused decode kernel: the grid barriers' arrival counter
    unsigned long long *exp_tab_dev = nullptr; // global-memory copy of the 2^(i/32) table
    const float *e4m3_lut_dev = nullptr;       // device address of the fmt 8 decode table
    int sticky_status = 0;                    // last non-zero kernel status seen by the host
    float last_ms = 0.f;
    int last_launches = 0;
    unsigned long long total_launches = 0;   // kernels launched by earlier calls (see coli_cuda_launch_total)
    int have_timing = 0;
    std::vector<cudaEvent_t> *kev = nullptr;   // per-launch event pairs of the streaming GEMV
    int kev_used = 0;
    uint64_t g_calls = 0, g_experts = 0, g_rows = 0;
    double g_h2d = 0, g_kern = 0, g_d2h = 0;
};

static DeviceCtx g_ctx[COLI_CUDA_MAX_DEVICES];
static UploadRing g_ring[COLI_CUDA_MAX_DEVICES];     // pinned pieces of the device's transfers
static UploadRing *ring_of(const DeviceCtx *c) { return &g_ring[c - g_ctx]; }
// Held by a blocking call from its rows' way in to its result's way out: io_x and io_y are the device's, and layer calls of
// two threads, or one beside a projection, may meet there.
static std::mutex g_io_mu[COLI_CUDA_MAX_DEVICES];
static std::mutex &io_mutex(const DeviceCtx *c) { return g_io_mu[c - g_ctx]; }
static int g_nctx = 0;
static std::mutex g_mu;
static int g_timing = 0;
static std::atomic<long> g_gpu_calls{0};
static thread_local int g_cur_dev = -1;
static int g_fp8_lut_ready = 0;           // the fmt 8 decode table has been handed over (coli_cuda_fp8_set_lut)
static int g_fp8_standard = 0;            // ... and is E4M3's own, NaN codes included

static int cuda_ok(cudaError_t e, const char *what) {
    if (e == cudaSuccess) return 1;
    std::fprintf(stderr, "[CUDA] %s: %s\n", what, cudaGetErrorString(e));
    (void)cudaGetLastError();   // consume: a failed call must not poison the next launch check
    return 0;
}
static DeviceCtx *find_ctx(int device) {
    for (int i = 0; i < g_nctx; i++) if (g_ctx[i].device == device) return &g_ctx[i];
    return nullptr;
}
static int select_ctx(DeviceCtx *c) {
    if (!c) return 0;
    c->chain = false;
    if (g_cur_dev == c->device) return 1;
    if (!cuda_ok(cudaSetDevice(c->device), "select device")) return 0;
    g_cur_dev = c->device;
    return 1;
}
// Grow-only device buffer. Growing waits for the stream first: queued work may
// still read the old allocation.
static int reserve(DeviceCtx *c, Buf *b, size_t bytes) {
    if (bytes <= b->cap) return 1;
    if (b->p) { cudaStreamSynchronize(c->stream); cudaFree(b->p); b->p = nullptr; b->cap = 0; }
    size_t want = bytes + bytes / 4;
    if (!cuda_ok(cudaMalloc(&b->p, want), "workspace allocation")) {
        if (!cuda_ok(cudaMalloc(&b->p, bytes), "workspace allocation")) { b->p = nullptr; return 0; }
        want = bytes;
    }
    b->cap = want;
    return 1;
}
// Pinned buffer for the rows of calls with host buffers, grow-only up to IO_PINNED_MAX, by a quarter more than asked
// for: pinning 8 MB takes 8 ms and 32 MB 19, which a row count that rises step by step would pay at each step. -> 0: more
// than that, or the system has none to give; the caller moves its rows through the ring of pieces instead.
#define IO_PINNED_MAX ((size_t)32 << 20)
static int reserve_pinned(DeviceCtx *c, float **p, size_t *cap, size_t bytes) {
    if (bytes <= *cap) return 1;
    if (bytes > IO_PINNED_MAX) return 0;
    if (*p) { cudaStreamSynchronize(c->stream); cudaFreeHost(*p); }
    *p = nullptr; *cap = 0;
    size_t want = bytes + bytes / 4 < IO_PINNED_MAX ? bytes + bytes / 4 : IO_PINNED_MAX;
    if (cudaMallocHost((void **)p, want) != cudaSuccess) {
        (void)cudaGetLastError();
        want = bytes;
        if (!cuda_ok(cudaMallocHost((void **)p, want), "pinned allocation")) { *p = nullptr; return 0; }
    }
    *cap = want;
    return 1;
}
// Rows that kernels read or write 16 bytes at a time: a caller's pointer that does not lie on such a boundary is refused
// here, on the GPU it would be a misaligned access.
static int rows_aligned(const char *call, const void *x, const void *y = nullptr, uintptr_t to = 16) {
    if (((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(y)) & (to - 1)) == 0) return 1;
    std::fprintf(stderr, "[CUDA] %s: rows must start on %d-byte boundaries\n", call, (int)to);
    return 0;
}
// Test hook of the reference (c/backend_cuda.cu:1340-1348): COLI_GPU_FAIL_AFTER=N
// makes every compute entry point report failure after N successful calls.
static int fault_injected() {
    const char *fa = std::getenv("COLI_GPU_FAIL_AFTER");
    return fa && g_gpu_calls++ >= std::atol(fa);
}

static size_t row_bytes(int fmt, int I) {
    switch (fmt) {
    case 0: return (size_t)I * 4;
    case 1: case 8: return (size_t)I;
    case 2: case 4: case 7: return ((size_t)I + 1) / 2;
    case 3: return ((size_t)I + 3) / 4;
    }
    return 0;
}

// ---------------------------------------------------------------------------
// Lifecycle
// ---------------------------------------------------------------------------
static void fill_exp2_table(uint64_t *tab) { coli_expf_fill_table(tab); }

// Launch of a kernel of the call's chain. Behind another kernel of the same call (c->chain) it does not wait for
// that one's end on the queue: its CTAs are placed while the other drains and wait in pdl_enter, which saves 2 to 4 us
// per launch in a chain of short kernels. A call's first kernel, and one behind a copy, is launched in the ordinary
// way, and what a chained kernel reads of its predecessors it reads by ordinary loads (not ld.global.nc, whose
// lines may be older than the wait).
template <class... P, class... A>
static void launch_pdl(DeviceCtx *c, void (*kern)(P...), dim3 grid, unsigned block, size_t smem, A &&...args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid; cfg.blockDim = dim3(block); cfg.dynamicSmemBytes = smem; cfg.stream = c->stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at; cfg.numAttrs = c->chain ? 1 : 0;
    (void)cudaLaunchKernelEx(&cfg, kern, std::forward<A>(args)...);      // (an error stays for cudaGetLastError)
    c->chain = true;
}

template <typename K>
static void set_smem(K kern, int bytes) {
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
}

// launch geometry of the streaming GEMV per column-set count
template <int NC> struct GemvCfg { static constexpr int WARPS = NC <= 2 ? 16 : 8; static constexpr int NST = NC <= 2 ? 3 : 6; };

template <int MODE, int NC>
static void setup_one() {
    constexpr int W = GemvCfg<NC>::WARPS, N = GemvCfg<NC>::NST;
    set_smem(k_gemv_stream<MODE, NC, W, N>, W * N * (chunk_bytes_of(MODE) + 8));
}
template <int MODE>
static void setup_mode() { setup_one<MODE, 2>(); setup_one<MODE, 4>(); setup_one<MODE, 8>(); }

extern "C" void coli_cuda_shutdown(void);

static int decode_smem_bytes(int mode) {
    return DEC_WARPS * DEC_NST * chunk_bytes_of(mode) + DEC_BAR_BYTES + (int)((sizeof(DecShared) + 127) & ~127) +
           2 * DEC_PART_BYTES + dec_act_bytes(mode);
}

template <int MODE>
static void setup_decode() {
    set_smem(k_moe_decode<MODE, false>, decode_smem_bytes(MODE)); set_smem(k_moe_decode<MODE, true>, decode_smem_bytes(MODE));
    set_smem(k_gemv_rows<MODE, 1>, rows_smem(MODE, 1, ROWS_MAX_X) + 4096); set_smem(k_gemv_rows<MODE, 2>, rows_smem(MODE, 1, ROWS_MAX_X) + 4096);
}

// The grouped GEMM's warps share out the registers of its launch: their number must be what the split was made for. Where it is not,
// no tensor qualifies for that kernel and the streaming one takes its calls.
template <int MODE, int PHASE>
static int setup_tc_phase() {
    set_smem(k_expert_gemm_tc<MODE, PHASE>, tc_smem_total(MODE));
    cudaFuncAttributes fa{};
    if (!cuda_ok(cudaFuncGetAttributes(&fa, k_expert_gemm_tc<MODE, PHASE>), "kernel attributes")) return 0;
    if ((fa.numRegs + 7) / 8 * 8 == TC_REGS_LAUNCH) return 1;
    std::fprintf(stderr, "[CUDA] grouped GEMM built with %d registers a thread, %d needed: not used\n", fa.numRegs, TC_REGS_LAUNCH);
    return 0;
}
template <int MODE>
static int setup_tc() { return setup_tc_phase<MODE, 1>() && setup_tc_phase<MODE, 2>(); }

extern "C" int coli_cuda_init(const int *devices, int count) {
    if (!devices || count < 1 || count > COLI_CUDA_MAX_DEVICES) return 0;
    if (g_nctx) coli_cuda_shutdown();
    int ndev = 0;
    if (!cuda_ok(cudaGetDeviceCount(&ndev), "device count") || ndev < 1) return 0;
    for (int i = 0; i < count; i++) {
        if (devices[i] < 0 || devices[i] >= ndev) return 0;
        for (int j = 0; j < i; j++) if (devices[j] == devices[i]) return 0;
    }
    uint64_t tab[32];
    fill_exp2_table(tab);
    for (int i = 0; i < count; i++) {
        DeviceCtx *c = &g_ctx[i];
        *c = DeviceCtx();
        c->device = devices[i];
        if (!cuda_ok(cudaSetDevice(c->device), "init device")) { g_nctx = i; coli_cuda_shutdown(); return 0; }
        g_cur_dev = c->device;
        cudaDeviceProp prop{};
        if (!cuda_ok(cudaGetDeviceProperties(&prop, c->device), "device properties")) { g_nctx = i; coli_cuda_shutdown(); return 0; }
        if (prop.major < 10) {
            std::fprintf(stderr, "[CUDA] device %d is sm_%d%d: this backend is built for sm_100a only\n",
                         c->device, prop.major, prop.minor);
            g_nctx = i; coli_cuda_shutdown(); return 0;
        }
        c->sms = prop.multiProcessorCount;
        if (!cuda_ok(cudaStreamCreate(&c->stream), "stream") ||
            !cuda_ok(cudaEventCreate(&c->ev0), "event") || !cuda_ok(cudaEventCreate(&c->ev1), "event") ||
            !cuda_ok(cudaEventCreateWithFlags(&c->ev_done, cudaEventDisableTiming), "event") ||
            !cuda_ok(cudaHostAlloc((void **)&c->status, sizeof(int), cudaHostAllocMapped | cudaHostAllocPortable), "status") ||
            !cuda_ok(cudaMalloc((void **)&c->dec_sync, DEC_SYNC_WORDS * sizeof(unsigned int)), "grid barrier") ||
            !cuda_ok(cudaMemset(c->dec_sync, 0, DEC_SYNC_WORDS * sizeof(unsigned int)), "grid barrier") ||
            !cuda_ok(cudaMalloc((void **)&c->check, 4 * sizeof(uint32_t)), "scale check") ||
            !cuda_ok(cudaMallocHost((void **)&c->check_host, 4 * sizeof(uint32_t)), "scale check") ||
            !cuda_ok(cudaMalloc((void **)&c->exp_tab_dev, sizeof(tab)), "exp table") ||
            !cuda_ok(cudaMemcpy(c->exp_tab_dev, tab, sizeof(tab), cudaMemcpyHostToDevice), "exp table") ||
            !cuda_ok(cudaMemcpyToSymbol(c_exp2_tab, tab, sizeof(tab)), "exp table")) {
            g_nctx = i + 1; coli_cuda_shutdown(); return 0;
        }
        *c->status = 0;
        setup_mode<SC_ROW>(); setup_mode<SC_H16>(); setup_mode<SC_F32>(); setup_mode<SC_MX>();
        set_smem(k_router_logits<16, 256>, router_smem(16, 256)); set_smem(k_router_logits<64, 64>, router_smem(64, 64));
        set_smem(k_dense_gemv<0>, DENSE_GEMV_SMEM); set_smem(k_dense_gemv<8>, DENSE_GEMV_SMEM);
        setup_decode<SC_ROW>(); setup_decode<SC_H16>(); setup_decode<SC_F32>(); setup_decode<SC_MX>();
        c->tc = setup_tc<SC_ROW>() && setup_tc<SC_H16>() && setup_tc<SC_MX>();
        set_smem(k_tc_plan, 33 * ROUTE_MAX_E * (int)sizeof(int));
        set_smem(k_route_build, ROUTE_BUILD_INTS * ROUTE_MAX_E * (int)sizeof(int));
        if (!cuda_ok(cudaGetLastError(), "kernel attributes")) { g_nctx = i + 1; coli_cuda_shutdown(); return 0; }
    }
    g_nctx = count;
    return 1;
}

static void free_buf(Buf *b) { if (b->p) cudaFree(b->p); b->p = nullptr; b->cap = 0; }

extern "C" void coli_cuda_shutdown(void) {
    for (int i = 0; i < g_nctx; i++) {
        DeviceCtx *c = &g_ctx[i];
        if (c->device < 0) continue;
        if (cudaSetDevice(c->device) != cudaSuccess) { (void)cudaGetLastError(); continue; }
        cudaDeviceSynchronize();
        Buf *bufs[] = {&c->stage_w, &c->stage_s, &c->x, &c->y, &c->bq, &c->bs, &c->pg, &c->pu, &c->hq,
                       &c->hs, &c->pd, &c->segs1, &c->segs2, &c->ctl, &c->gbuf, &c->ubuf, &c->misc,
                       &c->ep_ws, &c->ep_x, &c->ep_y};
        for (Buf *b : bufs) free_buf(b);
        for (int s = 0; s < 27; s++) free_buf(&c->pipe[s]);
        if (c->host_x) cudaFreeHost(c->host_x);
        if (c->host_y) cudaFreeHost(c->host_y);
        if (c->io_x) cudaFreeHost(c->io_x);
        if (c->io_y) cudaFreeHost(c->io_y);
        if (c->status) cudaFreeHost(c->status);
        if (c->dec_sync) cudaFree(c->dec_sync);
        if (c->check) cudaFree(c->check);
        if (c->check_host) cudaFreeHost(c->check_host);
        upload_ring_free(ring_of(c));
        c->io.free();
        if (c->exp_tab_dev) cudaFree(c->exp_tab_dev);
        if (c->ev0) cudaEventDestroy(c->ev0);
        if (c->ev1) cudaEventDestroy(c->ev1);
        if (c->ev_done) cudaEventDestroy(c->ev_done);
        if (c->kev) { for (cudaEvent_t e : *c->kev) cudaEventDestroy(e); delete c->kev; c->kev = nullptr; }
        if (c->stream) cudaStreamDestroy(c->stream);
        (void)cudaGetLastError();
        *c = DeviceCtx();
    }
    g_nctx = 0;
    g_cur_dev = -1;
    g_gpu_calls = 0;
    g_fp8_lut_ready = 0;
}

extern "C" int coli_cuda_device_count(void) { return g_nctx; }
extern "C" int coli_cuda_device_at(int index) { return index >= 0 && index < g_nctx ? g_ctx[index].device : -1; }
extern "C" int coli_cuda_mem_info(int device, size_t *free_bytes, size_t *total_bytes) {
    DeviceCtx *c = find_ctx(device);
    if (!free_bytes || !total_bytes || !select_ctx(c)) return 0;
    return cuda_ok(cudaMemGetInfo(free_bytes, total_bytes), "memory info");
}
extern "C" int coli_cuda_device_integrated(int device) {
    cudaDeviceProp prop{};
    if (!cuda_ok(cudaGetDeviceProperties(&prop, device), "device properties")) return 0;
    return prop.integrated ? 1 : 0;
}
extern "C" void coli_cuda_stats(int device, size_t *tensor_count, size_t *tensor_bytes) {
    std::lock_guard<std::mutex> lock(g_mu);
    size_t n = 0, b = 0;
    for (int i = 0; i < g_nctx; i++)
        if (device < 0 || g_ctx[i].device == device) { n += g_ctx[i].tensor_count; b += g_ctx[i].tensor_bytes; }
    if (tensor_count) *tensor_count = n;
    if (tensor_bytes) *tensor_bytes = b;
}
extern "C" size_t coli_cuda_physical_bytes(int device) {
    size_t b = 0;
    for (int i = 0; i < g_nctx; i++) if (device < 0 || g_ctx[i].device == device) b += g_ctx[i].physical_bytes;
    return b;
}
extern "C" void coli_cuda_group_stats(uint64_t *calls, uint64_t *experts, uint64_t *rows,
                                      double *h2d_ms, double *kernel_ms, double *d2h_ms) {
    std::lock_guard<std::mutex> lock(g_mu);
    uint64_t a = 0, b = 0, r = 0; double h = 0, k = 0, d = 0;
    for (int i = 0; i < g_nctx; i++) {
        a += g_ctx[i].g_calls; b += g_ctx[i].g_experts; r += g_ctx[i].g_rows;
        h += g_ctx[i].g_h2d; k += g_ctx[i].g_kern; d += g_ctx[i].g_d2h;
    }
    if (calls) *calls = a; if (experts) *experts = b; if (rows) *rows = r;
    if (h2d_ms) *h2d_ms = h; if (kernel_ms) *kernel_ms = k; if (d2h_ms) *d2h_ms = d;
}
extern "C" void coli_cuda_group_stats_device(int device, uint64_t *calls, uint64_t *experts,
                                             uint64_t *rows, double *h2d_ms, double *kernel_ms,
                                             double *d2h_ms) {
    std::lock_guard<std::mutex> lock(g_mu);
    DeviceCtx *c = find_ctx(device);
    if (calls) *calls = c ? c->g_calls : 0; if (experts) *experts = c ? c->g_experts : 0;
    if (rows) *rows = c ? c->g_rows : 0; if (h2d_ms) *h2d_ms = c ? c->g_h2d : 0;
    if (kernel_ms) *kernel_ms = c ? c->g_kern : 0; if (d2h_ms) *d2h_ms = c ? c->g_d2h : 0;
}
extern "C" int coli_cuda_e8_set_grid(const void *) { return 0; }
// fmt 8 (FP8 E4M3 bytes, one f32 scale per 128x128 block; c/quant.h:430-536): the engine
// hands over its 256-entry decode table once after init (c/backend_cuda.cu:918-927); uploads
// of fmt 8 are refused until it has (the kernels would read a zero table).
extern "C" int coli_cuda_fp8_set_lut(const float *lut) {
    if (!lut || g_nctx < 1) return 0;
    for (int i = 0; i < g_nctx; i++) {
        if (!select_ctx(&g_ctx[i])) return 0;
        if (!cuda_ok(cudaMemcpyToSymbol(d_e4m3_lut, lut, 256 * sizeof(float)), "e4m3 table upload")) return 0;
        void *p = nullptr;
        if (!cuda_ok(cudaGetSymbolAddress(&p, d_e4m3_lut), "e4m3 table address")) return 0;
        g_ctx[i].e4m3_lut_dev = static_cast<const float *>(p);
    }
    g_fp8_standard = 1;
    for (int i = 0; i < 256; i++) {
        const int e = (i >> 3) & 15, m = i & 7;
        float v = e ? std::ldexp(1.f + m / 8.f, e - 7) : std::ldexp(m / 8.f, -6);
        if (i & 128) v = -v;
        if ((i & 127) == 127 ? !std::isnan(lut[i]) : lut[i] != v) g_fp8_standard = 0;
    }
    g_fp8_lut_ready = 1;
    return 1;
}
extern "C" void coli_cuda_set_timing(int enabled) { g_timing = enabled ? 1 : 0; }
extern "C" int coli_cuda_last_timing(int device, float *kernel_ms, int *launches) {
    DeviceCtx *c = find_ctx(device);
    if (!c || !c->have_timing) return 0;
    if (kernel_ms) *kernel_ms = c->last_ms;
    if (launches) *launches = c->last_launches;
    return 1;
}
extern "C" unsigned long long coli_cuda_launch_total(int device) {
    DeviceCtx *c = find_ctx(device);
    return c ? c->total_launches + (unsigned long long)c->last_launches : 0;
}
extern "C" void *coli_cuda_stream(int device) {
    DeviceCtx *c = find_ctx(device);
    return c ? (void *)c->stream : nullptr;
}
extern "C" int coli_cuda_kernel_status(int device) {
    DeviceCtx *c = find_ctx(device);
    if (!select_ctx(c)) return -1;
    if (!cuda_ok(cudaStreamSynchronize(c->stream), "synchronize")) return -1;
    int v = *reinterpret_cast<volatile int *>(c->status);
    return v ? v : c->sticky_status;
}

// ---------------------------------------------------------------------------
// Tensors
// ---------------------------------------------------------------------------
// Decides from the scale facts that k_check_scales / k_check_mx left (kernels_misc.cuh) whether the
// tensor-core path can carry this tensor exactly and with which power-of-two pre-multiplier (gemm_tc.cuh):
//   SC_ROW  integer codes, no shift
//   SC_H16  scale * 2^shift puts the largest scale in [2^10, 2^11); every non-zero scale must
//           lie within 2^-12 of the largest so that the hi/lo split keeps its low bits
//   SC_MX   2^(e - 127 + shift) must be an fp16 power of two <= 2^13 for every group that holds a
//           non-zero code: shift = 140 - e_max, spread e_max - e <= TC_MX_SPREAD (down to 2^-11)
static void tensor_tc_params(const DeviceCtx *c, ColiCudaTensor *t, const uint32_t *f) {
    t->tc_ok = 0; t->tc_shift = 0;
    if (!c->tc || !t->packed || (t->O % 128) || (t->I % 128)) return;
    if (t->mode == SC_ROW) { t->tc_ok = 1; return; }
    if (t->mode == SC_H16) {
        float smax, smin;
        const uint32_t lo = 0x7FFFFFFFu - f[2];
        std::memcpy(&smax, &f[1], 4); std::memcpy(&smin, &lo, 4);
        if (f[3]) return;                             // inf / nan / beyond fp16
        if (f[1] == 0) { t->tc_ok = 1; return; }
        if (smin < smax * (1.0f / 4096.0f)) return;
        int ex; std::frexp(smax, &ex);             // smax = m * 2^ex, m in [0.5, 1)
        int shift = 11 - ex;                       // smax * 2^shift in [2^10, 2^11)
        if (shift < 0 || shift > 30) return;
        t->tc_shift = shift; t->tc_ok = 1;
        return;
    }
    if (t->mode == SC_MX) {
        const int emax = (int)f[0], emin = f[1] ? 255 - (int)f[1] : emax;      // emin over groups with a non-zero code
        if (f[2] || emax - emin > TC_MX_SPREAD) return;
        t->tc_shift = 140 - emax; t->tc_ok = 1;
    }
}

static void tensor_release(ColiCudaTensor *t) {
    if (t->raw_w) cudaFree(t->raw_w);
    if (t->raw_s) cudaFree(t->raw_s);
    if (t->pk) cudaFree(t->pk);
    if (t->rowscale) cudaFree(t->rowscale);
    t->raw_w = t->raw_s = nullptr; t->pk = nullptr; t->rowscale = nullptr;
}

// Copies weights/scales to the device in the tensor's storage class. `t` has
// fmt/I/O/gs/ng set; allocations are made when `allocate` is set (upload) and
// reused otherwise (update).
static int tensor_fill(DeviceCtx *c, ColiCudaTensor *t, const void *weights, const void *scales,
                       int allocate) {
    const size_t wbytes = row_bytes(t->fmt, t->I) * (size_t)t->O;
    const size_t scount = t->fmt == 0 ? 0 : t->fmt == 8 ? (size_t)((t->O + 127) / 128) * (size_t)t->ng
                                                        : (size_t)t->O * (size_t)t->ng;
    const size_t sbytes = t->fmt == 7 ? scount : scount * sizeof(float);
    if (!t->packed) {
        if (allocate) {
            // 16 spare bytes: the matmul reads whole words of rows that start anywhere
            if (!cuda_ok(cudaMalloc(&t->raw_w, wbytes + 16), "tensor allocation")) return 0;
            if (sbytes && !cuda_ok(cudaMalloc(&t->raw_s, sbytes), "scale allocation")) return 0;
            t->physical_bytes = wbytes + sbytes;
        }
        if (!cuda_ok(upload_staged(ring_of(c), t->raw_w, weights, wbytes, c->stream), "tensor upload")) return 0;
        if (sbytes && !cuda_ok(upload_staged(ring_of(c), t->raw_s, scales, sbytes, c->stream), "scale upload")) return 0;
        return cuda_ok(cudaStreamSynchronize(c->stream), "tensor upload sync");
    }
    if (!reserve(c, &c->stage_w, wbytes) || (sbytes && !reserve(c, &c->stage_s, sbytes))) return 0;
    // Scales first: what the storage class depends on is found on the device while the codes travel.
    // Nothing of an existing tensor is overwritten before its new scales have been accepted.
    if (!cuda_ok(upload_staged(ring_of(c), c->stage_s.p, scales, sbytes, c->stream), "scale upload")) return 0;
    if (t->fmt == 4) {
        cudaMemsetAsync(c->check, 0, 4 * sizeof(uint32_t), c->stream);
        k_check_scales<<<(unsigned)((scount + 1023) / 1024), 256, 0, c->stream>>>(c->check, static_cast<const float *>(c->stage_s.p), scount);
        cudaMemcpyAsync(c->check_host, c->check, 4 * sizeof(uint32_t), cudaMemcpyDeviceToHost, c->stream);
        cudaEventRecord(c->ev_done, c->stream);
    }
    if (!cuda_ok(upload_staged(ring_of(c), c->stage_w.p, weights, wbytes, c->stream), "tensor upload")) return 0;
    if (t->fmt == 7) {
        cudaMemsetAsync(c->check, 0, 4 * sizeof(uint32_t), c->stream);
        k_check_mx<<<(unsigned)((scount + 255) / 256), 256, 0, c->stream>>>(c->check, static_cast<const uint8_t *>(c->stage_w.p),
                                                                            static_cast<const uint8_t *>(c->stage_s.p), scount);
        cudaMemcpyAsync(c->check_host, c->check, 4 * sizeof(uint32_t), cudaMemcpyDeviceToHost, c->stream);
        cudaEventRecord(c->ev_done, c->stream);
    }
    if (t->fmt != 2 && !cuda_ok(cudaEventSynchronize(c->ev_done), "scale check")) return 0;
    int mode = t->mode;
    if (allocate) {
        mode = t->fmt == 2 ? SC_ROW : t->fmt == 7 ? SC_MX : c->check_host[0] == 0 ? SC_H16 : SC_F32;
        t->mode = mode;
    } else if (t->fmt == 4 && mode == SC_H16 && c->check_host[0]) {
        return 0;   // the refreshed scales no longer fit the storage chosen at upload
    }
    tensor_tc_params(c, t, c->check_host);
    const int ch = chunk_bytes_of(mode);
    const size_t nblk = (size_t)(t->O / TILE_ROWS) * (t->I / BLOCK_K);
    const size_t pkbytes = nblk * ch;
    if (allocate) {
        // behind the tile streams: the tensor shift, for kernels that find the tensor by its address
        if (!cuda_ok(cudaMalloc((void **)&t->pk, pkbytes + TC_TAIL_BYTES), "tensor allocation")) return 0;
        t->physical_bytes = pkbytes + TC_TAIL_BYTES;
        if (mode == SC_ROW) {
            if (!cuda_ok(cudaMalloc((void **)&t->rowscale, (size_t)t->O * sizeof(float)), "scale allocation")) return 0;
            t->physical_bytes += (size_t)t->O * sizeof(float);
        }
    }
    size_t words = nblk * 512;
    k_repack_codes<<<(unsigned)((words + 255) / 256), 256, 0, c->stream>>>(
        t->pk, static_cast<const uint8_t *>(c->stage_w.p), t->O, t->I, ch, t->fmt == 7, t->tc_shift);
    if (mode == SC_ROW) {
        if (!cuda_ok(cudaMemcpyAsync(t->rowscale, c->stage_s.p, (size_t)t->O * sizeof(float), cudaMemcpyDeviceToDevice, c->stream), "scale upload")) return 0;
    } else {
        size_t n = nblk * 128;
        k_repack_scales<<<(unsigned)((n + 255) / 256), 256, 0, c->stream>>>(
            t->pk, c->stage_s.p, t->O, t->I, ch, mode, t->gs > 0 ? t->gs : t->I, t->ng,
            mode == SC_MX && t->tc_ok ? 140 - t->tc_shift - TC_MX_SPREAD : 0);
    }
    if (!cuda_ok(cudaGetLastError(), "repack launch")) return 0;
    return cuda_ok(cudaStreamSynchronize(c->stream), "tensor upload sync");
}

static thread_local int g_upload_gs = 0;

extern "C" int coli_cuda_tensor_upload(ColiCudaTensor **tensor, const void *weights,
                                       const float *scales, int fmt, int I, int O, int device) {
    if (!tensor) return 0;
    const int want_gs = (fmt == 4 && g_upload_gs > 0) ? g_upload_gs : 0;
    if (*tensor) {
        ColiCudaTensor *t = *tensor;
        return t->fmt == fmt && t->I == I && t->O == O && t->device == device && t->gs == want_gs;
    }
    DeviceCtx *c = find_ctx(device);
    if (!weights || I < 1 || O < 1 || !select_ctx(c)) return 0;
    if (!(fmt == 0 || fmt == 1 || fmt == 2 || fmt == 3 || fmt == 4 || fmt == 7 || fmt == 8)) return 0;
    if (fmt && !scales) return 0;
    if (fmt == 8 && !g_fp8_lut_ready) return 0;
    ColiCudaTensor *t = static_cast<ColiCudaTensor *>(std::calloc(1, sizeof(*t)));
    if (!t) return 0;
    t->fmt = fmt; t->I = I; t->O = O; t->device = device; t->gs = want_gs;
    t->ng = fmt == 7 ? (I + 31) / 32 : fmt == 8 ? (I + 127) / 128 : (want_gs ? (I + want_gs - 1) / want_gs : 1);
    const size_t wbytes = row_bytes(fmt, I) * (size_t)O;
    t->logical_bytes = wbytes + (fmt == 0 ? 0 : fmt == 7 ? (size_t)O * t->ng
                                : fmt == 8 ? (size_t)((O + 127) / 128) * t->ng * sizeof(float)
                                           : (size_t)O * t->ng * sizeof(float));
    t->packed = (fmt == 2 || fmt == 7 || (fmt == 4 && (want_gs == 32 || want_gs == 64 || want_gs == 128))) &&
                I % BLOCK_K == 0 && O % TILE_ROWS == 0;
    if (!tensor_fill(c, t, weights, scales, 1)) {
        tensor_release(t);
        std::free(t);
        return 0;
    }
    {
        std::lock_guard<std::mutex> lock(g_mu);     // uploads may come from one host thread per device
        c->tensor_count++;
        c->tensor_bytes += t->logical_bytes;
        c->physical_bytes += t->physical_bytes;
    }
    *tensor = t;
    return 1;
}
extern "C" int coli_cuda_tensor_upload_g(ColiCudaTensor **tensor, const void *weights,
                                         const float *scales, int fmt, int I, int O, int device,
                                         int gs) {
    g_upload_gs = gs > 0 ? gs : 0;
    int r = coli_cuda_tensor_upload(tensor, weights, scales, fmt, I, O, device);
    g_upload_gs = 0;
    return r;
}
// The entropy-coded upload of builds with -DCOLI_ANS (c/backend_cuda.h:60-67): this backend
// holds no decoder for it and refuses, which the engine answers by uploading the plain bytes.
extern "C" int coli_cuda_tensor_upload_compressed(ColiCudaTensor **, const void *, const float *, int, int, int,
                                                  int) { return 0; }
extern "C" void coli_cuda_tensor_free(ColiCudaTensor *t) {
    if (!t) return;
    DeviceCtx *c = find_ctx(t->device);
    if (c) {
        select_ctx(c);
        cudaStreamSynchronize(c->stream);
        {
            std::lock_guard<std::mutex> lock(g_mu);
            if (c->tensor_count) c->tensor_count--;
            if (c->tensor_bytes >= t->logical_bytes) c->tensor_bytes -= t->logical_bytes;
            if (c->physical_bytes >= t->physical_bytes) c->physical_bytes -= t->physical_bytes;
        }
        tensor_release(t);
        (void)cudaGetLastError();
    }
    std::free(t);
}
extern "C" size_t coli_cuda_tensor_bytes(const ColiCudaTensor *t) { return t ? t->logical_bytes : 0; }
extern "C" int coli_cuda_tensor_device(const ColiCudaTensor *t) { return t ? t->device : -1; }
extern "C" int coli_cuda_tensor_update(ColiCudaTensor *t, const void *weights, const float *scales) {
    if (!t || !weights || (t->fmt && !scales)) return 0;
    DeviceCtx *c = find_ctx(t->device);
    if (!select_ctx(c)) return 0;
    cudaStreamSynchronize(c->stream);
    return tensor_fill(c, t, weights, scales, 0);
}

// ---------------------------------------------------------------------------
// Streaming GEMV launch helpers
// ---------------------------------------------------------------------------
template <int MODE, int NC>
static void launch_one(DeviceCtx *c, const GemvSeg *segs, const GemvCtl *ctl, const __half *bq,
                       const float *bs) {
    constexpr int W = GemvCfg<NC>::WARPS, N = GemvCfg<NC>::NST;
    size_t smem = (size_t)W * N * (chunk_bytes_of(MODE) + 8);
    launch_pdl(c, k_gemv_stream<MODE, NC, W, N>, c->sms, W * 32, smem, segs, ctl, bq, bs, c->status);
}
template <int MODE>
static void launch_mode(DeviceCtx *c, int nc, const GemvSeg *segs, const GemvCtl *ctl,
                        const __half *bq, const float *bs) {
    switch (nc) {
    case 2: launch_one<MODE, 2>(c, segs, ctl, bq, bs); break;
    case 4: launch_one<MODE, 4>(c, segs, ctl, bq, bs); break;
    default: launch_one<MODE, 8>(c, segs, ctl, bq, bs); break;
    }
}
static int g_kernel_events = 0;   // 1: bracket every streaming-GEMV launch with an event pair
#define KEV_MAX_PAIRS 8192
static void kernel_event_pair(DeviceCtx *c, cudaEvent_t *e0, cudaEvent_t *e1) {
    *e0 = *e1 = nullptr;
    if (!g_kernel_events || c->kev_used >= KEV_MAX_PAIRS) return;
    if (!c->kev) c->kev = new std::vector<cudaEvent_t>();
    while ((int)c->kev->size() < 2 * (c->kev_used + 1)) {
        cudaEvent_t e;
        if (cudaEventCreate(&e) != cudaSuccess) { (void)cudaGetLastError(); return; }
        c->kev->push_back(e);
    }
    *e0 = (*c->kev)[2 * c->kev_used]; *e1 = (*c->kev)[2 * c->kev_used + 1];
    c->kev_used++;
}
static void launch_gemv(DeviceCtx *c, int mode, int nc, const GemvSeg *segs, const GemvCtl *ctl,
                        const __half *bq, const float *bs) {
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    kernel_event_pair(c, &e0, &e1);
    if (e0) cudaEventRecord(e0, c->stream);
    if (e0) c->chain = false;
    switch (mode) {
    case SC_ROW: launch_mode<SC_ROW>(c, nc, segs, ctl, bq, bs); break;
    case SC_H16: launch_mode<SC_H16>(c, nc, segs, ctl, bq, bs); break;
    case SC_F32: launch_mode<SC_F32>(c, nc, segs, ctl, bq, bs); break;
    default: launch_mode<SC_MX>(c, nc, segs, ctl, bq, bs); break;
    }
    if (e1) cudaEventRecord(e1, c->stream);
    c->last_launches++;
}
extern "C" void coli_cuda_set_kernel_events(int enabled) {
    g_kernel_events = enabled ? 1 : 0;
    for (int i = 0; i < g_nctx; i++) g_ctx[i].kev_used = 0;
}
extern "C" int coli_cuda_kernel_events(int device, float *total_ms, int *launches) {
    DeviceCtx *c = find_ctx(device);
    if (!select_ctx(c)) return 0;
    if (!cuda_ok(cudaStreamSynchronize(c->stream), "synchronize")) return 0;
    float tot = 0.f;
    for (int i = 0; i < c->kev_used; i++) {
        float ms = 0.f;
        if (cudaEventElapsedTime(&ms, (*c->kev)[2 * i], (*c->kev)[2 * i + 1]) == cudaSuccess) tot += ms;
        else (void)cudaGetLastError();
    }
    if (total_ms) *total_ms = tot;
    if (launches) *launches = c->kev_used;
    c->kev_used = 0;
    return 1;
}

// column sets (4 rows each) per pass at most, for a given largest row count
static int pick_nc(int max_rows) { return max_rows <= 8 ? 2 : max_rows <= 16 ? 4 : 8; }

// Split of the contraction into k slices, a divisor of the block count: every warp of the grid works through
// its share of the tasks, so the time goes with the rounds that takes times a task's blocks, plus about two
// blocks' worth per task for starting it and storing its sums. At least two blocks per task.
static int pick_nkpart(int nkb, long base_tasks, int sms) {
    const long warps = (long)sms * 16;      // (8 with more than 8 rows a pass: the rounds only double)
    int best = 1;
    long best_cost = LONG_MAX;
    for (int k = 1; k == 1 || k <= nkb / 2; k++) {
        if (nkb % k) continue;
        const long cost = (base_tasks * k + warps - 1) / warps * (nkb / k + 2);
        if (cost < best_cost) { best_cost = cost; best = k; }
    }
    return best;
}

static void timing_begin(DeviceCtx *c) {
    c->total_launches += (unsigned long long)c->last_launches;
    c->last_launches = 0;
    c->have_timing = 0;
    if (g_timing) cudaEventRecord(c->ev0, c->stream);
}
static void timing_end(DeviceCtx *c) {
    if (g_timing) cudaEventRecord(c->ev1, c->stream);
}
static void timing_collect(DeviceCtx *c) {   // after a stream synchronize
    if (g_timing && cudaEventElapsedTime(&c->last_ms, c->ev0, c->ev1) == cudaSuccess) c->have_timing = 1;
    else (void)cudaGetLastError();
}

struct HostSegs {
    std::vector<GemvSeg> v[4];   // by scale mode
    int ntask[4] = {0, 0, 0, 0};
    int uniform[4] = {0, 0, 0, 0};   // tasks per segment when all segments of a mode agree, else -1
};

static void add_seg(HostSegs *hs, const ColiCudaTensor *t, float *out, const int *rowid, int nrows,
                    int pos0, int nkpart) {
    GemvSeg s;
    std::memset(&s, 0, sizeof(s));
    s.w = t->pk; s.rowscale = t->rowscale; s.out = out;
    for (int r = 0; r < nrows; r++) s.rowid[r] = rowid[r];
    s.nrows = nrows; s.pos0 = pos0;
    s.O = t->O; s.ntiles = t->O / TILE_ROWS; s.nkb = t->I / BLOCK_K;
    s.nkpart = nkpart; s.kb_per_part = s.nkb / nkpart;
    s.task0 = hs->ntask[t->mode];
    const int nt = s.ntiles * nkpart;
    if (hs->uniform[t->mode] == 0) hs->uniform[t->mode] = nt;
    else if (hs->uniform[t->mode] != nt) hs->uniform[t->mode] = -1;
    hs->ntask[t->mode] += nt;
    hs->v[t->mode].push_back(s);
}

// Segment lists of a call on the device: uploaded in one copy before its kernels.
struct SegLists {
    const GemvSeg *seg[2][4];
    const GemvCtl *ctl[2][4];
};
static int upload_segs(DeviceCtx *c, SegLists *sl, const HostSegs *const *hs, int n, Buf *buf, int npos) {
    size_t need = 0;
    for (int k = 0; k < n; k++) for (int m = 0; m < 4; m++) need += hs[k]->v[m].size() * sizeof(GemvSeg) + sizeof(GemvCtl);
    if (!reserve(c, buf, need)) return 0;
    // Pageable staging: cudaMemcpyAsync from pageable memory returns once the
    // source has been captured, so the vector can die with this call even
    // though the stream has not run yet.
    std::vector<uint8_t> stage(need);
    const uint8_t *dp = static_cast<const uint8_t *>(buf->p);
    size_t off = 0;
    for (int k = 0; k < n; k++)
        for (int m = 0; m < 4; m++) {
            const std::vector<GemvSeg> &v = hs[k]->v[m];
            if (!v.empty()) std::memcpy(stage.data() + off, v.data(), v.size() * sizeof(GemvSeg));
            sl->seg[k][m] = v.empty() ? nullptr : reinterpret_cast<const GemvSeg *>(dp + off);
            off += v.size() * sizeof(GemvSeg);
        }
    for (int k = 0; k < n; k++)
        for (int m = 0; m < 4; m++) {
            GemvCtl ctl;
            ctl.nseg = (int)hs[k]->v[m].size(); ctl.ntask = hs[k]->ntask[m]; ctl.npos = npos;
            ctl.tasks_per_seg = hs[k]->uniform[m] > 0 ? hs[k]->uniform[m] : 0;
            std::memcpy(stage.data() + off, &ctl, sizeof(ctl));
            sl->ctl[k][m] = reinterpret_cast<const GemvCtl *>(dp + off);
            off += sizeof(ctl);
        }
    c->chain = false;
    return cuda_ok(cudaMemcpyAsync(buf->p, stage.data(), need, cudaMemcpyHostToDevice, c->stream), "segment upload");
}
// One GEMV launch per scale mode present in list k.
static int run_segs(DeviceCtx *c, const SegLists &sl, int k, int nc, const __half *bq, const float *bs) {
    for (int m = 0; m < 4; m++)
        if (sl.seg[k][m]) launch_gemv(c, m, nc, sl.seg[k][m], sl.ctl[k][m], bq, bs);
    return cuda_ok(cudaGetLastError(), "gemv launch");
}

// Rows the one-launch kernel takes: up to 8, and up to 96 KB of split activations beside its weight ring.
template <int MODE, int NC>
static void launch_rows(DeviceCtx *c, const ColiCudaTensor *t, float *y, const float *x, int S) {
    launch_pdl(c, k_gemv_rows<MODE, NC>, t->O / 16, ROWS_WARPS * 32, rows_smem(MODE, S, t->I), y, x, t->pk, t->rowscale, S, t->I, t->O,
                                                                                              c->status);
}

// y_dev[S,O] = x_dev[S,I] @ W^T for a packed tensor, all on c->stream.
static int linear_packed(DeviceCtx *c, const ColiCudaTensor *t, float *y_dev, const float *x_dev, int S) {
    const int nkb = t->I / BLOCK_K;
    if (!rows_aligned("linear", x_dev)) return 0;
    if (S <= 8 && S * t->I <= ROWS_MAX_X) {
        switch (t->mode * 2 + (S > 4)) {
        case SC_ROW * 2: launch_rows<SC_ROW, 1>(c, t, y_dev, x_dev, S); break;
        case SC_ROW * 2 + 1: launch_rows<SC_ROW, 2>(c, t, y_dev, x_dev, S); break;
        case SC_H16 * 2: launch_rows<SC_H16, 1>(c, t, y_dev, x_dev, S); break;
        case SC_H16 * 2 + 1: launch_rows<SC_H16, 2>(c, t, y_dev, x_dev, S); break;
        case SC_F32 * 2: launch_rows<SC_F32, 1>(c, t, y_dev, x_dev, S); break;
        case SC_F32 * 2 + 1: launch_rows<SC_F32, 2>(c, t, y_dev, x_dev, S); break;
        case SC_MX * 2: launch_rows<SC_MX, 1>(c, t, y_dev, x_dev, S); break;
        default: launch_rows<SC_MX, 2>(c, t, y_dev, x_dev, S); break;
        }
        c->last_launches++;
        return cuda_ok(cudaGetLastError(), "linear launch");
    }
    if (!rows_aligned("linear", y_dev)) return 0;
    const int nc = pick_nc(S), rpp = 4 * nc;
    const int npass = (S + rpp - 1) / rpp;
    const int nkpart = pick_nkpart(nkb, (long)npass * (t->O / TILE_ROWS), c->sms);
    if (!reserve(c, &c->bq, (size_t)S * t->I * 2 * sizeof(__half)) ||
        !reserve(c, &c->bs, (size_t)S * nkb * sizeof(float)) ||
        !reserve(c, &c->pd, (size_t)nkpart * S * t->O * sizeof(float))) return 0;
    HostSegs hs;
    int rowid[SEG_MAX_ROWS];
    for (int p = 0; p < npass; p++) {
        int r0 = p * rpp, nr = S - r0 < rpp ? S - r0 : rpp;
        for (int r = 0; r < nr; r++) rowid[r] = r0 + r;
        add_seg(&hs, t, (float *)c->pd.p, rowid, nr, r0, nkpart);
    }
    SegLists sl;
    const HostSegs *lists[1] = {&hs};
    if (!upload_segs(c, &sl, lists, 1, &c->segs2, S)) return 0;
    int nw = S * nkb;
    launch_pdl(c, k_prep_rows, (nw * 32 + 255) / 256, 256, 0, (__half *)c->bq.p, (float *)c->bs.p, x_dev, S, t->I);
    c->last_launches++;
    if (!run_segs(c, sl, 0, nc, (const __half *)c->bq.p, (const float *)c->bs.p)) return 0;
    size_t n4 = (size_t)S * t->O / 4;
    launch_pdl(c, k_reduce_parts, (unsigned)((n4 + 255) / 256), 256, 0, y_dev, (const float *)c->pd.p, S, t->O, nkpart);
    c->last_launches++;
    return cuda_ok(cudaGetLastError(), "linear launch");
}

// CTAs that share an SM at up to four rows. A wave takes a CTA's loads one behind the other, so what counts is how many
// waves there are: the fewest CTAs an SM that need the fewest, between LO and HI. More of them leave a thread fewer
// registers (128, 80, 64 at 2, 3, 4), that is fewer words ahead: 8-bit formats spill at 64, and FP8, which gains most from them, at 80.
// One row, us at two / three / four an SM by O (columns in parentheses):
//   grouped int4 (6150)  8200: 56 / 58 / 58    9480: 77 / 58 / 58    12296: 101 / 60 / 60    18440: 103 / 109 / 67    32776: 194 / 159 / 118
//   MXFP4 (6150)         8200: 42 / 44 / 44    9480: 52 / 44 / 46    12296: 75 / 46 / 46     18440: 75 / 81 / 50      32776: 140 / 118 / 89
//   per-row int4 (6150)  9480: 42 / 42 / 42    14216: 54 / 54 / 44   18440: 75 / 77 / 48     21320: 77 / 77 / 79      32776: 110 / 110 / 83
//   2-bit (6144)         9504: 30 / 30 / 30    14208: 32 / 32 / 32   18432: 50 / 50 / 34     21312: 50 / 52 / 50      32768: 71 / 71 / 56
//   int8 (6144)          9472: 22 / 22 / 24    9504: 26 / 22 / 26    12288: 30 / 24 / 28     18432: 32 / 34 / 34      32768: 50 / 46 / 52
//   FP8 (6144)           9472: 19 / 22 / 26    9504: 24 / 22 / 26    12288: 26 / 26 / 28     18432: 28 / 36 / 38      32768: 44 / 52 / 54
// (2-bit and per-row int4 take 72 to 80 registers however many they may: two and three are one. 2-bit in more tiles than two an SM hold
// takes what the compiler chooses, 63: one row of 12288 20 / 19, 18432 27 / 25 us, capped for three and four / so. int8 off 16-byte
// rows has two: of 6150 x 32768 65, three 71.)
// Five to eight rows: capped for two an SM (128 registers) where that beats the 100 to 120 that the compiler takes: capped / not, 6144 x 8192
// FP8 16.6 / 18.6, 6150 x 12288 int8 36 / 43, 6150 x 4736 per-row int4 26 / 29; 6150 x 8192 MXFP4 34 / 31, 6150 x 2048 grouped int4 41 / 39, 6144 x 18432
// 2-bit 42 / 39, 6144 x 32768 int8 51 / 50.
template <int FMT, bool AL16> struct DenseCtas {
    static constexpr int LO = FMT == 2 ? 3 : 2, HI = FMT == 8 || (FMT == 1 && !AL16) ? 2 : FMT == 1 ? 3 : 4;
};
static int dense_ctas(int lo, int hi, long ctas, int sms) {
    int best = lo;
    for (int k = lo + 1; k <= hi; k++)
        if ((ctas + (long)k * sms - 1) / ((long)k * sms) < (ctas + (long)best * sms - 1) / ((long)best * sms)) best = k;
    return best;
}
template <int FMT, bool AL16>
static void launch_dense(DeviceCtx *c, const ColiCudaTensor *t, float *y, int S, const __half *bq, const float *bs) {
    const int nc = S <= 4 ? 1 : S <= 8 ? 2 : 4;
    const dim3 grid((unsigned)((t->O + 31) / 32), (unsigned)((S + 4 * nc - 1) / (4 * nc)));
    const long ctas = (long)grid.x * grid.y;
    const uint8_t *w = static_cast<const uint8_t *>(t->raw_w);
    const size_t rb = row_bytes(t->fmt, t->I);
    const int gs = t->gs > 0 ? t->gs : t->I;
    auto go = [&](auto kern) { launch_pdl(c, kern, grid, DENSE_WARPS * 32, 0, y, bq, bs, w, t->raw_s, S, t->I, t->O, rb, gs, t->ng); };
    // More than 8 rows, one CTA an SM: int8 runs faster in the 178 registers of the compiler's choice than in the 211 it may take (16 rows of
    // 6144 x 4736 17.4 / 18.6). 8-bit rows on 16 bytes: three waves of one CTA an SM against one of two and a rest (12 rows of 6144 x 9504 |
    // 12288 | 14208: int8 42 / 44 | 46 / 44 | 48 / 52, FP8 36 / 38 | 38 / 42 | 40 / 44 us; at two and four waves two an SM are as fast or faster)
    const bool three = ctas > 2L * c->sms && ctas <= 3L * c->sms;
    if (nc == 1) {
        constexpr int LO = DenseCtas<FMT, AL16>::LO, HI = DenseCtas<FMT, AL16>::HI;
        const int k = dense_ctas(LO, HI, ctas, c->sms);
        if (k == LO) go(k_dense_mma<FMT, 1, AL16, FMT == 3 ? 3 : LO>);
        else if (FMT == 3) go(k_dense_mma<FMT, 1, AL16, 0>);
        else if (k == HI) go(k_dense_mma<FMT, 1, AL16, HI>);
        else go(k_dense_mma<FMT, 1, AL16, (LO + HI) / 2>);
    } else if (nc == 2) go(k_dense_mma<FMT, 2, AL16, FMT == 2 || FMT == 8 || (FMT == 1 && !AL16) ? 2 : 0>);
    else if (ctas > c->sms && !(AL16 && three)) go(k_dense_mma<FMT, 4, AL16, 2>);
    else go(k_dense_mma<FMT, 4, AL16, FMT == 1 ? 0 : 1>);
}

static int linear_raw(DeviceCtx *c, const ColiCudaTensor *t, float *y_dev, const float *x_dev, int S) {
    // Quantised rows take the tensor-core kernel; scale groups must hold whole 32-column groups, and FP8
    // tables other than E4M3's own have no conversion instruction.
    const bool whole = t->fmt != 4 || t->ng == 1 || t->gs % 32 == 0;
    if (t->fmt != 0 && whole && (t->fmt != 8 || g_fp8_standard)) {
        const int nkb = (t->I + 127) / 128;
        if (!reserve(c, &c->bq, (size_t)S * nkb * 256 * sizeof(__half)) || !reserve(c, &c->bs, (size_t)S * nkb * sizeof(float))) return 0;
        __half *bq = (__half *)c->bq.p;
        float *bs = (float *)c->bs.p;
        launch_pdl(c, k_prep_dense, (S * nkb * 32 + 255) / 256, 256, 0, bq, bs, x_dev, S, t->I, t->fmt);
        switch (t->fmt) {
        case 1: if (t->I % 16 == 0) launch_dense<1, true>(c, t, y_dev, S, bq, bs); else launch_dense<1, false>(c, t, y_dev, S, bq, bs); break;
        case 8: if (t->I % 16 == 0) launch_dense<8, true>(c, t, y_dev, S, bq, bs); else launch_dense<8, false>(c, t, y_dev, S, bq, bs); break;
        case 2: launch_dense<2, false>(c, t, y_dev, S, bq, bs); break;
        case 3: launch_dense<3, false>(c, t, y_dev, S, bq, bs); break;
        case 4: launch_dense<4, false>(c, t, y_dev, S, bq, bs); break;
        default: launch_dense<7, false>(c, t, y_dev, S, bq, bs); break;
        }
        c->last_launches += 2;
        return cuda_ok(cudaGetLastError(), "matmul launch");
    }
    // rows that start 16-byte aligned take the streaming kernel (128-bit loads)
    const bool dense = (t->fmt == 0 && t->I % 4 == 0) || (t->fmt == 8 && t->I % 16 == 0);
    if (dense && (reinterpret_cast<uintptr_t>(x_dev) & 15) == 0 && (reinterpret_cast<uintptr_t>(t->raw_w) & 15) == 0) {
        dim3 grid((unsigned)((t->O + 31) / 32), (unsigned)((S + 7) / 8));
        const float *sc = static_cast<const float *>(t->raw_s);
        if (t->fmt == 0) launch_pdl(c, k_dense_gemv<0>, grid, 256, DENSE_GEMV_SMEM, y_dev, x_dev, t->raw_w, sc, nullptr, S, t->I, t->O);
        else launch_pdl(c, k_dense_gemv<8>, grid, 256, DENSE_GEMV_SMEM, y_dev, x_dev, t->raw_w, sc, c->e4m3_lut_dev, S, t->I, t->O);
        c->last_launches++;
        return cuda_ok(cudaGetLastError(), "matmul launch");
    }
    dim3 grid((unsigned)((t->O + 7) / 8), (unsigned)((S + 7) / 8));
    launch_pdl(c, k_generic_matmul, grid, 256, 0, y_dev, x_dev, t->raw_w, t->raw_s, t->fmt, S, t->I, t->O,
                                                  t->gs > 0 ? t->gs : t->I, t->ng);
    c->last_launches++;
    return cuda_ok(cudaGetLastError(), "matmul launch");
}
static int linear_any(DeviceCtx *c, const ColiCudaTensor *t, float *y_dev, const float *x_dev, int S) {
    return t->packed ? linear_packed(c, t, y_dev, x_dev, S) : linear_raw(c, t, y_dev, x_dev, S);
}

// after the call's kernels are done
static int kernels_ok(DeviceCtx *c) {
    const int v = *reinterpret_cast<volatile int *>(c->status);
    if (v) {
        std::fprintf(stderr, "[CUDA] kernel wait guard expired (status %d)\n", v);
        // the grid barrier's arrival count may be mid-way: start over
        cudaMemsetAsync(c->dec_sync, 0, DEC_SYNC_WORDS * sizeof(unsigned int), c->stream);
        *reinterpret_cast<volatile int *>(c->status) = 0;
        c->sticky_status = v;
        if (c->group_pending) c->group_pending = -1;      // it may have been that group's: its take reports it too
        return 0;
    }
    return 1;
}
static int check_status(DeviceCtx *c) {
    return cuda_ok(cudaStreamSynchronize(c->stream), "synchronize") && kernels_ok(c);
}

// Host rows of a blocking call. Everything passes through pinned memory (a copy out of the cache and a DMA
// are faster than the driver's pageable path, 21 us against 27 at 300 KB), and small rows are not copied to the
// device at all: the kernel that reads them once, or stores the result, addresses the pinned buffer.
#define IO_DIRECT_BYTES (64u << 10)
// A few rows out of pinned memory into device memory by a kernel: the kernel behind it starts 5 us earlier than
// behind a copy command, whose completion the stream has to be told by another engine. n4: float4s.
static int pull_rows(DeviceCtx *c, void *dst, const void *pinned, size_t bytes) {
    const int n4 = (int)(bytes / 16);
    launch_pdl(c, k_pull, (n4 + 255) / 256, 256, 0, static_cast<float4 *>(dst), static_cast<const float4 *>(pinned), n4);
    return cuda_ok(cudaGetLastError(), "input upload");
}
// Rows to the device by way of a pinned buffer of their size, or of the ring where there is none.
static int rows_in(DeviceCtx *c, void *dst, void *pinned, const void *src, size_t bytes) {
    return cuda_ok(pinned ? IoPieces::in(dst, pinned, src, bytes, c->stream) : upload_staged(ring_of(c), dst, src, bytes, c->stream), "input upload");
}
// ... and back, once the kernels are known to have done well. rows_out_start only enqueues; the ring's part waits for rows_out_finish.
static int rows_out_start(DeviceCtx *c, void *pinned, const void *src_dev, size_t bytes) {
    return !pinned || cuda_ok(c->io.out_start(pinned, src_dev, bytes, c->stream), "output download");
}
static int rows_out_finish(DeviceCtx *c, void *dst, void *pinned, const void *src_dev, size_t bytes) {
    if (pinned) return c->io.out_finish(dst, pinned, bytes, [c] { return kernels_ok(c) != 0; });
    bool ready = true;
    return cuda_ok(download_staged(ring_of(c), dst, src_dev, bytes, c->stream, [c, &ready] { return ready = kernels_ok(c) != 0; }),
                   "output download") && ready;
}
// -> where the kernels find x, or NULL. read_once: the first kernel reads every element once (not every CTA all of them).
static const float *io_in(DeviceCtx *c, const float *x, size_t bytes, bool read_once) {
    float *pinned = reserve_pinned(c, &c->io_x, &c->io_x_cap, bytes) ? c->io_x : nullptr;
    if (pinned && read_once && bytes <= IO_DIRECT_BYTES) {
        std::memcpy(pinned, x, bytes);
        return pinned;
    }
    if (!reserve(c, &c->x, bytes)) return nullptr;
    if (pinned && bytes <= IO_DIRECT_BYTES && bytes % 16 == 0) {
        std::memcpy(pinned, x, bytes);
        return pull_rows(c, c->x.p, pinned, bytes) ? (const float *)c->x.p : nullptr;
    }
    return rows_in(c, c->x.p, pinned, x, bytes) ? (const float *)c->x.p : nullptr;
}
static float *io_out(DeviceCtx *c, size_t bytes) {
    if (reserve_pinned(c, &c->io_y, &c->io_y_cap, bytes) && bytes <= IO_DIRECT_BYTES) return c->io_y;
    return reserve(c, &c->y, bytes) ? (float *)c->y.p : nullptr;
}
static int io_finish(DeviceCtx *c, float *y, const float *y_dev, size_t bytes) {
    if (y_dev == c->io_y) {
        if (!check_status(c)) return 0;
        std::memcpy(y, c->io_y, bytes);
        return 1;
    }
    float *pinned = bytes <= c->io_y_cap ? c->io_y : nullptr;
    return rows_out_start(c, pinned, y_dev, bytes) && rows_out_finish(c, y, pinned, y_dev, bytes);
}

extern "C" int coli_cuda_matmul(ColiCudaTensor **tensor, float *y, const float *x, const void *weights,
                                const float *scales, int fmt, int S, int I, int O, int device, int gs) {
    if (fault_injected()) return 0;
    if (fmt == 4 && gs <= 0) return 0;
    if (S < 1 || !tensor || !x || !y) return 0;
    if (gs > 0) { if (!coli_cuda_tensor_upload_g(tensor, weights, scales, fmt, I, O, device, gs)) return 0; }
    else if (!coli_cuda_tensor_upload(tensor, weights, scales, fmt, I, O, device)) return 0;
    ColiCudaTensor *t = *tensor;
    DeviceCtx *c = find_ctx(t->device);
    if (!select_ctx(c)) return 0;
    std::lock_guard<std::mutex> hold(io_mutex(c));
    size_t xb = (size_t)S * I * sizeof(float), yb = (size_t)S * O * sizeof(float);
    const float *xd = io_in(c, x, xb, t->packed ? S > 8 : t->fmt != 0);
    float *yd = io_out(c, yb);
    if (!xd || !yd) return 0;
    timing_begin(c);
    if (!linear_any(c, t, yd, xd, S)) return 0;
    timing_end(c);
    if (!io_finish(c, y, yd, yb)) return 0;
    timing_collect(c);
    return 1;
}

extern "C" int coli_cuda_matmul_mxfp4(float *y, const float *x, const unsigned char *q4,
                                      const unsigned char *e8s, int S, int I, int O) {
    if (S < 1 || I < 1 || O < 1 || !y || !x || !q4 || !e8s || g_nctx < 1) return 0;
    ColiCudaTensor *t = nullptr;
    int dev = g_ctx[0].device;
    // a stateless call: the temporary tensor is freed again before returning
    int ok = coli_cuda_matmul(&t, y, x, q4, reinterpret_cast<const float *>(e8s), 7, S, I, O, dev, 0);
    if (t) coli_cuda_tensor_free(t);
    return ok;
}

extern "C" int coli_cuda_pipe_gemm(ColiCudaTensor *t, float *y_dev, const float *x_dev, int S) {
    if (fault_injected()) return 0;
    if (!t || S < 1 || !y_dev || !x_dev) return 0;
    DeviceCtx *c = find_ctx(t->device);
    if (!select_ctx(c)) return 0;
    return linear_any(c, t, y_dev, x_dev, S);
}

// ---------------------------------------------------------------------------
// Expert FFN over a packed group (device buffers), all on c->stream:
//   x_dev [total, D] rows in call order -> y_dev [total, D]
// ---------------------------------------------------------------------------
static int group_shape_ok(ColiCudaTensor *const *gates, ColiCudaTensor *const *ups,
                          ColiCudaTensor *const *downs, const int *rows, int count, int *device,
                          int *D, int *I, int *total, int *max_rows, int *all_packed, int *any_packed) {
    if (!gates || !ups || !downs || count < 1 || !gates[0]) return 0;
    *device = gates[0]->device; *D = gates[0]->I; *I = gates[0]->O;
    *total = 0; *max_rows = 0; *all_packed = 1; *any_packed = 0;
    for (int cidx = 0; cidx < count; cidx++) {
        ColiCudaTensor *g = gates[cidx], *u = ups[cidx], *d = downs[cidx];
        int r = rows ? rows[cidx] : 1;
        if (!g || !u || !d || r < 1 || g->device != *device || u->device != *device || d->device != *device ||
            g->I != *D || u->I != *D || g->O != *I || u->O != *I || d->I != *I || d->O != *D) return 0;
        if ((g->fmt == 4 && g->gs <= 0) || (u->fmt == 4 && u->gs <= 0) || (d->fmt == 4 && d->gs <= 0)) return 0;
        int p = g->packed && u->packed && d->packed;
        *all_packed &= p;
        *any_packed |= g->packed | u->packed | d->packed;
        *total += r;
        if (r > *max_rows) *max_rows = r;
    }
    return 1;
}


// ---------------------------------------------------------------------------
// Tensor-core path of the expert group (gemm_tc.cuh): taken when some expert has
// more rows than one streaming pass holds and every tensor qualifies.
// ---------------------------------------------------------------------------
// 0: never; 1: when it pays (tc_pays); 2: whenever the tensors and shapes allow it (tests).
static int g_tc_enabled = 1;
extern "C" void coli_cuda_set_tensor_core(int enabled) { g_tc_enabled = enabled < 0 ? 0 : enabled > 2 ? 2 : enabled; }
// The streaming kernel's cost grows with the rows (one set of MMAs per 4 rows and block of weights, and a wider pass for all from a
// mean of 4 in layers), the tensor-core path's hardly does up to 30 rows per expert, but it starts higher, most of all where a
// weight takes two fp16 terms (grouped int4), and that in either phase. So the line, as the mean of rows per expert, follows both phases'
// formats. Measured, streaming / tensor cores in us, layers with random routing (M*K rows over E experts) at D x I
// 2048 x 1024 (E 64) | 6144 x 2048 (E 64) | 7168 x 2048 (E 256 and a shared expert):
//   per-row int4          mean 2.5: 80 / 82 | 261 / 275 | 1128 / 1121     3: 84 / 82 | 279 / 281 | 1341 / 1307     4: 89 / 83 | 310 / 296 | 1522 / 1352
//   MXFP4                 mean 3: 80 / 83 | 268 / 286 | 1306 / 1353     4: 85 / 83 | 299 / 306 | 1440 / 1383
//   grouped int4          mean 4: 92 / 109 | 334 / 452 | 1557 / 2093     4.5: 112 / 110 | 431 / 452 | 2029 / 1943     5: 118 / 109 | 455 / 452 | 2236 / 2002
//   down grouped int4, gate and up per row    mean 4: 90 / 92 | 320 / 347 | 1530 / 1592     4.5: 112 / 92 | 420 / 347 | 2055 / 1463
//   gate and up grouped int4, down per row    mean 4: 92 / 101 | 328 / 402 | 1525 / 1882     4.5: 113 / 101 | 430 / 401 | 2024 / 1722
// Layers of less than TC_LARGE weights a matrix are short of launches rather than of work and cross later, at a mean of 4.5 where streaming
// passes widen (1024 x 512, E 64: per row 4: 43 / 47, 4.5: 52 / 46; MXFP4 43 / 47, 50 / 47; down grouped 45 / 49, 53 / 50; gate and up grouped 5: 55 / 53;
// 1024 x 768: per row 53 / 55, 65 / 55; gate and up grouped 4.5: 65 / 65). A little above it the lines of large layers come early, by 2 to 10 %
// (per-row 3, MXFP4 4: 1024 x 1024 58 / 60, 58 / 61; 1152 x 1024 62 / 68, 62 / 68; 1280 x 1024 70 / 70, 72 / 71; 1536 x 768 67 / 65, 68 / 69); grouped int4 at 8 does not
// (1024 x 512 63 / 56; 512 x 256 40 / 41).
// Groups of experts with unevenly spread rows widen single passes instead of all (24 experts, 2048 x 1024 | 6144 x 2048): per-row 2.5:
// 42 / 42 | 118 / 137, 3: 43 / 42 | 144 / 138; MXFP4 3: 42 / 43 | 140 / 139, 4: 42 / 44 | 150 / 140; grouped 5: 48 / 56 | 174 / 211, 6: 63 / 56 |
// 232 / 209; down grouped 5: 47 / 50 | 161 / 162, 6: 61 / 49 | 220 / 159; gate and up grouped 5: 48 / 52 | 164 / 186, 6: 63 / 52 | 225 / 191.
// Below TC_LARGE the lines lie where those passes widen, at 6, whatever the format (per row | MXFP4 | down grouped | gate and up grouped, at 5.5 and 6:
// 1024 x 512 26 / 28, 32 / 28 | 25 / 28, 31 / 28 | 26 / 29, 32 / 29 | 26 / 31, 32 / 31; 768 x 384 24 / 25, 27 / 25 | 23 / 25, 26 / 25 | 24 / 26, 27 / 26 | 24 / 26, 27 / 26;
// 1152 x 768 32 / 33, 40 / 32 | 31 / 33, 38 / 32 | 32 / 35, 40 / 34 | 32 / 37, 39 / 36), above it they come early up to 1.5 million weights (1280 x 1024: per row 3:
// 33 / 35, 4.5: 36 / 36; MXFP4 3.5: 32 / 36, 5: 36 / 36; 1536 x 1024 37 / 36 and 36 / 36 at the lines). Below TC_TINY both sides take the same 22 to 23 us,
// from a mean of 2 to 8 (256 x 128, 512 x 256).
// Grouped int4 has its line above where the times cross. Its products fill the accumulator, which truncates: against 64 bits an
// expert of 2048 x 1024 is off by 2.9e-6 on the tensor cores and by 1.5e-7 in the streaming kernel (per-row int4 2.2e-7 | 1.3e-7, MXFP4
// 2.6e-7 | 1.1e-7: few bits a product, most sums exact). A call is not taken there for less than a good part of its time; the
// same goes for gate and up or down alone.
#define TC_LARGE (1L << 20)
#define TC_TINY (1L << 17)
static bool tc_pays(long rows, long experts, int mode_gu, int mode_d, bool layer, long weights) {
    const bool two_gu = mode_gu == SC_H16, two_d = mode_d == SC_H16;
    const int kind = two_gu && two_d ? 2 : two_gu ? 4 : two_d ? 3 : mode_gu == SC_MX || mode_d == SC_MX ? 1 : 0;
    // half rows: per-row int4, MXFP4, grouped int4, only down grouped, only gate and up grouped
    static const int layers[3][5] = {{9, 9, 16, 9, 11}, {9, 9, 16, 9, 11}, {6, 8, 16, 9, 11}};
    static const int groups[3][5] = {{5, 6, 16, 9, 11}, {12, 12, 16, 12, 12}, {6, 7, 16, 11, 12}};
    const int size = weights >= TC_LARGE ? 2 : weights >= TC_TINY ? 1 : 0;
    return 2 * rows >= (long)(layer ? layers : groups)[size][kind] * experts;
}

template <int MODE, int PHASE>
static void launch_tc_one(DeviceCtx *c, const TcArgs &a) {
    launch_pdl(c, k_expert_gemm_tc<MODE, PHASE>, c->sms, TC_THREADS, tc_smem_total(MODE), a);
}
static int launch_tc(DeviceCtx *c, int mode, int phase, const TcArgs &a) {
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    kernel_event_pair(c, &e0, &e1);
    if (e0) cudaEventRecord(e0, c->stream);
    if (e0) c->chain = false;
    switch (mode * 2 + phase - 1) {
    case SC_ROW * 2: launch_tc_one<SC_ROW, 1>(c, a); break;
    case SC_ROW * 2 + 1: launch_tc_one<SC_ROW, 2>(c, a); break;
    case SC_H16 * 2: launch_tc_one<SC_H16, 1>(c, a); break;
    case SC_H16 * 2 + 1: launch_tc_one<SC_H16, 2>(c, a); break;
    case SC_MX * 2: launch_tc_one<SC_MX, 1>(c, a); break;
    case SC_MX * 2 + 1: launch_tc_one<SC_MX, 2>(c, a); break;
    default: return 0;
    }
    if (e1) cudaEventRecord(e1, c->stream);
    c->last_launches++;
    return 1;
}

// Device memory of a pass list with its tables, cut out of one block. `pass` comes first, then everything the
// host may upload with it (grp_pass, rowsrc) and the rest.
static size_t tc_list_layout(TcList *l, void *mem, int npass_cap, int ngrp_cap, int nrow_cap) {
    uint8_t *p = static_cast<uint8_t *>(mem);
    l->pass = reinterpret_cast<TcPass *>(p);
    int *q = reinterpret_cast<int *>(l->pass + npass_cap);
    l->npass = q; l->ngrp = q + 1; q += 4;
    l->lo_x = q; q += npass_cap;
    l->lo_h = q; q += npass_cap;
    l->grp_pass = q; q += ngrp_cap;
    l->rowsrc = nrow_cap ? q : nullptr; q += nrow_cap;
    l->rowdst = nullptr;
    return reinterpret_cast<uint8_t *>(q) - p;
}

// The expert FFN over a pass list that is already on the device (built there by k_tc_plan, or
// uploaded): rows x -> prepared tiles -> gate/up with the SwiGLU -> prepared tiles -> down -> y.
//   npos_cap positions and ngrp_cap padded groups of 16 at most; x rows are bf16 when x_bf16.
static int tc_ffn(DeviceCtx *c, int mode_gu, int mode_d, const TcList &l, const void *x, int x_bf16, int npos_cap, int ngrp_cap,
                  int D, int I, float *y) {
    const size_t rows = (size_t)ngrp_cap * 16;
    if (!reserve(c, &c->bq, rows * D * 2 * sizeof(__half)) || !reserve(c, &c->bs, (size_t)npos_cap * 2 * sizeof(float)) ||
        !reserve(c, &c->pg, (size_t)npos_cap * I * sizeof(float)) || !reserve(c, &c->hq, rows * I * 2 * sizeof(__half))) return 0;
    __half *xq = (__half *)c->bq.p, *hq = (__half *)c->hq.p;
    float *xinv = (float *)c->bs.p, *hinv = xinv + npos_cap, *H = (float *)c->pg.p;
    launch_pdl(c, k_prep_tc, ngrp_cap * 8, TC_PREP_THREADS, 0, xq, xinv, l.lo_x, x, l.rowsrc, l.pass, l.grp_pass, l.ngrp, D, x_bf16);
    TcArgs a;
    a.pass = l.pass; a.npass = l.npass; a.status = c->status;
    a.lo = l.lo_x; a.q = xq; a.qinv = xinv; a.rowdst = nullptr; a.out = H; a.K = D; a.O = I; a.ntile = I / 64;
    if (!launch_tc(c, mode_gu, 1, a)) return 0;
    launch_pdl(c, k_prep_tc, ngrp_cap * 8, TC_PREP_THREADS, 0, hq, hinv, l.lo_h, H, nullptr, l.pass, l.grp_pass, l.ngrp, I, 0);
    a.lo = l.lo_h; a.q = hq; a.qinv = hinv; a.rowdst = l.rowdst; a.out = y; a.K = I; a.O = D; a.ntile = D / 128;
    if (!launch_tc(c, mode_d, 2, a)) return 0;
    c->last_launches += 2;
    return cuda_ok(cudaGetLastError(), "tensor-core gemm launch");
}

// whatever: also where it does not pay
static int group_tc_ok(ColiCudaTensor *const *gates, ColiCudaTensor *const *ups,
                       ColiCudaTensor *const *downs, int count, int max_rows, int total, bool whatever = false) {
    if (!g_tc_enabled || max_rows < 2) return 0;
    if (g_tc_enabled == 1 && !whatever && !tc_pays(total, count, gates[0]->mode, downs[0]->mode, false, (long)gates[0]->I * gates[0]->O)) return 0;
    for (int e = 0; e < count; e++)
        if (!gates[e]->tc_ok || !ups[e]->tc_ok || !downs[e]->tc_ok || gates[e]->mode != gates[0]->mode ||
            ups[e]->mode != gates[0]->mode || downs[e]->mode != downs[0]->mode) return 0;
    return 1;
}

// x_dev [total (or 1 when bcast), D] -> y_dev [total, D].
// rowmap (host, optional): row of x of every packed position (a gather), and the row of y its
// result goes to (the expert-parallel layer works in place on differently grouped rows).
// x_bf16: x_dev holds bf16 rows.
static int group_device_tc(DeviceCtx *c, ColiCudaTensor *const *gates, ColiCudaTensor *const *ups,
                           ColiCudaTensor *const *downs, const int *rows, int count, int D, int I,
                           int total, float *y_dev, const void *x_dev, int bcast, const int *rowmap = nullptr,
                           int x_bf16 = 0) {
    int npass = 0, ngrp = 0;
    for (int e = 0; e < count; e++) {
        const int re = rows ? rows[e] : 1;
        npass += (re + TC_ROWS - 1) / TC_ROWS; ngrp += tc_pass_groups(re);
    }
    const int nmap = rowmap || bcast ? total : 0;
    TcList dl, hl;
    const size_t need = tc_list_layout(&dl, nullptr, npass, ngrp, nmap);
    if (!reserve(c, &c->misc, need)) return 0;
    std::vector<uint8_t> stage(need, 0);   // pageable: captured by the copy call before it returns
    tc_list_layout(&hl, stage.data(), npass, ngrp, nmap);
    tc_list_layout(&dl, c->misc.p, npass, ngrp, nmap);
    int off = 0, p = 0, grp = 0;
    for (int e = 0; e < count; e++) {
        const int re = rows ? rows[e] : 1, rp = tc_pass_rows(re);
        for (int r0 = 0; r0 < re; r0 += rp, p++) {
            const int nr = re - r0 < rp ? re - r0 : rp, npad = (nr + 15) & ~15;
            hl.pass[p] = TcPass{gates[e]->pk, ups[e]->pk, downs[e]->pk, gates[e]->rowscale, ups[e]->rowscale, downs[e]->rowscale,
                                off + r0, nr, npad, grp * 16, gates[e]->tc_shift, ups[e]->tc_shift, downs[e]->tc_shift};
            for (int i = 0; i < npad / 16; i++) hl.grp_pass[grp++] = p;
        }
        off += re;
    }
    *hl.npass = p; *hl.ngrp = grp;
    if (rowmap) std::memcpy(hl.rowsrc, rowmap, (size_t)total * sizeof(int));   // (bcast: all zero)
    c->chain = false;
    if (!cuda_ok(cudaMemcpyAsync(c->misc.p, stage.data(), need, cudaMemcpyHostToDevice, c->stream), "pass list upload")) return 0;
    dl.rowdst = rowmap ? dl.rowsrc : nullptr;
    return tc_ffn(c, gates[0]->mode, downs[0]->mode, dl, x_dev, x_bf16, total, ngrp, D, I, y_dev);
}

static int g_fused_decode = 3;
extern "C" void coli_cuda_set_fused_decode(int enabled) { g_fused_decode = enabled; }
#ifdef COLI_DECODE_PROBE
// Development builds only (-DCOLI_DECODE_PROBE): phase timestamps of the fused kernel.
static unsigned long long *g_decode_probe = nullptr;
extern "C" void coli_cuda_set_decode_probe(void *dev_buffer) { g_decode_probe = static_cast<unsigned long long *>(dev_buffer); }
#endif

// Warps that share one unit of a phase of the fused decode kernel (4, 8 or 16): the count
// that wastes the fewest warp slots on the phase's nkb blocks, ties going to 8 for the
// gate/up phase (few units per CTA) and to 4 for the down phase (many). A function of the
// shape only: the order of every sum in the kernel follows from it.
static int dec_pick_wpk(int nkb, int phase) {
    const int pref[2][3] = {{8, 16, 4}, {4, 8, 16}};
    int best = 0, bw = 1 << 30;
    for (int i = 0; i < 3; i++) {
        const int w = pref[phase - 1][i];
        const int waste = (nkb + w - 1) / w * w - nkb;
        if (waste < bw) { bw = waste; best = w; }
    }
    return best;
}

// Launches the fused decode kernel; a carries the problem (rule, x, out, M and, for a layer, tables, logits and
// routing outputs), preset the pass list of a call whose routing the host knows. npos: packed rows at most.
static int launch_decode(DeviceCtx *c, int mode, DecodeArgs &a, const DecPreset *preset, int npos, Buf *xq, Buf *xs, Buf *hq,
                         Buf *hs, Buf *pd) {
    const int D = a.rule.D, I = a.rule.I, nkb1 = D / BLOCK_K, nkb2 = I / BLOCK_K;
    const size_t act_cap = (size_t)dec_act_bytes(mode);
    a.act_smem = (size_t)a.M * nkb1 * 516 <= act_cap;
    // Down phase with a local combine (a CTA owns 16 output rows over every pass): when every
    // pass row's activations fit one CTA's shared memory and D/16 slices spread well over the SMs.
    const long units2 = D / 16, waves2 = (units2 + c->sms - 1) / c->sms;
    a.wpk1 = dec_pick_wpk(nkb1, 1); a.wpk2 = dec_pick_wpk(nkb2, 2);
    a.local2 = (size_t)npos * ((size_t)I * 4 + (size_t)nkb2 * 16 + 64) <= act_cap && units2 * 100 >= 85 * waves2 * c->sms &&
               (size_t)npos * a.wpk2 * 64 <= (size_t)2 * DEC_PART_BYTES;
    if (!reserve(c, hq, (size_t)npos * I * 2 * sizeof(__half)) || !reserve(c, hs, (size_t)npos * (I / 32) * sizeof(float)) ||
        !reserve(c, pd, (size_t)npos * D * sizeof(float))) return 0;
    if (!a.act_smem) {
        // x does not fit the kernel's shared memory: split it once here, the kernel reads the fragments
        if (!reserve(c, xq, (size_t)a.M * D * 2 * sizeof(__half)) || !reserve(c, xs, (size_t)a.M * nkb1 * sizeof(float))) return 0;
        launch_pdl(c, k_prep_rows, (a.M * nkb1 * 32 + 255) / 256, 256, 0, (__half *)xq->p, (float *)xs->p, a.x, a.M, D);
        c->last_launches++;
    }
    a.xq = (const __half *)xq->p; a.xs = (const float *)xs->p;
    a.hq = (__half *)hq->p; a.hs = (float *)hs->p; a.Y = (float *)pd->p;
    a.sync = c->dec_sync; a.exp_tab = c->exp_tab_dev; a.status = c->status;
    a.mg_grid = dec_magic((unsigned int)c->sms); a.mg_nt1 = dec_magic((unsigned int)(I / TILE_ROWS));
    a.mg_nt2 = dec_magic((unsigned int)(D / TILE_ROWS));
#ifdef COLI_DECODE_PROBE
    a.probe = g_decode_probe;
#endif
    DecRouted routed;
    void *args[] = {&a, preset ? const_cast<DecPreset *>(preset) : static_cast<void *>(&routed)};
    static const void *const fns[4][2] = {
        {(const void *)k_moe_decode<SC_ROW, false>, (const void *)k_moe_decode<SC_ROW, true>},
        {(const void *)k_moe_decode<SC_H16, false>, (const void *)k_moe_decode<SC_H16, true>},
        {(const void *)k_moe_decode<SC_F32, false>, (const void *)k_moe_decode<SC_F32, true>},
        {(const void *)k_moe_decode<SC_MX, false>, (const void *)k_moe_decode<SC_MX, true>}};
    const void *fn = fns[mode][preset != nullptr];
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    kernel_event_pair(c, &e0, &e1);
    if (e0) cudaEventRecord(e0, c->stream);
    // 1: cooperative launch (co-residency of the grid guaranteed by the driver).
    // 2: plain launch (the grid is one CTA per SM, so it still fits the device).
    // 3: plain launch with programmatic stream serialisation: the next layer's CTAs are
    //    scheduled as this grid's CTAs exit and wait at griddepcontrol.wait, which hides
    //    most of the launch latency between back-to-back layer calls.
    cudaError_t err;
    const size_t smem = (size_t)decode_smem_bytes(mode);
    if (g_fused_decode == 3) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(c->sms); cfg.blockDim = dim3(DEC_WARPS * 32);
        cfg.dynamicSmemBytes = smem; cfg.stream = c->stream;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = at; cfg.numAttrs = 1;
        err = cudaLaunchKernelExC(&cfg, fn, args);
    } else if (g_fused_decode == 2) {
        err = cudaLaunchKernel(fn, dim3(c->sms), dim3(DEC_WARPS * 32), args, smem, c->stream);
    } else {
        err = cudaLaunchCooperativeKernel(fn, dim3(c->sms), dim3(DEC_WARPS * 32), args, smem, c->stream);
    }
    if (e1) cudaEventRecord(e1, c->stream);
    c->chain = !e1;
    c->last_launches++;
    return cuda_ok(err, "fused decode launch");
}
// What the fused kernel takes, apart from its row and expert counts.
static bool decode_shape_ok(const DeviceCtx *c, int D, int I, const void *out) {
    return g_fused_decode && D % BLOCK_K == 0 && I % BLOCK_K == 0 && I <= DEC_MAX_I && c->sms >= DEC_MAX_PASS && c->sms <= 256 &&
           (reinterpret_cast<uintptr_t>(out) & 15) == 0;
}

// A grouped call of at most 8 rows (or one row through up to 16 experts, weighted and added) as one launch of
// the fused decode kernel. -> 1 done, 0 failed, -1 not this kernel's. Against split + descriptors + two GEMVs +
// SwiGLU + reduction (six stream operations) it takes 41 us instead of 95 for 8 experts of a 6144 x 2048 layer.
//   rows: per expert (y gets one row per packed row), or NULL: x is one row, y = sum_i weights[i] * expert_i(x)
static int group_decode(DeviceCtx *c, ColiCudaTensor *const *gates, ColiCudaTensor *const *ups, ColiCudaTensor *const *downs,
                        const int *rows, const float *weights, int count, int D, int I, int total, float *y, const float *x) {
    if ((rows && total > DEC_MAX_M) || !decode_shape_ok(c, D, I, y) || (reinterpret_cast<uintptr_t>(x) & 15)) return -1;
    const int mode = gates[0]->mode;
    DecPreset p;
    std::memset(&p, 0, sizeof(p));
    int off = 0;
    for (int e = 0; e < count; e++) {
        if (gates[e]->mode != mode || ups[e]->mode != mode || downs[e]->mode != mode) return -1;
        const int re = rows ? rows[e] : 1;
        for (int r0 = 0; r0 < re; r0 += 4) {
            if (p.npass == DEC_PRESET_MAX) return -1;
            auto &ps = p.pass[p.npass++];
            ps.wg = gates[e]->pk; ps.wu = ups[e]->pk; ps.wd = downs[e]->pk;
            ps.rg = gates[e]->rowscale; ps.ru = ups[e]->rowscale; ps.rd = downs[e]->rowscale;
            ps.nrows = re - r0 < 4 ? re - r0 : 4; ps.pos0 = off + r0;
            for (int i = 0; i < ps.nrows; i++) ps.rowid[i] = (unsigned char)(rows ? off + r0 + i : 0);
        }
        off += re;
    }
    p.npos = off;
    for (int i = 0; i < off; i++) { p.w[i] = weights ? weights[i] : 1.f; p.pos[i] = (unsigned char)i; }
    DecodeArgs a;
    std::memset(&a, 0, sizeof(a));
    a.rule.D = D; a.rule.I = I; a.rule.K = rows ? 1 : off; a.rule.gating = 1;
    a.M = rows ? off : 1; a.x = x; a.out = y;
    return launch_decode(c, mode, a, &p, off, &c->bq, &c->bs, &c->hq, &c->hs, &c->pd);
}

static int group_device(DeviceCtx *c, ColiCudaTensor *const *gates, ColiCudaTensor *const *ups,
                        ColiCudaTensor *const *downs, const int *rows, int count, int D, int I,
                        int total, int max_rows, int all_packed, float *y_dev, const float *x_dev,
                        const int *bcast_src /* optional: every row reads x row 0 */) {
    if (all_packed && D % 128 == 0 && I % 128 == 0 && group_tc_ok(gates, ups, downs, count, max_rows, total))
        return group_device_tc(c, gates, ups, downs, rows, count, D, I, total, y_dev, x_dev, bcast_src != nullptr);
    if (all_packed) {
        if (!bcast_src && rows) {
            const int r = group_decode(c, gates, ups, downs, rows, nullptr, count, D, I, total, y_dev, x_dev);
            if (r >= 0) return r;
        }
        int nc = pick_nc(max_rows);
        auto passes = [&](int per) { long n = 0; for (int e = 0; e < count; e++) n += ((rows ? rows[e] : 1) + per - 1) / per; return n; };
        // a few experts above 8 rows: two passes for these cost less than the slower code for 16 rows costs all of them
        while (nc > 2 && 4 * passes(2 * nc) <= 5 * (long)count) nc >>= 1;
        const int rpp = 4 * nc;
        const long npass = passes(rpp);
        const int nkb1 = D / BLOCK_K, nkb2 = I / BLOCK_K;
        const int nkp1 = pick_nkpart(nkb1, 2 * npass * (I / TILE_ROWS), c->sms);
        const int nkp2 = pick_nkpart(nkb2, npass * (D / TILE_ROWS), c->sms);
        const int nxrows = bcast_src ? 1 : total;
        if (!reserve(c, &c->bq, (size_t)nxrows * D * 2 * sizeof(__half)) ||
            !reserve(c, &c->bs, (size_t)nxrows * nkb1 * sizeof(float)) ||
            !reserve(c, &c->pg, (size_t)nkp1 * total * I * sizeof(float)) ||
            !reserve(c, &c->pu, (size_t)nkp1 * total * I * sizeof(float)) ||
            !reserve(c, &c->hq, (size_t)total * I * 2 * sizeof(__half)) ||
            !reserve(c, &c->hs, (size_t)total * nkb2 * sizeof(float)) ||
            !reserve(c, &c->pd, (size_t)nkp2 * total * D * sizeof(float))) return 0;
        HostSegs h1, h2;
        int rowid[SEG_MAX_ROWS], posid[SEG_MAX_ROWS], off = 0;
        for (int e = 0; e < count; e++) {
            int re = rows ? rows[e] : 1;
            for (int r0 = 0; r0 < re; r0 += rpp) {
                int nr = re - r0 < rpp ? re - r0 : rpp;
                for (int r = 0; r < nr; r++) { rowid[r] = bcast_src ? 0 : off + r0 + r; posid[r] = off + r0 + r; }
                add_seg(&h1, gates[e], (float *)c->pg.p, rowid, nr, off + r0, nkp1);
                add_seg(&h1, ups[e], (float *)c->pu.p, rowid, nr, off + r0, nkp1);
                add_seg(&h2, downs[e], (float *)c->pd.p, posid, nr, off + r0, nkp2);
            }
            off += re;
        }
        SegLists sl;
        const HostSegs *lists[2] = {&h1, &h2};
        if (!upload_segs(c, &sl, lists, 2, &c->segs1, total)) return 0;
        int nw = nxrows * nkb1;
        launch_pdl(c, k_prep_rows, (nw * 32 + 255) / 256, 256, 0, (__half *)c->bq.p, (float *)c->bs.p, x_dev, nxrows, D);
        c->last_launches++;
        if (!run_segs(c, sl, 0, nc, (const __half *)c->bq.p, (const float *)c->bs.p)) return 0;
        int nw2 = total * nkb2;
        launch_pdl(c, k_swiglu_prep, (nw2 * 32 + 255) / 256, 256, 0, 
            (__half *)c->hq.p, (float *)c->hs.p, (const float *)c->pg.p, (const float *)c->pu.p, nullptr,
            total, I, nkp1);
        c->last_launches++;
        if (!run_segs(c, sl, 1, nc, (const __half *)c->hq.p, (const float *)c->hs.p)) return 0;
        size_t n4 = (size_t)total * D / 4;
        launch_pdl(c, k_reduce_parts, (unsigned)((n4 + 255) / 256), 256, 0, y_dev, (const float *)c->pd.p, total, D, nkp2);
        c->last_launches++;
        return cuda_ok(cudaGetLastError(), "expert group launch");
    }
    // raw tensors: three generic matmuls and the SwiGLU per expert
    if (!reserve(c, &c->gbuf, (size_t)max_rows * I * sizeof(float)) ||
        !reserve(c, &c->ubuf, (size_t)max_rows * I * sizeof(float))) return 0;
    int off = 0;
    for (int e = 0; e < count; e++) {
        int re = rows ? rows[e] : 1;
        if (gates[e]->packed || ups[e]->packed || downs[e]->packed) return 0;
        const float *xe = bcast_src ? x_dev : x_dev + (size_t)off * D;
        int rs = bcast_src ? 1 : re;
        if (!linear_raw(c, gates[e], (float *)c->gbuf.p, xe, rs) ||
            !linear_raw(c, ups[e], (float *)c->ubuf.p, xe, rs)) return 0;
        size_t n = (size_t)rs * I;
        launch_pdl(c, k_silu_mul, (unsigned)((n + 255) / 256), 256, 0, (float *)c->gbuf.p, (const float *)c->ubuf.p, n);
        c->last_launches++;
        if (!linear_raw(c, downs[e], y_dev + (size_t)off * D, (const float *)c->gbuf.p, rs)) return 0;
        off += re;
    }
    return cuda_ok(cudaGetLastError(), "expert group launch");
}

static void count_group(DeviceCtx *c, int count, int total) {
    std::lock_guard<std::mutex> lock(g_mu);
    c->g_calls++; c->g_experts += (uint64_t)count; c->g_rows += (uint64_t)total;
}

static int group_host(ColiCudaTensor *const *gates, ColiCudaTensor *const *ups,
                      ColiCudaTensor *const *downs, const int *rows, int count, float *y,
                      const float *x, int async_issue) {
    if (!gates || !ups || !downs || !rows || !x || count < 1 || count > 64) return 0;
    if (!async_issue && !y) return 0;
    int device, D, I, total, max_rows, all_packed, any_packed;
    if (!group_shape_ok(gates, ups, downs, rows, count, &device, &D, &I, &total, &max_rows, &all_packed, &any_packed)) return 0;
    if (!all_packed && any_packed) return 0;   // a group mixing packed and raw tensors is not handled
    if (async_issue && total > 8) return 0;
    DeviceCtx *c = find_ctx(device);
    if (!c || (async_issue && c->group_pending) || !select_ctx(c)) return 0;
    size_t xb = (size_t)total * D * sizeof(float);
    // A blocking call may come between issue and take: the issued group's rows stay where no other call puts its own.
    // (The issued rows have to be pinned: up to 8, nothing waits for them here.)
    std::unique_lock<std::mutex> hold(io_mutex(c), std::defer_lock);
    if (!async_issue) hold.lock();
    if (!reserve(c, &c->x, xb) || !reserve(c, &c->y, xb)) return 0;
    float *hx, *hy;
    if (async_issue) {
        if (!reserve_pinned(c, &c->host_x, &c->host_x_cap, xb) || !reserve_pinned(c, &c->host_y, &c->host_y_cap, xb)) return 0;
        hx = c->host_x; hy = c->host_y;
    } else {
        hx = reserve_pinned(c, &c->io_x, &c->io_x_cap, xb) ? c->io_x : nullptr;
        hy = reserve_pinned(c, &c->io_y, &c->io_y_cap, xb) ? c->io_y : nullptr;
    }
    const char *pe = std::getenv("COLI_CUDA_PROFILE");
    int profile = pe && std::atoi(pe);
    cudaEvent_t ev[4] = {};
    if (profile) for (int i = 0; i < 4; i++) if (!cuda_ok(cudaEventCreate(&ev[i]), "profile event")) {
        for (int j = 0; j < i; j++) cudaEventDestroy(ev[j]);
        profile = 0; break;
    }
    if (profile) cudaEventRecord(ev[0], c->stream);
    if (!rows_in(c, c->x.p, hx, x, xb)) return 0;
    if (profile) cudaEventRecord(ev[1], c->stream);
    timing_begin(c);
    if (!group_device(c, gates, ups, downs, rows, count, D, I, total, max_rows, all_packed,
                      (float *)c->y.p, (const float *)c->x.p, nullptr)) return 0;
    timing_end(c);
    if (profile) cudaEventRecord(ev[2], c->stream);
    if (!rows_out_start(c, hy, c->y.p, xb)) return 0;
    if (profile) cudaEventRecord(ev[3], c->stream);
    if (async_issue) {
        c->group_pending = 1;
        count_group(c, count, total);
        if (profile) for (int i = 0; i < 4; i++) cudaEventDestroy(ev[i]);
        return 1;
    }
    if (!rows_out_finish(c, y, hy, c->y.p, xb)) return 0;
    if (profile && !cuda_ok(cudaStreamSynchronize(c->stream), "synchronize")) return 0;
    timing_collect(c);
    if (profile) {
        float a = 0, b = 0, d = 0;
        cudaEventElapsedTime(&a, ev[0], ev[1]); cudaEventElapsedTime(&b, ev[1], ev[2]); cudaEventElapsedTime(&d, ev[2], ev[3]);
        { std::lock_guard<std::mutex> lock(g_mu); c->g_h2d += a; c->g_kern += b; c->g_d2h += d; }
        for (int i = 0; i < 4; i++) cudaEventDestroy(ev[i]);
    }
    count_group(c, count, total);
    return 1;
}

extern "C" int coli_cuda_expert_group(ColiCudaTensor *const *gates, ColiCudaTensor *const *ups,
                                      ColiCudaTensor *const *downs, const int *rows, int count,
                                      float *y, const float *x) {
    if (fault_injected()) return 0;
    return group_host(gates, ups, downs, rows, count, y, x, 0);
}
extern "C" int coli_cuda_expert_group_issue(ColiCudaTensor *const *gates, ColiCudaTensor *const *ups,
                                            ColiCudaTensor *const *downs, const int *rows, int count,
                                            const float *x) {
    return group_host(gates, ups, downs, rows, count, nullptr, x, 1);
}
extern "C" const float *coli_cuda_expert_group_take(int device) {
    DeviceCtx *c = find_ctx(device);
    if (!c || !c->group_pending) return nullptr;
    const bool expired = c->group_pending < 0;
    c->group_pending = 0;
    if (!select_ctx(c)) return nullptr;
    if (!check_status(c) || expired) return nullptr;
    timing_collect(c);
    return c->host_y;
}
extern "C" int coli_cuda_expert_mlp(ColiCudaTensor *gate, ColiCudaTensor *up, ColiCudaTensor *down,
                                    float *y, const float *x, int S) {
    if (fault_injected()) return 0;
    if (!gate || !up || !down || !x || !y || S < 1) return 0;
    ColiCudaTensor *g[1] = {gate}, *u[1] = {up}, *d[1] = {down};
    int rows[1] = {S};
    int device, D, I, total, max_rows, all_packed, any_packed;
    if (!group_shape_ok(g, u, d, rows, 1, &device, &D, &I, &total, &max_rows, &all_packed, &any_packed)) return 0;
    if (!all_packed && any_packed) return 0;
    DeviceCtx *c = find_ctx(device);
    if (!select_ctx(c)) return 0;
    std::lock_guard<std::mutex> hold(io_mutex(c));
    size_t xb = (size_t)S * D * sizeof(float);
    const float *xd = io_in(c, x, xb, all_packed && S > DEC_MAX_M);
    float *yd = io_out(c, xb);
    if (!xd || !yd) return 0;
    timing_begin(c);
    if (!group_device(c, g, u, d, rows, 1, D, I, total, max_rows, all_packed, yd, xd, nullptr)) return 0;
    timing_end(c);
    if (!io_finish(c, y, yd, xb)) return 0;
    timing_collect(c);
    return 1;
}
// The reference's W4A16 tensor-core shared-expert call (c/backend_cuda.cu:1457-1484)
// is the same function with per-row int4 tensors required.
extern "C" int coli_cuda_shared_mlp_w4a16(ColiCudaTensor *gate, ColiCudaTensor *up, ColiCudaTensor *down,
                                          float *y, const float *x, int S) {
    if (!gate || !up || !down || gate->fmt != 2 || up->fmt != 2 || down->fmt != 2) return 0;
    return coli_cuda_expert_mlp(gate, up, down, y, x, S);
}

// ---------------------------------------------------------------------------
// Attention / RoPE entry points: outside this backend's path ("not offloaded").
// ---------------------------------------------------------------------------
extern "C" int coli_cuda_attention_absorb(ColiCudaTensor *, float *, const float *, const float *, const float *, int, int, int, int, int, int, float) { return 0; }
extern "C" int coli_cuda_attention_absorb_batch(ColiCudaTensor *, float *, const float *, const float *, const float *, int, int, int, int, int, int, int, float) { return 0; }
extern "C" int coli_cuda_attention_project_batch(ColiCudaTensor *, ColiCudaTensor *, float *, const float *, const float *, const float *, int, int, int, int, int, int, int, float) { return 0; }
extern "C" int coli_cuda_attention_project_ragged(ColiCudaTensor *, ColiCudaTensor *, float *, const float *, const void *const *, const float *const *, const float *const *, const int *, int, int, int, int, int, int, int, float) { return 0; }
extern "C" int coli_cuda_attention_project_batch_dev(ColiCudaTensor *, ColiCudaTensor *, float *, const float *, const float *, const float *, int, int, int, int, int, int, int, float) { return 0; }
extern "C" int coli_cuda_attention_absorb_batch_dev(ColiCudaTensor *, float *, const float *, const float *, const float *, int, int, int, int, int, int, int, float) { return 0; }
extern "C" int coli_cuda_attention_absorb_kvdev(ColiCudaTensor *, float *, const float *, const float *, const float *, int, int, int, int, int, int, float) { return 0; }
extern "C" int coli_cuda_attention_project_batch_dev_out(ColiCudaTensor *, ColiCudaTensor *, float *, const float *, const float *, const float *, int, int, int, int, int, int, int, float) { return 0; }

// ---------------------------------------------------------------------------
// Resident-pipeline primitives
// ---------------------------------------------------------------------------
extern "C" float *coli_cuda_pipe_scratch(int device, int slot, size_t bytes) {
    DeviceCtx *c = find_ctx(device);
    if (slot < 0 || slot >= 27 || !select_ctx(c)) return nullptr;
    if (!reserve(c, &c->pipe[slot], bytes)) return nullptr;
    return (float *)c->pipe[slot].p;
}
extern "C" void *coli_cuda_pipe_alloc(int device, size_t bytes) {
    DeviceCtx *c = find_ctx(device);
    if (!select_ctx(c)) return nullptr;
    void *p = nullptr;
    if (!cuda_ok(cudaMalloc(&p, bytes), "pipe alloc")) return nullptr;
    return p;
}
extern "C" void coli_cuda_pipe_free(int device, void *p) {
    DeviceCtx *c = find_ctx(device);
    if (!p || !select_ctx(c)) return;
    cudaFree(p);
}
// Peer access to pipe_alloc'ed buffers across processes (one process per GPU): the owner
// exports a 64-byte handle, another process opens it and gets a pointer into the owner's HBM
// that this process's copies and kernels can use (NVLink / NVSwitch path).
extern "C" int coli_cuda_pipe_ipc_export(int device, void *dev_ptr, void *handle64) {
    DeviceCtx *c = find_ctx(device);
    if (!dev_ptr || !handle64 || !select_ctx(c)) return 0;
    static_assert(sizeof(cudaIpcMemHandle_t) == 64, "handle size");
    cudaIpcMemHandle_t h;
    if (!cuda_ok(cudaIpcGetMemHandle(&h, dev_ptr), "ipc export")) return 0;
    std::memcpy(handle64, &h, sizeof(h));
    return 1;
}
extern "C" void *coli_cuda_pipe_ipc_open(int device, const void *handle64) {
    DeviceCtx *c = find_ctx(device);
    if (!handle64 || !select_ctx(c)) return nullptr;
    cudaIpcMemHandle_t h;
    std::memcpy(&h, handle64, sizeof(h));
    void *p = nullptr;
    if (!cuda_ok(cudaIpcOpenMemHandle(&p, h, cudaIpcMemLazyEnablePeerAccess), "ipc open")) return nullptr;
    return p;
}
extern "C" int coli_cuda_pipe_ipc_close(int device, void *peer_ptr) {
    DeviceCtx *c = find_ctx(device);
    if (!peer_ptr || !select_ctx(c)) return 0;
    return cuda_ok(cudaIpcCloseMemHandle(peer_ptr), "ipc close");
}
// Asynchronous device-to-device copy (either side may be a peer pointer) on `stream`
// (a cudaStream_t; NULL = the backend's stream). Large copies run on the copy engines, beside
// whatever kernels are resident.
extern "C" int coli_cuda_pipe_copy_async(int device, void *dst, const void *src, size_t bytes, void *stream) {
    DeviceCtx *c = find_ctx(device);
    if (!select_ctx(c)) return 0;
    if (bytes == 0) return 1;
    if (!dst || !src) return 0;
    return cuda_ok(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToDevice,
                                   stream ? static_cast<cudaStream_t>(stream) : c->stream), "pipe copy");
}
// Both run on the legacy stream, which waits for, and is waited for by, the backend's stream and every other
// blocking stream of the device. An upload returns when the source has been read, a download when dst is filled; a
// download behind a kernel whose wait has expired leaves dst alone and returns 0, like every call that waits.
extern "C" int coli_cuda_pipe_upload(int device, void *dst, const void *src, size_t bytes) {
    DeviceCtx *c = find_ctx(device);
    if ((bytes && (!dst || !src)) || !select_ctx(c)) return 0;       // (the host reads src here, the runtime does not look at it first)
    return cuda_ok(upload_staged(ring_of(c), dst, src, bytes, cudaStreamLegacy), "pipe upload");
}
extern "C" int coli_cuda_pipe_download(int device, const void *src, void *dst, size_t bytes) {
    DeviceCtx *c = find_ctx(device);
    if ((bytes && (!dst || !src)) || !select_ctx(c)) return 0;
    bool ready = true;
    return cuda_ok(download_staged(ring_of(c), dst, src, bytes, cudaStreamLegacy, [c, &ready] { return ready = kernels_ok(c) != 0; }),
                   "pipe download") && ready;
}
extern "C" int coli_cuda_pipe_rmsnorm_s(int device, float *y_dev, const float *x_dev, const float *w_dev,
                                        int S, int D, float eps, int xstride, int ystride) {
    if (fault_injected()) return 0;
    DeviceCtx *c = find_ctx(device);
    if (S < 1 || D < 1 || xstride < D || ystride < D || !select_ctx(c)) return 0;
    launch_pdl(c, k_rmsnorm, S, RMSNORM_THREADS, 0, y_dev, x_dev, w_dev, D, eps, xstride, ystride);
    return cuda_ok(cudaGetLastError(), "pipe rmsnorm");
}
extern "C" int coli_cuda_pipe_rmsnorm(int device, float *y_dev, const float *x_dev, const float *w_dev,
                                      int S, int D, float eps) {
    return coli_cuda_pipe_rmsnorm_s(device, y_dev, x_dev, w_dev, S, D, eps, D, D);
}
extern "C" int coli_cuda_pipe_silu_mul(int device, float *gate_dev, const float *up_dev, size_t n) {
    if (fault_injected()) return 0;
    DeviceCtx *c = find_ctx(device);
    if (!n || !select_ctx(c)) return 0;
    launch_pdl(c, k_silu_mul, (unsigned)((n + 255) / 256), 256, 0, gate_dev, up_dev, n);
    return cuda_ok(cudaGetLastError(), "pipe silu mul");
}
extern "C" int coli_cuda_pipe_rope(int device, float *v_dev, const int *pos_dev, int rows, int stride, int offset,
                                   int R, int heads, float theta) {
    if (fault_injected()) return 0;
    DeviceCtx *c = find_ctx(device);
    if (!v_dev || !pos_dev || rows < 1 || R < 2 || R > 256 || heads < 1 || !select_ctx(c)) return 0;
    launch_pdl(c, k_rope_rows, rows, 128, 0, v_dev, pos_dev, 0, stride, offset, R, heads, theta);
    c->last_launches++;
    return cuda_ok(cudaGetLastError(), "pipe rope");
}
extern "C" int coli_cuda_pipe_rope_base(int device, float *v_dev, int pos_base, int rows, int stride, int offset,
                                        int R, int heads, float theta) {
    if (fault_injected()) return 0;
    DeviceCtx *c = find_ctx(device);
    if (!v_dev || rows < 1 || R < 2 || R > 256 || heads < 1 || !select_ctx(c)) return 0;
    launch_pdl(c, k_rope_rows, rows, 128, 0, v_dev, nullptr, pos_base, stride, offset, R, heads, theta);
    c->last_launches++;
    return cuda_ok(cudaGetLastError(), "pipe rope");
}
extern "C" int coli_cuda_pipe_add(int device, float *x_dev, const float *t_dev, size_t n) {
    if (fault_injected()) return 0;
    DeviceCtx *c = find_ctx(device);
    if (!n || !select_ctx(c)) return 0;
    launch_pdl(c, k_add, (unsigned)((n + 255) / 256), 256, 0, x_dev, t_dev, n);
    return cuda_ok(cudaGetLastError(), "pipe add");
}
extern "C" int coli_cuda_pipe_rows_add(int device, float *x_dev, const float *partial_dev,
                                       const int *rows_dev, int nrows, int D) {
    if (fault_injected()) return 0;
    DeviceCtx *c = find_ctx(device);
    if (nrows < 1 || D < 1 || !select_ctx(c)) return 0;
    launch_pdl(c, k_rows_add, nrows, 256, 0, x_dev, partial_dev, rows_dev, D);
    return cuda_ok(cudaGetLastError(), "pipe rows add");
}
extern "C" int coli_cuda_pipe_copy2d(int device, float *dst, int dpitch, const float *src, int spitch,
                                     int width, int height) {
    DeviceCtx *c = find_ctx(device);
    if (!select_ctx(c)) return 0;
    return cuda_ok(cudaMemcpy2DAsync(dst, (size_t)dpitch * 4, src, (size_t)spitch * 4, (size_t)width * 4,
                                     height, cudaMemcpyDeviceToDevice, c->stream), "pipe copy2d");
}
extern "C" int coli_cuda_pipe_peer_copy(int dst_dev, float *dst, int src_dev, const float *src, size_t bytes) {
    if (!dst || !src) return 0;
    DeviceCtx *cd = find_ctx(dst_dev), *cs = find_ctx(src_dev);
    if (!cd || !cs) return 0;
    if (!select_ctx(cs) || !cuda_ok(cudaStreamSynchronize(cs->stream), "peer copy sync")) return 0;
    if (dst_dev == src_dev)
        return cuda_ok(cudaMemcpy(dst, src, bytes, cudaMemcpyDeviceToDevice), "pipe intra copy");
    if (!select_ctx(cd) || !cuda_ok(cudaStreamSynchronize(cd->stream), "peer copy sync")) return 0;
    return cuda_ok(cudaMemcpyPeer(dst, dst_dev, src, src_dev, bytes), "pipe peer copy");
}
extern "C" int coli_cuda_pipe_sync(int device) {
    DeviceCtx *c = find_ctx(device);
    if (!select_ctx(c)) return 0;
    return cuda_ok(cudaDeviceSynchronize(), "pipe sync") && kernels_ok(c);
}
extern "C" int coli_cuda_expire_wait(int device) {
    DeviceCtx *c = find_ctx(device);
    if (!select_ctx(c)) return 0;
    k_expire_wait<<<1, 1, 0, c->stream>>>(c->status);
    return cuda_ok(cudaGetLastError(), "expire wait");
}

static void launch_router(DeviceCtx *c, float *logits, const float *x, const float *w, int M, int D, int E) {
    const int n = M * E;
    const bool aligned = D % 4 == 0 && ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w)) & 15) == 0;
    // up to two waves of CTAs: few outputs each, for the shortest chain time; beyond: more chains per SM
    if (aligned && n <= 16 * 2 * c->sms)
        launch_pdl(c, k_router_logits<16, 256>, (n + 15) / 16, 64, router_smem(16, 256), logits, x, w, M, D, E, c->status);
    else if (aligned)
        launch_pdl(c, k_router_logits<64, 64>, (n + 63) / 64, 96, router_smem(64, 64), logits, x, w, M, D, E, c->status);
    else
        launch_pdl(c, k_router_logits_any, (n + 63) / 64, 64, 0, logits, x, w, M, D, E);
}

extern "C" int coli_cuda_pipe_router(int device, const float *x_dev, const void *rw_dev, const void *rb_dev,
                                     int D, int E, int Ksel, float topp, int norm_topk, float routed_scale,
                                     int *idx_host, float *w_host, int *keff_host) {
    DeviceCtx *c = find_ctx(device);
    if (!x_dev || !rw_dev || !rb_dev || D < 1 || E < 1 || E > ROUTE_MAX_E || Ksel < 1 || Ksel > ROUTE_MAX_K ||
        Ksel > E || !idx_host || !w_host || !keff_host || !select_ctx(c)) return 0;
    // the selection goes straight to pinned memory where there is some: idx [Ksel] | w [Ksel] | keff
    const size_t sel = (size_t)Ksel * 8 + 4;
    std::lock_guard<std::mutex> hold(io_mutex(c));
    if (!reserve(c, &c->misc, (size_t)E * 4 + sel)) return 0;
    const bool pinned = reserve_pinned(c, &c->io_y, &c->io_y_cap, sel);
    float *logits = (float *)c->misc.p;
    int *idx = pinned ? (int *)c->io_y : (int *)(logits + E), *keff = idx + 2 * Ksel;
    float *w = (float *)(idx + Ksel);
    RouteRule rule{D, 0, E, Ksel, 1, norm_topk, routed_scale, topp};
    launch_router(c, logits, x_dev, (const float *)rw_dev, 1, D, E);
    launch_pdl(c, k_route_topk, route_grid(1), ROUTE_THREADS, route_smem(E), logits, (const float *)rb_dev, rule, 1, idx, w, keff);
    if (!cuda_ok(cudaGetLastError(), "pipe router launch") || !check_status(c)) return 0;
    int few[2 * ROUTE_MAX_K + 1];
    if (!pinned && !rows_out_finish(c, few, nullptr, idx, sel)) return 0;
    const int *got = pinned ? idx : few;
    std::memcpy(idx_host, got, (size_t)Ksel * 4);
    std::memcpy(w_host, got + Ksel, (size_t)Ksel * 4);
    std::memcpy(keff_host, got + 2 * Ksel, 4);
    return 1;
}

extern "C" int coli_cuda_expert_group_resident_issue(ColiCudaTensor *const *gates, ColiCudaTensor *const *ups,
                                                     ColiCudaTensor *const *downs, const float *weights,
                                                     int count, int home_device, const float *x_src_dev,
                                                     float *partial_slot_dev) {
    if (!gates || !ups || !downs || !weights || count < 1 || count > 64 || !x_src_dev || !partial_slot_dev) return 0;
    int device, D, I, total, max_rows, all_packed, any_packed;
    if (!group_shape_ok(gates, ups, downs, nullptr, count, &device, &D, &I, &total, &max_rows, &all_packed, &any_packed)) return 0;
    if (!all_packed && any_packed) return 0;
    DeviceCtx *c = find_ctx(device), *home = find_ctx(home_device);
    if (!home || !select_ctx(c)) return 0;
    if (device == home_device && all_packed) {
        const int r = group_decode(c, gates, ups, downs, nullptr, weights, count, D, I, total, partial_slot_dev, x_src_dev);
        if (r == 0) return 0;
        if (r > 0) return cuda_ok(cudaEventRecord(c->ev_done, c->stream), "resident event record");
    }
    // fixed capacities (64 experts) so that a re-issue never reallocates under queued work
    if (!reserve(c, &c->x, (size_t)64 * D * sizeof(float)) || !reserve(c, &c->y, (size_t)64 * D * sizeof(float)) ||
        !reserve(c, &c->misc, (size_t)(D + 64) * sizeof(float) + 4096)) return 0;
    float *partial_local = (float *)c->misc.p, *w_dev = partial_local + D;
    c->chain = false;
    // by way of the stack: a pageable source is captured before the call returns, the caller's own memory may be pinned
    float w_host[64];
    std::memcpy(w_host, weights, (size_t)count * sizeof(float));
    if (!cuda_ok(cudaMemcpyAsync(w_dev, w_host, (size_t)count * sizeof(float), cudaMemcpyHostToDevice, c->stream), "resident group weights")) return 0;
    cudaError_t e = device == home_device
        ? cudaMemcpyAsync(c->x.p, x_src_dev, (size_t)D * sizeof(float), cudaMemcpyDeviceToDevice, c->stream)
        : cudaMemcpyPeerAsync(c->x.p, device, x_src_dev, home_device, (size_t)D * sizeof(float), c->stream);
    if (!cuda_ok(e, "resident group x copy")) return 0;
    int one = 1;
    if (!group_device(c, gates, ups, downs, nullptr, count, D, I, total, 1, all_packed, (float *)c->y.p,
                      (const float *)c->x.p, &one)) return 0;
    launch_pdl(c, k_weighted_sum_rows, 48, 256, 0, partial_local, (const float *)c->y.p, w_dev, count, D);
    e = device == home_device
        ? cudaMemcpyAsync(partial_slot_dev, partial_local, (size_t)D * sizeof(float), cudaMemcpyDeviceToDevice, c->stream)
        : cudaMemcpyPeerAsync(partial_slot_dev, home_device, partial_local, device, (size_t)D * sizeof(float), c->stream);
    if (!cuda_ok(e, "resident partial copy")) return 0;
    if (!cuda_ok(cudaEventRecord(c->ev_done, c->stream), "resident event record")) return 0;
    return cuda_ok(cudaGetLastError(), "resident group launch");
}
extern "C" int coli_cuda_expert_group_resident_take(int home_device, const int *devices, int n_issued,
                                                    float *slots_dev, float *acc_dev, int D) {
    if (n_issued < 1 || !devices || !slots_dev || !acc_dev || D < 1) return 0;
    DeviceCtx *home = find_ctx(home_device);
    if (!select_ctx(home)) return 0;
    for (int i = 0; i < n_issued; i++) {
        DeviceCtx *src = find_ctx(devices[i]);
        if (!src) return 0;
        if (!cuda_ok(cudaStreamWaitEvent(home->stream, src->ev_done, 0), "resident take wait")) return 0;
    }
    launch_pdl(home, k_sum_slots, 48, 256, 0, acc_dev, slots_dev, n_issued, D);
    return cuda_ok(cudaGetLastError(), "resident take reduce");
}

#include "moe_layer.cuh"

// Device-pointer form of coli_cuda_expert_group (additive): x_dev and y_dev hold
// sum(rows) consecutive [D] rows in call order on the tensors' device; experts with
// zero rows are allowed and skipped; count is not limited to 64. Enqueues on the
// backend's stream and returns. Used by the expert-parallel layer, whose rows arrive
// from other ranks already in device memory.
extern "C" int coli_cuda_expert_group_dev(ColiCudaTensor *const *gates, ColiCudaTensor *const *ups,
                                          ColiCudaTensor *const *downs, const int *rows, int count,
                                          float *y_dev, const float *x_dev) {
    if (fault_injected()) return 0;
    if (!gates || !ups || !downs || !rows || !x_dev || !y_dev || count < 1) return 0;
    std::vector<ColiCudaTensor *> g, u, d;
    std::vector<int> r;
    for (int e = 0; e < count; e++) {
        if (rows[e] < 0) return 0;
        if (rows[e] == 0) continue;
        g.push_back(gates[e]); u.push_back(ups[e]); d.push_back(downs[e]); r.push_back(rows[e]);
    }
    if (g.empty()) return 1;
    int device, D, I, total, max_rows, all_packed, any_packed;
    if (!group_shape_ok(g.data(), u.data(), d.data(), r.data(), (int)g.size(), &device, &D, &I, &total,
                        &max_rows, &all_packed, &any_packed)) return 0;
    if (!all_packed && any_packed) return 0;
    if (all_packed && !rows_aligned("expert group", x_dev, y_dev)) return 0;
    DeviceCtx *c = find_ctx(device);
    if (!select_ctx(c)) return 0;
    timing_begin(c);
    int ok = group_device(c, g.data(), u.data(), d.data(), r.data(), (int)g.size(), D, I, total, max_rows,
                          all_packed, y_dev, x_dev, nullptr);
    timing_end(c);
    if (ok) count_group(c, (int)g.size(), total);
    return ok;
}

// idx_dev[s] = argmax of row s of x_dev [S, N] with the engine's first-largest rule.
extern "C" int coli_cuda_pipe_argmax(int device, int *idx_dev, const float *x_dev, int S, int N) {
    DeviceCtx *c = find_ctx(device);
    if (!idx_dev || !x_dev || S < 1 || N < 1 || !select_ctx(c)) return 0;
    launch_pdl(c, k_argmax_rows, S * ARGMAX_CLUSTER, 1024, 0, idx_dev, x_dev, N);
    c->last_launches++;
    return cuda_ok(cudaGetLastError(), "argmax launch");
}

// Weighted combine of an expert-parallel layer on device buffers: out[s] = sum over the
// first keff[s] selections of w[s,kk] * y[entry_of[s,kk]], then + shared[s] when given.
// entry_of and keff are 64-bit integers. Enqueues on the backend's stream.
extern "C" int coli_cuda_moe_combine_dev(int device, float *out_dev, const float *y_dev,
                                         const long long *entry_of_dev, const float *w_dev,
                                         const long long *keff_dev, const float *shared_dev, int M, int K,
                                         int D) {
    DeviceCtx *c = find_ctx(device);
    if (!out_dev || !entry_of_dev || !w_dev || !keff_dev || M < 1 || K < 1 || D < 4 || D % 4 || !select_ctx(c)) return 0;
    if ((reinterpret_cast<uintptr_t>(out_dev) | reinterpret_cast<uintptr_t>(y_dev) | reinterpret_cast<uintptr_t>(shared_dev)) & 15) return 0;
    size_t n4 = (size_t)M * D / 4;
    launch_pdl(c, k_combine_rows, (unsigned)((n4 + 255) / 256), 256, 0, out_dev, y_dev, entry_of_dev, w_dev, keff_dev,
                                                                     shared_dev, M, K, D);
    c->last_launches++;
    return cuda_ok(cudaGetLastError(), "combine launch");
}

// ---------------------------------------------------------------------------
// Expert-parallel layer, device side (additive; the reference has no collective path:
// it pins whole experts to devices and moves rows host -> device per call,
// c/colibri.c:4819-4839, 8367-8417). One process per GPU; the host issues the NCCL
// all-to-all exchanges between these calls. All work goes to the backend's stream.
// ---------------------------------------------------------------------------
// Plan + pack. From this rank's routing (idx [m,K], keff [m]) and the expert placement
// (dest[e] = owning rank, slot[e] = index among that rank's experts; G ranks, `slots`
// experts per rank at most) it produces, on the device:
//   counts [G*slots]   live entries per (destination rank, local expert)
//   entry_of [m*K]     position of every live entry in the send buffer, -1 for dead ones
//   send [n, D]        the rows in (destination rank, local expert, row order), as bf16
//                      (payload_bf16; *inexact is raised if a value is not exact in bf16,
//                      which would change results: the caller must then use f32) or f32
// The send buffer must hold m*K rows.
extern "C" int coli_cuda_ep_plan_dev(int device, const float *x_dev, int m, int D, int K, const int *idx_dev,
                                     const int *keff_dev, const int *dest_dev, const int *slot_dev, int E,
                                     int G, int slots, int payload_bf16, int *counts_dev, int *entry_of_dev,
                                     void *send_dev, int *inexact_dev) {
    if (fault_injected()) return 0;
    DeviceCtx *c = find_ctx(device);
    const int nb = G * slots;
    if (!x_dev || !idx_dev || !keff_dev || !dest_dev || !slot_dev || !counts_dev || !entry_of_dev || !send_dev ||
        !inexact_dev || m < 1 || K < 1 || K > 31 || E < 1 || G < 1 || slots < 1 || D < 4 || D % 4 || !rows_aligned("ep plan", x_dev) ||
        !rows_aligned("ep plan", send_dev, nullptr, payload_bf16 ? 8 : 16) || !select_ctx(c)) return 0;
    if (!reserve(c, &c->ep_ws, ((size_t)nb + 1 + (size_t)m * K) * sizeof(int))) return 0;
    int *off = static_cast<int *>(c->ep_ws.p), *row_of = off + nb + 1;
    c->chain = false;
    if (!cuda_ok(cudaMemsetAsync(counts_dev, 0, (size_t)nb * sizeof(int), c->stream), "ep plan") ||
        !cuda_ok(cudaMemsetAsync(entry_of_dev, 0xFF, (size_t)m * K * sizeof(int), c->stream), "ep plan")) return 0;
    const int n = m * K;
    launch_pdl(c, k_ep_count, (n + 255) / 256, 256, 0, counts_dev, idx_dev, keff_dev, dest_dev, slot_dev, m, K, slots);
    launch_pdl(c, k_ep_offsets, 1, 256, 0, off, counts_dev, nb);
    launch_pdl(c, k_ep_place, E, EP_PLACE_WARPS * 32, 0, entry_of_dev, row_of, off, idx_dev, keff_dev, dest_dev, slot_dev, m, K, slots);
    if (payload_bf16) launch_pdl(c, k_ep_gather<true>, n, 256, 0, send_dev, x_dev, row_of, off + nb, D, inexact_dev);
    else launch_pdl(c, k_ep_gather<false>, n, 256, 0, send_dev, x_dev, row_of, off + nb, D, inexact_dev);
    c->last_launches += 4;
    return cuda_ok(cudaGetLastError(), "ep plan launch");
}

// Expert FFN over the rows this rank received. x_dev holds them in receive order (source
// rank, local expert, row order), recv_counts (host) [nsrc][nslots] says how many; the
// results go to y_dev [n, D] f32 in the same receive order, ready to be sent back. With the
// tensor-core kernel the regrouping per expert is a gather in its activation preparation and
// a scatter in its read-back, so no row is copied; the streaming kernels get permuted copies.
extern "C" int coli_cuda_ep_expert_group_dev(ColiCudaTensor *const *gates, ColiCudaTensor *const *ups,
                                             ColiCudaTensor *const *downs, int nslots, const int *recv_counts,
                                             int nsrc, float *y_dev, const void *x_dev, int x_bf16) {
    if (fault_injected()) return 0;
    if (!gates || !ups || !downs || !recv_counts || nslots < 1 || nsrc < 1 || !y_dev || !x_dev) return 0;
    std::vector<int> seg_start((size_t)nsrc * nslots);
    int n = 0;
    for (int s = 0; s < nsrc; s++)
        for (int e = 0; e < nslots; e++) {
            if (recv_counts[s * nslots + e] < 0) return 0;
            seg_start[(size_t)s * nslots + e] = n; n += recv_counts[s * nslots + e];
        }
    if (n == 0) return 1;
    std::vector<ColiCudaTensor *> g, u, d;
    std::vector<int> rows, rowmap;
    rowmap.reserve(n);
    for (int e = 0; e < nslots; e++) {
        int re = 0;
        for (int s = 0; s < nsrc; s++) {
            const int cnt = recv_counts[s * nslots + e], st = seg_start[(size_t)s * nslots + e];
            for (int r = 0; r < cnt; r++) rowmap.push_back(st + r);
            re += cnt;
        }
        if (re) { g.push_back(gates[e]); u.push_back(ups[e]); d.push_back(downs[e]); rows.push_back(re); }
    }
    int device, D, I, total, max_rows, all_packed, any_packed;
    if (!group_shape_ok(g.data(), u.data(), d.data(), rows.data(), (int)g.size(), &device, &D, &I, &total,
                        &max_rows, &all_packed, &any_packed)) return 0;
    if (!all_packed && any_packed) return 0;
    // (raw experts may have D % 4 != 0, which the permuted copies do not take)
    if (D % 4 || !rows_aligned("ep expert group", y_dev) || !rows_aligned("ep expert group", x_dev, nullptr, x_bf16 ? 4 : 8)) return 0;
    DeviceCtx *c = find_ctx(device);
    if (!select_ctx(c)) return 0;
    timing_begin(c);
    int ok;
    // rows that start off the boundaries of the other path's loads: the tensor cores' preparation reads them, at any mean
    const bool odd = (reinterpret_cast<uintptr_t>(x_dev) & (x_bf16 ? 7 : 15)) != 0;
    if (all_packed && D % 128 == 0 && I % 128 == 0 &&
        group_tc_ok(g.data(), u.data(), d.data(), (int)g.size(), max_rows, total, odd)) {
        ok = group_device_tc(c, g.data(), u.data(), d.data(), rows.data(), (int)g.size(), D, I, total, y_dev, x_dev, 0,
                             rowmap.data(), x_bf16);
    } else {
        if (!rows_aligned("ep expert group", x_dev, nullptr, x_bf16 ? 8 : 16)) return 0;
        if (!reserve(c, &c->ep_ws, ((size_t)n) * sizeof(int)) || !reserve(c, &c->ep_x, (size_t)n * D * sizeof(float)) ||
            !reserve(c, &c->ep_y, (size_t)n * D * sizeof(float))) return 0;
        int *map_dev = static_cast<int *>(c->ep_ws.p);
        c->chain = false;
        if (!cuda_ok(cudaMemcpyAsync(map_dev, rowmap.data(), (size_t)n * sizeof(int), cudaMemcpyHostToDevice, c->stream), "ep row map")) return 0;
        if (x_bf16) launch_pdl(c, k_ep_permute<true, false>, n, 256, 0, (float *)c->ep_x.p, x_dev, map_dev, n, D);
        else launch_pdl(c, k_ep_permute<false, false>, n, 256, 0, (float *)c->ep_x.p, x_dev, map_dev, n, D);
        c->last_launches++;
        ok = group_device(c, g.data(), u.data(), d.data(), rows.data(), (int)g.size(), D, I, total, max_rows, all_packed,
                          (float *)c->ep_y.p, (const float *)c->ep_x.p, nullptr);
        if (ok) {
            launch_pdl(c, k_ep_permute<false, true>, n, 256, 0, y_dev, c->ep_y.p, map_dev, n, D);
            c->last_launches++;
            ok = cuda_ok(cudaGetLastError(), "ep permute launch");
        }
    }
    timing_end(c);
    if (ok) count_group(c, (int)g.size(), total);
    return ok;
}

// out[s] = sum over the first keff[s] selections of w[s,kk] * y[entry_of[s,kk]] (+ shared[s]):
// y holds the answers in send-buffer order, entry_of is the plan's table.
extern "C" int coli_cuda_ep_combine_dev(int device, float *out_dev, const float *y_dev, const int *entry_of_dev,
                                        const float *w_dev, const int *keff_dev, const float *shared_dev, int m,
                                        int K, int D) {
    DeviceCtx *c = find_ctx(device);
    if (!out_dev || !y_dev || !entry_of_dev || !w_dev || !keff_dev || m < 1 || K < 1 || D < 4 || D % 4 || !select_ctx(c)) return 0;
    if ((reinterpret_cast<uintptr_t>(out_dev) | reinterpret_cast<uintptr_t>(y_dev) | reinterpret_cast<uintptr_t>(shared_dev)) & 15) return 0;
    const size_t n4 = (size_t)m * D / 4;
    launch_pdl(c, k_ep_combine, (unsigned)((n4 + 255) / 256), 256, 0, out_dev, y_dev, entry_of_dev, w_dev, keff_dev,
                                                                   shared_dev, m, K, D);
    c->last_launches++;
    return cuda_ok(cudaGetLastError(), "ep combine launch");
}

// ---------------------------------------------------------------------------
// Allocation-free matmul on device pointers (no counterpart in the reference).
//
// Some callers may not allocate device memory when they reach the backend: an
// engine that has already handed every free byte of HBM to its KV cache and
// expert tier (a cudaMalloc would fail or force an eviction), or a decode loop
// that cannot afford the device-wide synchronisation a cudaMalloc / cudaFree
// implies. coli_cuda_pipe_gemm normally grows per-device workspaces on demand;
// this variant keeps all of its scratch (segment descriptors, the fp16 hi/lo
// split of the activations, their block scales and the partial sums of the
// contraction slices) in one fixed file-scope device array instead.
//
// The array is per device (every device that loads this library holds its
// 8 MiB until the process exits) and is shared by all calls: it keeps whatever
// the last call left there (nothing in it has to start at zero: every word a
// call reads it has written first), and two calls that overlap on the GPU, e.g.
// from two host threads or on two streams, race on it. The first call on a
// device looks up the array's device address (cudaGetSymbolAddress, with that
// device current); make that first call before any stream capture begins.
// ---------------------------------------------------------------------------
#define NOALLOC_SCRATCH_BYTES (8u << 20)
#define NOALLOC_MAX_ROWS 32
#define NOALLOC_HEADER_BYTES 4096          // one segment descriptor + the control block
#define NOALLOC_SCALE_BYTES 16384          // inverse block scales: rows * (I/128) floats
static __device__ __align__(256) unsigned char g_noalloc_scratch[NOALLOC_SCRATCH_BYTES];
static unsigned char *g_noalloc_dev[64];   // device address of the array, per CUDA ordinal

extern "C" int coli_cuda_pipe_gemm_noalloc(ColiCudaTensor *t, float *y_dev, const float *x_dev, int S) {
    if (fault_injected()) return 0;
    if (!t || !y_dev || !x_dev || S < 1 || !rows_aligned("pipe_gemm_noalloc", x_dev, y_dev)) return 0;
    DeviceCtx *c = find_ctx(t->device);
    if (!select_ctx(c)) return 0;
    if (!t->packed) {
        std::fprintf(stderr, "[CUDA] pipe_gemm_noalloc: tensor is not in the packed layout "
                             "(needs fmt 2/4/7, I %% 128 == 0, O %% 32 == 0)\n");
        return 0;
    }
    if (t->device < 0 || t->device >= 64) return 0;
    if (S > NOALLOC_MAX_ROWS) {
        std::fprintf(stderr, "[CUDA] pipe_gemm_noalloc: %d rows exceed the limit of %d\n", S, NOALLOC_MAX_ROWS);
        return 0;
    }
    const int nkb = t->I / BLOCK_K;
    const int nc = pick_nc(S);
    const size_t bs_bytes = (size_t)S * nkb * sizeof(float);
    const size_t bq_bytes = (size_t)S * t->I * 2 * sizeof(__half);
    auto scratch = [&](int k) { return NOALLOC_HEADER_BYTES + NOALLOC_SCALE_BYTES + bq_bytes + (size_t)k * S * t->O * sizeof(float); };
    int nkpart = pick_nkpart(nkb, (long)(t->O / TILE_ROWS), c->sms);
    while (nkpart > 1 && (nkb % nkpart || scratch(nkpart) > NOALLOC_SCRATCH_BYTES)) nkpart--;     // the partial sums have to fit
    const size_t need = scratch(nkpart);
    if (bs_bytes > NOALLOC_SCALE_BYTES || need > NOALLOC_SCRATCH_BYTES) {
        std::fprintf(stderr, "[CUDA] pipe_gemm_noalloc: S=%d I=%d O=%d needs %zu bytes of scratch, the fixed "
                             "array holds %u\n", S, t->I, t->O, need, NOALLOC_SCRATCH_BYTES);
        return 0;
    }
    if (!g_noalloc_dev[t->device]) {
        // once per device, with that device current (select_ctx above)
        void *p = nullptr;
        if (!cuda_ok(cudaGetSymbolAddress(&p, g_noalloc_scratch), "static scratch address") || !p) return 0;
        g_noalloc_dev[t->device] = static_cast<unsigned char *>(p);
    }
    unsigned char *base = g_noalloc_dev[t->device];
    GemvSeg *seg_dev = reinterpret_cast<GemvSeg *>(base);
    GemvCtl *ctl_dev = reinterpret_cast<GemvCtl *>(base + NOALLOC_HEADER_BYTES - 256);
    float *bs_dev = reinterpret_cast<float *>(base + NOALLOC_HEADER_BYTES);
    __half *bq_dev = reinterpret_cast<__half *>(base + NOALLOC_HEADER_BYTES + NOALLOC_SCALE_BYTES);
    float *pd_dev = reinterpret_cast<float *>(base + NOALLOC_HEADER_BYTES + NOALLOC_SCALE_BYTES + bq_bytes);
    // descriptor and control block from the stack (pageable source: captured before the call returns)
    struct { GemvSeg seg; } hs;
    GemvCtl hc;
    std::memset(&hs, 0, sizeof(hs));
    hs.seg.w = t->pk; hs.seg.rowscale = t->rowscale; hs.seg.out = pd_dev;
    for (int r = 0; r < S; r++) hs.seg.rowid[r] = r;
    hs.seg.nrows = S; hs.seg.pos0 = 0;
    hs.seg.O = t->O; hs.seg.ntiles = t->O / TILE_ROWS; hs.seg.nkb = nkb;
    hs.seg.nkpart = nkpart; hs.seg.kb_per_part = nkb / nkpart; hs.seg.task0 = 0;
    hc.nseg = 1; hc.ntask = hs.seg.ntiles * nkpart; hc.npos = S; hc.tasks_per_seg = hc.ntask;
    c->chain = false;
    if (!cuda_ok(cudaMemcpyAsync(seg_dev, &hs.seg, sizeof(GemvSeg), cudaMemcpyHostToDevice, c->stream), "noalloc segment") ||
        !cuda_ok(cudaMemcpyAsync(ctl_dev, &hc, sizeof(GemvCtl), cudaMemcpyHostToDevice, c->stream), "noalloc control")) return 0;
    const int nw = S * nkb;
    launch_pdl(c, k_prep_rows, (nw * 32 + 255) / 256, 256, 0, bq_dev, bs_dev, x_dev, S, t->I);
    switch (t->mode) {
    case SC_ROW: launch_mode<SC_ROW>(c, nc, seg_dev, ctl_dev, bq_dev, bs_dev); break;
    case SC_H16: launch_mode<SC_H16>(c, nc, seg_dev, ctl_dev, bq_dev, bs_dev); break;
    case SC_F32: launch_mode<SC_F32>(c, nc, seg_dev, ctl_dev, bq_dev, bs_dev); break;
    default: launch_mode<SC_MX>(c, nc, seg_dev, ctl_dev, bq_dev, bs_dev); break;
    }
    const size_t n4 = (size_t)S * t->O / 4;
    launch_pdl(c, k_reduce_parts, (unsigned)((n4 + 255) / 256), 256, 0, y_dev, pd_dev, S, t->O, nkpart);
    c->last_launches += 3;
    return cuda_ok(cudaGetLastError(), "pipe_gemm_noalloc launch");
}
