// Routing on the device: router logits, top-K selection that reproduces the
// CPU engine's result index for index, expert-union building and the row lists
// / work descriptors of the two GEMV phases.
//
// Bit-exactness rules followed here (the CPU engine selects on values AFTER the
// softmax / sigmoid, by strict '>' with the lowest index winning ties, so the
// values themselves have to be the same floats):
//  * the router dot product adds products in ascending column order with a
//    separately rounded multiply and add per term (the order of the engine's
//    plain C loop when the compiler does not contract it);
//  * expf is evaluated with the table-driven double-precision scheme that the
//    host C library uses for expf (reduce x*32/ln2 to k + r, 2^(k/32) from a
//    32-entry table, cubic in r, all in double, one rounding to float), so the
//    device value equals the host value;
//  * sums that the engine forms serially (softmax denominator, top-K weight
//    sum) are formed serially, divisions are IEEE.
#pragma once
#include "common.cuh"
#include "gemv_stream.cuh"
#include "expf_exact.h"

// 2^(i/32) table in the "bits minus (i<<47)" form the scheme wants; filled at init.
__constant__ uint64_t c_exp2_tab[32];

__device__ __forceinline__ float expf_host_exact(float x) { return coli_expf_exact(x, c_exp2_tab); }

// logits[s*E+e] = sum_i x[s,i]*W[e,i], ascending i, multiply and add rounded separately
// (the engine's order, so the sum is one dependent chain of D additions per output: about
// 4 cycles each, which is the floor: 13 us at D = 6144). One thread per (s,e), 16 outputs per CTA: few,
// because an SM takes in about 50 B per cycle and 64 weight rows at once were slower than their chains.
// A stage of the ring is 256 columns of the CTA's weight rows and of its x row(s) (row stride 260 floats:
// rows start 16-byte aligned and the 128-bit reads of 8 threads walking different rows do not collide).
// The additions run beside the products of the next 16 columns and the loads of those behind them. Measured (cold) at 256
// outputs of 6144 terms: 89 us with 64 outputs per CTA, products before additions and CTA barriers between tiles of 64; 30 us with 16
// outputs and copies ahead of the chains, the products of 64 columns formed from loads that the chain waited for; 24 so (2048 outputs of
// 7168: 35 -> 28). Six cycles an addition, where its latency is four.
// Two forms: k_router_logits, one copy warp with bulk copies of 256 columns per row and an mbarrier per stage
// (rows that start 16-byte aligned), and k_router_logits_any, plain loads, for the rest.
#define ROUTER_STAGES 6
__host__ __device__ constexpr int router_smem(int out, int tile) { return ROUTER_STAGES * 2 * out * (tile + 4) * 4; }
template <int OUT, int TILE>
__global__ void __launch_bounds__(OUT <= 32 ? 64 : OUT + 32) k_router_logits(float *__restrict__ logits, const float *x,
                                                                             const float *__restrict__ W, int M, int D, int E,
                                                                             int *status) {
    pdl_enter();
    extern __shared__ __align__(16) float rt[];         // [stage][w | x][OUT][TILE + 4]
    __shared__ __align__(8) unsigned long long s_full[ROUTER_STAGES], s_empty[ROUTER_STAGES];
    constexpr int LD = TILE + 4, NS = ROUTER_STAGES, CW = (OUT + 31) / 32;
    const int tid = threadIdx.x, lane = tid & 31, i0 = blockIdx.x * OUT, nrow = min(OUT, M * E - i0);
    // when all outputs of the CTA belong to one row of x, that row is staged once (tile row 0)
    const bool one_x = i0 / E == (i0 + nrow - 1) / E;
    const int ntile = (D + TILE - 1) / TILE;
    if (tid == 0) {
        for (int i = 0; i < NS; i++) { mbar_init(smem_u32(s_full + i), 1); mbar_init(smem_u32(s_empty + i), CW); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    if (tid >= CW * 32) {
        // copies: row j of the weights, or of x
        const int rows = nrow + (one_x ? 1 : nrow);
        int t = 0;
        for (; t < ntile; t++) {
            const int st = t % NS, width = min(TILE, D - t * TILE);
            const uint32_t bar = smem_u32(s_full + st);
            if (t >= NS && !mbar_wait_bounded(smem_u32(s_empty + st), (t / NS + 1) & 1)) break;
            if (lane == 0) mbar_expect_tx(bar, (uint32_t)rows * width * 4);
            __syncwarp();
            for (int j = lane; j < rows; j += 32) {
                const bool is_x = j >= nrow;
                const int r = is_x ? j - nrow : j, i = i0 + r, s = i / E;
                const float *src = (is_x ? x + (size_t)s * D : W + (size_t)(i - s * E) * D) + (size_t)t * TILE;
                bulk_g2s(smem_u32(rt + ((size_t)(st * 2 + is_x) * OUT + r) * LD), src, width * 4, bar);
            }
        }
        // copies in flight land before the shared memory goes away (bounded): chains that gave up no longer wait for them
        for (int i = max(0, t - NS); i < t; i++) mbar_wait_bounded(smem_u32(s_full + i % NS), (i / NS) & 1);
        return;
    }
    const int row = tid & (OUT - 1);                    // (lanes beyond OUT repeat a row)
    // Steps of 16 columns in three stages: while the products of one are added, those of the next are formed and the operands
    // of the one behind it are on their way, so the chain of additions waits for nothing. (A zero operand, or
    // a sum that starts with +0, changes no bit of it.)
    float a = 0.f;
    float4 w0[4], x0[4], w1[4], x1[4], p0[4], p1[4];
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int q = 0; q < 4; q++) w1[q] = x1[q] = p0[q] = zero;
    auto load = [](float4 (&w)[4], float4 (&xv)[4], const float4 *wt, const float4 *xt) {
#pragma unroll
        for (int q = 0; q < 4; q++) { w[q] = wt[q]; xv[q] = xt[q]; }
    };
    auto mul = [](float4 (&p)[4], const float4 (&w)[4], const float4 (&xv)[4]) {
#pragma unroll
        for (int q = 0; q < 4; q++)
            p[q] = make_float4(__fmul_rn(xv[q].x, w[q].x), __fmul_rn(xv[q].y, w[q].y), __fmul_rn(xv[q].z, w[q].z), __fmul_rn(xv[q].w, w[q].w));
    };
    auto add = [&](const float4 (&p)[4]) {
#pragma unroll
        for (int q = 0; q < 4; q++) {
            a = __fadd_rn(a, p[q].x); a = __fadd_rn(a, p[q].y);
            a = __fadd_rn(a, p[q].z); a = __fadd_rn(a, p[q].w);
        }
    };
    bool ok = true;
    for (int t = 0; t < ntile; t++) {
        const int st = t % NS, width = min(TILE, D - t * TILE);
        if (ok && !mbar_wait_bounded(smem_u32(s_full + st), (t / NS) & 1)) ok = false;      // (one expired wait, not one a tile)
        const float4 *wt = reinterpret_cast<const float4 *>(rt + ((size_t)(st * 2) * OUT + row) * LD);
        const float4 *xt = reinterpret_cast<const float4 *>(rt + ((size_t)(st * 2 + 1) * OUT + (one_x ? 0 : row)) * LD);
#pragma unroll 1
        for (int c = width >> 5; c > 0; c--, wt += 8, xt += 8) {
            load(w0, x0, wt, xt); mul(p1, w1, x1); add(p0);
            load(w1, x1, wt + 4, xt + 4); mul(p0, w0, x0); add(p1);
        }
        if (width < TILE || t == ntile - 1) {           // the end: what is under way, then up to 28 columns one by one
            mul(p1, w1, x1); add(p0); add(p1);
            for (int q = (width & 31) >> 2; q > 0; q--, wt++, xt++) {
                const float4 wv = *wt, xv = *xt;
                a = __fadd_rn(a, __fmul_rn(xv.x, wv.x)); a = __fadd_rn(a, __fmul_rn(xv.y, wv.y));
                a = __fadd_rn(a, __fmul_rn(xv.z, wv.z)); a = __fadd_rn(a, __fmul_rn(xv.w, wv.w));
            }
        }
        // the tile before has been multiplied: its last operands were in the first products of this one
        __syncwarp();
        if (t > 0 && lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(s_empty + (t - 1) % NS)) : "memory");
    }
    if (tid < nrow) logits[i0 + tid] = a;
    if (!ok && lane == 0) kstat_set(status, KSTAT_MBAR_TIMEOUT);
}
// One thread per output, operands straight from memory.
__global__ void k_router_logits_any(float *__restrict__ logits, const float *x, const float *__restrict__ W, int M, int D,
                                    int E) {
    pdl_enter();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= M * E) return;
    const int s = i / E;
    const float *xr = x + (size_t)s * D, *wr = W + (size_t)(i - s * E) * D;
    float a = 0.f;
#pragma unroll 8
    for (int k = 0; k < D; k++) a = __fadd_rn(a, __fmul_rn(xr[k], wr[k]));
    logits[i] = a;
}

#define ROUTE_MAX_E 1024
#define ROUTE_MAX_K 64

// Per-layer device tables the build kernel reads.
struct LayerTables {
    const uint8_t *const *gate_pk, *const *up_pk, *const *down_pk;     // [E] packed bases
    const float *const *gate_rs, *const *up_rs, *const *down_rs;       // [E] row scales (SC_ROW) or NULL
    const uint8_t *sh_gate_pk, *sh_up_pk, *sh_down_pk;                 // shared expert or NULL
    const float *sh_gate_rs, *sh_up_rs, *sh_down_rs;
};

struct BuildOut {
    GemvSeg *seg1, *seg2;      // gate/up interleaved; down
    GemvCtl *ctl1, *ctl2;
    int *pos_of;               // [M*K] packed row of (token, kk)
    int *uniq, *nu;            // union in first-appearance order
    int *npos, *shared_pos0;
    float *partG, *partU, *partD;
};

// One CTA of 1024 threads. Builds the union (first-appearance order), the packed row order (expert-major in union
// order, entries of an expert in ascending order) and the segment lists. A warp walks a contiguous slice of the entries; ranks
// come from match masks and per-warp counts, so no atomics decide an order. Bound by latency, a few dependent round trips:
// 512 entries of 256 experts in 13 us, where a warp per expert that searched all rows for it, and one thread that summed
// up the union, took 47. Dynamic shared memory: ROUTE_BUILD_INTS * E ints.
#define ROUTE_BUILD_INTS 37
__global__ void __launch_bounds__(1024) k_route_build(const int *idx, const int *keff, int M, RouteRule rule, LayerTables tab,
                                                      BuildOut out, int rpp, int nkpart1, int nkpart2, int seg_cap) {
    pdl_enter();
    extern __shared__ int sm_build[];
    const int E = rule.E, K = rule.K, D = rule.D, I = rule.I;
    int *hist = sm_build, *first = hist + 32 * E, *cnt = first + E, *base = cnt + E, *uniq = base + E, *passbase = uniq + E;
    __shared__ int s_a[32], s_b[32], s_c[32];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int n = M * K, slice = ((n + 31) / 32 + 31) & ~31, i0 = warp * slice, i1 = min(n, i0 + slice);
    for (int e = tid; e < 32 * E; e += 1024) hist[e] = 0;
    if (tid < E) first[tid] = 0x7fffffff;
    __syncthreads();
    auto entry = [&](int i) { const int s = i / K; return i < i1 && i - s * K < keff[s] ? idx[i] : -1; };
    // exclusive sums over the CTA's threads of two values, and the totals
    auto scan = [&](int &a, int &b, int &ta, int &tb) {
        int pa = a, pb = b;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int x = __shfl_up_sync(0xffffffffu, pa, d), y = __shfl_up_sync(0xffffffffu, pb, d);
            if (lane >= d) { pa += x; pb += y; }
        }
        if (lane == 31) { s_a[warp] = pa; s_b[warp] = pb; }
        __syncthreads();
        int wa = s_a[lane], wb = s_b[lane];
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int x = __shfl_up_sync(0xffffffffu, wa, d), y = __shfl_up_sync(0xffffffffu, wb, d);
            if (lane >= d) { wa += x; wb += y; }
        }
        ta = __shfl_sync(0xffffffffu, wa, 31); tb = __shfl_sync(0xffffffffu, wb, 31);
        a = pa - a + __shfl_sync(0xffffffffu, wa, warp) - s_a[warp];
        b = pb - b + __shfl_sync(0xffffffffu, wb, warp) - s_b[warp];
    };
    int *mine = hist + warp * E;
    for (int b = i0; b < i1; b += 32) {
        const int e = entry(b + lane);
        const unsigned m = __match_any_sync(0xffffffffu, e);
        if (e >= 0 && lane == __ffs(m) - 1) {
            if (mine[e] == 0) atomicMin(&first[e], b + lane);
            mine[e] += __popc(m);
        }
        __syncwarp();
    }
    __syncthreads();
    // union: entry i opens an expert iff it is that expert's first; its place is the number of such entries before it
    int opens = 0;
    for (int b = i0; b < i1; b += 32) {
        const int e = entry(b + lane);
        opens += __popc(__ballot_sync(0xffffffffu, e >= 0 && first[e >= 0 ? e : 0] == b + lane));
    }
    if (lane == 0) s_c[warp] = opens;
    if (tid < E) {
        int c = 0;
        for (int w = 0; w < 32; w++) { const int h = hist[w * E + tid]; hist[w * E + tid] = c; c += h; }
        cnt[tid] = c;
    }
    __syncthreads();
    int at = 0;
    for (int w = 0; w < 32; w++) { const int o = s_c[w]; at += w < warp ? o : 0; }
    for (int b = i0; b < i1; b += 32) {
        const int e = entry(b + lane);
        const bool op = e >= 0 && first[e] == b + lane;
        const unsigned m = __ballot_sync(0xffffffffu, op);
        if (op) uniq[at + __popc(m & ((1u << lane) - 1u))] = e;
        at += __popc(m);
    }
    int nu = 0;
    for (int w = 0; w < 32; w++) nu += s_c[w];
    __syncthreads();
    // packed rows and passes before expert number tid of the union
    const int e = tid < nu ? uniq[tid] : 0, c = tid < nu ? cnt[e] : 0, np = (c + rpp - 1) / rpp;
    int pos = c, pass = np, npos, npass;
    scan(pos, pass, npos, npass);
    if (tid < nu) { base[e] = pos; passbase[e] = pass; out.uniq[tid] = e; }
    const int nsh = tab.sh_gate_pk ? (M + rpp - 1) / rpp : 0;
    const int nseg = min(npass + nsh, seg_cap);      // capacity is sized for the worst case; never exceeded
    const int t1 = (I / TILE_ROWS) * nkpart1, t2 = (D / TILE_ROWS) * nkpart2;
    if (tid == 0) {
        const int all = npos + (nsh ? M : 0);
        *out.npos = all; *out.shared_pos0 = npos; *out.nu = nu;
        out.ctl1->nseg = 2 * nseg; out.ctl1->ntask = 2 * nseg * t1; out.ctl1->npos = all; out.ctl1->tasks_per_seg = t1;
        out.ctl2->nseg = nseg; out.ctl2->ntask = nseg * t2; out.ctl2->npos = all; out.ctl2->tasks_per_seg = t2;
    }
    auto put = [&](int si, int which, const uint8_t *w, const float *rs, int nrows, int pos0) {
        GemvSeg *sg = which == 2 ? &out.seg2[si] : &out.seg1[2 * si + which];
        const int O = which == 2 ? D : I, nkb = (which == 2 ? I : D) / BLOCK_K, nkpart = which == 2 ? nkpart2 : nkpart1;
        sg->w = w; sg->rowscale = rs; sg->out = which == 0 ? out.partG : which == 1 ? out.partU : out.partD;
        sg->nrows = nrows; sg->pos0 = pos0;
        sg->O = O; sg->ntiles = O / TILE_ROWS; sg->nkb = nkb; sg->nkpart = nkpart; sg->kb_per_part = nkb / nkpart;
        sg->task0 = which == 2 ? si * t2 : (2 * si + which) * t1;
    };
    if (tid < nu) {
        const uint8_t *wg = tab.gate_pk[e], *wu = tab.up_pk[e], *wd = tab.down_pk[e];
        const float *rg = tab.gate_rs ? tab.gate_rs[e] : nullptr, *ru = tab.up_rs ? tab.up_rs[e] : nullptr, *rd = tab.down_rs ? tab.down_rs[e] : nullptr;
        for (int p = 0; p < np && pass + p < nseg; p++) {
            const int nr = min(rpp, c - p * rpp), p0 = pos + p * rpp;
            put(pass + p, 0, wg, rg, nr, p0); put(pass + p, 1, wu, ru, nr, p0); put(pass + p, 2, wd, rd, nr, p0);
        }
    }
    for (int p = tid; p < nsh && npass + p < nseg; p += 1024) {
        const int si = npass + p, r0 = p * rpp, nr = min(rpp, M - r0);
        put(si, 0, tab.sh_gate_pk, tab.sh_gate_rs, nr, npos + r0);
        put(si, 1, tab.sh_up_pk, tab.sh_up_rs, nr, npos + r0);
        put(si, 2, tab.sh_down_pk, tab.sh_down_rs, nr, npos + r0);
    }
    for (int s = tid; s < (nsh ? M : 0); s += 1024) {
        const int si = npass + s / rpp, r = s % rpp;
        if (si < nseg) { out.seg1[2 * si].rowid[r] = s; out.seg1[2 * si + 1].rowid[r] = s; out.seg2[si].rowid[r] = npos + s; }
    }
    __syncthreads();
    for (int b = i0; b < i1; b += 32) {
        const int i = b + lane, s = i / K, e = entry(i);
        const unsigned m = __match_any_sync(0xffffffffu, e);
        if (e >= 0) {
            const int r = mine[e] + __popc(m & ((1u << lane) - 1u)), si = passbase[e] + r / rpp, q = r % rpp;
            out.pos_of[i] = base[e] + r;
            if (si < nseg) { out.seg1[2 * si].rowid[q] = s; out.seg1[2 * si + 1].rowid[q] = s; out.seg2[si].rowid[q] = base[e] + r; }
        }
        __syncwarp();
        if (e >= 0 && lane == __ffs(m) - 1) mine[e] += __popc(m);
        __syncwarp();
    }
}
