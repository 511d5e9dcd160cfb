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
// The products of 64 columns are formed while the additions of the 64 before run: the loads and
// multiplications fill the chain's gaps. Measured at 256 outputs of 6144 terms: 89 us with 64 outputs
// per CTA, products before additions and CTA barriers between tiles of 64; 39 us with 16 outputs, the barriers left.
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
        for (int t = 0; t < ntile; t++) {
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
        return;
    }
    const int row = tid & (OUT - 1);                    // (lanes beyond OUT repeat a row)
    float a = 0.f;
    float4 p[16];                                       // products of the 64 columns before
#pragma unroll
    for (int q = 0; q < 16; q++) p[q] = make_float4(0.f, 0.f, 0.f, 0.f);
    bool ok = true;
    for (int t = 0; t < ntile; t++) {
        const int st = t % NS, width = min(TILE, D - t * TILE);
        if (!mbar_wait_bounded(smem_u32(s_full + st), (t / NS) & 1)) ok = false;
        const float4 *wt = reinterpret_cast<const float4 *>(rt + ((size_t)(st * 2) * OUT + row) * LD);
        const float4 *xt = reinterpret_cast<const float4 *>(rt + ((size_t)(st * 2 + 1) * OUT + (one_x ? 0 : row)) * LD);
        for (int c = 0; c < width; c += 64, wt += 16, xt += 16) {
            const int n4 = min(16, (width - c) >> 2);
            // (the first round adds the zeros p starts with: the engine's sum starts from zero too)
            if (n4 == 16) {
#pragma unroll
                for (int q = 0; q < 16; q++) {
                    const float4 wv = wt[q], xv = xt[q], old = p[q];
                    p[q] = make_float4(__fmul_rn(xv.x, wv.x), __fmul_rn(xv.y, wv.y), __fmul_rn(xv.z, wv.z), __fmul_rn(xv.w, wv.w));
                    a = __fadd_rn(a, old.x); a = __fadd_rn(a, old.y);
                    a = __fadd_rn(a, old.z); a = __fadd_rn(a, old.w);
                }
            } else {                                    // the ragged end: nothing stays pending
#pragma unroll
                for (int q = 0; q < 16; q++) {
                    a = __fadd_rn(a, p[q].x); a = __fadd_rn(a, p[q].y);
                    a = __fadd_rn(a, p[q].z); a = __fadd_rn(a, p[q].w);
                    p[q] = make_float4(-0.f, -0.f, -0.f, -0.f);
                }
                for (int q = 0; q < n4; q++) {
                    const float4 wv = wt[q], xv = xt[q];
                    a = __fadd_rn(a, __fmul_rn(xv.x, wv.x)); a = __fadd_rn(a, __fmul_rn(xv.y, wv.y));
                    a = __fadd_rn(a, __fmul_rn(xv.z, wv.z)); a = __fadd_rn(a, __fmul_rn(xv.w, wv.w));
                }
            }
        }
        __syncwarp();
        if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(s_empty + st)) : "memory");
    }
#pragma unroll
    for (int q = 0; q < 16; q++) {
        a = __fadd_rn(a, p[q].x); a = __fadd_rn(a, p[q].y);
        a = __fadd_rn(a, p[q].z); a = __fadd_rn(a, p[q].w);
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

// One CTA. Builds the union, the packed row order (expert-major in union
// order, rows of an expert in ascending token order) and the segment lists.
__global__ void k_route_build(const int *idx, const int *keff, int M,
                              RouteRule rule, LayerTables tab, BuildOut out, int rpp, int nkpart1,
                              int nkpart2, int seg_cap) {
    pdl_enter();
    extern __shared__ int sm_build[];
    const int E = rule.E, K = rule.K, D = rule.D, I = rule.I;
    int *first = sm_build, *cnt = first + E, *base = cnt + E, *uniq = base + E, *passbase = uniq + E;
    __shared__ int s_nu, s_npass;
    const int tid = threadIdx.x, nth = blockDim.x;
    for (int e = tid; e < E; e += nth) { first[e] = 0x7fffffff; cnt[e] = 0; }
    if (tid == 0) s_nu = 0;
    __syncthreads();
    for (int i = tid; i < M * K; i += nth) {
        int s = i / K, kk = i - s * K;
        if (kk < keff[s]) {
            int e = idx[i];
            atomicMin(&first[e], i);
            atomicAdd(&cnt[e], 1);
        }
    }
    __syncthreads();
    for (int e = tid; e < E; e += nth) {
        if (cnt[e] > 0) {
            int rank = 0;
            for (int o = 0; o < E; o++) rank += (cnt[o] > 0 && first[o] < first[e]);
            uniq[rank] = e;
            atomicAdd(&s_nu, 1);
        }
    }
    __syncthreads();
    const int nu = s_nu;
    if (tid == 0) {
        int pos = 0, np = 0;
        for (int j = 0; j < nu; j++) {
            int e = uniq[j];
            base[e] = pos; passbase[e] = np;
            pos += cnt[e];
            np += (cnt[e] + rpp - 1) / rpp;
        }
        int shared_pos0 = pos;
        int np_routed = np;
        if (tab.sh_gate_pk) { pos += M; np += (M + rpp - 1) / rpp; }
        if (np > seg_cap) np = seg_cap;   // capacity is sized for the worst case; never exceeded
        s_npass = np;
        *out.npos = pos; *out.shared_pos0 = shared_pos0; *out.nu = nu;
        out.ctl1->nseg = 2 * np; out.ctl1->ntask = 2 * np * (I / TILE_ROWS) * nkpart1; out.ctl1->npos = pos;
        out.ctl1->tasks_per_seg = (I / TILE_ROWS) * nkpart1;
        out.ctl2->nseg = np; out.ctl2->ntask = np * (D / TILE_ROWS) * nkpart2; out.ctl2->npos = pos;
        out.ctl2->tasks_per_seg = (D / TILE_ROWS) * nkpart2;
        // shared expert segments
        if (tab.sh_gate_pk) {
            for (int p = 0; p < (M + rpp - 1) / rpp && np_routed + p < seg_cap; p++) {
                int sidx = np_routed + p;
                int r0 = p * rpp, nr = min(rpp, M - r0);
                GemvSeg *sg_ = &out.seg1[2 * sidx], *su_ = &out.seg1[2 * sidx + 1], *sd_ = &out.seg2[sidx];
                sg_->w = tab.sh_gate_pk; sg_->rowscale = tab.sh_gate_rs; sg_->out = out.partG;
                su_->w = tab.sh_up_pk; su_->rowscale = tab.sh_up_rs; su_->out = out.partU;
                sd_->w = tab.sh_down_pk; sd_->rowscale = tab.sh_down_rs; sd_->out = out.partD;
                for (int r = 0; r < nr; r++) {
                    sg_->rowid[r] = r0 + r; su_->rowid[r] = r0 + r; sd_->rowid[r] = shared_pos0 + r0 + r;
                }
                sg_->nrows = su_->nrows = sd_->nrows = nr;
                sg_->pos0 = su_->pos0 = sd_->pos0 = shared_pos0 + r0;
            }
        }
    }
    for (int j = tid; j < nu; j += nth) out.uniq[j] = uniq[j];
    __syncthreads();
    // row lists: one warp per union expert
    const int warp = tid >> 5, lane = tid & 31, nwarps = nth >> 5;
    for (int j = warp; j < nu; j += nwarps) {
        int e = uniq[j];
        int run = 0;
        for (int s0 = 0; s0 < M; s0 += 32) {
            int s = s0 + lane, hit = -1;
            if (s < M) {
                int ke = keff[s];
                for (int kk = 0; kk < ke; kk++) if (idx[s * K + kk] == e) { hit = kk; break; }
            }
            unsigned mask = __ballot_sync(0xffffffffu, hit >= 0);
            if (hit >= 0) {
                int r = run + __popc(mask & ((1u << lane) - 1));
                int pos = base[e] + r;
                out.pos_of[s * K + hit] = pos;
                int sidx = passbase[e] + r / rpp;
                if (sidx < seg_cap) {
                    out.seg1[2 * sidx].rowid[r % rpp] = s;
                    out.seg1[2 * sidx + 1].rowid[r % rpp] = s;
                    out.seg2[sidx].rowid[r % rpp] = pos;
                }
            }
            run += __popc(mask);
        }
        // per-pass constants of this expert
        int npass = (cnt[e] + rpp - 1) / rpp;
        for (int p = lane; p < npass; p += 32) {
            int sidx = passbase[e] + p;
            if (sidx >= seg_cap) continue;
            int nr = min(rpp, cnt[e] - p * rpp);
            GemvSeg *sg_ = &out.seg1[2 * sidx], *su_ = &out.seg1[2 * sidx + 1], *sd_ = &out.seg2[sidx];
            sg_->w = tab.gate_pk[e]; sg_->rowscale = tab.gate_rs ? tab.gate_rs[e] : nullptr; sg_->out = out.partG;
            su_->w = tab.up_pk[e]; su_->rowscale = tab.up_rs ? tab.up_rs[e] : nullptr; su_->out = out.partU;
            sd_->w = tab.down_pk[e]; sd_->rowscale = tab.down_rs ? tab.down_rs[e] : nullptr; sd_->out = out.partD;
            sg_->nrows = su_->nrows = sd_->nrows = nr;
            sg_->pos0 = su_->pos0 = sd_->pos0 = base[e] + p * rpp;
        }
    }
    __syncthreads();
    // shape constants and task offsets of every segment
    const int np = s_npass;
    const int t1 = (I / TILE_ROWS) * nkpart1, t2 = (D / TILE_ROWS) * nkpart2;
    for (int i = tid; i < 2 * np; i += nth) {
        GemvSeg *sgm = &out.seg1[i];
        sgm->O = I; sgm->ntiles = I / TILE_ROWS; sgm->nkb = D / BLOCK_K;
        sgm->nkpart = nkpart1; sgm->kb_per_part = (D / BLOCK_K) / nkpart1; sgm->task0 = i * t1;
    }
    for (int i = tid; i < np; i += nth) {
        GemvSeg *sgm = &out.seg2[i];
        sgm->O = D; sgm->ntiles = D / TILE_ROWS; sgm->nkb = I / BLOCK_K;
        sgm->nkpart = nkpart2; sgm->kb_per_part = (I / BLOCK_K) / nkpart2; sgm->task0 = i * t2;
    }
}
