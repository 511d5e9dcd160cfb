// y[S,O] = x[S,I] @ W^T for a packed tensor and up to 8 rows in ONE launch without descriptors: the
// dense projections of a decode step (shared expert, per-matrix calls of the resident pipeline).
//
// The streaming kernel (gemv_stream.cuh) needs a descriptor upload, an activation split, the GEMV
// and a reduction of its partial sums: four stream operations, 27 us for a 6 MB matrix that HBM
// delivers in one. Here a CTA owns 16 output rows (half a packed tile): its 8 warps take the
// contraction's 128-column blocks in turn, every warp requesting up to ROWS_NST half chunks by bulk
// copies before anything else; meanwhile the CTA splits x into fp16 hi/lo fragments in shared memory,
// and the warps' sums meet there at the end. Bound by the latency of the few loads in flight at these sizes.
#pragma once
#include "common.cuh"
#include "gemv_stream.cuh"
#include "kernels_misc.cuh"

#define ROWS_WARPS 8
#define ROWS_NST 8
#define ROWS_MAX_X 24576      // S * I at most: 96 KB of split activations beside the weight ring
__host__ __device__ constexpr int rows_smem(int mode, int S, int I) {
    return ROWS_WARPS * ROWS_NST * (half_bytes_of(mode) + 8) + S * I * 4 + S * (I / BLOCK_K) * 4 + ROWS_WARPS * 2 * 32 * 8;
}

template <int MODE, int NC>
__global__ void __launch_bounds__(ROWS_WARPS * 32) k_gemv_rows(float *__restrict__ y, const float *x,
                                                               const uint8_t *__restrict__ w, const float *rowscale,
                                                               int S, int I, int O, int *status) {
    constexpr int HS = half_bytes_of(MODE);
    // While the kernel before drains: ask for this CTA's weights to be brought into L2 (no value is read yet).
    if (threadIdx.x < 32) {
        const uint8_t *base = w + (size_t)(blockIdx.x >> 1) * (I / BLOCK_K) * 2 * HS + (blockIdx.x & 1) * HS;
        for (int kb = threadIdx.x; kb < I / BLOCK_K; kb += 32)
            asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(base + (size_t)kb * 2 * HS), "r"(HS) : "memory");
    }
    pdl_enter();
    extern __shared__ __align__(128) uint8_t smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3, nkb = I / BLOCK_K;
    const uint32_t ring = smem_u32(smem) + warp * ROWS_NST * HS;
    uint8_t *after = smem + ROWS_WARPS * ROWS_NST * HS;
    const uint32_t bars = smem_u32(after) + warp * ROWS_NST * 8;
    __half *xq = reinterpret_cast<__half *>(after + ROWS_WARPS * ROWS_NST * 8);
    float2 *part = reinterpret_cast<float2 *>(reinterpret_cast<uint8_t *>(xq) + (size_t)S * I * 4);
    float *xs = reinterpret_cast<float *>(part + ROWS_WARPS * 2 * 32);
    // half blockIdx.x & 1 of tile blockIdx.x / 2
    const uint8_t *src = w + (size_t)(blockIdx.x >> 1) * nkb * 2 * HS + (blockIdx.x & 1) * HS;
    int issued = warp;                                  // next block to request
    if (lane == 0) {
        for (int s = 0; s < ROWS_NST; s++) mbar_init(bars + s * 8, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        for (int s = 0; s < ROWS_NST && issued < nkb; s++, issued += ROWS_WARPS) {
            mbar_expect_tx(bars + s * 8, HS);
            bulk_g2s(ring + s * HS, src + (size_t)issued * 2 * HS, HS, bars + s * 8);
        }
    }
    for (int b = warp; b < S * nkb; b += ROWS_WARPS) {
        const float4 v = *reinterpret_cast<const float4 *>(x + (size_t)b * BLOCK_K + lane * 4);
        const float m = warp_max(fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w))));
        const float s = block_scale_from_max(m);
        store_split4(xq + (size_t)b * 256, lane, v, s);
        if (lane == 0) xs[b] = 1.f / s;
    }
    __syncthreads();
    const __half *bp[NC];
    const float *sp[NC];
#pragma unroll
    for (int cs = 0; cs < NC; cs++) {
        bp[cs] = xq + (size_t)min(cs * 4 + (g >> 1), S - 1) * nkb * 256 + (g & 1) * 32 + t * 8;
        sp[cs] = xs + (size_t)min(cs * 4 + t, S - 1) * nkb;
    }
    float R[NC][4];
#pragma unroll
    for (int cs = 0; cs < NC; cs++)
#pragma unroll
        for (int i = 0; i < 4; i++) R[cs][i] = 0.f;
    int s = 0;
    uint32_t par = 0;
    bool ok = true;
    for (int kb = warp; kb < nkb; kb += ROWS_WARPS) {
        // (behind an expired wait one try a block)
        if (!mbar_try_wait(bars + s * 8, par) && !(ok && mbar_wait_bounded(bars + s * 8, par))) ok = false;
        float bacc[NC][2][4];
        block_mma<MODE, NC, false, 1>(ring + s * HS, lane, g,
                                      [&](int grp, int cs) { return *reinterpret_cast<const uint4 *>(bp[cs] + (size_t)kb * 256 + grp * 64); },
                                      bacc);
#pragma unroll
        for (int cs = 0; cs < NC; cs++) {
            const float ix = sp[cs][kb];
#pragma unroll
            for (int i = 0; i < 4; i++) R[cs][i] = fmaf(bacc[cs][0][i], ix, R[cs][i]);
        }
        __syncwarp();
        if (lane == 0 && ok && issued < nkb) {
            mbar_expect_tx(bars + s * 8, HS);
            bulk_g2s(ring + s * HS, src + (size_t)issued * 2 * HS, HS, bars + s * 8);
            issued += ROWS_WARPS;
        }
        if (++s == ROWS_NST) { s = 0; par ^= 1; }
    }
#pragma unroll
    for (int cs = 0; cs < NC; cs++) part[(warp * 2 + cs) * 32 + lane] = make_float2(R[cs][0] + R[cs][1], R[cs][2] + R[cs][3]);
    __syncthreads();
    // row r of x, output o of the half: lane (o & 7)*4 + (r & 3) of set r / 4, component o >> 3
    for (int i = threadIdx.x; i < S * 16; i += ROWS_WARPS * 32) {
        const int r = i >> 4, o = i & 15;
        const float *p = reinterpret_cast<const float *>(part + (r >> 2) * 32 + (o & 7) * 4 + (r & 3)) + (o >> 3);
        float a = 0.f;
#pragma unroll
        for (int k = 0; k < ROWS_WARPS; k++) a += p[k * 2 * 32 * 2];
        if (MODE == SC_ROW) a *= rowscale[blockIdx.x * 16 + o];
        y[(size_t)r * O + blockIdx.x * 16 + o] = a;
    }
    if (!ok && lane == 0) {                             // (last, out of the way of the ordinary end)
        kstat_set(status, KSTAT_MBAR_TIMEOUT);
        // copies in flight land before the shared memory goes away (bounded): the last one of every stage
        const int n = (issued - warp) / ROWS_WARPS;
#pragma unroll 1
        for (int i = max(0, n - ROWS_NST); i < n; i++) mbar_wait_bounded(bars + i % ROWS_NST * 8, (i / ROWS_NST) & 1);
    }
}
