// Device side of the expert-parallel layer: the dispatch plan (which entry goes to
// which rank and local expert, at which position of the send buffer), the packing
// of the rows into that buffer, and the weighted combine of the answers.
//
// The reference has no collective path (experts are pinned to devices and rows go
// host -> device per call, c/colibri.c:4819-4839, 8367-8417); the exchange itself is
// NCCL's all-to-all, issued by the host between these kernels. Everything here is
// integer / copy work bound by latency or HBM; no atomics decide an order: positions
// follow from counts and a stable rank (expert bucket, then row order), so the plan is
// the same on every run.
#pragma once
#include "common.cuh"
#include <cuda_bf16.h>

// cnt[dest[e]*slots + slot[e]] += 1 for every live entry (row, kk < keff[row]).
__global__ void k_ep_count(int *__restrict__ cnt, const int *idx, const int *keff,
                           const int *dest, const int *slot, int m, int K, int slots) {
    pdl_enter();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m * K) return;
    const int s = i / K, kk = i - s * K;
    if (kk >= keff[s]) return;
    const int e = idx[i];
    atomicAdd(&cnt[dest[e] * slots + slot[e]], 1);      // integer counts: the result does not depend on the order
}

// One block: exclusive prefix sum of the nb bucket counts -> off[nb], total -> off[nb].
__global__ void k_ep_offsets(int *__restrict__ off, const int *cnt, int nb) {
    pdl_enter();
    __shared__ int part[1024];
    const int tid = threadIdx.x, nth = blockDim.x;
    const int per = (nb + nth - 1) / nth, b0 = tid * per, b1 = min(nb, b0 + per);
    int s = 0;
    for (int b = b0; b < b1; b++) s += cnt[b];
    part[tid] = s;
    __syncthreads();
    if (tid == 0) {
        int run = 0;
        for (int t = 0; t < nth; t++) { int v = part[t]; part[t] = run; run += v; }
        off[nb] = run;
    }
    __syncthreads();
    int run = part[tid];
    for (int b = b0; b < b1; b++) { off[b] = run; run += cnt[b]; }
}

// One CTA of 8 warps per expert e; a warp owns a contiguous slice of the rows and walks it twice, 32 rows at a time:
// counting, then placing behind the warps before it. The entries that select e
// get consecutive positions of e's bucket in row order (a row that selects e twice keeps
// its kk order). entry_of[row*K+kk] = position in the send buffer; row_of[position] = row.
// entry_of must hold -1 everywhere beforehand (dead entries keep it).
// Bound by the latency of the walk: one warp per expert took 80 us for 2048 rows, eight take a sixth of it.
#define EP_PLACE_WARPS 8
__global__ void __launch_bounds__(EP_PLACE_WARPS * 32) k_ep_place(int *__restrict__ entry_of, int *__restrict__ row_of, const int *off,
                           const int *idx, const int *keff,
                           const int *dest, const int *slot, int m, int K,
                           int slots) {
    pdl_enter();
    __shared__ int s_n[EP_PLACE_WARPS];
    const int e = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int per = ((m + EP_PLACE_WARPS - 1) / EP_PLACE_WARPS + 31) & ~31, r0 = warp * per, r1 = min(m, r0 + per);
    auto hits_of = [&](int s) {             // bit kk set: entry (s, kk) selects e
        int hits = 0;
        if (s < r1) {
#pragma unroll 8
            for (int kk = 0; kk < K; kk++) hits |= (idx[s * K + kk] == e) << kk;
            hits &= (1 << keff[s]) - 1;
        }
        return hits;
    };
    int cnt = 0;
    for (int s0 = r0; s0 < r1; s0 += 32) cnt += __popc(hits_of(s0 + lane));
    cnt = __reduce_add_sync(0xffffffffu, cnt);
    if (lane == 0) s_n[warp] = cnt;
    __syncthreads();
    int run = off[dest[e] * slots + slot[e]];
    for (int w = 0; w < warp; w++) run += s_n[w];
    if (cnt == 0) return;
    for (int s0 = r0; s0 < r1; s0 += 32) {
        const int s = s0 + lane;
        int hits = hits_of(s);
        const int n = __popc(hits);
        // exclusive prefix of n over the lanes
        int pre = n;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) { int v = __shfl_up_sync(0xffffffffu, pre, d); if (lane >= d) pre += v; }
        int pos = run + pre - n;
        while (hits) {
            const int kk = __ffs(hits) - 1;
            hits &= hits - 1;
            entry_of[s * K + kk] = pos;
            row_of[pos] = s;
            pos++;
        }
        run += __shfl_sync(0xffffffffu, pre, 31);
    }
}

// Block p copies row row_of[p] of x into position p of the send buffer, as bf16 (when the
// values are exact in bf16; any value that is not raises *inexact) or as f32.
// Launched for the largest possible count; blocks beyond *total leave.
template <bool BF16>
__global__ void k_ep_gather(void *__restrict__ send, const float *x, const int *row_of,
                            const int *total, int D, int *__restrict__ inexact) {
    pdl_enter();
    const int p = blockIdx.x;
    if (p >= *total) return;
    const float4 *src = reinterpret_cast<const float4 *>(x + (size_t)row_of[p] * D);
    int bad = 0;
    for (int i = threadIdx.x; i < D / 4; i += blockDim.x) {
        const float4 v = src[i];
        if (BF16) {
            const uint32_t a = __float_as_uint(v.x), b = __float_as_uint(v.y), c = __float_as_uint(v.z), d = __float_as_uint(v.w);
            bad |= (a | b | c | d) & 0xFFFFu;              // low mantissa bits a bf16 cannot hold
            reinterpret_cast<uint2 *>(static_cast<__nv_bfloat16 *>(send) + (size_t)p * D)[i] =
                make_uint2((a >> 16) | (b & 0xFFFF0000u), (c >> 16) | (d & 0xFFFF0000u));
        } else {
            reinterpret_cast<float4 *>(static_cast<float *>(send) + (size_t)p * D)[i] = v;
        }
    }
    if (BF16 && bad) *inexact = 1;
}

// dst[map[p]] = src[p] (FORWARD) or dst[p] = src[map[p]] (gather), rows of D floats; src may be bf16.
template <bool SRC_BF16, bool SCATTER>
__global__ void k_ep_permute(float *__restrict__ dst, const void *src, const int *map,
                             int n, int D) {
    pdl_enter();
    const int p = blockIdx.x;
    if (p >= n) return;
    const int q = map[p];
    const size_t so = (size_t)(SCATTER ? p : q) * D, dof = (size_t)(SCATTER ? q : p) * D;
    for (int i = threadIdx.x; i < D / 4; i += blockDim.x) {
        float4 v;
        if (SRC_BF16) {
            const uint2 r = reinterpret_cast<const uint2 *>(static_cast<const __nv_bfloat16 *>(src) + so)[i];
            v = make_float4(__uint_as_float(r.x << 16), __uint_as_float(r.x & 0xFFFF0000u),
                            __uint_as_float(r.y << 16), __uint_as_float(r.y & 0xFFFF0000u));
        } else {
            v = reinterpret_cast<const float4 *>(static_cast<const float *>(src) + so)[i];
        }
        reinterpret_cast<float4 *>(dst + dof)[i] = v;
    }
}

// out[s] = sum_{kk < keff[s]} w[s,kk] * y[entry_of[s,kk]]  (+ shared[s]): the row's selection
// order, shared expert last; the same arithmetic as the single-GPU layer's combine.
__global__ void k_ep_combine(float *__restrict__ out, const float *y, const int *entry_of,
                             const float *wts, const int *keff,
                             const float *shared, int m, int K, int D) {
    pdl_enter();
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int dq = D / 4;
    if (i >= (size_t)m * dq) return;
    const int s = i / dq, d4 = i - (size_t)s * dq;
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    const int ke = keff[s];
    int kk = 0;
    for (; kk + 4 <= ke; kk += 4) {         // four rows requested before the first is added
        float4 a[4];
        float wgt[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            wgt[j] = wts[s * K + kk + j];
            a[j] = reinterpret_cast<const float4 *>(y + (size_t)entry_of[s * K + kk + j] * D)[d4];
        }
#pragma unroll
        for (int j = 0; j < 4; j++) {
            acc.x = fmaf(wgt[j], a[j].x, acc.x); acc.y = fmaf(wgt[j], a[j].y, acc.y);
            acc.z = fmaf(wgt[j], a[j].z, acc.z); acc.w = fmaf(wgt[j], a[j].w, acc.w);
        }
    }
    for (; kk < ke; kk++) {
        const int pos = entry_of[s * K + kk];
        const float wgt = wts[s * K + kk];
        const float4 a = reinterpret_cast<const float4 *>(y + (size_t)pos * D)[d4];
        acc.x = fmaf(wgt, a.x, acc.x); acc.y = fmaf(wgt, a.y, acc.y);
        acc.z = fmaf(wgt, a.z, acc.z); acc.w = fmaf(wgt, a.w, acc.w);
    }
    if (shared) {
        const float4 a = reinterpret_cast<const float4 *>(shared + (size_t)s * D)[d4];
        acc.x += a.x; acc.y += a.y; acc.z += a.z; acc.w += a.w;
    }
    reinterpret_cast<float4 *>(out)[i] = acc;
}
