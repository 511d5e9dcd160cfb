// Small kernels around the streaming GEMV: upload-time repacking, activation
// preparation (f32 rows -> fp16 hi/lo B fragments with a power-of-two block
// scale), the SwiGLU and combine reductions of the partial sums, the generic
// warp-per-row matmul for tensors the packed layout does not cover, and the
// elementwise resident-pipeline primitives.
#pragma once
#include "common.cuh"

// ---------------------------------------------------------------------------
// Upload-time repack: raw row-major nibbles [O, I/2] -> tile streams.
// One thread per output 32-bit word.
// ---------------------------------------------------------------------------
// Facts about a tensor's scales that decide its storage and whether the tensor-core path can carry it;
// the words start at zero and only grow. Bound by HBM, a few us per tensor (one pass on a host thread: 2 ms
// for the 459 000 scales of a 7168 x 2048 matrix in groups of 32).
// f32 scales: [0] some value is not exact in fp16, [1] largest |s| (bits), [2] 0x7FFFFFFF - smallest
// non-zero |s| (bits), [3] some |s| is not at most 65504.
__global__ void __launch_bounds__(256) k_check_scales(uint32_t *__restrict__ out, const float *__restrict__ s, size_t n) {
    uint32_t inexact = 0, mx = 0, mn = 0, wild = 0;
    for (int j = 0; j < 4; j++) {
        const size_t i = (size_t)blockIdx.x * 1024 + j * 256 + threadIdx.x;
        if (i < n) {
            const float v = s[i], a = fabsf(v);
            inexact |= !(__half2float(__float2half_rn(v)) == v);
            wild |= !(a <= 65504.f);
            const uint32_t b = __float_as_uint(a);
            mx = max(mx, b);
            if (b) mn = max(mn, 0x7FFFFFFFu - b);
        }
    }
    inexact = __reduce_or_sync(0xffffffffu, inexact); wild = __reduce_or_sync(0xffffffffu, wild);
    mx = __reduce_max_sync(0xffffffffu, mx); mn = __reduce_max_sync(0xffffffffu, mn);
    if ((threadIdx.x & 31) == 0) {
        if (inexact) out[0] = 1;
        if (wild) out[3] = 1;
        atomicMax(&out[1], mx); atomicMax(&out[2], mn);
    }
}
// ue8m0 exponents with their 16 code bytes per group: [0] largest exponent, [1] 255 - smallest exponent of a
// group with a non-zero code, [2] some exponent is 255 (NaN).
__global__ void __launch_bounds__(256) k_check_mx(uint32_t *__restrict__ out, const uint8_t *__restrict__ codes,
                                                  const uint8_t *__restrict__ e8, size_t n) {
    const size_t i = (size_t)blockIdx.x * 256 + threadIdx.x;
    uint32_t mx = 0, mn = 0, nan = 0;
    if (i < n) {
        const uint32_t e = e8[i];
        const uint4 c = reinterpret_cast<const uint4 *>(codes)[i];
        mx = e; nan = e == 255;
        if ((c.x | c.y | c.z | c.w) & 0x77777777u) mn = 255 - e;
    }
    nan = __reduce_or_sync(0xffffffffu, nan);
    mx = __reduce_max_sync(0xffffffffu, mx); mn = __reduce_max_sync(0xffffffffu, mn);
    if ((threadIdx.x & 31) == 0) {
        if (nan) out[2] = 1;
        atomicMax(&out[0], mx); atomicMax(&out[1], mn);
    }
}

__global__ void k_repack_codes(uint8_t *__restrict__ pk, const uint8_t *__restrict__ raw, int O,
                               int I, int chunk_bytes, int is_mx, int tc_shift) {
    const int nkb = I / BLOCK_K, ntiles = O / TILE_ROWS;
    size_t total = (size_t)ntiles * nkb * 512;   // words
    size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= total) return;
    if (idx == 0) *reinterpret_cast<int *>(pk + (size_t)ntiles * nkb * chunk_bytes) = tc_shift;
    int grp = idx & 3;
    int lane = (idx >> 2) & 31;
    int j = (idx >> 7) & 3;
    size_t blk = idx >> 9;
    int kb = blk % nkb;
    int tile = blk / nkb;
    int g = lane >> 2, t = lane & 3;
    int row = tile * TILE_ROWS + (j >> 1) * 16 + (j & 1) * 8 + g;
    int k0 = kb * BLOCK_K + grp * 32 + t * 8;
    const uint8_t *src = raw + (size_t)row * (I / 2) + k0 / 2;
    uint32_t word = 0;
    if (is_mx) {
#pragma unroll
        for (int b = 0; b < 4; b++) word |= (uint32_t)src[b] << (8 * b);
    } else {
        uint32_t c[8];
#pragma unroll
        for (int b = 0; b < 4; b++) { c[2 * b] = src[b] & 15u; c[2 * b + 1] = src[b] >> 4; }
        const int order[8] = {0, 2, 4, 6, 1, 3, 5, 7};
#pragma unroll
        for (int f = 0; f < 8; f++) word |= c[order[f]] << (4 * f);
    }
    uint32_t *dst = reinterpret_cast<uint32_t *>(pk + blk * (size_t)chunk_bytes + (j >> 1) * (chunk_bytes / 2) + (j & 1) * 512 +
                                                 lane * 16 + grp * 4);
    *dst = word;
}

// Scales -> per-chunk scale part. One thread per (block, sub, g, h, grp). MXFP4: exponents below e_min
// (groups without a non-zero code, see tensor_tc_params) are stored as e_min.
__global__ void k_repack_scales(uint8_t *__restrict__ pk, const void *__restrict__ raw_s, int O, int I,
                                int chunk_bytes, int mode, int gs, int ng, int e_min) {
    const int nkb = I / BLOCK_K, ntiles = O / TILE_ROWS;
    size_t total = (size_t)ntiles * nkb * 128;
    size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= total) return;
    int grp = idx & 3, h = (idx >> 2) & 1, g = (idx >> 3) & 7, sub = (idx >> 6) & 1;
    size_t blk = idx >> 7;
    int kb = blk % nkb, tile = blk / nkb;
    int row = tile * TILE_ROWS + sub * 16 + h * 8 + g;
    int k = kb * BLOCK_K + grp * 32;
    uint8_t *sp = pk + blk * (size_t)chunk_bytes + sub * (chunk_bytes / 2) + 1024;
    int slot = ((g * 2 + (grp >> 1)) * 2 + h) * 2 + (grp & 1);
    if (mode == SC_MX) {
        const int e = static_cast<const uint8_t *>(raw_s)[(size_t)row * ng + k / 32];
        sp[slot] = (uint8_t)(e > e_min ? e : e_min);
    } else {
        float s = static_cast<const float *>(raw_s)[(size_t)row * ng + k / gs];
        if (mode == SC_H16) reinterpret_cast<__half *>(sp)[slot] = __float2half_rn(s);
        else reinterpret_cast<float *>(sp)[slot] = s;
    }
}

// ---------------------------------------------------------------------------
// Activation preparation. One warp per (row, 128-column block): find the
// block's largest magnitude, pick the power-of-two scale that puts it in
// [2^13, 2^14), split every scaled value into fp16 hi + fp16 lo (hi+lo keeps 22
// significant bits; lo may be subnormal, which tensor cores honour), and store
// both in B-fragment order: halfs[((grp*2 + hl)*4 + t)*8 + i] for column
// grp*32 + t*8 + i. The inverse scale goes to bscale[row*nkb + kb].
// ---------------------------------------------------------------------------
__device__ __forceinline__ float block_scale_from_max(float m) {
    // m >= 0. Returns 2^(13 - floor(log2 m)), clamped; 1 for zero / non-finite.
    uint32_t e = (__float_as_uint(m) >> 23) & 0xFFu;
    if (e == 0 || e == 255) return 1.f;
    int se = 267 - (int)e;            // biased exponent of the scale
    if (se > 247) se = 247;
    return __uint_as_float((uint32_t)se << 23);
}

__device__ __forceinline__ void store_split4(__half *blk, int lane, float4 v, float s) {
    // lane holds columns 4*lane .. 4*lane+3 of the block
    int k = lane * 4;
    int grp = k >> 5, t = (k & 31) >> 3, i0 = k & 7;
    float x[4] = {v.x * s, v.y * s, v.z * s, v.w * s};
    __half hi[4], lo[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        hi[i] = __float2half_rn(x[i]);
        lo[i] = __float2half_rn(x[i] - __half2float(hi[i]));
    }
    __half *ph = blk + ((grp * 2 + 0) * 4 + t) * 8 + i0;
    __half *pl = blk + ((grp * 2 + 1) * 4 + t) * 8 + i0;
    *reinterpret_cast<uint2 *>(ph) = make_uint2(
        (uint32_t)__half_as_ushort(hi[0]) | ((uint32_t)__half_as_ushort(hi[1]) << 16),
        (uint32_t)__half_as_ushort(hi[2]) | ((uint32_t)__half_as_ushort(hi[3]) << 16));
    *reinterpret_cast<uint2 *>(pl) = make_uint2(
        (uint32_t)__half_as_ushort(lo[0]) | ((uint32_t)__half_as_ushort(lo[1]) << 16),
        (uint32_t)__half_as_ushort(lo[2]) | ((uint32_t)__half_as_ushort(lo[3]) << 16));
}

__device__ __forceinline__ float warp_max(float m) {
#pragma unroll
    for (int o = 16; o; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    return m;
}

__global__ void k_prep_rows(__half *__restrict__ bq, float *__restrict__ bscale,
                            const float *x, int nrows, int K) {
    pdl_enter();
    const int nkb = K / BLOCK_K;
    int wid = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (wid >= nrows * nkb) return;
    int row = wid / nkb, kb = wid - row * nkb;
    float4 v = *reinterpret_cast<const float4 *>(x + (size_t)row * K + kb * BLOCK_K + lane * 4);
    float m = warp_max(fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w))));
    float s = block_scale_from_max(m);
    store_split4(bq + ((size_t)row * nkb + kb) * 256, lane, v, s);
    if (lane == 0) bscale[(size_t)row * nkb + kb] = 1.f / s;
}

// SwiGLU over the gate/up partial sums, fused with the preparation of the down
// projection's B operand. One warp per (pos, 128-wide block of I).
//   g = sum_kp pg[(kp*npos+pos)*I + o] (ascending kp), same for u;
//   h = g/(1+exp(-g)) * u
__global__ void k_swiglu_prep(__half *__restrict__ hq, float *__restrict__ hscale,
                              const float *pg, const float *pu,
                              const int *npos_p, int npos_cap, int I, int nkpart) {
    pdl_enter();
    const int npos = npos_p ? *npos_p : npos_cap;
    const int nkb = I / BLOCK_K;
    int wid = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (wid >= npos * nkb) return;
    int pos = wid / nkb, kb = wid - pos * nkb;
    float4 gsum = make_float4(0, 0, 0, 0), usum = gsum;
    for (int kp = 0; kp < nkpart; kp++) {
        size_t off = ((size_t)kp * npos + pos) * I + kb * BLOCK_K + lane * 4;
        float4 a = *reinterpret_cast<const float4 *>(pg + off);
        float4 b = *reinterpret_cast<const float4 *>(pu + off);
        gsum.x += a.x; gsum.y += a.y; gsum.z += a.z; gsum.w += a.w;
        usum.x += b.x; usum.y += b.y; usum.z += b.z; usum.w += b.w;
    }
    float4 h;
    h.x = (gsum.x / (1.0f + expf(-gsum.x))) * usum.x;
    h.y = (gsum.y / (1.0f + expf(-gsum.y))) * usum.y;
    h.z = (gsum.z / (1.0f + expf(-gsum.z))) * usum.z;
    h.w = (gsum.w / (1.0f + expf(-gsum.w))) * usum.w;
    float m = warp_max(fmaxf(fmaxf(fabsf(h.x), fabsf(h.y)), fmaxf(fabsf(h.z), fabsf(h.w))));
    float s = block_scale_from_max(m);
    store_split4(hq + ((size_t)pos * nkb + kb) * 256, lane, h, s);
    if (lane == 0) hscale[(size_t)pos * nkb + kb] = 1.f / s;
}

// y[pos, o] = sum_kp part[(kp*npos+pos)*O + o]  (ascending kp)
__global__ void k_reduce_parts(float *__restrict__ y, const float *part, int npos, int O,
                               int nkpart) {
    pdl_enter();
    size_t n = (size_t)npos * O / 4;
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float4 acc = make_float4(0, 0, 0, 0);
    for (int kp = 0; kp < nkpart; kp++) {
        float4 a = reinterpret_cast<const float4 *>(part + (size_t)kp * npos * O)[i];
        acc.x += a.x; acc.y += a.y; acc.z += a.z; acc.w += a.w;
    }
    reinterpret_cast<float4 *>(y)[i] = acc;
}

// Weighted combine of a layer: for token s,
//   out[s] = sum_{kk<keff[s]} w[s,kk] * Y[pos_of[s*K+kk]]  (+ Y[shared_pos0 + s])
// with Y[pos] = sum_kp part[(kp*npos+pos)*D + d]; selection order, shared last.
__global__ void k_combine(float *__restrict__ out, const float *part,
                          const int *pos_of, const float *wts,
                          const int *keff, const int *npos_p, int M, int K,
                          int D, int nkpart, const int *shared_pos0_p) {
    pdl_enter();
    const int npos = *npos_p;
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    int dq = D / 4;
    if (i >= (size_t)M * dq) return;
    int s = i / dq, d4 = i - (size_t)s * dq;
    float4 acc = make_float4(0, 0, 0, 0);
    int ke = keff[s], kk = 0;
    // one partial sum: four rows requested before the first is added (a row at a time, the two dependent loads of each
    // were waited for in turn)
    if (nkpart == 1) {
        for (; kk + 4 <= ke; kk += 4) {
            float4 y[4];
            float wgt[4];
#pragma unroll
            for (int j = 0; j < 4; j++) {
                wgt[j] = wts[s * K + kk + j];
                y[j] = reinterpret_cast<const float4 *>(part + (size_t)pos_of[s * K + kk + j] * D)[d4];
            }
#pragma unroll
            for (int j = 0; j < 4; j++) {
                acc.x += wgt[j] * (0.f + y[j].x); acc.y += wgt[j] * (0.f + y[j].y);
                acc.z += wgt[j] * (0.f + y[j].z); acc.w += wgt[j] * (0.f + y[j].w);
            }
        }
    }
    for (; kk < ke; kk++) {
        int pos = pos_of[s * K + kk];
        float wgt = wts[s * K + kk];
        float4 y = make_float4(0, 0, 0, 0);
        for (int kp = 0; kp < nkpart; kp++) {
            float4 a = reinterpret_cast<const float4 *>(part + ((size_t)kp * npos + pos) * D)[d4];
            y.x += a.x; y.y += a.y; y.z += a.z; y.w += a.w;
        }
        acc.x += wgt * y.x; acc.y += wgt * y.y; acc.z += wgt * y.z; acc.w += wgt * y.w;
    }
    if (shared_pos0_p) {
        int pos = *shared_pos0_p + s;
        float4 y = make_float4(0, 0, 0, 0);
        for (int kp = 0; kp < nkpart; kp++) {
            float4 a = reinterpret_cast<const float4 *>(part + ((size_t)kp * npos + pos) * D)[d4];
            y.x += a.x; y.y += a.y; y.z += a.z; y.w += a.w;
        }
        acc.x += y.x; acc.y += y.y; acc.z += y.z; acc.w += y.w;
    }
    reinterpret_cast<float4 *>(out)[i] = acc;
}

// Weighted combine over separate buffers (expert-parallel layer): for row s,
//   out[s] = sum_{kk<keff[s]} w[s,kk] * y[entry_of[s*K+kk]]  (+ shared[s]),
// selection order, shared expert last. entry_of is 64-bit (a torch index tensor).
__global__ void k_combine_rows(float *__restrict__ out, const float *y,
                               const long long *entry_of, const float *wts,
                               const long long *keff, const float *shared, int M,
                               int K, int D) {
    pdl_enter();
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    int dq = D / 4;
    if (i >= (size_t)M * dq) return;
    int s = i / dq, d4 = i - (size_t)s * dq;
    float4 acc = make_float4(0, 0, 0, 0);
    int ke = (int)keff[s];
    for (int kk = 0; kk < ke; kk++) {
        long long pos = entry_of[s * K + kk];
        float wgt = wts[s * K + kk];
        float4 a = reinterpret_cast<const float4 *>(y + (size_t)pos * D)[d4];
        acc.x += wgt * a.x; acc.y += wgt * a.y; acc.z += wgt * a.z; acc.w += wgt * a.w;
    }
    if (shared) {
        float4 a = reinterpret_cast<const float4 *>(shared + (size_t)s * D)[d4];
        acc.x += a.x; acc.y += a.y; acc.z += a.z; acc.w += a.w;
    }
    reinterpret_cast<float4 *>(out)[i] = acc;
}

// ---------------------------------------------------------------------------
// Generic matmul, for what the row-major kernels leave: f32 rows that are not 16-byte aligned, int4 groups that are not
// whole groups of 32 columns, and FP8 with a table other than E4M3's own whose rows are not 16-byte aligned. Any
// shape: one warp per output row o and chunk of up to 8 input rows; lanes stride over columns,
// products in f32, shuffle reduction. y[s*O+o].
// ---------------------------------------------------------------------------
__device__ float d_e4m3_lut[256];     // decode table of fmt 8, set by coli_cuda_fp8_set_lut

__device__ __forceinline__ float raw_weight(const void *w, const void *sc, int fmt, int I, int gs,
                                            int ng, int o, int i) {
    if (fmt == 0) return static_cast<const float *>(w)[(size_t)o * I + i];
    if (fmt == 8)      // ng = 128-column blocks per row; one scale per 128x128 block
        return d_e4m3_lut[static_cast<const uint8_t *>(w)[(size_t)o * I + i]] *
               static_cast<const float *>(sc)[(size_t)(o >> 7) * ng + (i >> 7)];
    const uint8_t v = static_cast<const uint8_t *>(w)[(size_t)o * ((I + 1) / 2) + (i >> 1)];      // fmt 4
    const int n = (i & 1) ? (v >> 4) : (v & 15);
    return (float)(n - 8) * static_cast<const float *>(sc)[(size_t)o * ng + i / gs];
}

__global__ void k_generic_matmul(float *__restrict__ y, const float *x, const void *w,
                                 const void *sc, int fmt, int S, int I, int O, int gs, int ng) {
    pdl_enter();
    int o = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    int lane = threadIdx.x & 31;
    int s0 = blockIdx.y * 8;
    if (o >= O) return;
    float acc[8];
#pragma unroll
    for (int r = 0; r < 8; r++) acc[r] = 0.f;
    int ns = min(8, S - s0);
    for (int i = lane; i < I; i += 32) {
        float wv = raw_weight(w, sc, fmt, I, gs, ng, o, i);
#pragma unroll
        for (int r = 0; r < 8; r++)
            if (r < ns) acc[r] = fmaf(x[(size_t)(s0 + r) * I + i], wv, acc[r]);
    }
#pragma unroll
    for (int r = 0; r < 8; r++) {
        float a = acc[r];
#pragma unroll
        for (int off = 16; off; off >>= 1) a += __shfl_xor_sync(0xffffffffu, a, off);
        if (lane == 0 && r < ns) y[(size_t)(s0 + r) * O + o] = a;
    }
}

// ---------------------------------------------------------------------------
// Streaming GEMV for row-major tensors whose rows are 16-byte aligned: fmt 0 (f32, e.g. a
// vocabulary head) and fmt 8 (FP8 bytes with one f32 scale per 128x128 block) with a decode
// table other than E4M3's own. Bound by HBM: every weight byte is read once with 128-bit loads.
//   y[s*O + o] = sum_i x[s,i] * w[o,i]
// One warp owns 4 output rows and up to 8 rows of x (blockIdx.y selects the group of 8);
// the CTA stages 1024 columns of those x rows in shared memory per round (two buffers, filled
// by asynchronous copies while the previous round is multiplied: one CTA barrier per round), a
// lane takes 16-byte pieces of its 4 weight rows, always one piece ahead of the one it
// multiplies (also across rounds, so weight loads stay in flight while x is staged), so x
// costs one shared-memory read per 4 output rows. Requires I % 16 == 0 (fmt 0: I % 4 == 0).
// Dynamic shared memory: DENSE_GEMV_SMEM bytes.
// ---------------------------------------------------------------------------
#define DENSE_GEMV_CK 1024
#define DENSE_GEMV_SMEM (2 * 8 * DENSE_GEMV_CK * 4)
template <int FMT>
__global__ void __launch_bounds__(256, FMT == 0 ? 3 : 2) k_dense_gemv(float *__restrict__ y, const float *x,
                                                    const void *__restrict__ w, const float *sc,
                                                    const float *lut, int S, int I, int O) {
    pdl_enter();
    constexpr int VPL = FMT == 0 ? 4 : 16;          // values in one 16-byte piece
    constexpr int CK = DENSE_GEMV_CK;               // columns of x staged per round
    constexpr int PIECES = CK / (32 * VPL);
    extern __shared__ __align__(16) float xs[];     // [2][8][CK]
    __shared__ float s_lut[256];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int s0 = blockIdx.y * 8, ns = min(8, S - s0);
    const int o0 = (blockIdx.x * 8 + warp) * 4;
    if (FMT == 8) s_lut[tid] = lut[tid];
    float acc[4][8];
#pragma unroll
    for (int r = 0; r < 4; r++)
#pragma unroll
        for (int q = 0; q < 8; q++) acc[r][q] = 0.f;
    const size_t rowb = FMT == 0 ? (size_t)I * 4 : (size_t)I;       // bytes per weight row
    const uint8_t *wb = static_cast<const uint8_t *>(w);
    const int nblk = (I + 127) >> 7;
    // rows of x this CTA does not have read as zeros, in both buffers, for good
    for (int idx = tid; idx < 2 * 8 * CK / 4; idx += 256) {
        const int q = (idx / (CK / 4)) & 7;
        if (q >= ns) reinterpret_cast<float4 *>(xs)[idx] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    auto stage = [&](int c0, int buf) {
        for (int idx = tid; idx < 8 * CK / 4; idx += 256) {
            const int q = idx / (CK / 4), j = idx - q * (CK / 4), col = c0 + j * 4;
            if (q < ns && col < I) {
                const uint32_t dst = (uint32_t)__cvta_generic_to_shared(xs + (size_t)buf * 8 * CK) + idx * 16;
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(x + (size_t)(s0 + q) * I + col) : "memory");
            }
        }
    };
    auto load_piece = [&](int col, uint4 (&raw)[4]) {
#pragma unroll
        for (int r = 0; r < 4; r++)
            raw[r] = (col < I && o0 + r < O)
                         ? __ldcs(reinterpret_cast<const uint4 *>(wb + (size_t)(o0 + r) * rowb + (size_t)col * (FMT == 0 ? 4 : 1)))
                         : make_uint4(0, 0, 0, 0);
    };
    uint4 cur[4], nxt[4];
    load_piece(lane * VPL, cur);
    stage(0, 0);
    int round = 0;
    for (int c0 = 0; c0 < I; c0 += CK, round++) {
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();            // this round's x is in place; nobody reads the other buffer any more
        if (c0 + CK < I) stage(c0 + CK, (round + 1) & 1);
        const float *xb = xs + (size_t)(round & 1) * 8 * CK;
#pragma unroll
        for (int p = 0; p < PIECES; p++) {
            const int col = c0 + (p * 32 + lane) * VPL;
            load_piece(col + 32 * VPL, nxt);        // the next piece, possibly the next round's first
            if (col < I) {
                if (FMT == 0) {
#pragma unroll
                    for (int q = 0; q < 8; q++) {
                        const float4 xv = reinterpret_cast<const float4 *>(xb)[q * (CK / 4) + ((col - c0) >> 2)];
#pragma unroll
                        for (int r = 0; r < 4; r++) {
                            const float4 wv = make_float4(__uint_as_float(cur[r].x), __uint_as_float(cur[r].y),
                                                          __uint_as_float(cur[r].z), __uint_as_float(cur[r].w));
                            acc[r][q] = fmaf(wv.w, xv.w, fmaf(wv.z, xv.z, fmaf(wv.y, xv.y, fmaf(wv.x, xv.x, acc[r][q]))));
                        }
                    }
                } else {
                    float wd[4][16];
#pragma unroll
                    for (int r = 0; r < 4; r++) {
                        const float bs = o0 + r < O ? sc[(size_t)((o0 + r) >> 7) * nblk + (col >> 7)] : 1.f;
                        const uint32_t wds[4] = {cur[r].x, cur[r].y, cur[r].z, cur[r].w};
#pragma unroll
                        for (int b = 0; b < 16; b++) {
                            const uint32_t byte = (wds[b >> 2] >> (8 * (b & 3))) & 0xFFu;
                            wd[r][b] = s_lut[byte] * bs;
                        }
                    }
#pragma unroll
                    for (int q = 0; q < 8; q++) {
                        float4 xv[4];
#pragma unroll
                        for (int k = 0; k < 4; k++)
                            xv[k] = reinterpret_cast<const float4 *>(xb)[q * (CK / 4) + ((col - c0) >> 2) + k];
#pragma unroll
                        for (int r = 0; r < 4; r++) {
                            float a = acc[r][q];
#pragma unroll
                            for (int k = 0; k < 4; k++) {
                                a = fmaf(wd[r][4 * k + 0], xv[k].x, a); a = fmaf(wd[r][4 * k + 1], xv[k].y, a);
                                a = fmaf(wd[r][4 * k + 2], xv[k].z, a); a = fmaf(wd[r][4 * k + 3], xv[k].w, a);
                            }
                            acc[r][q] = a;
                        }
                    }
                }
            }
#pragma unroll
            for (int r = 0; r < 4; r++) cur[r] = nxt[r];
        }
    }
#pragma unroll
    for (int r = 0; r < 4; r++)
#pragma unroll
        for (int q = 0; q < 8; q++) {
            float a = acc[r][q];
#pragma unroll
            for (int off = 16; off; off >>= 1) a += __shfl_xor_sync(0xffffffffu, a, off);
            if (lane == 0 && q < ns && o0 + r < O)
                y[(size_t)(s0 + q) * O + o0 + r] = a;
        }
}

// Interleaved rotary embedding of the resident pipeline (the arithmetic of
// c/backend_cuda.cu:2049-2063): block b rotates the R floats at v + b*stride + offset by
// the angle of position pos[b / heads] (or pos_base + b / heads): pair (2j, 2j+1) of the
// input lands at (j, R/2 + j).
__global__ void k_rope_rows(float *v, const int *pos, int pos_base, int stride, int offset, int R, int heads,
                            float theta) {
    pdl_enter();
    float *p = v + (size_t)blockIdx.x * stride + offset;
    const int half = R / 2;
    const int ps = pos ? pos[blockIdx.x / heads] : pos_base + (int)(blockIdx.x / heads);
    __shared__ float in[256];
    for (int j = threadIdx.x; j < R; j += blockDim.x) in[j] = p[j];
    __syncthreads();
    for (int j = threadIdx.x; j < half; j += blockDim.x) {
        const float inv = powf(theta, -2.0f * (float)j / (float)R);
        const float ang = (float)ps * inv;
        float sn, cs;
        sincosf(ang, &sn, &cs);
        const float a = in[2 * j], b = in[2 * j + 1];
        p[j] = a * cs - b * sn;
        p[half + j] = b * cs + a * sn;
    }
}

// ---------------------------------------------------------------------------
// Elementwise / row primitives of the resident pipeline.
// ---------------------------------------------------------------------------
// Rows from pinned host memory to device memory.
__global__ void k_pull(float4 *__restrict__ dst, const float4 *src, int n4) {
    pdl_enter();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n4) dst[i] = src[i];
}

__global__ void k_silu_mul(float *g, const float *u, size_t n) {
    pdl_enter();
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) { float v = g[i]; g[i] = (v / (1.0f + expf(-v))) * u[i]; }
}
__global__ void k_add(float *x, const float *t, size_t n) {
    pdl_enter();
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) x[i] += t[i];
}
// Block b adds partial row b into x row rows[b]; target rows are distinct.
__global__ void k_rows_add(float *x, const float *partial, const int *rows, int D) {
    pdl_enter();
    float *xr = x + (size_t)rows[blockIdx.x] * D;
    const float *pr = partial + (size_t)blockIdx.x * D;
    for (int i = threadIdx.x; i < D; i += blockDim.x) xr[i] += pr[i];
}
// y = (x * r) * w with r = 1 / sqrtf((float)(sum(x^2) / D) + eps), the sum in double and the
// rest in correctly rounded f32 operations (the arithmetic of c/colibri.c:1193-1196).
// One CTA of 1024 threads per row: with 256 the row's loads came 24 in a row per thread (20 us for one row of
// 6144 including the launch). 16-byte accesses when the rows allow them.
#define RMSNORM_THREADS 1024
__global__ void __launch_bounds__(RMSNORM_THREADS) k_rmsnorm(float *y, const float *x, const float *w, int D, float eps, int xstride,
                                                             int ystride) {
    pdl_enter();
    const float *xr = x + (size_t)blockIdx.x * xstride;
    float *yr = y + (size_t)blockIdx.x * ystride;
    __shared__ double sh[32];
    const bool v4 = D % 4 == 0 && ((reinterpret_cast<uintptr_t>(xr) | reinterpret_cast<uintptr_t>(yr) | reinterpret_cast<uintptr_t>(w)) & 15) == 0;
    double a = 0;
    float4 keep[2];                                     // rows up to 8192 stay in registers
    if (v4) {
#pragma unroll
        for (int j = 0; j < 2; j++) {
            const int i = threadIdx.x + j * RMSNORM_THREADS;
            keep[j] = i < D / 4 ? reinterpret_cast<const float4 *>(xr)[i] : make_float4(0.f, 0.f, 0.f, 0.f);
            a += (double)keep[j].x * keep[j].x + (double)keep[j].y * keep[j].y + (double)keep[j].z * keep[j].z + (double)keep[j].w * keep[j].w;
        }
        for (int i = threadIdx.x + 2 * RMSNORM_THREADS; i < D / 4; i += RMSNORM_THREADS) {
            const float4 v = reinterpret_cast<const float4 *>(xr)[i];
            a += (double)v.x * v.x + (double)v.y * v.y + (double)v.z * v.z + (double)v.w * v.w;
        }
    } else {
        for (int i = threadIdx.x; i < D; i += RMSNORM_THREADS) { double v = xr[i]; a += v * v; }
    }
#pragma unroll
    for (int off = 16; off; off >>= 1) a += __shfl_xor_sync(0xffffffffu, a, off);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = a;
    __syncthreads();
    double b = sh[threadIdx.x & 31];
#pragma unroll
    for (int off = 16; off; off >>= 1) b += __shfl_xor_sync(0xffffffffu, b, off);
    const float r = __fdiv_rn(1.f, __fsqrt_rn(__fadd_rn((float)(b / D), eps)));
    if (v4) {
        auto out = [&](int i, const float4 &v) {
            const float4 ww = reinterpret_cast<const float4 *>(w)[i];
            reinterpret_cast<float4 *>(yr)[i] = make_float4(__fmul_rn(__fmul_rn(v.x, r), ww.x), __fmul_rn(__fmul_rn(v.y, r), ww.y),
                                                            __fmul_rn(__fmul_rn(v.z, r), ww.z), __fmul_rn(__fmul_rn(v.w, r), ww.w));
        };
#pragma unroll
        for (int j = 0; j < 2; j++) if (threadIdx.x + j * RMSNORM_THREADS < D / 4) out(threadIdx.x + j * RMSNORM_THREADS, keep[j]);
        for (int i = threadIdx.x + 2 * RMSNORM_THREADS; i < D / 4; i += RMSNORM_THREADS) out(i, reinterpret_cast<const float4 *>(xr)[i]);
    } else {
        for (int i = threadIdx.x; i < D; i += RMSNORM_THREADS) yr[i] = __fmul_rn(__fmul_rn(xr[i], r), w[i]);
    }
}
// out[i] = sum_c w[c] * y[c*D+i] in call order (resident group accumulate)
__global__ void k_weighted_sum_rows(float *out, const float *y, const float *w, int count, int D) {
    pdl_enter();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < D; i += gridDim.x * blockDim.x) {
        float acc = 0.f;
        for (int c = 0; c < count; c++) acc += w[c] * y[(size_t)c * D + i];
        out[i] = acc;
    }
}
__global__ void k_sum_slots(float *dst, const float *slots, int n, int D) {
    pdl_enter();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < D; i += gridDim.x * blockDim.x) {
        float acc = 0.f;
        for (int s = 0; s < n; s++) acc += slots[(size_t)s * D + i];
        dst[i] = acc;
    }
}

// Row-wise argmax with the engine's scan semantics (c/olmoe.c:966-967, c/colibri.c greedy
// pick): best = 0, then every i with x[i] > x[best] in ascending order, i.e. the first index
// of the largest value, NaNs never winning; a NaN in x[0] keeps the answer at 0.
// A row is shared by a cluster of ARGMAX_CLUSTER CTAs whose answers meet in the first one's shared memory: one CTA
// per row took 35 us for 8 rows of 129280, waiting for its own loads. The first CTA's shared memory may be addressed
// only once that CTA is known to run: every CTA arrives at the cluster barrier on entry and waits for it before its
// answer leaves, with the row's loads in between.
#define ARGMAX_CLUSTER 8
__device__ __forceinline__ void argmax_take(float &bv, int &bi, float v, int i) {
    if (v > bv || (v == bv && i < bi)) { bv = v; bi = i; }
}
__global__ void __cluster_dims__(ARGMAX_CLUSTER, 1, 1) __launch_bounds__(1024) k_argmax_rows(int *__restrict__ out, const float *x,
                                                                                             int N) {
    pdl_enter();
    asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
    const int part = blockIdx.x % ARGMAX_CLUSTER, r = blockIdx.x / ARGMAX_CLUSTER, tid = threadIdx.x;
    const float *row = x + (size_t)r * N;
    __shared__ float sv[32];
    __shared__ int si[32];
    __shared__ float cv[ARGMAX_CLUSTER];
    __shared__ int ci[ARGMAX_CLUSTER];
    const int per = (N + ARGMAX_CLUSTER - 1) / ARGMAX_CLUSTER, i0 = part * per, i1 = min(N, i0 + per);
    float bv = -INFINITY;
    int bi = 0x7fffffff;
#pragma unroll 4
    for (int i = i0 + tid; i < i1; i += 1024) argmax_take(bv, bi, row[i], i);
    auto warp_best = [&]() {
#pragma unroll
        for (int off = 16; off; off >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, bv, off);
            const int oi = __shfl_xor_sync(0xffffffffu, bi, off);
            argmax_take(bv, bi, ov, oi);
        }
    };
    warp_best();
    if ((tid & 31) == 0) { sv[tid >> 5] = bv; si[tid >> 5] = bi; }
    __syncthreads();
    asm volatile("barrier.cluster.wait.aligned;" ::: "memory");         // every CTA of the cluster runs
    if (tid < 32) {
        bv = sv[tid]; bi = si[tid];
        warp_best();
        if (tid == 0) {
            uint32_t dv, di;
            asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(dv) : "r"((uint32_t)__cvta_generic_to_shared(cv + part)), "r"(0));
            asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(di) : "r"((uint32_t)__cvta_generic_to_shared(ci + part)), "r"(0));
            asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(dv), "f"(bv) : "memory");
            asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(di), "r"(bi) : "memory");
        }
        __syncwarp();
    }
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    if (part == 0 && tid == 0) {
        bv = -INFINITY; bi = 0x7fffffff;
        for (int i = 0; i < ARGMAX_CLUSTER; i++) argmax_take(bv, bi, cv[i], ci[i]);
        const float first = row[0];
        out[r] = (first != first || bi == 0x7fffffff) ? 0 : bi;
    }
}
