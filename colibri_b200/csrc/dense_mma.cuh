// Matmul of row-major quantised tensors (everything the packed layout does not cover except f32):
// int8, int4 (per row or grouped), int2, MXFP4 and FP8 E4M3, any shape, any number of rows.
//
//   y[s*O + o] = sum_i x[s,i] * w[o,i]
//
// A CTA owns 32 output rows and up to 4*NC rows of x; its 8 warps split the contraction by 128-column
// blocks and add their sums in shared memory. A lane's 16- or 4-byte loads of weight rows g, g+8, g+16,
// g+24 are tensor-core A fragments after an exact conversion to fp16 (the contraction order is a
// permutation that the activations are prepared in), the activations come as an fp16 (hi, lo) pair
// with a power-of-two scale per (row, 128 columns), laid out so that a lane reads its B fragments with
// 16-byte loads; column 2r of an MMA is row r's hi part, 2r+1 its lo part. Weight and activation scales are
// applied in f32 once per block (grouped formats: per 32 columns).
// Why: the scalar kernel before it decoded every weight to f32 and multiplied it with 8 rows by
// FFMA, through a 256-entry shared-memory table for FP8: 163 us at 6144 x 8192 FP8 and 12 rows, 22 so (50 MB at 2.3 TB/s). Bound by the
// latency of its loads (a warp multiplies a block with nothing of the next one requested), and 256 CTAs leave some of 148 SMs with
// two and some with one.
// CTAS: CTAs that share an SM; the registers of a thread are capped to that (0: the compiler's own choice). More than 8 rows take
// 180 to 245 of them, and with one CTA per SM a second wave runs behind the first; so when there are more CTAs than SMs the cap is for
// two (and spills a little: 1 % slower where there are fewer CTAs than SMs, so not there). Fewer rows take two to four by format and
// number of CTAs (launch_dense, with the figures). AHEAD: the activations' fragments are requested together before the decoding, except under
// that cap at more than 8 rows, where they cost more spills than they save waiting (ahead / not, 48 rows of 6144 x 8192: int8 68 / 57, FP8 56 / 53;
// of 6150 x 8192: MXFP4 128 / 119, per-row int4 114 / 109). Call times before both / with both, 12 rows of 6144 x 8192: FP8 43 / 33, 2-bit 67 /
// 42, of 6150 x 8200: grouped int4 116 / 71, MXFP4 90 / 61, per-row int4 102 / 57. Requesting
// half a block or a block ahead was slower for rows on 16 bytes (FP8 33 / 38), for the registers it takes.
// Rows need no alignment: without 16-byte rows, words come from aligned loads and funnel shifts, a run of 16 bytes from five (FP8, 6150
// columns: 12 rows 132 / 50 us, one row 67 / 34, with a pair of loads for every word 72 and 67); raw
// tensors carry 16 spare bytes at the end; columns beyond I are masked.
#pragma once
#include "common.cuh"
#include "gemv_stream.cuh"
#include "kernels_misc.cuh"

#define DENSE_WARPS 8

// formats whose lane run is 16 columns of a 64-column half block; else (4-bit) 8 columns of each 32-column group
__host__ __device__ constexpr bool dense_run16(int fmt) { return fmt == 1 || fmt == 3 || fmt == 8; }

// Where column k (0..127) of a block goes among its 256 halfs; the lo part lies dense_lo_off further.
__device__ __forceinline__ int dense_pos(int fmt, int k) {
    if (dense_run16(fmt)) {
        int i = k & 15;
        if (fmt == 3) i = (i & 7) * 2 + (i >> 3);              // 2-bit fields j and j + 8 of a word form a pair
        return ((k >> 6) * 8 + ((k >> 4) & 3)) * 16 + i;
    }
    int i = k & 7;
    if (fmt != 7) i = (i & 3) * 2 + (i >> 2);                  // nibbles j and j + 4
    return ((k >> 5) * 8 + ((k >> 3) & 3)) * 8 + i;
}
__host__ __device__ constexpr int dense_lo_off(int fmt) { return dense_run16(fmt) ? 64 : 32; }

// One warp per (row, block): power-of-two scale, hi and lo parts; columns beyond I are zero.
__global__ void k_prep_dense(__half *__restrict__ bq, float *__restrict__ bscale, const float *x, int S, int I, int fmt) {
    pdl_enter();
    const int nkb = (I + 127) / 128, wid = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (wid >= S * nkb) return;
    const int row = wid / nkb, kb = wid - row * nkb;
    float v[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int k = kb * 128 + i * 32 + lane;
        v[i] = k < I ? x[(size_t)row * I + k] : 0.f;
    }
    const float m = warp_max(fmaxf(fmaxf(fabsf(v[0]), fabsf(v[1])), fmaxf(fabsf(v[2]), fabsf(v[3]))));
    const float s = block_scale_from_max(m);
    __half *blk = bq + (size_t)wid * 256;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const float a = v[i] * s;
        const __half hi = __float2half_rn(a);
        const int p = dense_pos(fmt, i * 32 + lane);
        blk[p] = hi;
        blk[p + dense_lo_off(fmt)] = __float2half_rn(a - __half2float(hi));
    }
    if (lane == 0) bscale[wid] = 1.f / s;
}

// W values of a 32-bit word as half2 pairs, exact.
__device__ __forceinline__ void dense_i8x4(uint32_t q, uint32_t (&v)[2]) {
    // b + 128 as the low byte of 1024 + n, minus 1152
    const uint32_t u = q ^ 0x80808080u;
    const __half2 k1152 = __floats2half2_rn(1152.f, 1152.f);
    v[0] = h2_as_u32(__hsub2(u32_as_h2(__byte_perm(u, 0x64646464u, 0x4140)), k1152));
    v[1] = h2_as_u32(__hsub2(u32_as_h2(__byte_perm(u, 0x64646464u, 0x4342)), k1152));
}
__device__ __forceinline__ void dense_f8x4(uint32_t q, uint32_t (&v)[2]) {
    asm("{\n\t.reg .b16 a, b;\n\t"
        "mov.b32 {a, b}, %2;\n\t"
        "cvt.rn.f16x2.e4m3x2 %0, a;\n\t"
        "cvt.rn.f16x2.e4m3x2 %1, b;\n\t}"
        : "=r"(v[0]), "=r"(v[1]) : "r"(q));
}
__device__ __forceinline__ void dense_i4x8(uint32_t q, uint32_t (&v)[4]) {       // pairs (j, j + 4)
    const __half2 k1032 = __floats2half2_rn(1032.f, 1032.f);
#pragma unroll
    for (int j = 0; j < 4; j++) v[j] = h2_as_u32(__hsub2(u32_as_h2(((q >> (4 * j)) & 0x000F000Fu) | c_magic_1024), k1032));
}
__device__ __forceinline__ void dense_i2x16(uint32_t q, uint32_t (&v)[8]) {      // pairs (j, j + 8)
    const __half2 k1026 = __floats2half2_rn(1026.f, 1026.f);
#pragma unroll
    for (int j = 0; j < 8; j++) v[j] = h2_as_u32(__hsub2(u32_as_h2(((q >> (2 * j)) & 0x00030003u) | c_magic_1024), k1026));
}

template <int FMT, int NC, bool AL16, int CTAS>
__global__ void __launch_bounds__(DENSE_WARPS * 32, CTAS) k_dense_mma(float *__restrict__ y, const __half *bq,
                                                                const float *bscale, const uint8_t *__restrict__ w,
                                                                const void *sc, int S, int I, int O, size_t rowb,
                                                                int gs, int ng) {
    pdl_enter();
    constexpr bool RUN16 = dense_run16(FMT);
    constexpr bool AHEAD = NC < 4 || CTAS == 1;         // all sets' fragments are requested together, before the decoding
    constexpr int VPW = (FMT == 1 || FMT == 8) ? 4 : FMT == 3 ? 16 : 8;      // values per 32-bit word
    __shared__ float2 s_part[DENSE_WARPS][NC][2][32];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int o0 = blockIdx.x * 32, s0 = blockIdx.y * 4 * NC, nkb = (I + 127) >> 7;
    const uint8_t *wr[4];                              // rows g, g + 8, g + 16, g + 24 (the last row for those beyond O)
    int orow[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
        orow[j] = min(o0 + j * 8 + g, O - 1);
        wr[j] = w + (size_t)orow[j] * rowb;
    }
    // B fragments: column g of set cs is row cs*4 + g/2, part g & 1; results: this lane's columns are row cs*4 + t
    const __half *bp[NC];
    const float *sp[NC];
#pragma unroll
    for (int cs = 0; cs < NC; cs++) {
        const int rb = min(s0 + cs * 4 + (g >> 1), S - 1), rs = min(s0 + cs * 4 + t, S - 1);
        bp[cs] = bq + (size_t)rb * nkb * 256 + (g & 1) * dense_lo_off(FMT) + t * (RUN16 ? 16 : 8);
        sp[cs] = bscale + (size_t)rs * nkb;
    }
    auto word = [&](int j, int k) -> uint32_t {        // the 32-bit word of row j that holds columns k ...
        if (k >= I) return 0;
        const size_t b = (size_t)k * 4 / VPW;
        uint32_t q;
        const uint8_t *p = wr[j] + b;
        const uintptr_t a = reinterpret_cast<uintptr_t>(p);
        const uint32_t *pa = reinterpret_cast<const uint32_t *>(a & ~(uintptr_t)3);
        const int sh = (int)(a & 3) * 8;
        q = __ldg(pa);
        if (sh) q = __funnelshift_r(q, __ldg(pa + 1), sh);
        if (k + VPW > I) q &= 0xFFFFFFFFu >> ((VPW - (I - k)) * (32 / VPW));
        return q;
    };
    float R[NC][2][4];
#pragma unroll
    for (int cs = 0; cs < NC; cs++)
#pragma unroll
        for (int m = 0; m < 2; m++)
#pragma unroll
            for (int i = 0; i < 4; i++) R[cs][m][i] = 0.f;
    for (int kb = warp; kb < nkb; kb += DENSE_WARPS) {
        const int k0 = kb * 128;
        uint32_t q[4][RUN16 ? (FMT == 3 ? 2 : 8) : 4];         // this block's words, by row
#pragma unroll
        for (int j = 0; j < 4; j++) {
            if (FMT == 1 || FMT == 8) {
#pragma unroll
                for (int c = 0; c < 2; c++) {
                    const int k = k0 + c * 64 + t * 16;
                    if (AL16) {
                        const uint4 u = k < I ? __ldcs(reinterpret_cast<const uint4 *>(wr[j] + k)) : make_uint4(0, 0, 0, 0);
                        q[j][c * 4] = u.x; q[j][c * 4 + 1] = u.y; q[j][c * 4 + 2] = u.z; q[j][c * 4 + 3] = u.w;
                    } else {
                        // 16 bytes that start anywhere: five aligned words, of which none starts behind the row
                        const uintptr_t at = reinterpret_cast<uintptr_t>(wr[j]) + k, end = reinterpret_cast<uintptr_t>(wr[j]) + I;
                        const uint32_t *pa = reinterpret_cast<const uint32_t *>(at & ~(uintptr_t)3);
                        uint32_t r[5];
#pragma unroll
                        for (int i = 0; i < 5; i++) r[i] = reinterpret_cast<uintptr_t>(pa + i) < end ? __ldg(pa + i) : 0;
#pragma unroll
                        for (int i = 0; i < 4; i++) {
                            const int left = I - k - i * 4;        // bytes of the row in this word
                            q[j][c * 4 + i] = __funnelshift_r(r[i], r[i + 1], (int)(at & 3) * 8) &
                                              (left >= 4 ? 0xFFFFFFFFu : left <= 0 ? 0u : 0xFFFFFFFFu >> (32 - 8 * left));
                        }
                    }
                }
            } else if (FMT == 3) {
#pragma unroll
                for (int c = 0; c < 2; c++) q[j][c] = word(j, k0 + c * 64 + t * 16);
            } else {
#pragma unroll
                for (int c = 0; c < 4; c++) q[j][c] = word(j, k0 + c * 32 + t * 8);
            }
        }
        float ixs[NC];
#pragma unroll
        for (int cs = 0; cs < NC; cs++) ixs[cs] = sp[cs][kb];
        float bacc[NC][2][4];
#pragma unroll
        for (int cs = 0; cs < NC; cs++)
#pragma unroll
            for (int m = 0; m < 2; m++)
#pragma unroll
                for (int i = 0; i < 4; i++) bacc[cs][m][i] = 0.f;
        if (RUN16) {
#pragma unroll
            for (int c = 0; c < 2; c++) {
                uint4 b[NC][2];
#pragma unroll
                for (int cs = 0; AHEAD && cs < NC; cs++) {
                    b[cs][0] = ldg128(bp[cs] + (size_t)kb * 256 + c * 128);
                    b[cs][1] = ldg128(bp[cs] + (size_t)kb * 256 + c * 128 + 8);
                }
                uint32_t v[4][8];                              // by row: the run's 16 columns as 8 pairs
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    if (FMT == 3) dense_i2x16(q[j][c], v[j]);
                    else
#pragma unroll
                        for (int i = 0; i < 4; i++) {
                            uint32_t p[2];
                            if (FMT == 8) dense_f8x4(q[j][c * 4 + i], p); else dense_i8x4(q[j][c * 4 + i], p);
                            v[j][2 * i] = p[0]; v[j][2 * i + 1] = p[1];
                        }
                }
#pragma unroll
                for (int cs = 0; cs < NC; cs++) {
                    const uint4 b0 = AHEAD ? b[cs][0] : ldg128(bp[cs] + (size_t)kb * 256 + c * 128);
                    const uint4 b1 = AHEAD ? b[cs][1] : ldg128(bp[cs] + (size_t)kb * 256 + c * 128 + 8);
#pragma unroll
                    for (int m = 0; m < 2; m++) {
                        mma_f16(bacc[cs][m], v[2 * m][0], v[2 * m + 1][0], v[2 * m][1], v[2 * m + 1][1], b0.x, b0.y);
                        mma_f16(bacc[cs][m], v[2 * m][2], v[2 * m + 1][2], v[2 * m][3], v[2 * m + 1][3], b0.z, b0.w);
                        mma_f16(bacc[cs][m], v[2 * m][4], v[2 * m + 1][4], v[2 * m][5], v[2 * m + 1][5], b1.x, b1.y);
                        mma_f16(bacc[cs][m], v[2 * m][6], v[2 * m + 1][6], v[2 * m][7], v[2 * m + 1][7], b1.z, b1.w);
                    }
                }
            }
            if (FMT == 8) {                                    // one scale per 128 x 128 weights
                const float bs = static_cast<const float *>(sc)[(size_t)(o0 >> 7) * nkb + kb];
#pragma unroll
                for (int cs = 0; cs < NC; cs++) ixs[cs] *= bs;
            }
        } else {
#pragma unroll
            for (int c = 0; c < 4; c++) {
                uint4 bf[NC];
#pragma unroll
                for (int cs = 0; AHEAD && cs < NC; cs++) bf[cs] = ldg128(bp[cs] + (size_t)kb * 256 + c * 64);
                uint32_t v[4][4];
                float sw[4] = {1.f, 1.f, 1.f, 1.f};
                const int k = k0 + c * 32;
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    if (FMT == 7) decode_word<SC_MX>(q[j][c], v[j]); else dense_i4x8(q[j][c], v[j]);
                    if (FMT == 7) sw[j] = k < I ? __uint_as_float((uint32_t)static_cast<const uint8_t *>(sc)[(size_t)orow[j] * ng + (k >> 5)] << 23) : 0.f;
                    if (FMT == 4) sw[j] = k < I ? static_cast<const float *>(sc)[(size_t)orow[j] * ng + k / gs] : 0.f;
                }
#pragma unroll
                for (int cs = 0; cs < NC; cs++) {
                    const uint4 b = AHEAD ? bf[cs] : ldg128(bp[cs] + (size_t)kb * 256 + c * 64);
#pragma unroll
                    for (int m = 0; m < 2; m++) {
                        float acc[4] = {0.f, 0.f, 0.f, 0.f};
                        mma_f16(acc, v[2 * m][0], v[2 * m + 1][0], v[2 * m][1], v[2 * m + 1][1], b.x, b.y);
                        mma_f16(acc, v[2 * m][2], v[2 * m + 1][2], v[2 * m][3], v[2 * m + 1][3], b.z, b.w);
#pragma unroll
                        for (int i = 0; i < 4; i++) bacc[cs][m][i] = fmaf(acc[i], sw[2 * m + (i >> 1)], bacc[cs][m][i]);
                    }
                }
            }
        }
#pragma unroll
        for (int cs = 0; cs < NC; cs++)
#pragma unroll
            for (int m = 0; m < 2; m++)
#pragma unroll
                for (int i = 0; i < 4; i++) R[cs][m][i] = fmaf(bacc[cs][m][i], ixs[cs], R[cs][m][i]);
    }
#pragma unroll
    for (int cs = 0; cs < NC; cs++) {
        s_part[warp][cs][0][lane] = make_float2(R[cs][0][0] + R[cs][0][1], R[cs][0][2] + R[cs][0][3]);
        s_part[warp][cs][1][lane] = make_float2(R[cs][1][0] + R[cs][1][1], R[cs][1][2] + R[cs][1][3]);
    }
    __syncthreads();
    // element (row r of x, output o): lane g*4 + (r & 3) of set r / 4, tile half (o >> 4), component (o >> 3) & 1
    for (int i = threadIdx.x; i < 4 * NC * 32; i += DENSE_WARPS * 32) {
        const int r = i >> 5, ol = i & 31, o = o0 + ol;
        if (s0 + r >= S || o >= O) continue;
        const float *p = reinterpret_cast<const float *>(&s_part[0][r >> 2][ol >> 4][(ol & 7) * 4 + (r & 3)]) + ((ol >> 3) & 1);
        float a = 0.f;
#pragma unroll
        for (int k = 0; k < DENSE_WARPS; k++) a += p[(size_t)k * NC * 2 * 32 * 2];
        if (FMT == 1 || FMT == 2 || FMT == 3) a *= static_cast<const float *>(sc)[o];
        y[(size_t)(s0 + r) * O + o] = a;
    }
}
