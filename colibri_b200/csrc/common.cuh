// Shared definitions of the B200 MoE expert-FFN backend: resident tensor
// record, per-device context, the packed weight layout and the work
// descriptors the streaming GEMV kernels consume.
#pragma once

#include <cuda_runtime.h>
#include <cuda_fp16.h>
#include <stdint.h>
#include <stddef.h>

// ---------------------------------------------------------------------------
// Packed weight layout ("tile stream").
//
// A matrix W[O, I] (O output rows, I = contraction length) is cut into tiles
// of 32 output rows; a tile is cut along I into blocks of 128 columns. One
// block is stored as one contiguous chunk of two halves of 16 rows each,
//     [1024 B of 4-bit codes][scale bytes] [1024 B of 4-bit codes][scale bytes]
// and the chunks of a tile follow each other in ascending column order, so a
// tile's whole contraction is one linear stream (bulk-copyable without a
// tensor map), any column range of it is contiguous, and so is one half of a
// block (kernels that work on 16 rows copy just that).
//
// Inside the 1024 code bytes of a half the order is the register order of the
// m16n8k16 tensor-core A fragment, so a lane's 128-bit shared-memory load
// yields finished fragments: with lane = g*4+t (g = 0..7, t = 0..3), slot
// h (row g or g+8 of the half) sits at byte h*512 + lane*16 and holds four
// 32-bit words, one per 32-column group. Word (h, lane, grp) carries row
// h*8+g, columns grp*32 + 8t + {0..7}, as eight 4-bit fields:
//   int4 (fmt 2, 4): the stored offset-binary nibbles (value+8) in the order
//                    {0,2,4,6,1,3,5,7} (field f at bits 4f..4f+3), which lets
//                    two mask operations split a word into the (k, k+1) half2
//                    pairs the fragment wants.
//   MXFP4 (fmt 7):   the container's bytes (columns 2b and 2b+1 in byte b): one
//                    e2m1x2 -> f16x2 conversion per pair (12 issue cycles per word with
//                    its multiply, against 18 for shifts and masks that place the fields).
//
// Scale part of a half, by mode (always four 32-column slots per block; a group
// size of 64 or 128 repeats its scale), in the order [g][pair][h][i] for column
// group grp = 2*pair + i:
//   SC_ROW   nothing (one f32 per output row lives in a separate array)
//   SC_H16   fp16 (128 B)  int4 scales that are exact in fp16
//   SC_F32   f32  (256 B)  any other int4 scale
//   SC_MX    u8   (64 B)   ue8m0 exponents; of a tensor that qualifies for the
//                          tensor-core path, groups without a non-zero code hold an
//                          exponent of its fp16 range instead of their own
// ---------------------------------------------------------------------------
enum ScaleMode { SC_ROW = 0, SC_H16 = 1, SC_F32 = 2, SC_MX = 3 };

#define TILE_ROWS 32
#define BLOCK_K 128
#define CODE_BYTES 2048
#define TC_MX_SPREAD 24         // widest exponent spread of an MXFP4 tensor the tensor-core path carries exactly
#define TC_TAIL_BYTES 16          // behind a packed tensor's tile streams: its tensor-core shift (int)

__host__ __device__ inline int scale_bytes_of(int mode) {
    return mode == SC_H16 ? 256 : mode == SC_F32 ? 512 : mode == SC_MX ? 128 : 0;
}
__host__ __device__ inline int chunk_bytes_of(int mode) { return CODE_BYTES + scale_bytes_of(mode); }
// one half of a chunk: 16 rows, 1024 B of codes and their scales
__host__ __device__ constexpr int half_bytes_of(int mode) {
    return 1024 + (mode == SC_H16 ? 128 : mode == SC_F32 ? 256 : mode == SC_MX ? 64 : 0);
}

struct ColiCudaTensor {
    int fmt, I, O, device, gs, ng;
    size_t logical_bytes;     // what coli_cuda_stats reports: container weights + scales
    size_t physical_bytes;    // what is actually allocated on the device
    // raw storage (tensors the packed layout does not cover)
    void *raw_w;              // bytes as uploaded
    void *raw_s;              // f32 scales, or ue8m0 bytes for fmt 7
    // packed storage
    int packed;               // 1: tile-stream layout below is the only copy
    int mode;                 // ScaleMode
    uint8_t *pk;              // tile streams
    float *rowscale;          // SC_ROW only
    // tensor-core path (gemm_tc.cuh): usable for this tensor, and the power of two its
    // fp16 weight terms are pre-multiplied with
    int tc_ok, tc_shift;
};

// One matrix x one pass of rows for the streaming GEMV kernel.
#define SEG_MAX_ROWS 32
struct GemvSeg {
    const uint8_t *w;         // packed tensor base
    const float *rowscale;    // SC_ROW: [O]
    float *out;               // partial sums: out[(kpart*npos + pos0 + r)*O + o]
    int rowid[SEG_MAX_ROWS];  // rows of the B operand this pass multiplies
    int nrows, pos0;
    int O, ntiles, nkb;       // output rows, tiles (O/32), blocks along I (I/128)
    int nkpart, kb_per_part;  // split of the contraction into partial sums
    int task0;                // index of this segment's first task
};

// Control block of one GEMV launch (device memory).
struct GemvCtl {
    int nseg, ntask, npos;
    int tasks_per_seg;   // > 0 when every segment has this many tasks (then seg = task / tasks_per_seg)
};

// First statement of every kernel launched by launch_pdl: lets the stream's next kernel take its place on the SMs as
// soon as this one's CTAs all have theirs, and waits until the kernel before has finished and its writes are
// visible. Without the launch attribute both do nothing.
__device__ __forceinline__ void pdl_enter() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

#define KSTAT_MBAR_TIMEOUT 1

// The status word lives in pinned host memory that the device addresses directly, so the
// host reads it after a stream synchronisation without a copy. Kernels only ever store a
// non-zero code into it (a plain store: no atomics across the bus are needed for that).
__device__ __forceinline__ void kstat_set(int *status, int code) {
    *reinterpret_cast<volatile int *>(status) = code;
    __threadfence_system();
}

// Routing rule of a layer (device-visible mirror of ColiCudaMoeDesc).
struct RouteRule {
    int D, I, E, K;
    int gating, norm_topk;
    float routed_scale, topp;
};
