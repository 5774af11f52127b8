// From accumulator rows in registers to rows in global memory: the stored-tile epilogue of the tensor-core kernels
// (gemm_tcgen05.cu, bool_tcgen05.cu).
//
// A thread holds 16 columns of one row.  Written from there, every store would touch 32 rows, so the four warps that share a TMEM
// lane quarter (32 rows) lay their columns side by side in shared memory, and each then writes eight of the 32 rows.
// Aligned results go 64 columns at a time, in segments of 256 bytes a row, through two buffers that take turns: one barrier of the
// four warps per 64 columns.  Rows that start on no 16-byte boundary (ragged results) are written in 128-byte lines as they lie in
// memory, lane l word l of the line.  What those cost is the sectors that two stores complete between them: written one after the
// other by one warp they cost little, with other rows' stores in between several times as much (stores alone, [30011, 10007]:
// 32 words a row 397 us, 64 words 345, 128 words 318, 256 words 295; aligned 217 to 197), so of a ragged tile 128 columns are laid
// down, or, where shared memory has the room, all 256, and a warp writes one row after another.
#pragma once
#include "common.cuh"

namespace tpw {
namespace {

constexpr int kStoreCols = 64;                                 // columns per pass of four warps
constexpr int kStoreBuffer = 32 * kStoreCols * 4;              // bytes: 32 rows, 16-byte chunks XOR-swizzled by the row
constexpr int kStoreBytes = 4 * 2 * kStoreBuffer;              // four lane quarters, two buffers each

// barrier of the four warps of lane quarter q (barrier 0 is __syncthreads'), alone or with a vote
__device__ __forceinline__ void quarter_sync(int q) { asm volatile("barrier.cta.sync %0, 128;" ::"r"(q + 1) : "memory"); }
__device__ __forceinline__ bool quarter_all(int q, bool ok) {
    uint32_t r;
    asm volatile(
        "{\n\t.reg .pred p, s;\n\t"
        "setp.ne.u32 s, %2, 0;\n\t"
        "barrier.cta.red.and.pred p, %1, 128, s;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(r)
        : "r"(q + 1), "r"((uint32_t)ok)
        : "memory");
    return r != 0;
}

// this thread's 16 values, columns col .. col + 15 (a multiple of 16) of row `lane` of a block of COLS columns
template <int COLS>
__device__ __forceinline__ void stage_values(float *buf, const float (&o)[16], int col, int lane) {
#pragma unroll
    for (int v = 0; v < 4; ++v)
        *reinterpret_cast<float4 *>(buf + lane * COLS + ((((col >> 2) + v) ^ (lane & 7)) << 2)) =
            make_float4(o[4 * v], o[4 * v + 1], o[4 * v + 2], o[4 * v + 3]);
}

// rows 8 cq .. 8 cq + 7 of a staged block to dst (row 0, column 0 of the block); rows, cols: how many of them exist; vec: every row
// starts on a 16-byte boundary and cols is a multiple of 4; STREAM: nobody reads the result soon
template <int COLS, bool STREAM>
__device__ __forceinline__ void store_rows(const float *buf, float *dst, long long pitch, int rows, int cols, bool vec, int cq, int lane) {
    if (vec && COLS == kStoreCols) {
        const int cc = lane & 15;
#pragma unroll
        for (int it = 0; it < 4; ++it) {
            const int r = cq * 8 + it * 2 + (lane >> 4);
            const float4 v = *reinterpret_cast<const float4 *>(buf + r * COLS + ((cc ^ (r & 7)) << 2));
            if (r < rows && cc * 4 < cols) {
                float4 *p = reinterpret_cast<float4 *>(dst + r * pitch) + cc;
                if (STREAM) __stcs(p, v); else *p = v;
            }
        }
    } else {
        const int width = cols < COLS ? cols : COLS;
#pragma unroll 1
        for (int it = 0; it < 8; ++it) {
            const int r = cq * 8 + it;
            if (r >= rows) break;
            float *p = dst + r * pitch;
            const int w0 = lane - (int)((reinterpret_cast<uintptr_t>(p) >> 2) & 31u);   // words before the row's segment: negative
#pragma unroll
            for (int k = 0; k < COLS / 32 + 1; ++k) {
                const int w = w0 + 32 * k;
                if (w >= 0 && w < width) {
                    const float v = buf[r * COLS + (((w >> 2) ^ (r & 7)) << 2) + (w & 3)];
                    if (STREAM) __stcs(p + w, v); else p[w] = v;
                }
            }
        }
    }
}

} // namespace
} // namespace tpw
