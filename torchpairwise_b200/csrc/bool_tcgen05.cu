// Boolean pairwise metrics with the pair counts taken on the tensor cores.
//
// n11[i,j] = |x_i & y_j| is the dot product of two 0/1 vectors.  One-byte booleans are exactly the unsigned 8-bit
// operands of tcgen05.mma.kind::i8, whose 32-bit integer accumulators hold the counts exactly (D <= 2^24 < 2^31),
// so the contingency table of every pair is the same set of integers the popcount kernel produces and the shared
// epilogue (bool_epilogue.cuh) turns it into the same float32 bits.  What changes is the bound: the popcount tile
// is pinned at the POPC issue rate (C3, 65536 x 16384 x 1024 bits: 7.9 ms), the integer contraction leaves only
// the operand stream from L2 and the 4-byte output write.
//
// Kernel: persistent, one CTA per SM, by itself or in pairs (clusters of two, cta_group::2; pick_form), 576 threads -- warp 0
// issues TMA (one lane), warp 1 owns tensor memory and, in rank 0, issues the MMAs for both CTAs (one lane), warps 2..17 drain the
// accumulators (TMEM lane quarter = warp % 4).  A tile has 256 x2 rows and 128 x1 rows for every CTA; a k-step is
// 128 features = one 128-byte swizzled row per operand row, consumed by four MMAs of K = 32; stages of 16 KB (the CTA's x1
// rows) + 16 KB (a pair's CTA: its half of the x2 rows) or 32; two 256-column accumulators in tensor memory, so the epilogue of tile t overlaps
// the MMAs of tile t + 1.  Bound: operand reads and result writes share the way between L2 and the SMs (jaccard [32768, 16384,
// 1024] in pairs: 440 us without the stores, 494 without the operand copies, 356 of MMAs and copies alone, 694 together; with 128 x 256
// tiles per CTA, which read half as much again, and an epilogue of 23 instructions a distance, 720).  The operands are the caller's boolean
// matrices as they lie in memory when their rows start on 16-byte boundaries, else copies with the rows padded by zeros
// to a multiple of 16 bytes (bool_rows_kernel, which also counts the rows); the TMA unit zero-fills rows and features
// past the edge, and zeros add nothing to a count.  Every CTA loads its own tiles with plain per-CTA TMA loads from
// this GPU's memory.
//
// Results leave through shared memory: a pair's by four warps together (tile_store.cuh), a single CTA's in blocks of 32 x 32 that each
// warp writes by itself or hands to the copy engine.  [65536, 16384, 1024] jaccard 1447 -> 1315 us, [30011, 10007, 167] hamming
// 564 -> 429 us (pairs); [65536, 16384, 512] dice 1340 -> 1256, jaccard 1076 -> 915, hamming 943 -> 880 (single, packed epilogues).
//
// Every mbarrier wait is bounded; a role that gives up raises the pair's abort flag, everybody falls through to the
// final barrier, what is under way arrives (pair_exit.cuh; a CTA by itself is a pair whose other half has issued the same), tensor memory is released and the device status word reports the site.
#include "bool_epilogue.cuh"
#include "common.cuh"
#include "tcgen05.cuh"
#include "tile_store.cuh"

#include <type_traits>

#include <stdlib.h>

namespace tpw {
namespace {

constexpr int BM = 128;             // x1 rows per CTA (TMEM lanes); a pair's tile has twice as many
constexpr int BN = 256;             // x2 rows per tile (TMEM columns per accumulator)
constexpr int BKB = 128;            // features (bytes) per k-step
constexpr int A_BYTES = BM * BKB;       // 16 KB
constexpr int kEpilogueWarps = 16;            // four per TMEM lane quarter
// The forms of the kernel.  PAIR_SEGMENTS, PAIR_ROWS: two CTAs to a tile of 256 x 256, results through four warps' common staging
// (tile_store.cuh), 64 columns at a time where rows of the result start on 16-byte boundaries, the whole tile's rows at a time, with two
// operand stages instead of four, where they do not.  SINGLE: a CTA by itself, 128 x 256, three stages of the whole x2 tile; every warp
// drains 64 columns in blocks of 32 x 32 and stores them without meeting another.
enum Form { PAIR_SEGMENTS, PAIR_ROWS, SINGLE };
template <int FORM> struct Layout {
    static constexpr bool PAIR = FORM != SINGLE;
    static constexpr int kStages = FORM == PAIR_ROWS ? 2 : FORM == SINGLE ? 3 : 4;
    static constexpr int B_ROWS = PAIR ? BN / 2 : BN;    // x2 rows that a CTA stages
    static constexpr int STAGE_BYTES = A_BYTES + B_ROWS * BKB;
    static constexpr int OFF_BAR = kStages * STAGE_BYTES;
    // barriers: full, empty [kStages], tmem_full[2], tmem_empty[2]; then the TMEM base address, the abort flag and the pair's counts
    static constexpr int OFF_TMEM_PTR = OFF_BAR + (2 * kStages + 4) * 8;
    static constexpr int OFF_ABORT = OFF_TMEM_PTR + 4;
    static constexpr int OFF_COUNTS = OFF_ABORT + 4;
    static constexpr int OFF_STAGE = (OFF_COUNTS + (int)sizeof(PairCounts) + 1023) / 1024 * 1024;   // SINGLE: also the source of swizzled TMA stores
    static constexpr int OFF_POP = OFF_STAGE + (FORM == PAIR_ROWS ? BM * BN * 4 : kStoreBytes);   // per epilogue warp the x2 row counts of its 64 columns
    static constexpr int SMEM_ALLOC = OFF_POP + kEpilogueWarps * 256 + 1024;
    static_assert(SMEM_ALLOC <= 232448, "exceeds the dynamic shared memory of one CTA");
};
static_assert(kStoreBytes >= kEpilogueWarps * 4096, "room for the warps' blocks");
constexpr int kThreads = 64 + 32 * kEpilogueWarps;
constexpr uint32_t kTmemCols = 512;

struct BoolTcParams {
    const int32_t *pop1, *pop2;
    float *out;
    long long B, N1, N2, D;
    long long tiles_m, tiles_n, tiles;
    int metric;
    int vec;         // SINGLE: rows of the result start on 16-byte boundaries
    int stream;      // SINGLE: words of ragged rows are written past L2
    int tma_store;   // SINGLE: whole blocks leave through the output's tensor map
    float inv_d;     // 1/D when D is a power of two, else 0
    int *status;
};

// D[tmem] (+)= A[smem] * B[smem]^T on unsigned 8-bit operands, 32-bit integer accumulate (K = 32 per instruction)
template <bool PAIR>
__device__ __forceinline__ void tc_mma_i8(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    if (PAIR)
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "setp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::2.kind::i8 [%0], %1, %2, %3, p;\n\t}"
            ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
            : "memory");
    else
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "setp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}"
            ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
            : "memory");
}
// Instruction descriptor of kind::i8: D = signed 32-bit (bits [4,6) = 2), A and B unsigned 8-bit (bits [7,10) and
// [10,13) = 0), both K-major (bits 15 and 16 = 0), N >> 3 in bits [17,23), M >> 4 in bits [24,29); dense, no saturation.
__device__ __forceinline__ uint32_t make_idesc_i8(int M, int N) {
    return (2u << 4) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

// Row counts of one-byte booleans and, when dst is given, the rows as 0 / 1 bytes padded with zeros to `pitch` bytes.  One
// warp per row; reads the rows once, which is the bound (the bit-packing pass it replaces in front of this kernel read
// one byte per lane: 81920 x 1024 bytes 73 -> 30 us).  VEC: rows start on 16-byte boundaries and D is a multiple of 16.
template <bool VEC>
__global__ void __launch_bounds__(256)
bool_rows_kernel(const uint8_t *__restrict__ src, uint8_t *__restrict__ dst, int32_t *__restrict__ row_pop, long long rows,
                 long long D, long long pitch) {
    const int lane = threadIdx.x & 31;
    const long long warp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
    for (long long row = warp; row < rows; row += nwarps) {
        const uint8_t *s = src + row * D;
        int pop = 0;
        if (VEC) {
            for (long long k = lane * 16; k < D; k += 512) {
                const uint4 v = __ldg(reinterpret_cast<const uint4 *>(s + k));
                pop += __popc(__vcmpne4(v.x, 0u) & 0x01010101u) + __popc(__vcmpne4(v.y, 0u) & 0x01010101u) +
                       __popc(__vcmpne4(v.z, 0u) & 0x01010101u) + __popc(__vcmpne4(v.w, 0u) & 0x01010101u);
            }
        } else {
            for (long long k = lane * 4; k < pitch; k += 128) {
                uint32_t w = 0;
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (k + e < D && s[k + e] != 0) w |= 1u << (8 * e);
                pop += __popc(w);
                *reinterpret_cast<uint32_t *>(dst + row * pitch + k) = w;
            }
        }
        pop = __reduce_add_sync(0xffffffffu, pop);
        if (lane == 0) row_pop[row] = pop;
    }
}

// One instantiation per metric: with the metric a compile-time constant the epilogue's switch folds to the one case,
// which keeps the unrolled per-element code small enough for the instruction cache (with a run-time metric the 32
// inlined copies of the whole switch made the epilogue, not the contraction, the bound).
template <int METRIC, int FORM>
__global__ void __cluster_dims__(FORM == SINGLE ? 1 : 2, 1, 1) __launch_bounds__(kThreads, 1)
bool_count_tcgen05_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_y,
                          const __grid_constant__ CUtensorMap map_out, const BoolTcParams P) {
    typedef Layout<FORM> L;
    constexpr bool PAIR = L::PAIR;
    constexpr int kStages = L::kStages, STAGE_BYTES = L::STAGE_BYTES, kCtas = PAIR ? 2 : 1, kTileRows = kCtas * BM;
    extern __shared__ unsigned char smem_raw[];
    unsigned char *smem = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t *full = reinterpret_cast<uint64_t *>(smem + L::OFF_BAR);   // rank 0's: both CTAs' copies of a stage have landed
    uint64_t *empty = full + kStages;
    uint64_t *tmem_full = empty + kStages;
    uint64_t *tmem_empty = tmem_full + 2;                                // rank 0's: both CTAs have drained the accumulator
    uint32_t *tmem_ptr = reinterpret_cast<uint32_t *>(smem + L::OFF_TMEM_PTR);
    int *abort_flag = reinterpret_cast<int *>(smem + L::OFF_ABORT);
    PairCounts *counts = reinterpret_cast<PairCounts *>(smem + L::OFF_COUNTS);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = PAIR ? cluster_rank() : 0;       // the pair's tile: rows of rank 0, then rows of rank 1
    const int pair = blockIdx.x / kCtas, pairs = gridDim.x / kCtas, tiles = (int)P.tiles;   // 2^31 tiles would be a result of 2^49 bytes
    auto place = [&](int tile, int &tn, int &tm, int &b) {
        tn = tile % (int)P.tiles_n; tile /= (int)P.tiles_n;
        tm = tile % (int)P.tiles_m;
        b = tile / (int)P.tiles_m;
    };
    const int nkb = (int)((P.D + BKB - 1) / BKB);

    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
        for (int a = 0; a < 2; ++a) { mbar_init(&tmem_full[a], 1); mbar_init(&tmem_empty[a], kCtas * kEpilogueWarps); }
        *abort_flag = 0;
        mbar_init_fence();
        tma_prefetch_descriptor(&map_x);
        tma_prefetch_descriptor(&map_y);
    }
    if (warp == 1) {
        if (PAIR) tmem_alloc_pair(tmem_ptr, kTmemCols); else tmem_alloc(tmem_ptr, kTmemCols);
    }
    tc_fence_before();
    __syncthreads();
    if (PAIR) cluster_sync();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_ptr;
    auto give_up = [&](int site) {
        raise_abort(abort_flag, kCtas);
        if (P.status) atomicCAS(P.status, 0, (10 << 16) | site);
    };

    if (warp == 0) {
        // ---------------- TMA producer: this CTA's rows of x1, its half of the x2 rows ----------------
        if (lane == 0) {
            uint32_t it = 0;
            bool ok = true;
            for (int tile = pair; tile < tiles && ok; tile += pairs) {
                int tn, tm, b;
                place(tile, tn, tm, b);
                for (int kb = 0; kb < nkb; ++kb, ++it) {
                    const int s = it % kStages;
                    const uint32_t use = it / kStages;
                    if (use > 0 && !wait_or_abort(&empty[s], (use - 1) & 1, abort_flag)) {
                        give_up(1);
                        ok = false;
                        break;
                    }
                    unsigned char *st = smem + s * STAGE_BYTES;
                    const uint32_t bar = PAIR ? cluster_addr(&full[s], 0) : 0;
                    if (rank == 0) mbar_expect_tx(&full[s], kCtas * STAGE_BYTES);
                    const int row = tm * kTileRows + (int)rank * BM, col = tn * BN + (int)rank * (BN / 2);
                    if constexpr (PAIR) {
                        tma_load_3d_pair(st, &map_x, bar, kb * BKB, row, b);
                        tma_load_3d_pair(st + A_BYTES, &map_y, bar, kb * BKB, col, b);
                    } else {
                        tma_load_3d(st, &map_x, &full[s], kb * BKB, row, b);
                        tma_load_3d(st + A_BYTES, &map_y, &full[s], kb * BKB, col, b);
                    }
                }
            }
            if (ok && !wait_for_releases(empty, it, kStages, abort_flag)) give_up(5);
            publish(&counts->issued[rank], it, kCtas);
            if (!PAIR) publish(&counts->issued[1], it, 1);
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer: rank 0, for both ----------------
        if (lane == 0 && rank == 0) {
            const uint32_t idesc = make_idesc_i8(kTileRows, BN);
            uint32_t it = 0, acount = 0;
            bool ok = true;
            for (int tile = pair; tile < tiles && ok; tile += pairs, ++acount) {
                const uint32_t a = acount & 1, ause = acount >> 1;
                if (ause > 0 && !wait_or_abort<PAIR>(&tmem_empty[a], (ause - 1) & 1, abort_flag)) {
                    give_up(2);
                    ok = false;
                    break;
                }
                tc_fence_after();
                const uint32_t d_tmem = tmem_base + a * BN;
                for (int kb = 0; kb < nkb; ++kb, ++it) {
                    const int s = it % kStages;
                    if (!wait_or_abort<PAIR>(&full[s], (it / kStages) & 1, abort_flag)) {
                        give_up(3);
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t sb = smem_u32(smem + s * STAGE_BYTES);
                    const uint64_t dx = make_smem_desc(sb), dy = make_smem_desc(sb + A_BYTES);
                    // one MMA consumes 32 bytes of the swizzled row: the start address advances by 2 units of 16 bytes; the
                    // last k-step leaves out the MMAs that would only see zero fill
                    const int kmma = kb + 1 < nkb ? BKB / 32 : (int)((P.D - (long long)kb * BKB + 31) / 32);
#pragma unroll
                    for (int k = 0; k < BKB / 32; ++k)
                        if (k < kmma) tc_mma_i8<PAIR>(d_tmem, dx + 2 * k, dy + 2 * k, idesc, (kb | k) != 0);
                    tc_commit<PAIR>(&empty[s]);   // the stage may be refilled, in both CTAs, once these MMAs have read it
                }
                if (!ok) break;      // acount: accumulators handed over
                tc_commit<PAIR>(&tmem_full[a]);
            }
            publish(&counts->used, it, kCtas);
            publish(&counts->filled, acount, kCtas);
        }
    } else {
        // ---------------- epilogue: warps 2..17 ----------------
        const int q = warp & 3;
        const int cq = (warp - 2) >> 2;              // which 16 of every 64 columns; SINGLE: which 64 columns
        constexpr int kPasses = BN / kStoreCols;
        uint32_t tcount = 0;
        const int D = (int)P.D, N2 = (int)P.N2;
        // metrics with a packed form, on counts small enough for it: the row counts are kept as floats
        const bool packed = kPackedEpilogue<METRIC> && P.D < kQuotientMax;
        float *stage = reinterpret_cast<float *>(smem + L::OFF_STAGE + (PAIR ? q * (FORM == PAIR_ROWS ? 32 * BN * 4 : 2 * kStoreBuffer) : (warp - 2) * 4096));
        int32_t *popw = reinterpret_cast<int32_t *>(smem + L::OFF_POP + (warp - 2) * 256);
        const uint32_t drained[2] = {PAIR ? cluster_addr(&tmem_empty[0], 0) : 0, PAIR ? cluster_addr(&tmem_empty[1], 0) : 0};
        for (int tile = pair; tile < tiles; tile += pairs, ++tcount) {
            int tn, tm, b;
            place(tile, tn, tm, b);
            const uint32_t a = tcount & 1;
            // What the epilogue needs besides the counts depends on the tile index alone: fetch it before waiting for the
            // accumulator, so that the L2 round trip hides behind the contraction instead of sitting in every column block.
            const int row_base = tm * kTileRows + (int)rank * BM + q * 32;
            const int rows = (int)P.N1 - row_base;      // of this quarter's block, if not all 32
            const int pa = lane < rows ? __ldg(P.pop1 + b * P.N1 + row_base + lane) : 0;
            {
                // 64 counts per warp, two per lane: entry e is column 64 (e / 16) + 16 cq + e % 16, or 64 cq + e
                const int jc = tn * BN + (PAIR ? (lane >> 3) * kStoreCols + cq * 16 + (lane & 7) * 2 : cq * 64 + lane * 2);
                const int32_t *pb = P.pop2 + b * P.N2;
                int2 v = make_int2(0, 0);
                if (jc < N2) v.x = __ldg(pb + jc);
                if (jc + 1 < N2) v.y = __ldg(pb + jc + 1);
                if (packed) v = make_int2(__float_as_int((float)v.x), __float_as_int((float)v.y));
                __syncwarp();   // the previous tile's reads of this area are done
                *reinterpret_cast<int2 *>(popw + lane * 2) = v;
            }
            const bool here = wait_or_abort(&tmem_full[a], (tcount >> 1) & 1, abort_flag);
            if (!here && lane == 0) give_up(4);
            // a pair: all four warps of the quarter, or none, as they meet at the stores' barriers
            if (PAIR ? !quarter_all(q, here) : !__all_sync(0xffffffffu, here)) break;
            if (!PAIR) __syncwarp();
            tc_fence_after();
            float *out = P.out + (b * P.N1 + row_base) * P.N2 + tn * BN;
            const uint32_t acc = tmem_base + ((uint32_t)(q * 32) << 16) + a * BN + cq * (PAIR ? 16 : 64);
            const int cols = N2 - tn * BN;
            auto release = [&]() {                       // this warp has drained its part of accumulator `a`
                tc_fence_before();
                __syncwarp();
                if (lane == 0) {
                    if (PAIR) mbar_arrive_cluster(drained[a]); else mbar_arrive(&tmem_empty[a]);
                }
            };
            // the mean metrics multiply by 1 / D where D is a power of two and divide otherwise: decided here, once per
            // tile, so that the per-element code holds one of the two
            auto drain = [&](auto packed_tag, auto inv_tag, float inv_d) {
                constexpr bool PACKED = decltype(packed_tag)::value;
                constexpr int INV = decltype(inv_tag)::value;
                // four neighbouring columns of this thread's row, nb: their row counts
                auto four = [&](const uint32_t *r, int4 nb) {
                    float4 o;
                    if constexpr (PACKED) {
                        const f32x2 a2 = pack2((float)pa, (float)pa);
                        unpack2(bool_epilogue_packed<METRIC, INV>(r[0], r[1], a2, pack2(__int_as_float(nb.x), __int_as_float(nb.y)), (float)D, inv_d), o.x, o.y);
                        unpack2(bool_epilogue_packed<METRIC, INV>(r[2], r[3], a2, pack2(__int_as_float(nb.z), __int_as_float(nb.w)), (float)D, inv_d), o.z, o.w);
                    } else {
                        o.x = bool_epilogue<true, INV>(METRIC, (int)r[0], pa, nb.x, D, inv_d);
                        o.y = bool_epilogue<true, INV>(METRIC, (int)r[1], pa, nb.y, D, inv_d);
                        o.z = bool_epilogue<true, INV>(METRIC, (int)r[2], pa, nb.z, D, inv_d);
                        o.w = bool_epilogue<true, INV>(METRIC, (int)r[3], pa, nb.w, D, inv_d);
                    }
                    return o;
                };
                if constexpr (PAIR) {
                    const int passes = cols < BN ? (cols + kStoreCols - 1) / kStoreCols : kPasses;
#pragma unroll 1
                    for (int p = 0; p < passes; ++p) {
                        uint32_t r[16];
                        tmem_ld16(acc + p * kStoreCols, r);
                        tmem_ld_wait();
                        if (p + 1 == passes) release();
                        float o[16];
#pragma unroll
                        for (int v = 0; v < 4; ++v) {
                            const float4 t = four(r + 4 * v, *reinterpret_cast<const int4 *>(popw + p * 16 + 4 * v));
                            o[4 * v] = t.x; o[4 * v + 1] = t.y; o[4 * v + 2] = t.z; o[4 * v + 3] = t.w;
                        }
                        if constexpr (FORM == PAIR_ROWS) {
                            stage_values<BN>(stage, o, p * kStoreCols + cq * 16, lane);
                        } else {
                            // the vote ahead of the next tile keeps its first pass from a buffer that is still read
                            float *buf = stage + (p & 1) * (32 * kStoreCols);
                            stage_values<kStoreCols>(buf, o, cq * 16, lane);
                            quarter_sync(q);
                            store_rows<kStoreCols, true>(buf, out + p * kStoreCols, P.N2, rows, cols - p * kStoreCols, true, cq, lane);
                        }
                    }
                    if constexpr (FORM == PAIR_ROWS) {
                        quarter_sync(q);
                        store_rows<BN, true>(stage, out, P.N2, rows, cols, false, cq, lane);
                    }
                } else {
#pragma unroll 1
                    for (int c = 0; c < 2; ++c) {
                        const int first = cq * 64 + c * 32;
                        uint32_t r[32];
                        tmem_ld32(acc + c * 32, r);
                        tmem_ld_wait();
                        if (c == 1) release();
                        if (first >= cols || rows <= 0) continue;
                        if (P.tma_store) {
                            // by now the copy engine has read the previous block out of the staging area
                            if (lane == 0) tma_store_wait_read();
                            __syncwarp();
                        }
#pragma unroll
                        for (int v = 0; v < 8; ++v)
                            *reinterpret_cast<float4 *>(stage + lane * 32 + ((v ^ (lane & 7)) << 2)) = four(r + 4 * v, *reinterpret_cast<const int4 *>(popw + c * 32 + 4 * v));
                        const bool whole = P.vec && first + 32 <= cols;
                        if (whole && P.tma_store) {
                            // the staged block is what a 128-byte swizzled 32 x 32 box looks like: one lane hands it to the copy engine
                            // (the tensor map clips rows past N1) and the warp goes on
                            fence_proxy_async_smem();
                            __syncwarp();
                            if (lane == 0) {
                                tma_store_3d(&map_out, stage, tn * BN + first, row_base, b);
                                tma_store_commit();
                            }
                            continue;
                        }
                        __syncwarp();
                        if (whole) {
                            const int cc = lane & 7;
#pragma unroll
                            for (int it = 0; it < 8; ++it) {
                                const int row = it * 4 + (lane >> 3);
                                const float4 v = *reinterpret_cast<const float4 *>(stage + row * 32 + ((cc ^ (row & 7)) << 2));
                                if (row < rows) __stcs(reinterpret_cast<float4 *>(out + row * P.N2 + first) + cc, v);
                            }
                        } else if (first + lane < cols) {
                            const int n = rows < 32 ? rows : 32;
                            float *p = out + first + lane;
                            auto word = [&](int row) { return stage[row * 32 + (((lane >> 2) ^ (row & 7)) << 2) + (lane & 3)]; };
                            if (P.stream) {
#pragma unroll 8
                                for (int row = 0; row < n; ++row) __stcs(p + row * P.N2, word(row));
                            } else {
#pragma unroll 8
                                for (int row = 0; row < n; ++row) p[row * P.N2] = word(row);
                            }
                        }
                        __syncwarp();
                    }
                }
            };
            typedef std::integral_constant<bool, kPackedEpilogue<METRIC>> Packed;   // never taken where the metric has no such form
            if (METRIC == TPW_BOOL_EQ_MEAN || METRIC == TPW_BOOL_NE_MEAN) {
                if (packed && P.inv_d != 0.f) drain(Packed{}, std::integral_constant<int, 1>{}, P.inv_d);
                else if (packed) drain(Packed{}, std::integral_constant<int, 2>{}, approximate_reciprocal((float)P.D));
                else if (P.inv_d != 0.f) drain(std::false_type{}, std::integral_constant<int, 1>{}, P.inv_d);
                else drain(std::false_type{}, std::integral_constant<int, 0>{}, 0.f);
            } else if (packed) {
                drain(Packed{}, std::integral_constant<int, 2>{}, 0.f);
            } else {
                drain(std::false_type{}, std::integral_constant<int, -1>{}, P.inv_d);
            }
        }
    }

    if (!PAIR && P.tma_store && warp >= 2 && lane == 0) tma_store_wait_read();   // shared memory stays until the last block is read
    tc_fence_before();
    __syncthreads();
    if (PAIR) cluster_sync();   // neither CTA's shared memory goes while the other may still read it or arrive in it
    if (*reinterpret_cast<volatile int *>(abort_flag)) {   // raised in both CTAs or in neither
        if (threadIdx.x == 0) drain_pair(full, empty, tmem_full, kStages, counts, rank, [](uint32_t) { return (uint32_t)STAGE_BYTES; });
        __syncthreads();
        if (PAIR) cluster_sync();
    }
    if (warp == 1) {
        tc_fence_after();
        if (PAIR) tmem_dealloc_pair(tmem_base, kTmemCols); else tmem_dealloc(tmem_base, kTmemCols);
    }
}

} // namespace
} // namespace tpw

using namespace tpw;

// Which form runs, by times over a CTA by itself with one tile of 128 x 256 and the epilogues without packed arithmetic.  A pair saves a third
// of the operands but couples its 32 epilogue warps, four by four at the stores' barriers and all of them at the accumulators, which
// costs more than that where results rather than operands are the bound.
// Rows of the result on the 16-byte grid, at 2 to 4300 MB of them:
//   packed metrics, up to 1024 features    SINGLE 0.79 to 1.06 (jaccard 0.82 to 1.07), pairs 0.86 to 1.36
//                   above                  SINGLE 0.95 to 1.06, pairs 0.79 to 1.0
//                   1024, from 2 GB on     SINGLE 0.95 to 1.06, pairs 0.91 to 0.97
//   the others, up to 1536                 SINGLE 0.88 to 1.06 (kulczynski1 1.07), pairs 0.91 to 1.3
//               2048                       SINGLE 0.95 to 0.99, pairs 0.80 to 0.89 (yule 0.99 and 1.04);   4096  1.0 and 0.82 to 0.94
// Off the grid:
//   packed metrics, up to 1024 features    beyond L2's size pairs 0.65 to 1.05, SINGLE 1.0 to 1.2; below it pairs 0.98 to 1.16, SINGLE 0.81 to 1.0
//   russellrao, of short arithmetic too    beyond L2's size, 167 and 512 features, pairs 0.89 and 0.97, SINGLE 1.05 and 1.12; 1024  1.17 and 1.13
//   everything else                        SINGLE 0.95 to 1.04, pairs 1.02 to 1.36
static Form pick_form(int metric, bool aligned, double bytes, int64_t D) {
    const bool packed = has_packed_epilogue(metric) && D < kQuotientMax;
    if (!aligned) return D <= (packed ? 1024 : metric == TPW_BOOL_RUSSELLRAO ? 768 : 0) && bytes > 134217728.0 ? PAIR_ROWS : SINGLE;
    if (!packed) return D > (metric == TPW_BOOL_YULE ? 2048 : 1792) ? PAIR_SEGMENTS : SINGLE;
    return D > 1024 || (D > 960 && bytes >= 2147483648.0) ? PAIR_SEGMENTS : SINGLE;
}
// The copy engine takes a warp's blocks off its hands where the arithmetic is long enough to hide it and the operands leave it the way
// to L2 (over 128-bit stores: the metrics without packed arithmetic 0.83 to 0.97 to 1024 features, 1.08 to 1.14 at 1536, yule 0.9; jaccard to 512
// 0.92 to 0.95, 768 1.1 to 1.3; means by a division 167 features 0.9, 640 1.1; sums 1.0 to 1.35).
static bool copy_engine_stores(int metric, int64_t D) {
    const bool mean = metric == TPW_BOOL_EQ_MEAN || metric == TPW_BOOL_NE_MEAN;
    if (!has_packed_epilogue(metric)) return D <= (metric == TPW_BOOL_YULE ? 2048 : 1152);
    return D <= 512 && (metric == TPW_BOOL_JACCARD || (mean && (D & (D - 1)) != 0));
}

static bool tc_serves(int64_t B, int64_t N1, int64_t N2, int64_t D) {
    if (getenv("TPW_DISABLE_BOOL_TC")) return false;
    // up to 128 features the few-words popcount kernel is faster; the epilogue converts counts below 2^23 exactly with
    // one logic operation and one addition instead of the quarter-rate conversion instruction
    if (B <= 0 || N1 < BM || N2 < BN || D <= 128 || D >= (1 << 23)) return false;
    if (N1 >= (1ll << 31) || N2 >= (1ll << 31) || B >= (1ll << 31)) return false;
    return (double)B * (double)N1 * (double)N2 * (double)D >= 268435456.0;
}

// 1 when tpw_bool_metric_forward_tc serves this problem: rows of at least 128 bytes whose pitch keeps every row
// 16-byte aligned (a TMA requirement), counts that stay exact, and enough pairs to fill the persistent grid.
extern "C" int tpw_bool_metric_tc_eligible(int64_t B, int64_t N1, int64_t N2, int64_t D) {
    return D % 16 == 0 && tc_serves(B, N1, N2, D) ? 1 : 0;
}

// Any other row length of those problems goes the same way on padded rows.  The padded copy costs two passes over the
// operands, (N1 + N2) D bytes, against B N1 N2 outputs of at least 4 bytes each; the popcount tile, the other route, is
// several times slower wherever this one applies: hamming [30011, 10007, 167] 2.01 -> 0.55 ms.
extern "C" int64_t tpw_bool_rows_pitch(int64_t B, int64_t N1, int64_t N2, int64_t D) {
    return tc_serves(B, N1, N2, D) ? (D + 15) / 16 * 16 : 0;
}

extern "C" int tpw_bool_rows(const uint8_t *src, uint8_t *dst, int32_t *row_popcount, int64_t rows, int64_t D, int64_t pitch,
                             tpw_stream_t stream) {
    clear_error();
    TPW_CHECK_ARG(rows >= 0 && D > 0, "tpw_bool_rows: negative size");
    if (rows == 0) return TPW_OK;
    TPW_CHECK_ARG(src && row_popcount, "tpw_bool_rows: NULL pointer");
    TPW_CHECK_ARG(dst ? pitch >= D && pitch % 16 == 0 && aligned16(dst) : D % 16 == 0 && aligned16(src),
                  "tpw_bool_rows: padded rows need a 16-byte aligned copy and a pitch that is a multiple of 16, rows used in place "
                  "have to be 16-byte aligned themselves");
    long long blocks = (rows + 7) / 8;
    const long long cap = (long long)sm_count() * 16;
    if (blocks > cap) blocks = cap;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (dst) bool_rows_kernel<false><<<(unsigned)blocks, 256, 0, s>>>(src, dst, row_popcount, rows, D, pitch);
    else bool_rows_kernel<true><<<(unsigned)blocks, 256, 0, s>>>(src, nullptr, row_popcount, rows, D, D);
    TPW_LAUNCH_OK("bool_rows_kernel");
    return TPW_OK;
}

extern "C" int tpw_bool_metric_forward_tc(int metric, const uint8_t *x1, const uint8_t *x2,
                                          const int32_t *x1_popcount, const int32_t *x2_popcount, float *out,
                                          int64_t B, int64_t N1, int64_t N2, int64_t D, tpw_stream_t stream) {
    return tpw_bool_metric_forward_rows(metric, x1, x2, x1_popcount, x2_popcount, out, B, N1, N2, D, D, stream);
}

extern "C" int tpw_bool_metric_forward_rows(int metric, const uint8_t *x1, const uint8_t *x2,
                                            const int32_t *x1_popcount, const int32_t *x2_popcount, float *out,
                                            int64_t B, int64_t N1, int64_t N2, int64_t D, int64_t pitch, tpw_stream_t stream) {
    clear_error();
    TPW_CHECK_ARG(metric >= 0 && metric < TPW_BOOL_METRIC_COUNT, "tpw_bool_metric_forward_tc: unknown metric %d", metric);
    TPW_CHECK_ARG(B >= 0 && N1 >= 0 && N2 >= 0 && D >= 0, "tpw_bool_metric_forward_tc: negative size");
    if (B == 0 || N1 == 0 || N2 == 0) return TPW_OK;
    TPW_CHECK_ARG(D > 0 && D < (1 << 23), "tpw_bool_metric_forward_tc: D must be in [1, 2^23) (exact float32 counts)");
    TPW_CHECK_ARG(pitch >= D && pitch % 16 == 0, "tpw_bool_metric_forward_tc: D (the row pitch in bytes) must be a multiple of 16; use tpw_bool_metric_forward or padded rows");
    TPW_CHECK_ARG(x1 && x2 && x1_popcount && x2_popcount && out, "tpw_bool_metric_forward_tc: NULL pointer");
    TPW_CHECK_ARG(aligned16(x1) && aligned16(x2), "tpw_bool_metric_forward_tc: the boolean matrices must be 16-byte aligned");
    TPW_CHECK_ARG(N1 < (1ll << 31) && N2 < (1ll << 31) && B < (1ll << 31), "tpw_bool_metric_forward_tc: a dimension exceeds 2^31-1");
    BoolTcParams P;
    memset(&P, 0, sizeof(P));
    P.pop1 = x1_popcount; P.pop2 = x2_popcount; P.out = out;
    P.B = B; P.N1 = N1; P.N2 = N2; P.D = D;
    P.metric = metric;
    P.inv_d = (D & (D - 1)) == 0 ? 1.0f / (float)D : 0.f;
    const bool aligned = N2 % 4 == 0 && aligned16(out);
    const Form form = pick_form(metric, aligned, 4.0 * B * N1 * N2, D);
    P.tma_store = form == SINGLE && aligned && copy_engine_stores(metric, D);
    // long rows want L2 for the operands: streaming over plain words 0.89 to 1.0 at 1536 and 2048 features, 0.99 to 1.02 at 1100 and 4096, 0.97 to 1.01 below
    P.stream = D > 1024;
    const int rows = form == SINGLE ? BM : 2 * BM;
    P.tiles_m = (N1 + rows - 1) / rows;
    P.tiles_n = (N2 + BN - 1) / BN;
    P.tiles = B * P.tiles_m * P.tiles_n;
    P.status = device_status_ptr();
    CUtensorMap mx, my, mo;
    int st = make_tensor_map_3d(&mx, x1, 1, pitch, N1, B, BKB, BM, true);
    if (st != TPW_OK) return st;
    st = make_tensor_map_3d(&my, x2, 1, pitch, N2, B, BKB, form == SINGLE ? BN : BN / 2, true);
    if (st != TPW_OK) return st;
    memset(&mo, 0, sizeof(mo));
    P.vec = aligned ? 1 : 0;
    if (P.tma_store) {
        st = make_tensor_map_3d(&mo, out, 4, N2, N1, B, 32, 32, true);
        if (st != TPW_OK) return st;
    }
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const long long ctas = form == SINGLE ? 1 : 2, most = sm_count() / ctas, grid = ctas * (P.tiles < most ? P.tiles : most);
#define TPW_BOOL_TC_LAUNCH(M, FORM)                                                                                            \
    do {                                                                                                                       \
        auto kern = bool_count_tcgen05_kernel<M, FORM>;                                                                        \
        TPW_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Layout<FORM>::SMEM_ALLOC));        \
        kern<<<(unsigned)grid, kThreads, Layout<FORM>::SMEM_ALLOC, s>>>(mx, my, mo, P);                                        \
    } while (0)
#define TPW_BOOL_TC_CASE(M)                                                                                                    \
    case M:                                                                                                                    \
        if (form == SINGLE) TPW_BOOL_TC_LAUNCH(M, SINGLE);                                                                     \
        else if (form == PAIR_ROWS) TPW_BOOL_TC_LAUNCH(M, PAIR_ROWS);                                                          \
        else TPW_BOOL_TC_LAUNCH(M, PAIR_SEGMENTS);                                                                             \
        break
    switch (metric) {
        TPW_BOOL_TC_CASE(TPW_BOOL_AND_SUM); TPW_BOOL_TC_CASE(TPW_BOOL_OR_SUM); TPW_BOOL_TC_CASE(TPW_BOOL_XOR_SUM);
        TPW_BOOL_TC_CASE(TPW_BOOL_EQ_SUM); TPW_BOOL_TC_CASE(TPW_BOOL_NE_SUM); TPW_BOOL_TC_CASE(TPW_BOOL_EQ_MEAN);
        TPW_BOOL_TC_CASE(TPW_BOOL_NE_MEAN); TPW_BOOL_TC_CASE(TPW_BOOL_JACCARD); TPW_BOOL_TC_CASE(TPW_BOOL_KULSINSKI);
        TPW_BOOL_TC_CASE(TPW_BOOL_KULCZYNSKI1); TPW_BOOL_TC_CASE(TPW_BOOL_YULE); TPW_BOOL_TC_CASE(TPW_BOOL_DICE);
        TPW_BOOL_TC_CASE(TPW_BOOL_ROGERSTANIMOTO); TPW_BOOL_TC_CASE(TPW_BOOL_RUSSELLRAO); TPW_BOOL_TC_CASE(TPW_BOOL_SOKALMICHENER);
        TPW_BOOL_TC_CASE(TPW_BOOL_SOKALSNEATH);
        default: return fail(TPW_ERR_INVALID, "tpw_bool_metric_forward_tc: unknown metric %d", metric);
    }
#undef TPW_BOOL_TC_CASE
#undef TPW_BOOL_TC_LAUNCH
    TPW_LAUNCH_OK("bool_count_tcgen05_kernel");
    return TPW_OK;
}
