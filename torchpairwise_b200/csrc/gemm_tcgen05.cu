// Dense-contraction metrics (sqeuclidean, euclidean, cosine similarity / distance, correlation,
// linear kernel) on the 5th-generation tensor cores: TMA -> shared memory -> tcgen05.mma with fp32
// accumulators in tensor memory -> tcgen05.ld -> fused epilogue -> global.
//
// Precision.  The inputs are fp32 and the parity contract is rtol 1e-4 / atol 1e-5, which a single
// bf16 or tf32 pass does not meet.  Each operand is therefore split once into a bf16 "high" part
// and a bf16 "low" part (x = xh + xl up to 2^-17 relative) and the cross term is accumulated as
// xh.yh + xh.yl + xl.yh (three MMAs per k-step into the same fp32 accumulator; xl.yl is below the
// fp32 rounding of the sum).  Row norms are summed in fp32 from the unsplit values by the same
// pre-pass.
//
// Kernel.  Persistent, one CTA per SM, in pairs (clusters of two, cta_group::2) or by itself (single_pays), 576 threads: warp 0 = TMA producer
// (one lane), warp 1 = tensor-memory owner and, in rank 0, MMA issuer for both CTAs (one lane), warps 2..17 = epilogue.  A pair's output
// tile is 256 x 256, 128 rows to a CTA; k-step 64 bf16 = one 128-byte swizzled row.  The ring has five slots of 32 KB: the CTA's 128
// rows of x and its half, 128 rows, of y, high and low parts in turn.  The 512 TMEM columns hold two 128 x 256 fp32
// accumulators per CTA, so the epilogue of tile t overlaps the MMAs of tile t + 1.  Where a pair's tile is stored all sixteen
// epilogue warps drain it, four to a TMEM lane quarter, each 16 of every 64 columns; of the row-minimum and top-k epilogues
// eight warps own each accumulator, two to a lane quarter, each half of the columns.
// Why pairs: L2 -> SM traffic stands at 35 to 43 bytes a clock and SM whatever runs beside it.  A 128 x 256 tile per CTA takes 96 KB of
// operands per 1536 tensor-core clocks; a pair takes 64 KB, which the tensor cores wait for no longer (sqeuclidean [16384, 16384,
// 512] without its stores: 700 thousand clocks where the MMAs alone are 688), and less energy: under the power cap sqeuclidean [131072,
// 16384, 512] 6.15 -> 5.55 ms.  Every CTA fetches its own rows, with plain TMA loads, from this GPU's memory.
// A CTA by itself has a tile of 128 x 256 and three slots of 48 KB; each of its warps drains 64 columns (of the plain products of
// tf32 parts, eight warps, 128 columns and four slots) and stores them in blocks of 32 x 32 without meeting another.
//
// Three more instantiations share the pipeline: (1) kind::tf32 operands (high/low tf32 parts in fp32
// containers, 32 elements per k-step) for the gradient products of the backward and for plain dot
// products, with the reduction cut into chunks of 64 elements whose accumulators the epilogue warps
// add, rounded to nearest, into register-resident sums (the tensor cores add into tensor memory with
// truncation; see dense_backward_tensor below); (2) a row-minimum epilogue that folds each thread's
// accumulator row into one 64-bit key and stores no tile; (3) SELF, which zeroes the diagonal.
//
// Every wait (mbarrier) is bounded; a warp that gives up raises the pair's abort flag that the other
// roles poll, everybody falls through to the final barrier, what is under way arrives (pair_exit.cuh),
// tensor memory is released, and the device status word reports the site.
#include "common.cuh"
#include "packed_f32x2.cuh"
#include "tcgen05.cuh"
#include "tile_store.cuh"

#include <cuda_bf16.h>
#include <math.h>

#include <type_traits>

namespace tpw {
namespace {

constexpr int BM = 128;           // rows of x1 per CTA (TMEM lanes)
constexpr int TM = 2 * BM;        // rows of x1 per tile of a pair
constexpr int BN = 256;           // rows of x2 per tile (TMEM columns per accumulator)
constexpr int HN = BN / 2;        // of which each CTA stages half
constexpr int BK = 64;            // bf16 per k-step: 128 bytes
constexpr int kMmasPerStep = 4;    // a 128-byte operand row feeds four MMAs of 32 bytes (16 bf16 or 8 tf32) each
constexpr int A_BYTES = BM * BK * 2;          // 16 KB
// Shared memory of a pair's CTA and of a CTA by itself (single_pays): the ring of operand slots, one part (high or low) of a k-step each,
// barriers full, empty [kSlots], tmem_full[2], tmem_empty[2], the TMEM base address, the abort flag and the pair's counts; staging
// of the stored tiles (tile_store.cuh; 4 KB to a warp of a CTA by itself), where the top-k epilogue keeps its keys, 4 KB to a warp.
template <bool PAIR, bool TF32 = false> struct Ring {
    // a tf32 product by itself has eight epilogue warps, half of the staging, and with it a fourth slot: a tile of 64 features
    static constexpr int kSlots = PAIR ? 5 : TF32 ? 4 : 3, kWarps = PAIR || !TF32 ? 16 : 8, kThreads = 64 + 32 * kWarps;
    static constexpr int B_BYTES = (PAIR ? HN : BN) * BK * 2;
    static constexpr int SLOT_BYTES = A_BYTES + B_BYTES;
    static constexpr int OFF_BAR = kSlots * SLOT_BYTES;
    static constexpr int OFF_TMEM_PTR = OFF_BAR + (2 * kSlots + 4) * 8;
    static constexpr int OFF_ABORT = OFF_TMEM_PTR + 4;
    static constexpr int OFF_COUNTS = OFF_ABORT + 4;
    static constexpr int OFF_STAGE = (OFF_COUNTS + (int)sizeof(PairCounts) + 127) / 128 * 128;
    static constexpr int SMEM_ALLOC = OFF_STAGE + (PAIR ? kStoreBytes : kWarps * 4096) + 1024;
    static_assert(SMEM_ALLOC <= 232448, "exceeds the dynamic shared memory of one CTA");
};
static_assert(kStoreBytes >= Ring<true>::kWarps * 4096, "room for the top-k keys");
constexpr int SMEM_ALLOC = Ring<true>::SMEM_ALLOC, kThreads = Ring<true>::kThreads;
constexpr uint32_t kTmemCols = 512;

struct GemmParams {
    const float *n1sq, *n2sq; // squared row norms [B*N1], [B*N2]
    float *out;
    long long B, N1, N2, D;
    long long tiles_m, tiles_n, tiles;
    int epilogue;
    int self;                 // x2 is x1: the diagonal of the distance epilogues is exactly zero
    int vec_store;            // N2 % 4 == 0 and out 16-byte aligned
    int kchunk;               // k-steps accumulated in tensor memory before the sum moves to registers (0: all)
    unsigned long long *rowmin_keys; // ROWMIN instantiation: [B*N1] keys (float bits << 32 | x2 row), nothing is stored to out
    // TOPK > 0: [B*N1] upper bounds of the row's k-th smallest key (lowered by every tile half that finds k keys), [B*N1]
    // numbers of keys written so far, and per row room for k keys from every (column tile, half), [B*N1][topk_L * topk_k],
    // filled from the front
    unsigned long long *topk_lists, *topk_thr;
    int *topk_count;
    int topk_k, topk_L;
    // TOPK < 0: the columns of this launch are every col_step-th x2 row, cols of them; [B*N1][32 or 8 per column tile] minima of
    // groups of col_group columns (8: equal modulo 16 in a tile half, 32: modulo 4)
    float *gmin;
    int col_step, col_group;
    long long cols;
    const int *lo_any;        // [2] whether any low part of the x (y) operand is non-zero; NULL: treat both as non-zero
    int lo_always;            // bit 0 / 1: the x / y operand's low parts are used whatever lo_any says
    float *partial;           // tf32: [pair][2][TM][BN] sums of the tiles that a pair has only a part of (NULL: whole tiles only)
    int *status;
};

// D[tmem] (+)= A[smem] * B[smem]^T, fp32 accumulate; TF32 = false: bf16 operands (K = 16 per
// instruction), true: tf32 operands in 32-bit containers (K = 8 per instruction)
template <bool TF32, bool PAIR>
__device__ __forceinline__ void tc_mma(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
#define TPW_MMA(GROUP, KIND)                                                                                              \
    asm volatile(                                                                                                         \
        "{\n\t.reg .pred p;\n\t"                                                                                          \
        "setp.ne.b32 p, %4, 0;\n\t"                                                                                       \
        "tcgen05.mma.cta_group::" GROUP ".kind::" KIND " [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),                        \
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)                                                               \
        : "memory")
    if (TF32 && PAIR) TPW_MMA("2", "tf32");
    else if (TF32) TPW_MMA("1", "tf32");
    else if (PAIR) TPW_MMA("2", "f16");
    else TPW_MMA("1", "f16");
#undef TPW_MMA
}
// MN-major 32-bit tile: the only layout tcgen05 takes for it is the 128-byte swizzle with 32-byte
// atoms (layout type 1): rows of 128 bytes are k, four rows form one 512-byte atom (stride between
// 4-row groups in bits [32,46)), and the 32-value blocks along M/N follow each other at the leading
// byte offset in bits [16,30) (here 4096: 32 k-rows of 128 bytes).
__device__ __forceinline__ uint64_t make_smem_desc_mn(uint32_t smem_addr) {
    uint64_t d = 0;
    d |= (uint64_t)((smem_addr & 0x3FFFF) >> 4);
    d |= (uint64_t)(4096 >> 4) << 16;
    d |= (uint64_t)(512 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)1 << 61;
    return d;
}
// Instruction descriptor: D = fp32 (bits [4,6) = 1); A and B formats in bits [7,10) and [10,13):
// 1 = bf16 under kind::f16, 2 = tf32 under kind::tf32; bit 15 = 1 when A is MN-major
// (0: K-major; B is K-major, bit 16 = 0); N >> 3 in bits [17,23), M >> 4 in bits [24,29).
__device__ __forceinline__ uint32_t make_idesc(int M, int N, bool tf32, bool a_mn) {
    const uint32_t fmt = tf32 ? 2u : 1u;
    return (1u << 4) | (fmt << 7) | (fmt << 10) | ((a_mn ? 1u : 0u) << 15) |
           ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

// n1, n2: squared row norms for the two distance epilogues, reciprocal row norms (0 for an all-zero
// row, whose dot products are exactly 0 anyway) for the cosine family.
template <int EPI>
__device__ __forceinline__ float dot_epilogue(float dot, float n1, float n2, bool diag) {
    if (EPI == TPW_DOT_LINEAR) return dot;
    if (EPI == TPW_DOT_SQEUCLIDEAN) return diag ? 0.f : fmaxf(fmaf(-2.f, dot, n1 + n2), 0.f);
    if (EPI == TPW_DOT_EUCLIDEAN) return diag ? 0.f : sqrtf(fmaxf(fmaf(-2.f, dot, n1 + n2), 0.f));
    const float s = dot * (n1 * n2);
    if (EPI == TPW_DOT_COSINE_SIM) return s;
    const float dist = 1.f - s;
    if (EPI == TPW_DOT_COSINE_DIST) return fminf(fmaxf(dist, 0.f), 2.f);
    return dist;
}

// sqrt(x) for x = 0 or 2^-100 <= x < infinity, two at a time: one step of Newton's iteration for the square root from the
// approximate reciprocal square root (relative error below 2^-22, so the step leaves only its own rounding: within one float32 of
// sqrtf).  The term added under the root keeps it away from 1 / 0 and, 2^-126, changes no x of that range.
__device__ __forceinline__ f32x2 newton_sqrt(f32x2 x) {
    const f32x2 tiny = pack2(1.17549435e-38f, 1.17549435e-38f);
    float a, b, ra, rb;
    unpack2(add2(x, tiny), a, b);
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(ra) : "f"(a));
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(rb) : "f"(b));
    const f32x2 r = pack2(ra, rb), root = mul2(x, r), half = mul2(r, pack2(0.5f, 0.5f));
    return fma2(fma2(mul2(root, pack2(-1.f, -1.f)), root, x), half, root);
}
constexpr float kRootLow = 7.88860905e-31f;   // 2^-100

// dot_epilogue for 16 columns of one row, two lanes to an instruction (the same values, the root excepted as above).  With the
// scalar form, 23 instructions per Euclidean distance, the epilogue and not the contraction was the bound: euclidean
// [16, 4096, 4096, 256] forward 700 -> 445 us.
template <int EPI>
__device__ __forceinline__ void dot_epilogue16(const uint32_t (&dot)[16], float n1, const float (&n2)[16], float (&o)[16]) {
    const f32x2 row = pack2(n1, n1);
    f32x2 v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
        const f32x2 d = pack2(__uint_as_float(dot[2 * u]), __uint_as_float(dot[2 * u + 1])), col = pack2(n2[2 * u], n2[2 * u + 1]);
        if (EPI == TPW_DOT_LINEAR) v[u] = d;
        else if (EPI == TPW_DOT_SQEUCLIDEAN || EPI == TPW_DOT_EUCLIDEAN) v[u] = fma2(d, pack2(-2.f, -2.f), add2(row, col));
        else v[u] = mul2(d, mul2(row, col));
        if (EPI == TPW_DOT_COSINE_DIST || EPI == TPW_DOT_ONE_MINUS_SIM) v[u] = sub2(pack2(1.f, 1.f), v[u]);
        unpack2(v[u], o[2 * u], o[2 * u + 1]);
    }
    if (EPI == TPW_DOT_SQEUCLIDEAN || EPI == TPW_DOT_EUCLIDEAN) {
#pragma unroll
        for (int u = 0; u < 16; ++u) o[u] = fmaxf(o[u], 0.f);
    }
    if (EPI == TPW_DOT_COSINE_DIST) {
#pragma unroll
        for (int u = 0; u < 16; ++u) o[u] = fminf(fmaxf(o[u], 0.f), 2.f);
    }
    if (EPI == TPW_DOT_EUCLIDEAN) {
        float most = 0.f, least = INFINITY;
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            most = max3_abs(most, o[2 * u], o[2 * u + 1]);
            least = min3(least, o[2 * u], o[2 * u + 1]);
        }
        if (__any_sync(0xffffffffu, most > 3.402823466e+38f || least < kRootLow)) {
            // A distance somewhere in the warp that newton_sqrt does not take.  Small ones are rooted 2^80 times as large, where the
            // term under the root changes none of them (the smallest subnormal is 2^-149) and multiplying by either power of two is
            // exact; infinity is its own root.
#pragma unroll
            for (int u = 0; u < 16; u += 2) {
                const bool small0 = o[u] < kRootLow, small1 = o[u + 1] < kRootLow;
                const f32x2 up = pack2(small0 ? 1.2089258196146292e24f : 1.f, small1 ? 1.2089258196146292e24f : 1.f);
                const f32x2 down = pack2(small0 ? 9.0949470177292824e-13f : 1.f, small1 ? 9.0949470177292824e-13f : 1.f);   // 2^-40
                float a, b;
                unpack2(mul2(newton_sqrt(mul2(pack2(o[u], o[u + 1]), up)), down), a, b);
                o[u] = o[u] > 3.402823466e+38f ? o[u] : a;
                o[u + 1] = o[u + 1] > 3.402823466e+38f ? o[u + 1] : b;
            }
        } else {
#pragma unroll
            for (int u = 0; u < 8; ++u) unpack2(newton_sqrt(pack2(o[2 * u], o[2 * u + 1])), o[2 * u], o[2 * u + 1]);
        }
    }
}

// dot_epilogue without the cosine distance's upper clamp, for the top-k epilogue: columns are ordered the same way as long as
// the limit they are compared with lies below 2, so only the few that pass are clamped.
template <int EPI>
__device__ __forceinline__ float raw_distance(float dot, float n1, float n2) {
    return EPI == TPW_DOT_SQEUCLIDEAN ? dot_epilogue<EPI>(dot, n1, n2, false) : fmaxf(1.f - dot * (n1 * n2), 0.f);
}
template <int EPI>
__device__ __forceinline__ float clamp_distance(float raw) {
    return EPI == TPW_DOT_SQEUCLIDEAN ? raw : fminf(raw, 2.f);
}

// TF32 = false: operands are bf16 high/low parts, 64 per k-step; true: tf32 high/low parts in fp32
// containers, 32 per k-step.  Either way a k-step is one 128-byte swizzled row per operand row and
// four MMAs per operand pair, so the pipeline below is the same.
// Tile index -> (column tile, row tile, batch).  Column tiles vary fastest, so that consecutive tiles
// share the x1 rows and stream the (usually L2-resident) x2 rows -- except for the top-k epilogue, where
// row tiles vary fastest: a row's column tiles are then visited one after another over the run, and the
// bound that its earlier column tiles have lowered prunes the later ones.
template <bool ROW_TILES_FASTEST>
__device__ __forceinline__ void decode_tile(long long tile, const GemmParams &P, long long &tn, long long &tm, long long &b) {
    if (ROW_TILES_FASTEST) {
        tm = tile % P.tiles_m; tile /= P.tiles_m;
        tn = tile % P.tiles_n;
        b = tile / P.tiles_n;
    } else {
        tn = tile % P.tiles_n; tile /= P.tiles_n;
        tm = tile % P.tiles_m;
        b = tile / P.tiles_m;
    }
}

// Sorted insertion into an ascending register-resident list (branch-free: slot t becomes
// min(max(previous slot, key), slot t)); the largest entry falls off the end.
template <int N>
__device__ __forceinline__ void sorted_insert(unsigned long long (&lst)[N], unsigned long long key) {
#pragma unroll
    for (int t = N - 1; t > 0; --t) {
        const unsigned long long hi = lst[t - 1] > key ? lst[t - 1] : key;
        lst[t] = hi < lst[t] ? hi : lst[t];
    }
    lst[0] = key < lst[0] ? key : lst[0];
}

// The k smallest of a lane's n >= k keys (32 words apart), moved to its first k places; returns the largest of them and its slot.
// Not inlined: few tile halves come here.
struct KeySlot {
    unsigned long long key;
    int slot;
};
__device__ __noinline__ KeySlot keep_smallest(unsigned long long *buf, int n, int k) {
    KeySlot m{0, 0};
    for (;; --n) {
        m = {0, 0};
#pragma unroll 1
        for (int t = 0; t < n; t += 8) {   // eight loads under way together
            unsigned long long held[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) held[u] = t + u < n ? buf[(t + u) * 32] : 0;
#pragma unroll
            for (int u = 0; u < 8; ++u)
                if (t + u < n && held[u] >= m.key) m = {held[u], t + u};
        }
        if (n == k) return m;
        buf[m.slot * 32] = buf[(n - 1) * 32];
    }
}

// The share of a product that falls to one pair: whole tiles, every pairs-th.  With a scratch for partial tiles (tf32) only
// the full waves go that way; the chunks of the tiles that are left over are dealt out evenly, and a tile cut by the end of
// a share is finished by product_fixup_kernel.
template <typename I>
struct ProductShare {
    I tile_at, tile_last, base;   // whole tiles; first tile of those dealt out
    int stride, nch;
    int at, last;                 // this pair's chunks of the tiles dealt out
    __device__ __forceinline__ ProductShare(const GemmParams &P, int nch_, int ctas) {   // ctas: 2, or 1 where a CTA works by itself
        nch = nch_;
        const int pair = (int)blockIdx.x / ctas;
        stride = (int)gridDim.x / ctas;
        const long long left = P.partial ? P.tiles % stride : 0, all = left * nch;
        base = (I)(P.tiles - left);
        tile_at = (I)pair;
        tile_last = base;
        at = (int)(all * pair / stride);
        last = (int)(all * (pair + 1) / stride);
    }
    // the next piece: chunks [c0, c1) of a tile
    __device__ __forceinline__ bool next(I &tile, int &c0, int &c1) {
        if (tile_at < tile_last) {
            tile = tile_at;
            c0 = 0;
            c1 = nch;
            tile_at += stride;
            return true;
        }
        if (at >= last) return false;
        tile = base + at / nch;
        c0 = at % nch;
        c1 = last - at < nch - c0 ? c0 + (last - at) : nch;
        at += c1 - c0;
        return true;
    }
};

// Row minima, whose bound is the epilogue: where the last tile of a batch has no rows for rank 1, both CTAs work on rank 0's rows, and
// each drains half of the columns.  Nearest of [300, 50000, 64], 128 of 512 rows past the end: 52.8 -> 47.7 us.
__device__ __forceinline__ bool rank_1_is_idle(long long tm, const GemmParams &P) { return tm * TM + BM >= P.N1; }

// AMN (tf32 only): the x operand is MN-major, i.e. its global rows run along k and each row holds
// the tile's M values contiguously, so a matrix can be contracted over its row index without a
// transposed copy.  Such a tile is staged as blocks of {32 values, 32 k-rows} (one TMA box each, 4 KB,
// 128-byte swizzle with 32-byte atoms): block m holds values 32m..32m+31, an MMA consumes 8 k-rows = 1024 bytes.
template <int EPI, bool SELF, bool TF32, bool ROWMIN = false, bool AMN = false, int TOPK = 0, bool PAIR = true>
__global__ void __cluster_dims__(PAIR ? 2 : 1, 1, 1) __launch_bounds__(Ring<PAIR, TF32>::kThreads, 1)
gemm_metric_kernel(const __grid_constant__ CUtensorMap map_xh, const __grid_constant__ CUtensorMap map_xl,
                   const __grid_constant__ CUtensorMap map_yh, const __grid_constant__ CUtensorMap map_yl,
                   const GemmParams P) {
    typedef Ring<PAIR, TF32> L;
    constexpr int kSlots = L::kSlots, B_BYTES = L::B_BYTES, SLOT_BYTES = L::SLOT_BYTES, kCtas = PAIR ? 2 : 1, kTileRows = kCtas * BM;
    extern __shared__ unsigned char smem_raw[];
    unsigned char *smem = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t *full = reinterpret_cast<uint64_t *>(smem + L::OFF_BAR);   // rank 0's: both CTAs' copies of a slot have landed
    uint64_t *empty = full + kSlots;
    uint64_t *tmem_full = empty + kSlots;
    uint64_t *tmem_empty = tmem_full + 2;                             // rank 0's: both CTAs have drained the accumulator
    uint32_t *tmem_ptr = reinterpret_cast<uint32_t *>(smem + L::OFF_TMEM_PTR);
    int *abort_flag = reinterpret_cast<int *>(smem + L::OFF_ABORT);
    PairCounts *counts = reinterpret_cast<PairCounts *>(smem + L::OFF_COUNTS);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = PAIR ? cluster_rank() : 0;
    constexpr int BKE = TF32 ? BK / 2 : BK; // operand elements per k-step
    constexpr bool STORED = !ROWMIN && TOPK == 0;
    static_assert(PAIR || (STORED && !AMN), "a CTA by itself stores plain tiles");
    constexpr int kDrains = STORED ? L::kWarps : L::kWarps / 2;   // warps of a CTA that drain one accumulator
    typedef std::conditional_t<TF32, int, long long> Index;   // a stored product has fewer than 2^31 tiles
    const int nkb = (int)((P.D + BKE - 1) / BKE);

    if (threadIdx.x == 0) {
        for (int s = 0; s < kSlots; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
        for (int a = 0; a < 2; ++a) { mbar_init(&tmem_full[a], 1); mbar_init(&tmem_empty[a], kCtas * kDrains); }
        *abort_flag = 0;
        mbar_init_fence();
        tma_prefetch_descriptor(&map_xh);
        tma_prefetch_descriptor(&map_xl);
        tma_prefetch_descriptor(&map_yh);
        tma_prefetch_descriptor(&map_yl);
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
        if (P.status) atomicCAS(P.status, 0, (4 << 16) | site);
    };
    // Operands that the high parts hold exactly (16-bit inputs, small integers) have no low parts: their tiles are neither
    // loaded nor multiplied.  The products left out are zeros added to a finished sum; an infinite or NaN input has a NaN low part.
    // cosine of bfloat16 [5000, 768] x [4111, 768], forward and backward: 707 -> 652 us.
    const bool need_xl = !P.lo_any || (P.lo_always & 1) || P.lo_any[0] != 0;
    const bool need_yl = !P.lo_any || (P.lo_always & 2) || P.lo_any[1] != 0;
    const int parts = need_xl || need_yl ? 2 : 1;   // slots per k-step

    if (warp == 0) {
        // ---------------- TMA producer: this CTA's rows of x, its half of the rows of y ----------------
        if (lane == 0) {
            uint32_t s = 0, use = 0, issued = 0;     // slot, how often it has been filled before
            bool ok = true;
            const int kchunk = (P.kchunk > 0 && P.kchunk < nkb) ? P.kchunk : nkb;
            ProductShare<Index> share(P, (nkb + kchunk - 1) / kchunk, kCtas);
            Index tile;
            for (int c0, c1; ok && share.next(tile, c0, c1);) {
                long long tn, tm, b;
                decode_tile<TOPK != 0>(tile, P, tn, tm, b);
                const int row = (int)(tm * kTileRows) + (ROWMIN && rank_1_is_idle(tm, P) ? 0 : (int)rank * BM), col = (int)(tn * BN) + (int)rank * HN;
                const int kend = c1 * kchunk < nkb ? c1 * kchunk : nkb;
                for (int kb = c0 * kchunk; kb < kend && ok; ++kb) {
                    for (int part = 0; part < parts; ++part) {
                        if (use > 0 && !wait_or_abort(&empty[s], (use - 1) & 1, abort_flag)) {
                            give_up(1);
                            ok = false;
                            break;
                        }
                        unsigned char *st = smem + s * SLOT_BYTES;
                        const uint32_t bar = PAIR ? cluster_addr(&full[s], 0) : 0;
                        const bool load_x = part == 0 || need_xl, load_y = part == 0 || need_yl;
                        if (rank == 0) mbar_expect_tx(&full[s], kCtas * ((load_x ? A_BYTES : 0) + (load_y ? B_BYTES : 0)));
                        static_assert(TF32 || !AMN, "MN-major staging is laid out for 32-bit operands");
                        if (load_x) {
                            const CUtensorMap *map = part == 0 ? &map_xh : &map_xl;
                            if constexpr (AMN) {
#pragma unroll
                                for (int m = 0; m < BM / 32; ++m) tma_load_3d_pair(st + m * 4096, map, bar, row + 32 * m, kb * BKE, (int)b);
                            } else {
                                if constexpr (PAIR) tma_load_3d_pair(st, map, bar, kb * BKE, row, (int)b);
                                else tma_load_3d(st, map, &full[s], kb * BKE, row, (int)b);
                            }
                        }
                        if (load_y) {
                            const CUtensorMap *map = part == 0 ? &map_yh : &map_yl;
                            if constexpr (PAIR) tma_load_3d_pair(st + A_BYTES, map, bar, kb * BKE, col, (int)b);
                            else tma_load_3d(st + A_BYTES, map, &full[s], kb * BKE, col, (int)b);
                        }
                        ++issued;
                        if (++s == kSlots) { s = 0; ++use; }
                    }
                }
            }
            if (ok && !wait_for_releases(empty, issued, kSlots, abort_flag)) give_up(7);
            publish(&counts->issued[rank], issued, kCtas);
            if (!PAIR) publish(&counts->issued[1], issued, 1);
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer: rank 0, for both CTAs ----------------
        if (lane == 0 && rank == 0) {
            const uint32_t idesc = make_idesc(kTileRows, BN, TF32, AMN);
            uint32_t s = 0, phase = 0, acount = 0, used = 0;
            bool ok = true;
            const int kchunk = (P.kchunk > 0 && P.kchunk < nkb) ? P.kchunk : nkb;
            ProductShare<Index> share(P, (nkb + kchunk - 1) / kchunk, kCtas);
            Index tile;
            auto arrived = [&](int site) {
                if (!wait_or_abort<PAIR>(&full[s], phase, abort_flag)) {
                    give_up(site);
                    return false;
                }
                tc_fence_after();
                return true;
            };
            auto x_desc = [&](uint32_t slot) {
                const uint32_t at = smem_u32(smem + slot * SLOT_BYTES);
                return AMN ? make_smem_desc_mn(at) : make_smem_desc(at);
            };
            auto y_desc = [&](uint32_t slot) { return make_smem_desc(smem_u32(smem + slot * SLOT_BYTES + A_BYTES)); };
            for (int c0, c1; ok && share.next(tile, c0, c1);) {
                // one accumulator per chunk of k-steps: the tensor cores add into tensor memory with
                // truncation, so long reductions are cut into chunks that the epilogue sums in registers
                const int kend = c1 * kchunk < nkb ? c1 * kchunk : nkb;
                for (int kb0 = c0 * kchunk; kb0 < kend && ok; kb0 += kchunk, ++acount) {
                    const uint32_t a = acount & 1, ause = acount >> 1;
                    if (ause > 0 && !wait_or_abort<PAIR>(&tmem_empty[a], (ause - 1) & 1, abort_flag)) {
                        give_up(2);
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t d_tmem = tmem_base + a * BN;
                    const int kb1 = kb0 + kchunk < nkb ? kb0 + kchunk : nkb;
                    for (int kb = kb0; kb < kb1; ++kb) {
                        if (!arrived(3)) {
                            ok = false;
                            break;
                        }
                        const uint32_t hi = s;
                        const uint64_t dxh = x_desc(hi), dyh = y_desc(hi);
                        // K-major: one MMA consumes 32 bytes of the swizzled row (16 bf16 or 8 tf32), so the start
                        // address advances by 2 units of 16 bytes; MN-major: 8 k-rows = 1024 bytes = 64 units
                        constexpr uint64_t ka = AMN ? 64 : 2, kbn = 2;
#pragma unroll
                        for (int k = 0; k < kMmasPerStep; ++k)
                            tc_mma<TF32, PAIR>(d_tmem, dxh + ka * k, dyh + kbn * k, idesc, ((kb - kb0) | k) != 0);
                        if (++s == kSlots) { s = 0; phase ^= 1; }
                        if (parts == 1) {
                            tc_commit<PAIR>(&empty[hi]);
                            ++used;
                            continue;
                        }
                        if (!arrived(5)) {
                            tc_commit<PAIR>(&empty[hi]);   // for drain_pair: the MMAs above are under way
                            ++used;
                            ok = false;
                            break;
                        }
                        const uint32_t lo = s;
                        const uint64_t dxl = x_desc(lo), dyl = y_desc(lo);
                        if (need_xl && need_yl) {
#pragma unroll
                            for (int k = 0; k < kMmasPerStep; ++k) {
                                tc_mma<TF32, PAIR>(d_tmem, dxh + ka * k, dyl + kbn * k, idesc, 1);
                                tc_mma<TF32, PAIR>(d_tmem, dxl + ka * k, dyh + kbn * k, idesc, 1);
                            }
                        } else {
                            const uint64_t da = need_xl ? dxl : dxh, db = need_xl ? dyh : dyl;
#pragma unroll
                            for (int k = 0; k < kMmasPerStep; ++k) tc_mma<TF32, PAIR>(d_tmem, da + ka * k, db + kbn * k, idesc, 1);
                        }
                        tc_commit<PAIR>(&empty[hi]); // both slots may be refilled, in both CTAs, once these MMAs have read them
                        tc_commit<PAIR>(&empty[lo]);
                        used += 2;
                        if (++s == kSlots) { s = 0; phase ^= 1; }
                    }
                    if (!ok) break;      // acount: accumulators handed over
                    tc_commit<PAIR>(&tmem_full[a]);
                }
            }
            publish(&counts->used, used, kCtas);
            publish(&counts->filled, acount, kCtas);
        }
    } else {
        // ---------------- epilogue: warps 2..17, TMEM lanes 32*(warp % 4) .. +31 ----------------
        const int q = warp & 3;
        const uint32_t drained[2] = {PAIR ? cluster_addr(&tmem_empty[0], 0) : 0, PAIR ? cluster_addr(&tmem_empty[1], 0) : 0};
        uint32_t tcount = 0;
        bool ok = true;
        auto release = [&](uint32_t a) {   // this warp has drained its part of accumulator a
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {
                if (PAIR) mbar_arrive_cluster(drained[a]); else mbar_arrive(&tmem_empty[a]);
            }
        };
        auto ready = [&](uint32_t a, uint32_t parity, int site) {
            const bool here = wait_or_abort(&tmem_full[a], parity, abort_flag);
            if (!here && lane == 0) give_up(site);
            tc_fence_after();
            return here;
        };
        const long long pairs = gridDim.x / kCtas;
        // A pair's warps meet at the barriers of the stores: all four of a lane quarter go on, or none.  A CTA's own: the warp by itself.
        auto together = [&](bool here) { return PAIR ? quarter_all(q, here) : __all_sync(0xffffffffu, here) != 0; };
        // a CTA by itself: 32 staged columns of this warp, from column `first` of the tile on, to the result
        auto store_block = [&](const float *block, float *dst, long long pitch, int first, int rows, int cols) {
            __syncwarp();
            if (P.vec_store && first + 32 <= cols) {
                const int cc = lane & 7;
#pragma unroll
                for (int it = 0; it < 8; ++it) {
                    const int row = it * 4 + (lane >> 3);
                    const float4 v = *reinterpret_cast<const float4 *>(block + row * 32 + ((cc ^ (row & 7)) << 2));
                    if (row < rows) reinterpret_cast<float4 *>(dst + row * pitch + first)[cc] = v;
                }
            } else if (first + lane < cols) {
                const int n = rows < 32 ? rows : 32;
                float *p = dst + first + lane;
#pragma unroll 8
                for (int row = 0; row < n; ++row) p[row * pitch] = block[row * 32 + (((lane >> 2) ^ (row & 7)) << 2) + (lane & 3)];
            }
            __syncwarp();
        };
        if constexpr (STORED) {
            // which 16 of every 64 columns; a CTA by itself: which kCols
            const int cq = (warp - 2) >> 2;
            constexpr int kCols = 4 * BN / L::kWarps, kFirst = PAIR ? 16 : kCols, kStep = PAIR ? kStoreCols : 16;
            float *stage = reinterpret_cast<float *>(smem + L::OFF_STAGE + (PAIR ? q * 2 * kStoreBuffer : (warp - 2) * 4096));
            const uint32_t acc = tmem_base + ((uint32_t)(q * 32) << 16);
            if constexpr (TF32) {
                // Chunked reduction (plain products only): every chunk's accumulator is added, rounded to
                // nearest, into 64 register-resident sums per thread; the tile is stored after its last chunk.
                static_assert(!TF32 || EPI == TPW_DOT_LINEAR, "the tf32 pipeline serves the plain products");
                const int kchunk = (P.kchunk > 0 && P.kchunk < nkb) ? P.kchunk : nkb;
                const int nchunks = (nkb + kchunk - 1) / kchunk;
                uint32_t acount = 0;
                ProductShare<Index> share(P, nchunks, kCtas);
                const int start = share.at;
                Index tile;
                for (int c0, c1; ok && share.next(tile, c0, c1);) {
                    long long t = tile;
                    const long long tn = t % P.tiles_n; t /= P.tiles_n;
                    const long long tm = t % P.tiles_m;
                    const long long b = t / P.tiles_m;
                    float sums[kCols / 16][16];
#pragma unroll
                    for (int p = 0; p < kCols / 16; ++p)
#pragma unroll
                        for (int v = 0; v < 16; ++v) sums[p][v] = 0.f;
                    for (int ch = c0; ch < c1; ++ch, ++acount) {
                        const uint32_t a = acount & 1;
                        ok = ready(a, (acount >> 1) & 1, 6);
                        if (!ok) break;
#pragma unroll
                        for (int p = 0; p < kCols / 16; p += 2) {   // two loads under way: the sums leave few registers
                            uint32_t r0[16], r1[16];
                            tmem_ld16(acc + a * BN + p * kStep + cq * kFirst, r0);
                            tmem_ld16(acc + a * BN + (p + 1) * kStep + cq * kFirst, r1);
                            tmem_ld_wait();
#pragma unroll
                            for (int v = 0; v < 16; ++v) sums[p][v] += __uint_as_float(r0[v]);
#pragma unroll
                            for (int v = 0; v < 16; ++v) sums[p + 1][v] += __uint_as_float(r1[v]);
                        }
                        release(a);
                    }
                    ok = together(ok);
                    if (!ok) break;
                    const long long row_base = tm * kTileRows + rank * BM + q * 32;
                    if constexpr (!PAIR) {
                        const int rows = row_base < P.N1 ? (int)(P.N1 - row_base < 32 ? P.N1 - row_base : 32) : 0;
                        const int cols = P.N2 - tn * BN < BN ? (int)(P.N2 - tn * BN) : BN;
#pragma unroll
                        for (int p = 0; p < kCols / 16; p += 2) {
                            stage_values<32>(stage, sums[p], 0, lane);
                            stage_values<32>(stage, sums[p + 1], 16, lane);
                            store_block(stage, P.out + (b * P.N1 + row_base) * P.N2 + tn * BN, P.N2, cq * kCols + p * 16, rows, cols);
                        }
                        continue;
                    }
                    const bool part = c1 - c0 < nchunks;
                    // a share holds at most two parts of tiles, one at its start and one at its end
                    const long long slot = (long long)(blockIdx.x >> 1) * 2 + ((tile - share.base) * nchunks + c0 == start ? 0 : 1);
                    float *dst = part ? P.partial + (slot * TM + rank * BM + q * 32) * BN : P.out + (b * P.N1 + row_base) * P.N2 + tn * BN;
                    const long long pitch = part ? BN : P.N2;
                    const int rows = row_base < P.N1 ? (int)(P.N1 - row_base) : 0, cols = P.N2 - tn * BN < BN ? (int)(P.N2 - tn * BN) : BN;
#pragma unroll
                    for (int p = 0; p < BN / kStoreCols; ++p) {
                        if (p * kStoreCols >= cols) continue;
                        float *buf = stage + (p & 1) * (32 * kStoreCols);
                        stage_values<kStoreCols>(buf, sums[p], cq * 16, lane);
                        quarter_sync(q);
                        // a part is stored in whole 64-column segments and finished by product_fixup_kernel
                        store_rows<kStoreCols, false>(buf, dst + p * kStoreCols, pitch, part ? 32 : rows, part ? kStoreCols : cols - p * kStoreCols,
                                                      part || P.vec_store, cq, lane);
                    }
                }
            } else {
                for (long long tile = blockIdx.x / kCtas; tile < P.tiles; tile += pairs, ++tcount) {
                    long long tn, tm, b;
                    decode_tile<false>(tile, P, tn, tm, b);
                    const uint32_t a = tcount & 1;
                    // the row's norm depends on the tile index alone: fetched before the wait
                    const long long row_base = tm * kTileRows + rank * BM + q * 32, i = row_base + lane;
                    const float n1 = (EPI != TPW_DOT_LINEAR && i < P.N1) ? P.n1sq[b * P.N1 + i] : 0.f;
                    if (!together(ready(a, (tcount >> 1) & 1, 4))) break;
                    const int rows = row_base < P.N1 ? (int)(P.N1 - row_base < 32 ? P.N1 - row_base : 32) : 0;
                    const int cols = P.N2 - tn * BN < BN ? (int)(P.N2 - tn * BN) : BN, passes = (cols + kStoreCols - 1) / kStoreCols;
                    const float *n2p = P.n2sq + b * P.N2 + tn * BN;
                    float *out = P.out + (b * P.N1 + row_base) * P.N2 + tn * BN;
                    // this thread's 16 columns from col (a multiple of 16) on
                    auto columns = [&](int col, bool last, float (&o)[16]) {
                        const int left = cols - col;
                        float n2[16];
                        if (EPI != TPW_DOT_LINEAR) {
                            if (P.vec_store && left >= 16) {
#pragma unroll
                                for (int v = 0; v < 4; ++v) {
                                    const float4 t = __ldg(reinterpret_cast<const float4 *>(n2p + col) + v);
                                    n2[4 * v] = t.x; n2[4 * v + 1] = t.y; n2[4 * v + 2] = t.z; n2[4 * v + 3] = t.w;
                                }
                            } else {
#pragma unroll
                                for (int v = 0; v < 16; ++v) n2[v] = v < left ? __ldg(n2p + col + v) : 0.f;
                            }
                        }
                        uint32_t r[16];
                        tmem_ld16(acc + a * BN + col, r);
                        tmem_ld_wait();
                        if (last) release(a);
                        dot_epilogue16<EPI>(r, n1, n2, o);
                        if constexpr (SELF) {
                            const long long j0 = tn * BN + col;
                            if (row_base < j0 + 16 && j0 < row_base + 32) {
#pragma unroll
                                for (int v = 0; v < 16; ++v)
                                    if (i == j0 + v) o[v] = 0.f;
                            }
                        }
                    };
                    if constexpr (!PAIR) {
#pragma unroll 1
                        for (int c = 0; c < kCols / 16; ++c) {
                            float o[16];
                            columns(cq * kCols + c * 16, c + 1 == kCols / 16, o);
                            stage_values<32>(stage, o, (c & 1) * 16, lane);
                            if (c & 1) store_block(stage, out, P.N2, cq * kCols + (c - 1) * 16, rows, cols);
                        }
                    } else if (P.vec_store) {
#pragma unroll 1
                        for (int p = 0; p < passes; ++p) {
                            float o[16];
                            columns(p * kStoreCols + cq * 16, p + 1 == passes, o);
                            float *buf = stage + (p & 1) * (32 * kStoreCols);
                            stage_values<kStoreCols>(buf, o, cq * 16, lane);
                            quarter_sync(q);
                            store_rows<kStoreCols, false>(buf, out + p * kStoreCols, P.N2, rows, cols - p * kStoreCols, true, cq, lane);
                        }
                    } else {
                        constexpr int kWide = 2 * kStoreCols;   // both buffers as one
#pragma unroll 1
                        for (int p = 0; p < passes; ++p) {
                            float o[16];
                            columns(p * kStoreCols + cq * 16, p + 1 == passes, o);
                            stage_values<kWide>(stage, o, (p & 1) * kStoreCols + cq * 16, lane);
                            if ((p & 1) == 0 && p + 1 < passes) continue;
                            const int first = (p & ~1) * kStoreCols;
                            quarter_sync(q);
                            store_rows<kWide, false>(stage, out + first, P.N2, rows, cols - first, false, cq, lane);
                            quarter_sync(q);
                        }
                    }
                }
            }
        } else {
            // warps 2..9 own the even accumulators, warps 10..17 the odd ones; each drains half of the columns
            const int chalf = ((warp - 2) >> 2) & 1;
            const uint32_t a = (uint32_t)(warp - 2) >> 3;
            const uint32_t acc = tmem_base + ((uint32_t)(q * 32) << 16) + a * BN + chalf * (BN / 2);
            constexpr int kLast = BN / 64 - 1;
            for (long long tile = (long long)(blockIdx.x >> 1) + a * pairs; tile < P.tiles; tile += 2 * pairs, ++tcount) {
                long long tn, tm, b;
                decode_tile<TOPK != 0>(tile, P, tn, tm, b);
                const bool same_rows = ROWMIN && rank_1_is_idle(tm, P);
                const long long i = tm * TM + (same_rows ? 0 : rank * BM) + q * 32 + lane;
                const bool row_ok = i < P.N1;
                const float n1 = row_ok ? P.n1sq[b * P.N1 + i] : 0.f;
                const float *n2p = P.n2sq + b * P.N2;
                const long long col0 = tn * BN + chalf * (BN / 2);
                if (!ready(a, tcount & 1, 4)) break;
                if constexpr (ROWMIN) {
                    // streaming row minimum: this thread owns row i and folds its columns into one key
                    // (the epilogue value is non-negative, so its bit pattern orders like an unsigned integer)
                    unsigned long long best = ~0ull;
                    const int last = same_rows ? 2 * (int)rank + 1 : kLast;
#pragma unroll 1
                    for (int c = same_rows ? 2 * (int)rank : 0; c <= last; ++c) {
                        const long long j0 = col0 + c * 32;
                        uint32_t r[32];
                        tmem_ld32(acc + c * 32, r);
                        tmem_ld_wait();
                        if (c == last) release(a);
                        if (j0 >= P.N2) continue;
#pragma unroll
                        for (int v = 0; v < 32; ++v) {
                            const long long j = j0 + v;
                            const float nn = j < P.N2 ? __ldg(n2p + j) : 0.f;
                            const float o = dot_epilogue<EPI>(__uint_as_float(r[v]), n1, nn, false);
                            const unsigned long long key = ((unsigned long long)__float_as_uint(o) << 32) | (unsigned long long)(uint32_t)j;
                            if (j < P.N2 && key < best) best = key;
                        }
                    }
                    if (row_ok && best != ~0ull) atomicMin(P.rowmin_keys + b * P.N1 + i, best);
                }
                if constexpr (TOPK != 0) {
                    // Columns past the last count as NaN, which no minimum takes and no comparison passes.  TOPK < 0 keeps the minimum
                    // of every group of columns.  TOPK > 0: the minimum of eight distances decides for all of them whether any lane of the
                    // warp has one within its limit; if so, every lane appends its passing columns to its own words of the
                    // staging area, eight predicated stores without a loop.  Room for 16 keys a lane: a lane that holds more than 8
                    // (a row whose bound is loose) sends the warp's next groups through the loop below, which keeps the k smallest.
                    // (One passing column per trip of such a loop for every group: 10 nearest of [50000, 20000, 128], the pass over all
                    // columns 1.07 -> 0.95 ms; without any candidates it takes 0.45.)
                    const int k = P.topk_k;
                    const long long cols = TOPK < 0 ? P.cols : P.N2;
                    unsigned long long *buf = reinterpret_cast<unsigned long long *>(smem + L::OFF_STAGE + (warp - 2) * 4096) + lane;   // [16][32 lanes]
                    float *norms = reinterpret_cast<float *>(smem + L::OFF_STAGE + (warp - 2) * 4096);                                  // TOPK < 0: [128]
                    int cnt = 0;                                  // keys held
                    // keys have to stay below the bound of the row's k-th smallest; any value read while other tiles lower it is one
                    unsigned long long limit = 0;
                    if constexpr (TOPK > 0) {
                        if (row_ok) limit = *reinterpret_cast<volatile unsigned long long *>(P.topk_thr + b * P.N1 + i);
                    }
                    auto limit_value = [&]() {                    // every distance whose key is below the limit is at most this
                        const uint32_t hi = (uint32_t)(limit >> 32);
                        // a limit at or above the upper clamp lets every raw value through
                        return hi >= 0x7f800000u || (EPI == TPW_DOT_COSINE_DIST && hi >= 0x40000000u) ? INFINITY : __uint_as_float(hi);
                    };
                    float lim = row_ok ? limit_value() : -1.f;    // rows past N1: nothing passes
                    float gm[16];                                 // TOPK < 0: minima of the half's columns of every residue modulo 16
#pragma unroll
                    for (int t = 0; t < 16; ++t) gm[t] = INFINITY;
                    if constexpr (TOPK < 0) {
                        // the sampled rows' norms lie apart: fetched once per tile half (NaN past the last column)
                        __syncwarp();
#pragma unroll
                        for (int t = 0; t < 4; ++t) {
                            const long long j = col0 + t * 32 + lane;
                            norms[t * 32 + lane] = j < cols ? __ldg(n2p + j * P.col_step) : NAN;
                        }
                        __syncwarp();
                    }
#pragma unroll 1
                    for (int c = 0; c <= kLast; ++c) {
                        const long long j0 = col0 + c * 32;
                        uint32_t r[32];
                        tmem_ld32(acc + c * 32, r);
                        tmem_ld_wait();
                        if (c == kLast) release(a);
                        if (j0 >= cols) continue;
                        const bool whole = TOPK > 0 && P.vec_store && j0 + 32 <= cols;
#pragma unroll
                        for (int g = 0; g < 4; ++g) {
                            float nn[8], o[8];
                            if (whole || TOPK < 0) {
#pragma unroll
                                for (int u = 0; u < 2; ++u) {
                                    const float4 v4 = TOPK < 0 ? reinterpret_cast<const float4 *>(norms + c * 32 + 8 * g)[u]
                                                               : __ldg(reinterpret_cast<const float4 *>(n2p + j0 + 8 * g) + u);
                                    nn[4 * u] = v4.x; nn[4 * u + 1] = v4.y; nn[4 * u + 2] = v4.z; nn[4 * u + 3] = v4.w;
                                }
                            } else {
#pragma unroll
                                for (int v = 0; v < 8; ++v) nn[v] = j0 + 8 * g + v < cols ? __ldg(n2p + (j0 + 8 * g + v)) : 0.f;
                            }
#pragma unroll
                            for (int v = 0; v < 8; ++v) {
                                o[v] = raw_distance<EPI>(__uint_as_float(r[8 * g + v]), n1, nn[v]);
                                if (TOPK < 0 ? isnan(nn[v]) : !whole && j0 + 8 * g + v >= cols) o[v] = NAN;
                            }
                            if constexpr (TOPK < 0) {
#pragma unroll
                                for (int v = 0; v < 8; ++v) gm[(g & 1) * 8 + v] = fminf(gm[(g & 1) * 8 + v], o[v]);
                            } else {
                                const float m = min3(min3(o[0], o[1], o[2]), min3(o[3], o[4], o[5]), fminf(o[6], o[7]));
                                if (!__any_sync(0xffffffffu, m <= lim)) continue;
                                if (__all_sync(0xffffffffu, cnt <= 8)) {
                                    uint32_t at = smem_u32(buf) + cnt * 256;
#pragma unroll
                                    for (int v = 0; v < 8; ++v)
                                        if (o[v] <= lim) {
                                            asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(at), "r"((uint32_t)(j0 + 8 * g + v)),
                                                         "r"(__float_as_uint(clamp_distance<EPI>(o[v])))
                                                         : "memory");
                                            at += 256;
                                        }
                                    cnt = (at - smem_u32(buf)) >> 8;
                                    continue;
                                }
                                uint32_t mask = 0;
#pragma unroll
                                for (int v = 0; v < 8; ++v)
                                    if (o[v] <= lim) mask |= 1u << v;
                                int worst = 0;
                                auto shrink = [&]() {
                                    const KeySlot last = keep_smallest(buf, cnt, k);
                                    cnt = k;
                                    limit = last.key;
                                    worst = last.slot;
                                    lim = limit_value();
                                };
                                if (cnt >= k) shrink();
#pragma unroll 1
                                while (__any_sync(0xffffffffu, mask != 0)) {
                                    const int v = __ffs(mask) - 1;       // -1: nothing left in this lane
                                    mask &= mask - 1;
                                    float ov = o[0];
#pragma unroll
                                    for (int u = 1; u < 8; ++u)
                                        if (v == u) ov = o[u];
                                    const unsigned long long key = ((unsigned long long)__float_as_uint(clamp_distance<EPI>(ov)) << 32) |
                                                                   (unsigned long long)(uint32_t)(j0 + 8 * g + v);
                                    if (v < 0 || key >= limit) continue;
                                    buf[(cnt < k ? cnt : worst) * 32] = key;
                                    if (cnt < k) ++cnt;
                                    if (cnt == k) shrink();
                                }
                            }
                        }
                    }
                    if constexpr (TOPK < 0) {
#pragma unroll
                        for (int t = 0; t < 16; ++t) gm[t] = clamp_distance<EPI>(gm[t]);
                        const long long at = ((b * P.N1 + i) * P.tiles_n + tn) * 2 + chalf;
                        float4 *dst = reinterpret_cast<float4 *>(P.gmin) + (P.col_group == 8 ? at * 4 : at);
                        if (!row_ok) {
                        } else if (P.col_group == 8) {
#pragma unroll
                            for (int t = 0; t < 4; ++t) dst[t] = make_float4(gm[4 * t], gm[4 * t + 1], gm[4 * t + 2], gm[4 * t + 3]);
                        } else {
                            auto least = [&](int t) { return fminf(min3(gm[t], gm[t + 4], gm[t + 8]), gm[t + 12]); };
                            dst[0] = make_float4(least(0), least(1), least(2), least(3));
                        }
                    }
                    if constexpr (TOPK > 0) {
                        if (cnt >= k) {
                            limit = keep_smallest(buf, cnt, k).key;
                            cnt = k;
                            atomicMin(P.topk_thr + b * P.N1 + i, limit);   // k keys up to it, which are written here
                        }
                        // behind the keys that other tile halves have written (their order does not matter: the keys are unique
                        // and the merge looks at all of them)
                        if (cnt > 0) {
                            const int at = atomicAdd(P.topk_count + b * P.N1 + i, cnt);
                            unsigned long long *dst = P.topk_lists + (b * P.N1 + i) * P.topk_L * k + at;
#pragma unroll 1
                            for (int t = 0; t < cnt; ++t) dst[t] = buf[t * 32];
                        }
                        __syncwarp();
                    }
                }
            }
        }
    }

    tc_fence_before();
    __syncthreads();
    if (PAIR) cluster_sync();   // neither CTA's shared memory goes while the other may still read it or arrive in it
    if (*reinterpret_cast<volatile int *>(abort_flag)) {   // raised in both CTAs or in neither
        if (threadIdx.x == 0)
            drain_pair(full, empty, tmem_full, kSlots, counts, rank, [&](uint32_t u) {
                const bool high = u % parts == 0;
                return (uint32_t)((high || need_xl ? A_BYTES : 0) + (high || need_yl ? B_BYTES : 0));
            });
        __syncthreads();
        if (PAIR) cluster_sync();
    }
    if (warp == 1) {
        tc_fence_after();
        if (PAIR) tmem_dealloc_pair(tmem_base, kTmemCols); else tmem_dealloc(tmem_base, kTmemCols);
    }
}

// Tiles whose chunks several pairs share: the parts' sums, added in the order of the chunks; ROWS rows of a tile to a CTA.  What it takes is
// the parts' latency.  A tile or two left over lie in many parts (one for every chunk or two) and make few CTAs: four rows and eight parts in
// flight; many tiles lie in two or three each: sixteen rows.  [15, 1131, 1393, 192], 1 and 16 tiles left over: 47 us for both launches when
// parts were read one at a time, each behind three 64-bit divisions for its place; 14 now.
template <int ROWS>
__global__ void __launch_bounds__(BN)
product_fixup_kernel(const GemmParams P, int nch, long long pairs) {
    constexpr int PARTS = 32 / ROWS;
    __shared__ int parts[BN], before[BN / 32];      // deals_chunks: no more pairs than threads
    const long long left = P.tiles % pairs, base = P.tiles - left, local = blockIdx.x / (TM / ROWS), tile = base + local;
    const int row0 = (int)(blockIdx.x % (TM / ROWS)) * ROWS, col = threadIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const long long all = left * nch, u0 = local * nch, u1 = u0 + nch;
    // the shares that hold chunks of this tile, shares without chunks (fewer chunks than pairs) left out: one thread looks at each
    const int c = threadIdx.x;
    const bool narrow = all * BN < (1ll << 31);     // 32-bit divisions do
    const long long begin = narrow ? (int)all * c / (int)pairs : all * c / pairs, end = narrow ? (int)all * (c + 1) / (int)pairs : all * (c + 1) / pairs;
    const bool holds = c < pairs && begin < end && begin < u1 && end > u0;
    const uint32_t vote = __ballot_sync(0xffffffffu, holds);
    if (lane == 0) before[warp] = __popc(vote);
    __syncthreads();
    int n = 0, at = __popc(vote & ((1u << lane) - 1));
#pragma unroll
    for (int w = 0; w < BN / 32; ++w) {
        if (w < warp) at += before[w];
        n += before[w];
    }
    if (holds) parts[at] = c * 2 + (begin >= u0 ? 0 : 1);
    __syncthreads();
    if (n == 1) return;                             // one pair had the whole tile
    long long t = tile;
    const long long tn = t % P.tiles_n; t /= P.tiles_n;
    const long long tm = t % P.tiles_m;
    const long long b = t / P.tiles_m;
    const long long j = tn * BN + col;
    const int rows = P.N1 - tm * TM - row0 < ROWS ? (int)(P.N1 - tm * TM - row0) : ROWS;
    if (j >= P.N2 || rows <= 0) return;
    const float *src = P.partial + row0 * BN + col;
    float s[ROWS] = {};
    for (int k = 0; k < n; k += PARTS) {
        float v[PARTS][ROWS];
#pragma unroll
        for (int u = 0; u < PARTS; ++u)
#pragma unroll
            for (int r = 0; r < ROWS; ++r) v[u][r] = k + u < n && r < rows ? src[(long long)parts[k + u] * (TM * BN) + r * BN] : 0.f;
#pragma unroll
        for (int u = 0; u < PARTS; ++u)
#pragma unroll
            for (int r = 0; r < ROWS; ++r) s[r] += v[u][r];
    }
#pragma unroll
    for (int r = 0; r < ROWS; ++r)
        if (r < rows) P.out[(b * P.N1 + tm * TM + row0 + r) * P.N2 + j] = s[r];
}

// fp32 rows -> bf16 high/low parts (row pitch Dp, zero padded) and a per-row fp32 scalar: the
// squared norm, or (recip != 0) the reciprocal norm with 0 for an all-zero row; one warp per row
struct SplitRows {
    const float *x;
    __nv_bfloat16 *hi, *lo;
    float *nsq;
    int *lo_any;
    long long rows;
};
__global__ void split_rows_kernel(const SplitRows first, const SplitRows second, long long D, long long Dp, int recip) {
    // both operands in one launch: the clearing of lo_any in front of it then costs no launch more than two splits did
    const SplitRows &P = blockIdx.y == 0 ? first : second;
    const float *__restrict__ x = P.x;
    __nv_bfloat16 *__restrict__ hi = P.hi, *__restrict__ lo = P.lo;
    float *__restrict__ nsq = P.nsq;
    int *lo_any = P.lo_any;
    const long long rows = P.rows;
    const int lane = threadIdx.x & 31;
    const long long warp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
    uint32_t any = 0;                     // bits of all low parts but their signs: zero where they are all zero
    const bool vec = D == Dp && (reinterpret_cast<uintptr_t>(x) & 15u) == 0;   // D a multiple of 8: 16 bytes in, 8 and 8 out
    for (long long r = warp; r < rows; r += nwarps) {
        const float *row = x + r * D;
        float s = 0.f;
        auto split = [&](float v, uint32_t &hb, uint32_t &lb) {
            const __nv_bfloat16 h = __float2bfloat16_rn(v), l = __float2bfloat16_rn(v - __bfloat162float(h));
            hb = __bfloat16_as_ushort(h);
            lb = __bfloat16_as_ushort(l);
        };
        if (vec) {
            for (long long k = lane * 4; k < D; k += 128) {
                const float4 v = __ldg(reinterpret_cast<const float4 *>(row + k));
                uint32_t h[4], l[4];
                split(v.x, h[0], l[0]); split(v.y, h[1], l[1]); split(v.z, h[2], l[2]); split(v.w, h[3], l[3]);
                const uint2 hv = make_uint2(h[0] | (h[1] << 16), h[2] | (h[3] << 16)), lv = make_uint2(l[0] | (l[1] << 16), l[2] | (l[3] << 16));
                *reinterpret_cast<uint2 *>(hi + r * Dp + k) = hv;
                *reinterpret_cast<uint2 *>(lo + r * Dp + k) = lv;
                any |= (lv.x | lv.y) & 0x7fff7fffu;
                s = fmaf(v.x, v.x, s); s = fmaf(v.y, v.y, s); s = fmaf(v.z, v.z, s); s = fmaf(v.w, v.w, s);
            }
        } else {
            for (long long k = lane; k < Dp; k += 32) {
                const float v = k < D ? row[k] : 0.f;
                uint32_t h, l;
                split(v, h, l);
                hi[r * Dp + k] = __ushort_as_bfloat16((unsigned short)h);
                lo[r * Dp + k] = __ushort_as_bfloat16((unsigned short)l);
                any |= l & 0x7fffu;
                s = fmaf(v, v, s);
            }
        }
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
        if (lane == 0) {
            if (recip) {
                const float nrm = sqrtf(s);
                nsq[r] = nrm != 0.f ? __fdiv_rn(1.f, nrm) : 0.f;
            } else {
                nsq[r] = s;
            }
        }
    }
    // one store per CTA: one per warp, 19 thousand to one address, queued up for 50 us
    if (__syncthreads_or(any != 0) && threadIdx.x == 0) *lo_any = 1;
}

inline long long align_up(long long v, long long a) { return (v + a - 1) / a * a; }

// TPW_ENGINE_AUTO: the tensor-core engine pays for its split pre-pass and its tiles, 128 or 256 rows by 256, only on
// large fp32 problems; everything else stays on the exact fp32/fp64 CUDA-core tile.  Euclidean at 2^28 terms, tensor cores over CUDA cores:
// 1.2 with 128 rows and up to 256 features, 0.7 to 1.2 with 129 to 2048 rows, 0.3 to 0.6 from 1024 features on; at 2^27 1.1 to 1.2.
inline bool auto_picks_tensor_cores(int dtype, long long B, long long N1, long long N2, long long D) {
    return dtype == TPW_F32 && D >= 64 && N1 >= 128 && N2 >= 256 && (double)B * N1 * N2 * D >= (double)(1ll << 28);
}

// Stored bf16 tiles: whether a CTA works by itself, on 128 x 256, instead of in a pair.  A pair saves operand copies but couples its 32 epilogue
// warps, at the stores' barriers and at the accumulators; with few features the results are the bound.  Times of pairs and of single
// CTAs over tiles of 128 x 256 with eight epilogue warps and word-wise ragged stores, sqeuclidean (euclidean) of [131072, 16384, D],
// [30011, 10008, D] and [8000, 4000, D]:
//   64 features   1.0 to 1.16 (0.6 to 0.7) and 0.71 to 0.81 (0.45 to 0.51);   128  0.92 to 1.05 (0.61 to 0.66) and 0.79 to 0.87 (0.51 to 0.54)
//   160           1.02 (0.67 to 0.72) and 0.98 to 1.0 (0.63 to 0.67);   256  0.93 to 0.99 (0.7 to 0.78) and 1.01 to 1.1 (0.7 to 0.83)
// and where rows of the result start on no 16-byte boundary, [30011, 10007, D] and [8000, 4001, D]:
//   64            1.05 to 1.06 (0.75 to 0.78) and 1.11 to 1.22 (0.71 to 0.73), results within L2 0.96 (0.61): of larger ones two warps' stores
//                 complete a sector only after it has left L2, the more the faster they follow each other;   96  1.03 and 1.03
//   128 to 256    0.98 to 1.04 (0.75 to 0.79) and 0.88 to 0.97 (0.6 to 0.67);   500  0.86 and 1.14
inline bool single_pays(bool aligned, double bytes, long long D) {
    return aligned ? D <= 160 : D <= 256 && (D >= 96 || bytes <= 134217728.0);
}

struct ScratchLayout {
    long long Dp, off_xh, off_xl, off_yh, off_yl, off_n1, off_n2, off_lo, total;
};

inline ScratchLayout scratch_layout(long long B, long long N1, long long N2, long long D, bool self) {
    ScratchLayout L;
    L.Dp = align_up(D, 8); // 16-byte row pitch for the tensor maps
    const long long xa = align_up(B * N1 * L.Dp * 2, 1024), ya = self ? 0 : align_up(B * N2 * L.Dp * 2, 1024);
    L.off_xh = 0;
    L.off_xl = xa;
    L.off_yh = self ? L.off_xh : 2 * xa;
    L.off_yl = self ? L.off_xl : 2 * xa + ya;
    L.off_n1 = 2 * xa + 2 * ya;
    L.off_n2 = self ? L.off_n1 : L.off_n1 + align_up(B * N1 * 4, 1024);
    L.off_lo = L.off_n2 + align_up(B * N2 * 4, 1024);
    L.total = L.off_lo + 1024;
    return L;
}


// ---- gradient products on the tensor cores (tf32 x 3) ---------------------------------------------
//
// grad_x1 = s_mm * (C . X2) + s_row * x1 * rowsum(C),  grad_x2 = s_mm * (C^T . X1) + s_row * x2 * colsum(C)
// with C = g (squared Euclidean, plain products) or g / o (Euclidean).  Each operand is split into
// two tf32 numbers, hi = rn_tf32(v) and lo = rn_tf32(v - hi), and hi.hi + hi.lo + lo.hi is
// accumulated in fp32: 22 bits of every factor take part, so the products carry about 2^-21 of
// relative error, two orders below the float32 parity tolerance even for sums that cancel.

__device__ __forceinline__ float rn_tf32(float v) {
    uint32_t u;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(u) : "f"(v));
    return __uint_as_float(u);
}

enum { COEF_ID = 0, COEF_DIV_AUX = 1, COEF_COSINE = 2 };
constexpr int PT = 64;        // pre-pass tile edge

struct SplitParams {
    const float *a, *aux;       // [B,R,C]
    const float *n1, *n2;       // COEF_COSINE: row norms [B,R], [B,C]
    float *hi, *lo;             // [B,R,Cp]   (STRAIGHT)
    int *clear;                 // four words to set to 0 for the launches that follow; may be NULL
    float *rowpart, *colpart;   // [B,TC,R], [B,TR,C]   (SUMS)
    long long R, C, Cp, TR, TC;
    int vec_in;                 // C % 4 == 0 and 16-byte aligned inputs
    int epilogue;               // COEF_COSINE: what aux holds (tpw_dot_epilogue)
};

// Coefficient of one element and the summands of its row and column sums.
//   COEF_ID:      c = a
//   COEF_DIV_AUX: c = a / aux, 0 where aux == 0                     (Euclidean: g / o)
//   COEF_COSINE:  S = M / (n1 n2) with the "identity" safe divide, aux = S or 1 - S, a = upstream
//                 gradient: c = dM = gs / (n1 n2) (gs where that is 0), and with dd = -c S (0 where
//                 the denominator is 0) the row summand is dd n2[j], the column summand dd n1[i]
//                 (the gradients of the two norm vectors)
template <int MODE>
__device__ __forceinline__ void coefficient(float a, float aux, float na, float nb, int epilogue, float &c, float &rs, float &cs) {
    if (MODE == COEF_ID) {
        c = rs = cs = a;
    } else if (MODE == COEF_DIV_AUX) {
        c = aux != 0.f ? __fdiv_rn(a, aux) : 0.f;
        rs = cs = c;
    } else {
        const float S = epilogue == TPW_DOT_COSINE_SIM ? aux : 1.f - aux;
        const float gs = epilogue == TPW_DOT_COSINE_SIM ? a : -a;
        const float denom = na * nb;
        float dd = 0.f;
        if (denom != 0.f) {
            c = __fdiv_rn(gs, denom);
            dd = -c * S;
        } else {
            c = gs;
        }
        rs = dd * nb;
        cs = dd * na;
    }
}

// One 64 x 64 tile per CTA of 256 threads: coefficient, tf32 high/low copies (row pitch padded to a
// multiple of 4 and zero filled), per-tile row and column sums.
template <int MODE, bool SUMS>
__global__ void __launch_bounds__(256)
split_tile_kernel(const SplitParams P) {
    __shared__ float colacc[SUMS ? 16 * PT : 1];
    const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
    const long long b = blockIdx.z;
    const long long r0 = (long long)blockIdx.y * PT, c0 = (long long)blockIdx.x * PT;
    if (P.clear && tid < 4 && blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0) P.clear[tid] = 0;
    const float *a = P.a + b * P.R * P.C;
    const float *aux = MODE != COEF_ID ? P.aux + b * P.R * P.C : nullptr;
    const long long col = c0 + 4 * tx;
    float nb[4] = {0.f, 0.f, 0.f, 0.f};
    if (MODE == COEF_COSINE) {
#pragma unroll
        for (int e = 0; e < 4; ++e)
            if (col + e < P.C) nb[e] = P.n2[b * P.C + col + e];
    }
    float colp[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const long long row = r0 + ty + 16 * r;
        float v[4] = {0.f, 0.f, 0.f, 0.f}, rs[4] = {0.f, 0.f, 0.f, 0.f};
        if (row < P.R) {
            float av[4] = {0.f, 0.f, 0.f, 0.f}, ov[4] = {0.f, 0.f, 0.f, 0.f};
            const bool vec = P.vec_in && col + 3 < P.C;
            if (vec) {
                const float4 t = *reinterpret_cast<const float4 *>(a + row * P.C + col);
                av[0] = t.x; av[1] = t.y; av[2] = t.z; av[3] = t.w;
                if (MODE != COEF_ID) {
                    const float4 o = *reinterpret_cast<const float4 *>(aux + row * P.C + col);
                    ov[0] = o.x; ov[1] = o.y; ov[2] = o.z; ov[3] = o.w;
                }
            } else {
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (col + e < P.C) {
                        av[e] = a[row * P.C + col + e];
                        if (MODE != COEF_ID) ov[e] = aux[row * P.C + col + e];
                    }
            }
            const float na = MODE == COEF_COSINE ? P.n1[b * P.R + row] : 0.f;
#pragma unroll
            for (int e = 0; e < 4; ++e)
                if (col + e < P.C) {
                    float cs;
                    coefficient<MODE>(av[e], ov[e], na, nb[e], P.epilogue, v[e], rs[e], cs);
                    colp[e] += cs;
                }
        }
        if (row < P.R && col < P.Cp) {
            float4 h, l;
            h.x = rn_tf32(v[0]); l.x = rn_tf32(v[0] - h.x);
            h.y = rn_tf32(v[1]); l.y = rn_tf32(v[1] - h.y);
            h.z = rn_tf32(v[2]); l.z = rn_tf32(v[2] - h.z);
            h.w = rn_tf32(v[3]); l.w = rn_tf32(v[3] - h.w);
            *reinterpret_cast<float4 *>(P.hi + (b * P.R + row) * P.Cp + col) = h;
            *reinterpret_cast<float4 *>(P.lo + (b * P.R + row) * P.Cp + col) = l;
        }
        if (SUMS) {
            float s = (rs[0] + rs[1]) + (rs[2] + rs[3]);
#pragma unroll
            for (int off = 1; off < 16; off <<= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
            if (tx == 0 && row < P.R) P.rowpart[(b * P.TC + blockIdx.x) * P.R + row] = s;
        }
    }
    if constexpr (SUMS) {
#pragma unroll
        for (int e = 0; e < 4; ++e) colacc[ty * PT + 4 * tx + e] = colp[e];
        __syncthreads();
        if (tid < PT && c0 + tid < P.C) {
            float s = 0.f;
#pragma unroll
            for (int y = 0; y < 16; ++y) s += colacc[y * PT + tid];
            P.colpart[(b * P.TR + blockIdx.y) * P.C + c0 + tid] = s;
        }
    }
}

// tf32 high/low copies of a matrix's transpose, [B,C,Rp]: rows of the copy run along the source's row index, zero filled to Rp.
// The product's other operand then lies K-major, staged by one copy of 128 rows instead of four of {32 values, 32 rows}: C^T x1 of
// [16, 4096, 4096, 256] 620 -> 570 us.  (The products' bound is the copies' latency: with neither MMAs nor epilogue they take as long.)
struct Transposed {
    const float *src;
    float *hi, *lo;
    int *lo_any;
    long long R, Rp;
    int vec_in;
};
__global__ void __launch_bounds__(256)
split_transposed_kernel(const Transposed first, const Transposed second, long long C, int operands) {
    __shared__ float tile[PT][PT + 1];
    const Transposed &P = blockIdx.z % operands == 0 ? first : second;   // both in one launch
    const long long R = P.R, Rp = P.Rp;
    float *__restrict__ hi = P.hi, *__restrict__ lo = P.lo;
    int *lo_any = P.lo_any;
    const int vec_in = P.vec_in, tid = threadIdx.x;
    const long long b = blockIdx.z / operands, r0 = (long long)blockIdx.y * PT, c0 = (long long)blockIdx.x * PT;
    if (r0 >= Rp) return;
    const float *__restrict__ a = P.src + b * R * C;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        const int r = u * 16 + (tid >> 4), c = (tid & 15) * 4;
        const long long row = r0 + r, col = c0 + c;
        float v[4] = {0.f, 0.f, 0.f, 0.f};
        if (row < R) {
            if (vec_in && col + 3 < C) {
                const float4 t = *reinterpret_cast<const float4 *>(a + row * C + col);
                v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
            } else {
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (col + e < C) v[e] = a[row * C + col + e];
            }
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) tile[c + e][r] = v[e];
    }
    __syncthreads();
    uint32_t any = 0;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        const int c = u * 16 + (tid >> 4), r = (tid & 15) * 4;
        const long long col = c0 + c, row = r0 + r;
        if (col >= C || row >= Rp) continue;
        float4 h, l;
        h.x = rn_tf32(tile[c][r]); l.x = rn_tf32(tile[c][r] - h.x);
        h.y = rn_tf32(tile[c][r + 1]); l.y = rn_tf32(tile[c][r + 1] - h.y);
        h.z = rn_tf32(tile[c][r + 2]); l.z = rn_tf32(tile[c][r + 2] - h.z);
        h.w = rn_tf32(tile[c][r + 3]); l.w = rn_tf32(tile[c][r + 3] - h.w);
        *reinterpret_cast<float4 *>(hi + (b * C + col) * Rp + row) = h;
        *reinterpret_cast<float4 *>(lo + (b * C + col) * Rp + row) = l;
        any |= (__float_as_uint(l.x) | __float_as_uint(l.y) | __float_as_uint(l.z) | __float_as_uint(l.w)) & 0x7fffffffu;
    }
    if (__syncthreads_or(any != 0) && tid == 0) *lo_any = 1;
}

// sums[b,n] = part[b,0,n] + part[b,1,n] + ... in that order (deterministic); the row sums and, in the second row of CTAs, the
// column sums
struct Partials {
    const float *part;
    float *sums;
    long long T, N;
};
__global__ void reduce_partials_kernel(const Partials first, const Partials second, long long B) {
    const Partials &P = blockIdx.y == 0 ? first : second;
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (t >= B * P.N) return;
    const long long b = t / P.N, n = t % P.N;
    float s = 0.f;
    for (long long k = 0; k < P.T; ++k) s += P.part[(b * P.T + k) * P.N + n];
    P.sums[t] = s;
}

// g[r,k] = s_mm * g[r,k] + s_row * x[r,k] * sums[r] for one gradient or, in the second row of CTAs, the other; VEC elements of a
// row to a thread
struct Finish {
    float *g;
    const float *x, *sums;
    long long rows;
};
template <int VEC>
__global__ void grad_finish_kernel(const Finish first, const Finish second, long long D, float s_mm, float s_row) {
    struct alignas(VEC * 4) Pack { float v[VEC]; };
    const Finish &P = blockIdx.y == 0 ? first : second;
    const long long per = D / VEC, n = P.rows * per;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
        const float sum = P.sums[t / per];
        Pack g = reinterpret_cast<Pack *>(P.g)[t];
        const Pack x = reinterpret_cast<const Pack *>(P.x)[t];
#pragma unroll
        for (int u = 0; u < VEC; ++u) g.v[u] = fmaf(s_row * x.v[u], sum, s_mm * g.v[u]);
        reinterpret_cast<Pack *>(P.g)[t] = g;
    }
}

// How a tf32 product of M x N outputs over K is cut.  Whole tiles, one wave of persistent CTAs after another, leave the last
// wave as empty as it happens to be.  Where it is less than 0.92 full, its tiles' chunks of 64 are dealt out evenly instead, at least four to
// a CTA, and the parts of split tiles (two at most per CTA) are added by a kernel of their own, 5 to 15 us.  (Dealing out all
// tiles scatters the CTAs over batches whose operands do not fit L2 together: 660 -> 880 us a product of euclidean
// [16, 4096, 4096, 256].)  cosine bfloat16 [5000, 4111, 768], both products: 302 -> 277 us; euclidean [2, 1500, 1100, 192]: 100 -> 50 us.
constexpr int kProductChunk = 2;               // k-steps of 32
constexpr long long kPartialBytes = 2ll * TM * BN * 4;   // per pair
inline long long pair_count() { return sm_count() / 2; }
inline long long product_chunks(long long K) { return ((K + BK / 2 - 1) / (BK / 2) + kProductChunk - 1) / kProductChunk; }
inline long long product_tiles(long long B, long long M, long long N) { return B * ((M + TM - 1) / TM) * ((N + BN - 1) / BN); }
inline bool deals_chunks(long long B, long long M, long long N, long long K) {
    const long long tiles = product_tiles(B, M, N), pairs = pair_count(), left = tiles % pairs;
    // one wave more or less in a long queue, or a tile of a few chunks, is not worth the second kernel
    return pairs <= BN && tiles <= 8 * pairs && product_chunks(K) >= 16 && product_chunks(K) < (1 << 20) && left > 0 && left * 100 < pairs * 92;
}
inline long long product_pairs(long long B, long long M, long long N, long long K, bool room) {
    const long long tiles = product_tiles(B, M, N), pairs = pair_count();
    if (tiles >= pairs) return pairs;
    const long long most = room && deals_chunks(B, M, N, K) ? tiles * product_chunks(K) / 4 : tiles;
    return most < pairs ? (most > tiles ? most : tiles) : pairs;
}

struct BwdScratch {
    long long N1p, N2p, TR, TC;
    long long off_chi, off_clo, off_x1hi, off_x1lo, off_x2hi, off_x2lo;
    long long off_rowpart, off_colpart, off_rowsum, off_colsum, off_lo, total;
    long long off_part, with_part;   // partial tiles of the products, where they are worth it (with_part == total: not)
};

inline BwdScratch bwd_scratch_layout(long long B, long long N1, long long N2, long long D) {
    BwdScratch L;
    L.N2p = align_up(N2, 4);
    L.N1p = align_up(N1, 4);
    L.TR = (N1 + PT - 1) / PT;
    L.TC = (N2 + PT - 1) / PT;
    long long off = 0;
    auto take = [&](long long bytes) { const long long o = off; off += align_up(bytes, 1024); return o; };
    L.off_chi = take(B * N1 * L.N2p * 4);
    L.off_clo = take(B * N1 * L.N2p * 4);
    L.off_x1hi = take(B * D * L.N1p * 4);
    L.off_x1lo = take(B * D * L.N1p * 4);
    L.off_x2hi = take(B * D * L.N2p * 4);
    L.off_x2lo = take(B * D * L.N2p * 4);
    L.off_rowpart = take(B * L.TC * N1 * 4);
    L.off_colpart = take(B * L.TR * N2 * 4);
    L.off_rowsum = take(B * N1 * 4);
    L.off_colsum = take(B * N2 * 4);
    L.off_lo = take(4 * sizeof(int));
    L.total = off;
    L.off_part = off;
    L.with_part = deals_chunks(B, N1, D, N2) || deals_chunks(B, N2, D, N1) ? off + pair_count() * kPartialBytes : off;
    return L;
}

// The tensor-core gradient products pay for their split pre-pass only on large fp32 problems.
inline bool auto_picks_tensor_backward(int dtype, long long B, long long N1, long long N2, long long D) {
    return dtype == TPW_F32 && D >= 64 && N1 >= 256 && N2 >= 256 && (double)B * N1 * N2 * D >= (double)(1ll << 28);
}

template <int MODE, bool SUMS>
int launch_split(const SplitParams &P, long long B, cudaStream_t s) {
    const long long gx = (P.C + PT - 1) / PT, gy = (P.R + PT - 1) / PT;
    TPW_CHECK_ARG(gy <= 65535 && B <= 65535, "dense backward: more than 65535 row tiles or batches");
    split_tile_kernel<MODE, SUMS><<<dim3((unsigned)gx, (unsigned)gy, (unsigned)B), 256, 0, s>>>(P);
    TPW_LAUNCH_OK("split_tile_kernel");
    return TPW_OK;
}

// One operand of a tf32 product as high/low parts.  K-major (mn = false): rows are the M (or N) index,
// `pitch` elements per row hold k (zero padded).  MN-major (mn = true): rows are k, `pitch` elements
// per row hold the M (or N) index.
struct Tf32Operand {
    const float *hi, *lo;
    long long pitch;
    bool mn;
};

// out[b,m,n] = sum_k A[b](m,k) * Bm[b](n,k), Bm K-major; K = length of the reduction.  A K-major operand holds
// `pitch` >= K elements per row (zero beyond K), an MN-major operand has exactly K rows per batch.
// lo_any (may be NULL): lo_any[1] says whether Bm has any low part; A's are always used.
// partial (may be NULL): kPartialBytes per pair of SMs, for products that deal out chunks instead of whole tiles.
// single: tiles of a CTA by itself instead of pairs' (A K-major, no partial tiles).
int launch_tf32_product(const Tf32Operand &A, const Tf32Operand &Bm, float *out, const int *lo_any, float *partial, bool single,
                        long long B, long long M, long long N, long long K, cudaStream_t s) {
    CUtensorMap mah, mal, mbh, mbl;
    int st;
    auto encode = [&](CUtensorMap *m, const float *p, const Tf32Operand &o, long long rows, int box_rows) {
        return o.mn ? make_tensor_map_3d_atom32(m, p, 4, o.pitch, K, B, 32, 32)
                    : make_tensor_map_3d(m, p, 4, o.pitch, rows, B, BK / 2, box_rows, true);
    };
    if ((st = encode(&mah, A.hi, A, M, BM)) != TPW_OK) return st;
    if ((st = encode(&mal, A.lo, A, M, BM)) != TPW_OK) return st;
    if ((st = encode(&mbh, Bm.hi, Bm, N, single ? BN : HN)) != TPW_OK) return st;
    if ((st = encode(&mbl, Bm.lo, Bm, N, single ? BN : HN)) != TPW_OK) return st;
    GemmParams P;
    memset(&P, 0, sizeof(P));
    P.out = out;
    P.B = B; P.N1 = M; P.N2 = N; P.D = K; // K-major tails beyond K are zero padding or zero fill
    P.tiles_m = single ? (M + BM - 1) / BM : (M + TM - 1) / TM;
    P.tiles_n = (N + BN - 1) / BN;
    P.tiles = B * P.tiles_m * P.tiles_n;
    P.epilogue = TPW_DOT_LINEAR;
    P.lo_any = lo_any;
    P.lo_always = 1;
    // 64 elements per chunk: measured against float64, the products are then as accurate as the fp32
    // FMA chain of the CUDA-core kernel (the error grows in proportion to the chunk length) at no cost in time
    P.kchunk = kProductChunk;
    P.vec_store = (N % 4 == 0 && aligned16(out)) ? 1 : 0;
    P.status = device_status_ptr();
    const long long pairs = product_pairs(B, M, N, K, partial != nullptr);
    P.partial = !single && partial != nullptr && deals_chunks(B, M, N, K) ? partial : nullptr;
    const unsigned grid = single ? (unsigned)(P.tiles < sm_count() ? P.tiles : sm_count()) : 2 * (unsigned)pairs;
#define TPW_TF32_LAUNCH(AMN, PAIR)                                                                                        \
    do {                                                                                                                  \
        auto kern = gemm_metric_kernel<TPW_DOT_LINEAR, false, true, false, AMN, 0, PAIR>;                                 \
        typedef Ring<PAIR, true> L;                                                                                       \
        TPW_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, L::SMEM_ALLOC));              \
        kern<<<grid, L::kThreads, L::SMEM_ALLOC, s>>>(mah, mal, mbh, mbl, P);                                             \
    } while (0)
    if (single) TPW_TF32_LAUNCH(false, false);
    else if (A.mn) TPW_TF32_LAUNCH(true, true);
    else TPW_TF32_LAUNCH(false, true);
#undef TPW_TF32_LAUNCH
    TPW_LAUNCH_OK("gemm_metric_kernel (tf32)");
    if (P.partial && P.tiles % pairs != 0) {
        const long long left = P.tiles % pairs;
        if (left * (TM / 16) < 2 * sm_count()) product_fixup_kernel<4><<<(unsigned)(left * (TM / 4)), BN, 0, s>>>(P, (int)product_chunks(K), pairs);
        else product_fixup_kernel<16><<<(unsigned)(left * (TM / 16)), BN, 0, s>>>(P, (int)product_chunks(K), pairs);
        TPW_LAUNCH_OK("product_fixup_kernel");
    }
    return TPW_OK;
}

} // namespace
} // namespace tpw

using namespace tpw;

extern "C" int tpw_dot_metric_forward_simt(int dtype, int epilogue, const void *x1, const void *x2, void *out,
                                           int64_t B, int64_t N1, int64_t N2, int64_t D, tpw_stream_t stream);

// tf32 x 3 forward (plain dot products only): straight hi/lo copies of both operands
static long long tf32_forward_scratch(long long B, long long N1, long long N2, long long D) {
    const long long Dp = align_up(D, 4);
    return 2 * align_up(B * N1 * Dp * 4, 1024) + 2 * align_up(B * N2 * Dp * 4, 1024);
}

namespace tpw {
namespace {
// keys -> (smallest value, optionally its square root; its x2 row)
__global__ void dot_rowmin_finish_kernel(const unsigned long long *__restrict__ keys, float *__restrict__ min_out,
                                         long long *__restrict__ arg_out, long long n, int take_sqrt) {
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (t >= n) return;
    const unsigned long long key = keys[t];
    const bool none = key == ~0ull;
    float v = none ? __int_as_float(0x7f800000) : __uint_as_float((uint32_t)(key >> 32));
    if (take_sqrt) v = sqrtf(v);
    if (min_out) min_out[t] = v;
    if (arg_out) arg_out[t] = none ? -1ll : (long long)(uint32_t)key;
}
} // namespace
} // namespace tpw

namespace tpw {
namespace {
// A warp takes the k smallest of the n keys that key_of(e) returns, ascending: take(r, key), key the same in all lanes, ~0 where
// there are fewer.  Keys are unique (the x2 row, or the group, is part of the key).  Up to 128 keys, the usual case, lie
// four to a lane as they come, and each round costs two warp-wide minimum reductions; of more keys every lane first
// keeps the TOPK smallest of its share.  (Sorted insertion and 64-bit shuffles for every row, as it was: 104 keys a row,
// 50000 rows, 127 -> 40 us.)
__device__ __forceinline__ unsigned long long warp_min(unsigned long long v) {
    const uint32_t hi = __reduce_min_sync(0xffffffffu, (uint32_t)(v >> 32));
    const uint32_t lo = __reduce_min_sync(0xffffffffu, (uint32_t)(v >> 32) == hi ? (uint32_t)v : 0xffffffffu);
    return ((unsigned long long)hi << 32) | lo;
}
template <int TOPK, typename K, typename F>
__device__ __forceinline__ void warp_smallest(long long n, int k, K key_of, F take) {
    const int lane = threadIdx.x & 31;
    if (n <= 128) {
        unsigned long long mine[4];
#pragma unroll
        for (int t = 0; t < 4; ++t) mine[t] = t * 32 + lane < n ? key_of(t * 32 + lane) : ~0ull;
        for (int r = 0; r < k; ++r) {
            const unsigned long long a = mine[0] < mine[1] ? mine[0] : mine[1], b = mine[2] < mine[3] ? mine[2] : mine[3];
            const unsigned long long m = warp_min(a < b ? a : b);
#pragma unroll
            for (int t = 0; t < 4; ++t)
                if (mine[t] == m) mine[t] = ~0ull;
            take(r, m);
        }
        return;
    }
    unsigned long long mine[TOPK];
#pragma unroll
    for (int t = 0; t < TOPK; ++t) mine[t] = ~0ull;
    for (long long e = lane; e < n; e += 32) {
        const unsigned long long key = key_of(e);
        if (key < mine[TOPK - 1]) sorted_insert<TOPK>(mine, key);
    }
    for (int r = 0; r < k; ++r) {
        const unsigned long long m = warp_min(mine[0]);
        if (m != ~0ull && mine[0] == m) { // the owner pops its head
#pragma unroll
            for (int t = 0; t < TOPK - 1; ++t) mine[t] = mine[t + 1];
            mine[TOPK - 1] = ~0ull;
        }
        take(r, m);
    }
}

// One warp per row: the row's k smallest keys out of those the top-k epilogue wrote, ascending.
template <int TOPK>
__global__ void topk_merge_kernel(const unsigned long long *__restrict__ lists, const int *__restrict__ counts,
                                  float *__restrict__ val_out, long long *__restrict__ idx_out,
                                  long long rows, long long row_stride, int k, int take_sqrt) {
    const int lane = threadIdx.x & 31;
    const long long row = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (row >= rows) return;
    const unsigned long long *src = lists + row * row_stride;
    unsigned long long out = ~0ull;      // lane r: the r-th key
    warp_smallest<TOPK>(counts[row], k, [&](long long e) { return src[e]; }, [&](int r, unsigned long long m) { if (lane == r) out = m; });
    if (lane >= k) return;
    const bool none = out == ~0ull;
    float v = none ? __int_as_float(0x7f800000) : __uint_as_float((uint32_t)(out >> 32));
    if (take_sqrt) v = sqrtf(v);
    if (val_out) val_out[row * k + lane] = v;
    if (idx_out) idx_out[row * k + lane] = none ? -1ll : (long long)(uint32_t)out;
}

// One warp per row: an upper bound of the row's k-th smallest key from the minima of n groups of columns.  Each lane takes the
// smallest of its groups' minima, 32 distances of different columns, so k columns are no farther than the k-th smallest of them;
// the bound is the first key above all keys of that distance (~0: fewer than k lanes hold a finite distance).  Neighbouring
// columns belong to different groups and lanes, so that a row whose neighbours lie side by side in x2 is bounded like any other.
__global__ void topk_bound_kernel(const float *__restrict__ gmin, unsigned long long *__restrict__ bound, int *__restrict__ counts, long long rows,
                                  int n, int k) {
    const int lane = threadIdx.x & 31;
    const long long row = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (row >= rows) return;
    const float *src = gmin + row * n;
    float least = INFINITY;
#pragma unroll 4
    for (int e = lane; e < n; e += 32) least = fminf(least, src[e]);
    uint32_t mine = __float_as_uint(least), kth = 0;     // not negative: bits order like values
    for (int r = 0; r < k; ++r) {
        kth = __reduce_min_sync(0xffffffffu, mine);
        if (lane == __ffs(__ballot_sync(0xffffffffu, mine == kth)) - 1) mine = 0xffffffffu;
    }
    if (lane == 0) {
        bound[row] = kth < 0x7f800000u ? (unsigned long long)(kth + 1) << 32 : ~0ull;
        counts[row] = 0;
    }
}

constexpr int kTopkMax = 16;      // a tile half's keys fit the warp's 4 KB of staging

struct TopkScratch {
    long long L, off_lists, off_thr, off_count, total;
};
inline TopkScratch topk_scratch_layout(long long B, long long N1, long long N2, long long D, long long k) {
    TopkScratch T;
    T.L = 2 * ((N2 + BN - 1) / BN);
    const long long gemm = scratch_layout(B, N1, N2, D, false).total;
    T.off_lists = gemm;
    T.off_thr = gemm + align_up(B * N1 * T.L * k * 8, 1024);
    T.off_count = T.off_thr + align_up(B * N1 * 8, 1024);
    T.total = T.off_count + align_up(B * N1 * 4, 1024);
    return T;
}
} // namespace
} // namespace tpw

namespace tpw {
namespace {
// Common front end of the bf16 x 3 launches: splits x1 and x2 into the scratch (bf16 high/low parts, row
// norms: squared, or reciprocal for the cosine family), encodes the four tensor maps and fills the
// problem sizes of `P`.  The caller sets the epilogue-specific fields and launches.
struct Bf16Operands {
    CUtensorMap mxh, mxl, myh, myl;
};
int prepare_bf16_operands(const void *x1, const void *x2, void *scratch, bool reciprocal_norms,
                          long long B, long long N1, long long N2, long long D, cudaStream_t s,
                          Bf16Operands &M, GemmParams &P, bool pairs = true) {
    const ScratchLayout L = scratch_layout(B, N1, N2, D, false);
    unsigned char *base = static_cast<unsigned char *>(scratch);
    __nv_bfloat16 *xh = reinterpret_cast<__nv_bfloat16 *>(base + L.off_xh), *xl = reinterpret_cast<__nv_bfloat16 *>(base + L.off_xl);
    __nv_bfloat16 *yh = reinterpret_cast<__nv_bfloat16 *>(base + L.off_yh), *yl = reinterpret_cast<__nv_bfloat16 *>(base + L.off_yl);
    float *n1 = reinterpret_cast<float *>(base + L.off_n1), *n2 = reinterpret_cast<float *>(base + L.off_n2);
    int *lo_any = reinterpret_cast<int *>(base + L.off_lo);
    TPW_CUDA_OK(cudaMemsetAsync(lo_any, 0, 2 * sizeof(int), s));
    const int threads = 256;
    const long long cap = (long long)sm_count() * 16;
    const long long blocks = (B * (N1 > N2 ? N1 : N2) * 32 + threads - 1) / threads;
    const SplitRows first{(const float *)x1, xh, xl, n1, lo_any, B * N1}, second{(const float *)x2, yh, yl, n2, lo_any + 1, B * N2};
    split_rows_kernel<<<dim3((unsigned)(blocks < cap ? blocks : cap), 2), threads, 0, s>>>(first, second, D, L.Dp, reciprocal_norms ? 1 : 0);
    TPW_LAUNCH_OK("split_rows_kernel");
    int st;
    if ((st = make_tensor_map_3d(&M.mxh, xh, 2, L.Dp, N1, B, BK, BM, true)) != TPW_OK) return st;
    if ((st = make_tensor_map_3d(&M.mxl, xl, 2, L.Dp, N1, B, BK, BM, true)) != TPW_OK) return st;
    if ((st = make_tensor_map_3d(&M.myh, yh, 2, L.Dp, N2, B, BK, pairs ? HN : BN, true)) != TPW_OK) return st;
    if ((st = make_tensor_map_3d(&M.myl, yl, 2, L.Dp, N2, B, BK, pairs ? HN : BN, true)) != TPW_OK) return st;
    memset(&P, 0, sizeof(P));
    P.n1sq = n1; P.n2sq = n2;
    P.lo_any = lo_any;
    P.B = B; P.N1 = N1; P.N2 = N2; P.D = L.Dp;
    P.tiles_m = pairs ? (N1 + TM - 1) / TM : (N1 + BM - 1) / BM;
    P.tiles_n = (N2 + BN - 1) / BN;
    P.tiles = B * P.tiles_m * P.tiles_n;
    P.status = device_status_ptr();
    return TPW_OK;
}
} // namespace
} // namespace tpw

extern "C" int tpw_dot_topk_max_k(void) { return kTopkMax; }

extern "C" int64_t tpw_dot_topk_scratch_bytes(int64_t k, int64_t B, int64_t N1, int64_t N2, int64_t D) {
    if (k <= 0 || k > kTopkMax || B <= 0 || N1 <= 0 || N2 <= 0 || D <= 0) return 0;
    return topk_scratch_layout(B, N1, N2, D, k).total;
}

extern "C" int tpw_dot_topk_forward_ws(int epilogue, int k, const void *x1, const void *x2, float *val_out, int64_t *idx_out,
                                       void *scratch, int64_t scratch_bytes,
                                       int64_t B, int64_t N1, int64_t N2, int64_t D, tpw_stream_t stream) {
    clear_error();
    TPW_CHECK_ARG(epilogue == TPW_DOT_SQEUCLIDEAN || epilogue == TPW_DOT_EUCLIDEAN || epilogue == TPW_DOT_COSINE_DIST,
                  "tpw_dot_topk_forward_ws: epilogue must be TPW_DOT_SQEUCLIDEAN, TPW_DOT_EUCLIDEAN or TPW_DOT_COSINE_DIST");
    TPW_CHECK_ARG(k >= 1 && k <= kTopkMax, "tpw_dot_topk_forward_ws: k must be in [1, %d] (got %d)", kTopkMax, k);
    TPW_CHECK_ARG(B > 0 && N1 > 0 && N2 > 0 && D > 0, "tpw_dot_topk_forward_ws: sizes must be positive");
    TPW_CHECK_ARG(x1 && x2 && (val_out || idx_out), "tpw_dot_topk_forward_ws: NULL pointer");
    TPW_CHECK_ARG(N1 < (1ll << 31) && N2 < (1ll << 31) && B < (1ll << 31) && D < (1ll << 31),
                  "tpw_dot_topk_forward_ws: a dimension exceeds 2^31-1");
    const bool cosine = epilogue == TPW_DOT_COSINE_DIST;
    const TopkScratch T = topk_scratch_layout(B, N1, N2, D, k);
    const ScratchLayout L = scratch_layout(B, N1, N2, D, false);
    TPW_CHECK_ARG(scratch != nullptr && scratch_bytes >= T.total && aligned16(scratch),
                  "tpw_dot_topk_forward_ws: needs %lld bytes of 16-byte aligned scratch (got %lld)", T.total, (long long)scratch_bytes);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    unsigned char *base = static_cast<unsigned char *>(scratch);
    unsigned long long *lists = reinterpret_cast<unsigned long long *>(base + T.off_lists);
    unsigned long long *thr = reinterpret_cast<unsigned long long *>(base + T.off_thr);
    int *counts = reinterpret_cast<int *>(base + T.off_count);
    Bf16Operands M;
    GemmParams P;
    int st;
    if ((st = prepare_bf16_operands(x1, x2, scratch, cosine, B, N1, N2, D, s, M, P)) != TPW_OK) return st;
    P.epilogue = cosine ? TPW_DOT_COSINE_DIST : TPW_DOT_SQEUCLIDEAN;
    P.topk_lists = lists; P.topk_thr = thr; P.topk_count = counts; P.topk_k = k; P.topk_L = (int)T.L;
    P.vec_store = N2 % 4 == 0 ? 1 : 0;   // the squared x2 norms of a batch start on 16-byte boundaries
    const long long pairs = pair_count();
    const long long tiles_n_all = (N2 + BN - 1) / BN;
    const long long rows = B * N1;
    const unsigned mblocks = (unsigned)((rows * 32 + 255) / 256);
    long long *idx64 = reinterpret_cast<long long *>(idx_out);
    const int take_sqrt = epilogue == TPW_DOT_EUCLIDEAN ? 1 : 0;
#define TPW_TOPK_LAUNCH(EPI, CAP)                                                                                         \
    do {                                                                                                                  \
        auto kern = gemm_metric_kernel<EPI, false, false, false, false, CAP>;                                             \
        TPW_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_ALLOC));                 \
        kern<<<grid, kThreads, SMEM_ALLOC, s>>>(M.mxh, M.mxl, M.myh, M.myl, P);                                           \
        TPW_LAUNCH_OK("gemm_metric_kernel (top-k)");                                                                      \
    } while (0)
    // An insertion costs the whole warp as soon as one lane has one, so first a bound: the contraction over a sample of the x2 rows
    // keeps only the minima of groups of 8, and the k-th smallest of 32 of those bounds a row's k-th smallest distance almost as
    // closely as the distances themselves would; the pass over all columns then inserts about 5 k keys a row.  The sample is every
    // step-th row, through a tensor map of that pitch, so that the order of x2 does not matter: of 20 clusters one after another,
    // the first sixth of the columns bounded 17 of them not at all.  A quarter of the rows (an eighth for k up to 3, which inserts
    // little) was the fastest or within 3 % over 90 shapes and orders; at least one column tile.  Fewer than 8 column
    // tiles and k = 1 or 2 need no bound.  Microseconds with lists that bound each other / the first sixth, sampled from 8 tiles on / now:
    //   [50000, 20000, 128] k = 10 3989 / 1440 / 1469;  [50000, 1536, 128] k = 8 387 / 642 / 253, k = 16 806 / 1262 / 376;
    //   [20000, 20000, 64] in 20 clusters, k = 16 2338 / 4414 / 802;  [50000, 300, 128] k = 2 122 / 108 / 112
    const long long per = (k <= 3 ? 8 : 4) * BN;
    const long long sample_tiles = N2 > per ? N2 / per : 1, even = (N2 + sample_tiles * BN - 1) / (sample_tiles * BN), step = even > 1 ? even : 2;
    const long long cols = (N2 + step - 1) / step, sample = (cols + BN - 1) / BN;
    // the minima lie where the keys will, in groups as small as fit there (one column tile and k = 1: none do)
    const long long room = T.L * k * 8 / 4;
    const int group = BN / 8 * sample <= room ? 8 : BN / 32 * sample <= room ? 32 : 0;
    const long long groups = group ? (cols + group - 1) / group : 0;
    if ((tiles_n_all >= 8 || k > 2) && (groups < 32 ? groups : 32) >= k) {
        const CUtensorMap all_h = M.myh, all_l = M.myl;
        const unsigned char *yh = base + L.off_yh, *yl = base + L.off_yl;
        if ((st = make_tensor_map_3d_pitched(&M.myh, yh, 2, L.Dp, cols, B, step * L.Dp * 2, N2 * L.Dp * 2, BK, HN)) != TPW_OK) return st;
        if ((st = make_tensor_map_3d_pitched(&M.myl, yl, 2, L.Dp, cols, B, step * L.Dp * 2, N2 * L.Dp * 2, BK, HN)) != TPW_OK) return st;
        P.tiles_n = sample;
        P.tiles = B * P.tiles_m * P.tiles_n;
        P.cols = cols; P.col_step = (int)step; P.col_group = group;
        P.gmin = reinterpret_cast<float *>(lists);
        const unsigned grid = 2 * (unsigned)(P.tiles < pairs ? P.tiles : pairs);
        if (cosine) TPW_TOPK_LAUNCH(TPW_DOT_COSINE_DIST, -1); else TPW_TOPK_LAUNCH(TPW_DOT_SQEUCLIDEAN, -1);
        topk_bound_kernel<<<mblocks, 256, 0, s>>>(P.gmin, thr, counts, rows, (int)(BN / group * sample), k);
        TPW_LAUNCH_OK("topk_bound_kernel");
        M.myh = all_h; M.myl = all_l;
    } else {
        TPW_CUDA_OK(cudaMemsetAsync(thr, 0xFF, (size_t)rows * 8, s));
        TPW_CUDA_OK(cudaMemsetAsync(counts, 0, (size_t)rows * 4, s));
    }
    P.tiles_n = tiles_n_all;
    P.tiles = B * P.tiles_m * P.tiles_n;
    const unsigned grid = 2 * (unsigned)(P.tiles < pairs ? P.tiles : pairs);
    if (cosine) TPW_TOPK_LAUNCH(TPW_DOT_COSINE_DIST, 1); else TPW_TOPK_LAUNCH(TPW_DOT_SQEUCLIDEAN, 1);
    if (k <= 8) topk_merge_kernel<8><<<mblocks, 256, 0, s>>>(lists, counts, val_out, idx64, rows, T.L * k, k, take_sqrt);
    else topk_merge_kernel<16><<<mblocks, 256, 0, s>>>(lists, counts, val_out, idx64, rows, T.L * k, k, take_sqrt);
#undef TPW_TOPK_LAUNCH
    TPW_LAUNCH_OK("topk_merge_kernel");
    return TPW_OK;
}

extern "C" int64_t tpw_dot_rowmin_scratch_bytes(int64_t B, int64_t N1, int64_t N2, int64_t D) {
    if (B <= 0 || N1 <= 0 || N2 <= 0 || D <= 0) return 0;
    return scratch_layout(B, N1, N2, D, false).total + align_up(B * N1 * 8, 1024);
}

extern "C" int tpw_dot_rowmin_forward_ws(int epilogue, const void *x1, const void *x2, float *min_out, int64_t *arg_out,
                                         void *scratch, int64_t scratch_bytes,
                                         int64_t B, int64_t N1, int64_t N2, int64_t D, tpw_stream_t stream) {
    clear_error();
    TPW_CHECK_ARG(epilogue == TPW_DOT_SQEUCLIDEAN || epilogue == TPW_DOT_EUCLIDEAN || epilogue == TPW_DOT_COSINE_DIST,
                  "tpw_dot_rowmin_forward_ws: epilogue must be TPW_DOT_SQEUCLIDEAN, TPW_DOT_EUCLIDEAN or TPW_DOT_COSINE_DIST");
    const bool cosine = epilogue == TPW_DOT_COSINE_DIST;
    TPW_CHECK_ARG(B > 0 && N1 > 0 && N2 > 0 && D > 0, "tpw_dot_rowmin_forward_ws: sizes must be positive");
    TPW_CHECK_ARG(x1 && x2 && (min_out || arg_out), "tpw_dot_rowmin_forward_ws: NULL pointer");
    TPW_CHECK_ARG(N1 < (1ll << 31) && N2 < (1ll << 31) && B < (1ll << 31) && D < (1ll << 31),
                  "tpw_dot_rowmin_forward_ws: a dimension exceeds 2^31-1");
    const ScratchLayout L = scratch_layout(B, N1, N2, D, false);
    const long long need = L.total + align_up(B * N1 * 8, 1024);
    TPW_CHECK_ARG(scratch != nullptr && scratch_bytes >= need && aligned16(scratch),
                  "tpw_dot_rowmin_forward_ws: needs %lld bytes of 16-byte aligned scratch (got %lld)", need, (long long)scratch_bytes);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    unsigned long long *keys = reinterpret_cast<unsigned long long *>(static_cast<unsigned char *>(scratch) + L.total);
    TPW_CUDA_OK(cudaMemsetAsync(keys, 0xFF, (size_t)(B * N1) * 8, s));
    Bf16Operands M;
    GemmParams P;
    int st;
    if ((st = prepare_bf16_operands(x1, x2, scratch, cosine, B, N1, N2, D, s, M, P)) != TPW_OK) return st;
    P.epilogue = cosine ? TPW_DOT_COSINE_DIST : TPW_DOT_SQEUCLIDEAN;
    P.rowmin_keys = keys;
    const long long pairs = pair_count();
    const unsigned grid = 2 * (unsigned)(P.tiles < pairs ? P.tiles : pairs);
    if (cosine) {
        auto kern = gemm_metric_kernel<TPW_DOT_COSINE_DIST, false, false, true>;
        TPW_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_ALLOC));
        kern<<<grid, kThreads, SMEM_ALLOC, s>>>(M.mxh, M.mxl, M.myh, M.myl, P);
    } else {
        auto kern = gemm_metric_kernel<TPW_DOT_SQEUCLIDEAN, false, false, true>;
        TPW_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_ALLOC));
        kern<<<grid, kThreads, SMEM_ALLOC, s>>>(M.mxh, M.mxl, M.myh, M.myl, P);
    }
    TPW_LAUNCH_OK("gemm_metric_kernel (row minimum)");
    dot_rowmin_finish_kernel<<<(unsigned)((B * N1 + 255) / 256), 256, 0, s>>>(keys, min_out, reinterpret_cast<long long *>(arg_out), B * N1,
                                                                             epilogue == TPW_DOT_EUCLIDEAN ? 1 : 0);
    TPW_LAUNCH_OK("dot_rowmin_finish_kernel");
    return TPW_OK;
}

extern "C" int64_t tpw_dot_metric_scratch_bytes(int dtype, int engine, int64_t B, int64_t N1, int64_t N2, int64_t D) {
    if (B <= 0 || N1 <= 0 || N2 <= 0 || D <= 0 || dtype != TPW_F32) return 0;
    if (engine == TPW_ENGINE_TCGEN05_TF32X3) return tf32_forward_scratch(B, N1, N2, D);
    if (engine == TPW_ENGINE_TCGEN05_BF16X3 || (engine == TPW_ENGINE_AUTO && auto_picks_tensor_cores(dtype, B, N1, N2, D)))
        return scratch_layout(B, N1, N2, D, false).total;
    return 0;
}

extern "C" int tpw_dot_metric_forward_ws(int dtype, int epilogue, int engine,
                                         const void *x1, const void *x2, void *out, void *scratch, int64_t scratch_bytes,
                                         int64_t B, int64_t N1, int64_t N2, int64_t D, tpw_stream_t stream) {
    clear_error();
    TPW_CHECK_ARG(engine >= TPW_ENGINE_AUTO && engine <= TPW_ENGINE_TCGEN05_TF32X3, "tpw_dot_metric_forward_ws: bad engine %d", engine);
    if (engine == TPW_ENGINE_TCGEN05_TF32X3) {
        // x1 . x2^T with fp32-chain accuracy: tf32 high/low parts, chunked accumulation (see the gradient products)
        TPW_CHECK_ARG(dtype == TPW_F32 && epilogue == TPW_DOT_LINEAR,
                      "tpw_dot_metric_forward_ws: the tf32 engine computes float32 plain dot products (TPW_DOT_LINEAR) only");
        TPW_CHECK_ARG(B >= 0 && N1 >= 0 && N2 >= 0 && D >= 0, "tpw_dot_metric_forward_ws: negative size");
        if (B == 0 || N1 == 0 || N2 == 0) return TPW_OK;
        TPW_CHECK_ARG(x1 && x2 && out && D > 0, "tpw_dot_metric_forward_ws: NULL pointer or empty feature dimension");
        TPW_CHECK_ARG(N1 < (1ll << 31) && N2 < (1ll << 31) && D < (1ll << 31), "tpw_dot_metric_forward_ws: a dimension exceeds 2^31-1");
        const long long need = tf32_forward_scratch(B, N1, N2, D);
        TPW_CHECK_ARG(scratch != nullptr && scratch_bytes >= need && aligned16(scratch),
                      "tpw_dot_metric_forward_ws: the tf32 engine needs %lld bytes of 16-byte aligned scratch (got %lld)", need, (long long)scratch_bytes);
        cudaStream_t s = static_cast<cudaStream_t>(stream);
        const long long Dp = align_up(D, 4), xa = align_up(B * N1 * Dp * 4, 1024), ya = align_up(B * N2 * Dp * 4, 1024);
        unsigned char *base = static_cast<unsigned char *>(scratch);
        float *xhi = reinterpret_cast<float *>(base), *xlo = reinterpret_cast<float *>(base + xa);
        float *yhi = reinterpret_cast<float *>(base + 2 * xa), *ylo = reinterpret_cast<float *>(base + 2 * xa + ya);
        int st;
        for (int side = 0; side < 2; ++side) {
            SplitParams X;
            memset(&X, 0, sizeof(X));
            X.a = static_cast<const float *>(side == 0 ? x1 : x2);
            X.hi = side == 0 ? xhi : yhi;
            X.lo = side == 0 ? xlo : ylo;
            X.R = side == 0 ? N1 : N2; X.C = D; X.Cp = Dp;
            X.vec_in = (D % 4 == 0 && aligned16(X.a)) ? 1 : 0;
            if ((st = launch_split<COEF_ID, false>(X, B, s)) != TPW_OK) return st;
        }
        // Over pairs', plain products of [131072, 16384, D], [30011, 10007 or 10008, D] and [8000, 4000 or 4001, D]: 64 to 128 features 0.64 to
        // 0.98, 256 0.76 to 0.98, 384 0.83 to 1.01, 500 0.98 to 1.13 as the operands become the bound.
        const bool single = D <= 384;
        return launch_tf32_product(Tf32Operand{xhi, xlo, Dp, false}, Tf32Operand{yhi, ylo, Dp, false}, static_cast<float *>(out), nullptr, nullptr, single, B, N1, N2, Dp, s);
    }
    if (engine == TPW_ENGINE_AUTO && auto_picks_tensor_cores(dtype, B, N1, N2, D) && scratch != nullptr &&
        scratch_bytes >= scratch_layout(B, N1, N2, D, false).total)
        engine = TPW_ENGINE_TCGEN05_BF16X3;
    if (engine != TPW_ENGINE_TCGEN05_BF16X3 || dtype != TPW_F32) {
        TPW_CHECK_ARG(engine != TPW_ENGINE_TCGEN05_BF16X3 || dtype == TPW_F64,
                      "tpw_dot_metric_forward_ws: bad dtype %d", dtype);
        return tpw_dot_metric_forward_simt(dtype, epilogue, x1, x2, out, B, N1, N2, D, stream);
    }
    TPW_CHECK_ARG(epilogue >= TPW_DOT_LINEAR && epilogue <= TPW_DOT_EUCLIDEAN, "tpw_dot_metric_forward_ws: bad epilogue %d", epilogue);
    TPW_CHECK_ARG(B >= 0 && N1 >= 0 && N2 >= 0 && D >= 0, "tpw_dot_metric_forward_ws: negative size");
    if (B == 0 || N1 == 0 || N2 == 0) return TPW_OK;
    TPW_CHECK_ARG(x1 && x2 && out, "tpw_dot_metric_forward_ws: NULL pointer");
    TPW_CHECK_ARG(D > 0, "tpw_dot_metric_forward_ws: D must be positive");
    TPW_CHECK_ARG(N1 < (1ll << 31) && N2 < (1ll << 31) && B < (1ll << 31) && D < (1ll << 31),
                  "tpw_dot_metric_forward_ws: a dimension exceeds 2^31-1");
    const bool self = (x1 == x2) && (N1 == N2);
    const ScratchLayout L = scratch_layout(B, N1, N2, D, false);
    TPW_CHECK_ARG(scratch != nullptr && scratch_bytes >= L.total,
                  "tpw_dot_metric_forward_ws: the tensor-core engine needs %lld bytes of scratch (got %lld)",
                  L.total, (long long)scratch_bytes);
    TPW_CHECK_ARG(aligned16(scratch), "tpw_dot_metric_forward_ws: scratch must be 16-byte aligned");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const bool recip = epilogue == TPW_DOT_COSINE_SIM || epilogue == TPW_DOT_COSINE_DIST || epilogue == TPW_DOT_ONE_MINUS_SIM;
    Bf16Operands M;
    GemmParams P;
    int st;
    const bool single = single_pays(N2 % 4 == 0 && aligned16(out), 4.0 * B * N1 * N2, D);
    if ((st = prepare_bf16_operands(x1, x2, scratch, recip, B, N1, N2, D, s, M, P, !single)) != TPW_OK) return st;
    P.out = static_cast<float *>(out);
    P.epilogue = epilogue;
    P.self = self ? 1 : 0;
    P.vec_store = (N2 % 4 == 0 && aligned16(out)) ? 1 : 0;
    TPW_CHECK_ARG(P.tiles < (1ll << 40), "tpw_dot_metric_forward_ws: too many tiles");
    const long long ctas = single ? 1 : 2, most = sm_count() / ctas;
    const unsigned grid = (unsigned)(ctas * (P.tiles < most ? P.tiles : most));
#define TPW_GEMM_LAUNCH_FORM(EPI, SELF, PAIR)                                                                             \
    do {                                                                                                                  \
        auto kern = gemm_metric_kernel<EPI, SELF, false, false, false, 0, PAIR>;                                          \
        TPW_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Ring<PAIR>::SMEM_ALLOC));     \
        kern<<<grid, Ring<PAIR>::kThreads, Ring<PAIR>::SMEM_ALLOC, s>>>(M.mxh, M.mxl, M.myh, M.myl, P);                     \
    } while (0)
#define TPW_GEMM_LAUNCH(EPI, SELF)                                                                                        \
    do {                                                                                                                  \
        if (single) TPW_GEMM_LAUNCH_FORM(EPI, SELF, false); else TPW_GEMM_LAUNCH_FORM(EPI, SELF, true);                   \
    } while (0)
    switch (epilogue) {
        case TPW_DOT_LINEAR: TPW_GEMM_LAUNCH(TPW_DOT_LINEAR, false); break;
        case TPW_DOT_COSINE_SIM: TPW_GEMM_LAUNCH(TPW_DOT_COSINE_SIM, false); break;
        case TPW_DOT_COSINE_DIST: TPW_GEMM_LAUNCH(TPW_DOT_COSINE_DIST, false); break;
        case TPW_DOT_ONE_MINUS_SIM: TPW_GEMM_LAUNCH(TPW_DOT_ONE_MINUS_SIM, false); break;
        case TPW_DOT_SQEUCLIDEAN:
            if (self) TPW_GEMM_LAUNCH(TPW_DOT_SQEUCLIDEAN, true); else TPW_GEMM_LAUNCH(TPW_DOT_SQEUCLIDEAN, false);
            break;
        default:
            if (self) TPW_GEMM_LAUNCH(TPW_DOT_EUCLIDEAN, true); else TPW_GEMM_LAUNCH(TPW_DOT_EUCLIDEAN, false);
            break;
    }
#undef TPW_GEMM_LAUNCH
#undef TPW_GEMM_LAUNCH_FORM
    TPW_LAUNCH_OK("gemm_metric_kernel");
    return TPW_OK;
}

static bool backward_uses_tensor_cores(int dtype, int mode, int engine, int64_t B, int64_t N1, int64_t N2, int64_t D) {
    if (dtype != TPW_F32 || B <= 0 || N1 <= 0 || N2 <= 0 || D <= 0) return false;
    if (mode != TPW_LP_BWD_CDIST && mode != TPW_LP_BWD_PPMINKOWSKI && mode != TPW_LP_BWD_MATMUL) return false;
    if (engine == TPW_ENGINE_TCGEN05_BF16X3 || engine == TPW_ENGINE_TCGEN05_TF32X3) return true;
    return engine == TPW_ENGINE_AUTO && auto_picks_tensor_backward(dtype, B, N1, N2, D);
}

extern "C" int64_t tpw_dot_backward_scratch_bytes(int dtype, int mode, int engine, int64_t B, int64_t N1, int64_t N2, int64_t D) {
    if (!backward_uses_tensor_cores(dtype, mode, engine, B, N1, N2, D)) return 0;
    return bwd_scratch_layout(B, N1, N2, D).with_part;
}

extern "C" int tpw_cosine_backward_finish(int dtype, void *grad_x, const void *x, const void *norm, const void *term,
                                          int64_t rows, int64_t D, tpw_stream_t stream);

// Shared body of the two entry points below.  coef: COEF_ID / COEF_DIV_AUX / COEF_COSINE.
static int dense_backward_tensor(int coef, int epilogue, bool sums, float s_mm, float s_row,
                                 const void *grad, const void *aux, const void *norm1, const void *norm2,
                                 const void *x1, const void *x2, void *grad_x1, void *grad_x2, void *scratch, int64_t scratch_bytes,
                                 int64_t B, int64_t N1, int64_t N2, int64_t D, cudaStream_t s) {
    const BwdScratch L = bwd_scratch_layout(B, N1, N2, D);
    unsigned char *base = static_cast<unsigned char *>(scratch);
    auto F = [&](long long off) { return reinterpret_cast<float *>(base + off); };
    float *partial = L.with_part > L.total && scratch_bytes >= L.with_part ? F(L.off_part) : nullptr;
    int st;

    // coefficient matrix C [N1,N2] as tf32 high/low parts, written once: grad_x1 = C . X2 reads it K-major
    // (reduction along its rows), grad_x2 = C^T . X1 reads the same copy MN-major (reduction over its row index)
    SplitParams C;
    memset(&C, 0, sizeof(C));
    C.a = static_cast<const float *>(grad);
    C.aux = static_cast<const float *>(aux);
    C.n1 = static_cast<const float *>(norm1);
    C.n2 = static_cast<const float *>(norm2);
    C.epilogue = epilogue;
    int *lo_any = reinterpret_cast<int *>(base + L.off_lo);   // [side][coefficients (not used), x]
    C.hi = F(L.off_chi); C.lo = F(L.off_clo);
    C.clear = lo_any;
    C.rowpart = F(L.off_rowpart); C.colpart = F(L.off_colpart);
    C.R = N1; C.C = N2; C.Cp = L.N2p; C.TR = L.TR; C.TC = L.TC;
    C.vec_in = (N2 % 4 == 0 && aligned16(grad) && (coef == COEF_ID || aligned16(aux))) ? 1 : 0;
    if (coef == COEF_COSINE) st = launch_split<COEF_COSINE, true>(C, B, s);
    else if (coef == COEF_DIV_AUX) st = launch_split<COEF_DIV_AUX, true>(C, B, s);
    else if (sums) st = launch_split<COEF_ID, true>(C, B, s);
    else st = launch_split<COEF_ID, false>(C, B, s);
    if (st != TPW_OK) return st;
    if (sums) {
        const long long most = B * (N1 > N2 ? N1 : N2);
        reduce_partials_kernel<<<dim3((unsigned)((most + 255) / 256), 2), 256, 0, s>>>(
            Partials{F(L.off_rowpart), F(L.off_rowsum), L.TC, N1}, Partials{F(L.off_colpart), F(L.off_colsum), L.TR, N2}, B);
        TPW_LAUNCH_OK("reduce_partials_kernel");
    }
    const Tf32Operand Ck{F(L.off_chi), F(L.off_clo), L.N2p, false}, Cmn{F(L.off_chi), F(L.off_clo), L.N2p, true};
    // side 0: grad_x1[N1,D] = C . X2; side 1: grad_x2[N2,D] = C^T . X1.  xk: operand contracted against (its transpose is the K-major
    // one); xo: rows that receive the gradient
    Transposed T[2];
    Finish fin[2];
    int sides = 0;
    bool vec = D % 4 == 0;
    long long most = 0;
    for (int side = 0; side < 2; ++side) {
        void *gout = side == 0 ? grad_x1 : grad_x2;
        if (!gout) continue;
        const void *xk = side == 0 ? x2 : x1, *xo = side == 0 ? x1 : x2;
        T[sides] = Transposed{static_cast<const float *>(xk), F(side == 0 ? L.off_x2hi : L.off_x1hi), F(side == 0 ? L.off_x2lo : L.off_x1lo),
                              lo_any + 2 * side + 1, side == 0 ? N2 : N1, side == 0 ? L.N2p : L.N1p, D % 4 == 0 && aligned16(xk) ? 1 : 0};
        fin[sides] = Finish{static_cast<float *>(gout), static_cast<const float *>(xo), F(side == 0 ? L.off_rowsum : L.off_colsum), B * (side == 0 ? N1 : N2)};
        vec = vec && aligned16(gout) && aligned16(xo);
        if (T[sides].Rp > most) most = T[sides].Rp;
        ++sides;
    }
    const long long gx = (D + PT - 1) / PT, gy = (most + PT - 1) / PT;
    TPW_CHECK_ARG(gy <= 65535 && B <= 65535, "dense backward: more than 65535 row tiles or batches");
    if (B * sides <= 65535) {
        split_transposed_kernel<<<dim3((unsigned)gx, (unsigned)gy, (unsigned)(B * sides)), 256, 0, s>>>(T[0], T[sides - 1], D, sides);
    } else {
        for (int at = 0; at < sides; ++at)
            split_transposed_kernel<<<dim3((unsigned)gx, (unsigned)gy, (unsigned)B), 256, 0, s>>>(T[at], T[at], D, 1);
    }
    TPW_LAUNCH_OK("split_transposed_kernel");
    for (int side = 0, at = 0; side < 2; ++side) {
        void *gout = side == 0 ? grad_x1 : grad_x2;
        if (!gout) continue;
        const Tf32Operand Xk{T[at].hi, T[at].lo, T[at].Rp, false};
        if (side == 0) st = launch_tf32_product(Ck, Xk, static_cast<float *>(gout), lo_any, partial, false, B, N1, D, N2, s);
        else st = launch_tf32_product(Cmn, Xk, static_cast<float *>(gout), lo_any + 2, partial, false, B, N2, D, N1, s);
        if (st != TPW_OK) return st;
        if (coef == COEF_COSINE) {
            // the norm part of the chain: g[r,:] += term[r] * x[r,:] / norm[r]
            if ((st = tpw_cosine_backward_finish(TPW_F32, gout, fin[at].x, side == 0 ? norm1 : norm2, fin[at].sums, fin[at].rows, D, s)) != TPW_OK) return st;
        }
        ++at;
    }
    if (sums && coef != COEF_COSINE) {
        const long long rows = fin[0].rows > fin[sides - 1].rows ? fin[0].rows : fin[sides - 1].rows, cap = (long long)sm_count() * 8;
        const long long blocks = (rows * (vec ? D / 4 : D) + 255) / 256;
        const dim3 grid((unsigned)(blocks < cap ? blocks : cap), (unsigned)sides);
        if (vec) grad_finish_kernel<4><<<grid, 256, 0, s>>>(fin[0], fin[sides - 1], D, s_mm, s_row);
        else grad_finish_kernel<1><<<grid, 256, 0, s>>>(fin[0], fin[sides - 1], D, s_mm, s_row);
        TPW_LAUNCH_OK("grad_finish_kernel");
    }
    return TPW_OK;
}

extern "C" int tpw_dot_backward_ws(int dtype, int mode, int engine, const void *grad, const void *aux,
                                   const void *x1, const void *x2, void *grad_x1, void *grad_x2,
                                   void *scratch, int64_t scratch_bytes,
                                   int64_t B, int64_t N1, int64_t N2, int64_t D, tpw_stream_t stream) {
    clear_error();
    TPW_CHECK_ARG(engine >= TPW_ENGINE_AUTO && engine <= TPW_ENGINE_TCGEN05_TF32X3, "tpw_dot_backward_ws: bad engine %d", engine);
    TPW_CHECK_ARG(mode == TPW_LP_BWD_CDIST || mode == TPW_LP_BWD_PPMINKOWSKI || mode == TPW_LP_BWD_MATMUL,
                  "tpw_dot_backward_ws: mode %d has no contraction form (p = 2 modes and the plain products only)", mode);
    TPW_CHECK_ARG(B >= 0 && N1 >= 0 && N2 >= 0 && D >= 0, "tpw_dot_backward_ws: negative size");
    bool tensor = backward_uses_tensor_cores(dtype, mode, engine, B, N1, N2, D);
    if (tensor && engine == TPW_ENGINE_AUTO && (scratch == nullptr || scratch_bytes < bwd_scratch_layout(B, N1, N2, D).total))
        tensor = false;
    if (!tensor) {
        TPW_CHECK_ARG(engine == TPW_ENGINE_AUTO || engine == TPW_ENGINE_SIMT_FP32 || dtype == TPW_F64,
                      "tpw_dot_backward_ws: the tensor-core engine takes float32 only");
        return tpw_lp_backward(dtype, mode, grad, aux, x1, x2, nullptr, grad_x1, grad_x2, B, N1, N2, D, 2.0, stream);
    }
    TPW_CHECK_ARG(grad && x1 && x2 && (grad_x1 || grad_x2), "tpw_dot_backward_ws: NULL pointer");
    TPW_CHECK_ARG(mode != TPW_LP_BWD_CDIST || aux != nullptr, "tpw_dot_backward_ws: the Euclidean mode needs the forward output");
    TPW_CHECK_ARG(N1 < (1ll << 31) && N2 < (1ll << 31) && D < (1ll << 31), "tpw_dot_backward_ws: a dimension exceeds 2^31-1");
    const long long need = bwd_scratch_layout(B, N1, N2, D).total;
    TPW_CHECK_ARG(scratch != nullptr && scratch_bytes >= need,
                  "tpw_dot_backward_ws: the tensor-core engine needs %lld bytes of scratch (got %lld)", need, (long long)scratch_bytes);
    TPW_CHECK_ARG(aligned16(scratch), "tpw_dot_backward_ws: scratch must be 16-byte aligned");
    const float s_mm = mode == TPW_LP_BWD_MATMUL ? 1.f : (mode == TPW_LP_BWD_PPMINKOWSKI ? -2.f : -1.f);
    const float s_row = mode == TPW_LP_BWD_PPMINKOWSKI ? 2.f : 1.f;
    return dense_backward_tensor(mode == TPW_LP_BWD_CDIST ? COEF_DIV_AUX : COEF_ID, 0, mode != TPW_LP_BWD_MATMUL, s_mm, s_row,
                                 grad, aux, nullptr, nullptr, x1, x2, grad_x1, grad_x2, scratch, scratch_bytes, B, N1, N2, D,
                                 static_cast<cudaStream_t>(stream));
}

extern "C" int tpw_cosine_backward_ws(int epilogue, const void *grad, const void *out, const void *norm1, const void *norm2,
                                      const void *x1, const void *x2, void *grad_x1, void *grad_x2,
                                      void *scratch, int64_t scratch_bytes,
                                      int64_t B, int64_t N1, int64_t N2, int64_t D, tpw_stream_t stream) {
    clear_error();
    TPW_CHECK_ARG(epilogue == TPW_DOT_COSINE_SIM || epilogue == TPW_DOT_COSINE_DIST || epilogue == TPW_DOT_ONE_MINUS_SIM,
                  "tpw_cosine_backward_ws: bad epilogue %d", epilogue);
    TPW_CHECK_ARG(B > 0 && N1 > 0 && N2 > 0 && D > 0, "tpw_cosine_backward_ws: sizes must be positive");
    TPW_CHECK_ARG(grad && out && norm1 && norm2 && x1 && x2 && (grad_x1 || grad_x2), "tpw_cosine_backward_ws: NULL pointer");
    TPW_CHECK_ARG(N1 < (1ll << 31) && N2 < (1ll << 31) && D < (1ll << 31), "tpw_cosine_backward_ws: a dimension exceeds 2^31-1");
    const long long need = bwd_scratch_layout(B, N1, N2, D).total;
    TPW_CHECK_ARG(scratch != nullptr && scratch_bytes >= need,
                  "tpw_cosine_backward_ws: needs %lld bytes of scratch (got %lld)", need, (long long)scratch_bytes);
    TPW_CHECK_ARG(aligned16(scratch), "tpw_cosine_backward_ws: scratch must be 16-byte aligned");
    return dense_backward_tensor(COEF_COSINE, epilogue, true, 1.f, 0.f, grad, out, norm1, norm2, x1, x2, grad_x1, grad_x2, scratch, scratch_bytes,
                                 B, N1, N2, D, static_cast<cudaStream_t>(stream));
}
