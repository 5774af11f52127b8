// Directed Hausdorff distance between point sets, fused so that the [M1, M2] distance matrix is
// never written.
//
// Fast path (float32, D <= 16): a thread keeps a few points of x1 in registers and streams the x2 cloud
// through shared memory, every load a broadcast to the whole warp.  Only the running row minimum is kept in
// the hot loop.  Row minima are ordered by (float bits << 32 | visiting position of m): the float bits of a
// non-negative value order like the value, and the low word makes the LAST visited m win ties, which is the
// rule of the reference loop.  A finishing kernel then recomputes the winning row to find the FIRST visited n
// reaching its minimum, and writes sqrt(max), m*, n*.
//
// Squared distances are accumulated coordinate by coordinate with separately rounded multiply and
// add (no FMA contraction), i.e. bit-for-bit what the reference's CPU loop computes, so the
// selected indices agree with it whenever they are determined at all.
//
// With caller-provided scratch the hot loop (hausdorff_rowmin_fused_kernel) does not pay for that: it stores
// every row's approximate minimum, and the refining kernel then re-evaluates, with the exact arithmetic, only
// the rows whose approximate minimum lies within the approximation's error of the largest one (usually one
// to three per set pair) and applies the tie rules to them, so values and indices are still bit-identical to
// the exact path.  Two approximations:
//   expanded   |y|^2 - 2 x.y + |x|^2 about a point of the x2 cloud: D fused multiply-adds per point pair.  Its error is
//              bounded by the clouds' extent, not by the distance, so where more rows than the refining kernel should
//              look at lie that close together (well registered clouds, voxel shells), those rows are handed over to the
//              other one, and where a sample of rows says that most do (equal clouds, a far outlier, coordinates that are
//              not finite) the set pair skips this one;
//   direct     sum of squared differences with fused multiply-adds, 2 D per point pair, within a few units in the last
//              place of the separately rounded value.
//
// Any other dtype / feature count runs a plain one-CTA-per-set-pair kernel with the same rules.
#include "common.cuh"
#include "packed_f32x2.cuh"

#include <math.h>
#include <stdlib.h>

#include <atomic>

namespace tpw {
namespace {

constexpr int kThreads = 256;
constexpr int PM = 4;            // x1 points per thread
constexpr int CHUNK_VECS = 2048; // float4 slots staged per pass (32 KB): 2048 x2 points of up to 4 features, 1024 of up to 8

__device__ __forceinline__ float sqdist_exact(const float *a, const float *b, int D) {
    float d = 0.f;
    for (int k = 0; k < D; ++k) {
        const float diff = __fsub_rn(a[k], b[k]);
        d = __fadd_rn(d, __fmul_rn(diff, diff));
    }
    return d;
}
__device__ __forceinline__ double sqdist_exact(const double *a, const double *b, int D) {
    double d = 0.0;
    for (int k = 0; k < D; ++k) {
        const double diff = __dsub_rn(a[k], b[k]);
        d = __dadd_rn(d, __dmul_rn(diff, diff));
    }
    return d;
}

struct HdParams {
    const void *x1, *x2;
    const long long *order1, *order2;
    void *out;
    long long *idx1, *idx2;
    unsigned long long *keys;
    float *rowmins;   // [pairs, M1] approximate row minima (fused path only)
    long long B, N1, N2, M1, M2, D;
    long long mtiles;
    int splits;       // CTAs that share the x2 points of one row block (fused path)
    int handed_over;  // direct form: only the set pairs, and of those the rows, that the expanded form has handed over
    unsigned int *list;   // [pairs, M1] those rows; before, per sampling CTA of the pair, what it found (kSampleWords)
    int samples;      // sampling CTAs per set pair (0: none)
};

// An upper bound on the relative difference between the fused and the separately rounded sum of up to 8 squares
// (each is within D roundings of the real sum, all terms non-negative), with room to spare; below kTiny the
// relative bound gives way to an absolute one (products that underflow).
constexpr float kFusedSlack = 3.8146973e-6f;   // 2^-18
constexpr float kTiny = 1e-35f;
// 9 to 16 squares: (3 D - 1) roundings of 2^-24 between the two sums stay below 2^-17
template <int D> __device__ __forceinline__ constexpr float fused_slack() { return D <= 8 ? kFusedSlack : 2.f * kFusedSlack; }
constexpr int kMaxFastD = 16;                  // widest point the streamed kernels are instantiated for

// keys[pair] = max over m of (bits(rowmin) << 32 | position(m)), every product and sum rounded separately: the
// loop of the entry that has no room for the row minima.
template <int D>
__global__ void __launch_bounds__(kThreads)
hausdorff_rowmin_kernel(const HdParams P) {
    constexpr int V = (D + 3) / 4;           // float4 slots per x2 point
    constexpr int CHUNK = CHUNK_VECS / V;
    __shared__ float4 pts[CHUNK_VECS];
    const int tid = threadIdx.x;
    long long blk = blockIdx.x;
    const long long mt = blk % P.mtiles;
    blk /= P.mtiles;
    const long long pair = blk; // (b*N1 + i)*N2 + j
    const long long j = pair % P.N2;
    const long long bi = pair / P.N2;
    const long long b = bi / P.N1;
    const float *x1 = reinterpret_cast<const float *>(P.x1) + bi * P.M1 * D;
    const float *x2 = reinterpret_cast<const float *>(P.x2) + (b * P.N2 + j) * P.M2 * D;

    float px[PM][D];
    float rowmin[PM];
    long long mm[PM];
#pragma unroll
    for (int q = 0; q < PM; ++q) {
        mm[q] = mt * (kThreads * PM) + q * kThreads + tid;
        rowmin[q] = INFINITY;
#pragma unroll
        for (int k = 0; k < D; ++k) px[q][k] = mm[q] < P.M1 ? x1[mm[q] * D + k] : 0.f;
    }

    for (long long n0 = 0; n0 < P.M2; n0 += CHUNK) {
        const int cnt = (int)((P.M2 - n0) < CHUNK ? (P.M2 - n0) : CHUNK);
        __syncthreads();
        for (int e = tid; e < cnt; e += kThreads) {
            const float *s = x2 + (n0 + e) * D;
            float c[4 * V];
#pragma unroll
            for (int k = 0; k < 4 * V; ++k) c[k] = k < D ? s[k] : 0.f;
#pragma unroll
            for (int v = 0; v < V; ++v) pts[e * V + v] = make_float4(c[4 * v], c[4 * v + 1], c[4 * v + 2], c[4 * v + 3]);
        }
        __syncthreads();
#pragma unroll 4
        for (int e = 0; e < cnt; ++e) {
            float c[4 * V];
#pragma unroll
            for (int v = 0; v < V; ++v) {
                const float4 t = pts[e * V + v];
                c[4 * v] = t.x; c[4 * v + 1] = t.y; c[4 * v + 2] = t.z; c[4 * v + 3] = t.w;
            }
#pragma unroll
            for (int q = 0; q < PM; ++q) {
                float d = 0.f;
#pragma unroll
                for (int k = 0; k < D; ++k) {
                    const float diff = __fsub_rn(px[q][k], c[k]);
                    d = __fadd_rn(d, __fmul_rn(diff, diff));
                }
                rowmin[q] = fminf(rowmin[q], d);
            }
        }
    }

    unsigned long long key = 0ull;
#pragma unroll
    for (int q = 0; q < PM; ++q) {
        if (mm[q] < P.M1) {
            const unsigned long long pos =
                (unsigned long long)(P.order1 ? P.order1[b * P.M1 + mm[q]] : mm[q]);
            const unsigned long long kq = ((unsigned long long)__float_as_uint(rowmin[q]) << 32) | (pos & 0xffffffffull);
            key = kq > key ? kq : key;
        }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        const unsigned long long other = __shfl_xor_sync(0xffffffffu, key, off);
        key = other > key ? other : key;
    }
    if ((tid & 31) == 0) atomicMax(P.keys + pair, key);
}

// The fused loop.  Bound: FP32 issue.  Two x2 points lie side by side in shared memory, coordinate by coordinate, so that
// one packed instruction serves two point pairs, and one three-operand minimum folds both distances in: at D = 3 a
// point pair costs 3 lane-operations of the FMA pipe (direct: 6) in 1.5 (3) instructions and half a minimum, where it
// took 7 instructions.  A lone last point is paired with a point of NaNs, whose distance no minimum takes.
// CTAs of 128 threads (512 rows) leave a smaller last wave than 256 threads would; where a small batch has fewer row
// blocks than fill the GPU, `splits` CTAs share the x2 points of a row block and merge by an integer minimum
// (order-independent: the result does not depend on the split).
// Measured at 64 pairs of 8192-point clouds, D = 3: 1.17 ms scalar, 0.92 ms direct, 0.56 ms expanded.
constexpr int kFThreads = 128;
constexpr int FCHUNK_BYTES = 16384;
template <int D> struct Fused {
    static constexpr int PM = D <= 8 ? 4 : 2;            // x1 points per thread, both lanes of a packed register
    static constexpr int ROWS = kFThreads * PM;
};

// What the kernels agree on per set pair, in the eight bytes the exact path uses for its key: the largest squared norm
// about the centre (infinite: not bounded) and how many of its rows are handed over to the direct form (kAllRows: no list).
struct PairState {
    unsigned int extent, direct;
};
constexpr unsigned int kAllRows = 0xffffffffu;
constexpr float kExtentMax = 1e36f;   // beyond it the products could overflow
constexpr unsigned int kMaxCandidates = 32;    // rows that one CTA evaluates one after another, 4 us each at 8192 points
constexpr unsigned int kMaxExpanded = 8;       // more rows within the expanded form's error of the largest are handed over

// EXPAND: with R^2 the largest squared norm about the centre, the centred coordinates' roundings change a squared distance by at
// most 8 u R^2 (u = 2^-24), the two norms' by 2 D u R^2, the D multiply-adds' by 3 D u R^2 and the last addition's by 4 u R^2:
// E = (5 D + 12) u R^2.  A row of the largest distance lies within 2 E of the largest minimum; 16 D + 64 leaves room.
template <int D> __device__ __forceinline__ float expanded_slack(float extent) { return 2.f * (float)(8 * (D + 1) + 24) * 5.9604645e-8f * extent; }

// Whether the expanded form is worth trying on a set pair: the direct minima of 16 rows over all x2 points.  Where most of them lie
// within 0.4 of the expanded form's error of the largest, most of all rows will lie within the error of the largest of all
// (which is about 2.5 times as far from the low ones as the largest of 16 is, for noise), and the expanded pass would be thrown
// away.  The answer decides the time alone, not the result.  `samples` CTAs share the x2 points of a set pair, each half of a CTA
// with eight rows in registers; every CTA of the expanded pass combines what they found.
// Microseconds at 64 pairs of 8192 points in the unit cube, x2 = x1 plus noise, before any expanded form / with it and whole pairs
// handed over / with the sample and the listed rows: sigma 0.05 1222 / 569 / 602, 0.003 1222 / 1056 / 666, 0.002 1222 / 1537 / 972,
// equal clouds 1214 / 1476 / 938, two voxel shells 1289 / 622 / 909.
constexpr int kSampleRows = 16, kSampleWords = kSampleRows + 1;   // minima, and the largest squared norm about the centre
template <int D>
__global__ void __launch_bounds__(kThreads)
hausdorff_sample_kernel(const HdParams P) {
    constexpr int kRows = kSampleRows / 2, kHalf = kThreads / 2;
    __shared__ unsigned int s_found[kSampleWords];
    const int tid = threadIdx.x, half = tid / kHalf;
    const int part = (int)(blockIdx.x % P.samples);
    const long long pair = blockIdx.x / P.samples;
    const long long j = pair % P.N2;
    const long long bi = pair / P.N2;
    const long long b = bi / P.N1;
    const float *x1 = reinterpret_cast<const float *>(P.x1) + bi * P.M1 * D;
    const float *x2 = reinterpret_cast<const float *>(P.x2) + (b * P.N2 + j) * P.M2 * D;
    if (tid < kSampleWords) s_found[tid] = tid < kSampleRows ? 0x7f800000u : 0u;
    __syncthreads();
    float x[kRows][D], least[kRows], centre[D], extent = 0.f;
    bool unbounded = false;
    auto grow = [&](const float *v) {
        float n = 0.f;
#pragma unroll
        for (int k = 0; k < D; ++k) n = fmaf(v[k] - centre[k], v[k] - centre[k], n);
        extent = fmaxf(extent, n);
        unbounded |= !(n < kExtentMax);
    };
#pragma unroll
    for (int k = 0; k < D; ++k) centre[k] = x2[k];
#pragma unroll
    for (int r = 0; r < kRows; ++r) {
        const long long m = ((half * kRows + r) * 2 + 1) * P.M1 / (2 * kSampleRows);     // the middles of 16 equal ranges
        least[r] = INFINITY;
#pragma unroll
        for (int k = 0; k < D; ++k) x[r][k] = x1[m * D + k];
        grow(x[r]);
    }
    const long long per = (P.M2 + P.samples - 1) / P.samples, end = (part + 1) * per < P.M2 ? (part + 1) * per : P.M2;
#pragma unroll 4
    for (long long n = part * per + tid % kHalf; n < end; n += kHalf) {
        float y[D];
#pragma unroll
        for (int k = 0; k < D; ++k) y[k] = x2[n * D + k];
        grow(y);
#pragma unroll
        for (int r = 0; r < kRows; ++r) {
            float d = 0.f;
#pragma unroll
            for (int k = 0; k < D; ++k) d = fmaf(x[r][k] - y[k], x[r][k] - y[k], d);
            least[r] = fminf(least[r], d);
        }
    }
    // not negative: bits order like values
    const unsigned int bits = __reduce_max_sync(0xffffffffu, unbounded ? 0x7f800000u : __float_as_uint(extent));
    if ((tid & 31) == 0) atomicMax(&s_found[kSampleRows], bits);
#pragma unroll
    for (int r = 0; r < kRows; ++r) {
        const unsigned int m = __reduce_min_sync(0xffffffffu, __float_as_uint(least[r]));
        if ((tid & 31) == 0) atomicMin(&s_found[half * kRows + r], m);
    }
    __syncthreads();
    if (tid < kSampleWords) P.list[pair * P.M1 + part * kSampleWords + tid] = s_found[tid];
    if (part == 0 && tid == 0) reinterpret_cast<PairState *>(P.keys)[pair] = PairState{0, 0};
}

// One warp: whether the sample says that the set pair should go to the direct form at once (the same in all lanes).
template <int D>
__device__ __forceinline__ bool sample_says_direct(const HdParams &P, long long pair) {
    const int lane = threadIdx.x & 31;
    const unsigned int *found = P.list + pair * P.M1;
    unsigned int v = lane < kSampleRows ? 0x7f800000u : 0u;
    for (int s = 0; s < P.samples && lane < kSampleWords; ++s) {
        const unsigned int w = found[s * kSampleWords + lane];
        v = lane < kSampleRows ? min(v, w) : max(v, w);
    }
    __syncwarp();
    const float extent = __uint_as_float(__shfl_sync(0xffffffffu, v, kSampleRows));
    const float most = __uint_as_float(__reduce_max_sync(0xffffffffu, lane < kSampleRows ? v : 0u));
    const float lower = most * (1.f - fused_slack<D>()) - kTiny - 0.4f * expanded_slack<D>(extent);
    const int close = __popc(__ballot_sync(0xffffffffu, lane < kSampleRows && __uint_as_float(v) >= lower));
    return !(extent < kExtentMax) || close >= 10;
}

template <int D, bool EXPAND>
__global__ void __launch_bounds__(kFThreads)
hausdorff_rowmin_fused_kernel(const HdParams P) {
    typedef Fused<D> F;
    // packed words per pair of x2 points, an even number for 16-byte loads: the coordinates (EXPAND: times -2, and the squared norm)
    constexpr int W = EXPAND ? D + 1 : D, DP = (W + 1) / 2 * 2;
    constexpr int CHUNK = FCHUNK_BYTES / (DP * 8);   // pairs of x2 points staged per pass
    __shared__ ulonglong2 pts[FCHUNK_BYTES / 16];
    const int tid = threadIdx.x;
    const long long each = P.mtiles * P.splits, pair = blockIdx.x / each; // (b*N1 + i)*N2 + j
    const int part = (int)(blockIdx.x % each);
    PairState *state = reinterpret_cast<PairState *>(P.keys) + pair;
    long long mt = part / P.splits, rows = P.M1;
    int sp = part % P.splits, splits = P.splits;
    const unsigned int *list = nullptr;
    if (EXPAND) {
        __shared__ bool s_direct;
        if (P.samples > 0) {
            if (tid < 32) {
                const bool direct = sample_says_direct<D>(P, pair);
                if (tid == 0) {
                    s_direct = direct;
                    if (direct && part == 0) state->direct = kAllRows;
                }
            }
            __syncthreads();
            if (s_direct) return;
        }
    } else if (P.handed_over) {
        const unsigned int n = state->direct;
        if (n == 0) return;
        if (n != kAllRows) {
            // the pair's CTAs share the x2 points of the listed rows
            list = P.list + pair * P.M1;
            rows = n;
            const long long tiles = (rows + F::ROWS - 1) / F::ROWS;
            splits = (int)(each / tiles);
            mt = part / splits;
            sp = part % splits;
            if (mt >= tiles) return;
        }
    }
    const long long j = pair % P.N2;
    const long long bi = pair / P.N2;
    const long long b = bi / P.N1;
    const float *x1 = reinterpret_cast<const float *>(P.x1) + bi * P.M1 * D;
    const float *x2 = reinterpret_cast<const float *>(P.x2) + (b * P.N2 + j) * P.M2 * D;
    float centre[D];
#pragma unroll
    for (int k = 0; k < D; ++k) centre[k] = EXPAND ? x2[k] : 0.f;
    float extent = 0.f;          // largest squared norm this thread has seen
    bool unbounded = false;
    // this CTA's range of x2 points, cut at even positions
    const long long per = ((P.M2 + 1) / 2 + splits - 1) / splits * 2;
    const long long n_end = (sp + 1) * per < P.M2 ? (sp + 1) * per : P.M2;

    f32x2 px[F::PM][D];
    float rowmin[F::PM], xsq[F::PM];
#pragma unroll
    for (int q = 0; q < F::PM; ++q) {
        const long long c = mt * F::ROWS + q * kFThreads + tid, m = !EXPAND && list && c < rows ? list[c] : c;
        rowmin[q] = INFINITY;
        xsq[q] = 0.f;
#pragma unroll
        for (int k = 0; k < D; ++k) {
            const float v = c < rows ? x1[m * D + k] - centre[k] : 0.f;
            px[q][k] = pack2(v, v);
            xsq[q] = fmaf(v, v, xsq[q]);
        }
        extent = fmaxf(extent, xsq[q]);
        unbounded |= !(xsq[q] < kExtentMax);
    }

    for (long long n0 = sp * per; n0 < n_end; n0 += 2 * CHUNK) {
        const int cnt = (int)((n_end - n0 + 1) / 2 < CHUNK ? (n_end - n0 + 1) / 2 : CHUNK);
        __syncthreads();
        for (int e = tid; e < cnt; e += kFThreads) {
            const float *s = x2 + (n0 + 2 * e) * D;
            const bool two = n0 + 2 * e + 1 < n_end;
            f32x2 *dst = reinterpret_cast<f32x2 *>(pts) + e * DP;
            if (EXPAND) {
                float lo = 0.f, hi = 0.f;
#pragma unroll
                for (int k = 0; k < D; ++k) {
                    const float u = s[k] - centre[k], v = two ? s[D + k] - centre[k] : 0.f;
                    lo = fmaf(u, u, lo);
                    hi = fmaf(v, v, hi);
                    dst[k] = pack2(-2.f * u, -2.f * v);
                }
                extent = fmaxf(extent, fmaxf(lo, hi));
                unbounded |= !(lo < kExtentMax) || !(hi < kExtentMax);
                dst[D] = pack2(lo, two ? hi : NAN);
            } else {
#pragma unroll
                for (int k = 0; k < D; ++k) dst[k] = pack2(s[k], two ? s[D + k] : NAN);
            }
        }
        __syncthreads();
#pragma unroll 4
        for (int e = 0; e < cnt; ++e) {
            f32x2 c[DP];
#pragma unroll
            for (int v = 0; v < DP / 2; ++v) {
                const ulonglong2 t = pts[e * (DP / 2) + v];
                c[2 * v] = t.x; c[2 * v + 1] = t.y;
            }
#pragma unroll
            for (int q = 0; q < F::PM; ++q) {
                f32x2 d;
                if (EXPAND) {
                    d = fma2(px[q][0], c[0], c[D]);
#pragma unroll
                    for (int k = 1; k < D; ++k) d = fma2(px[q][k], c[k], d);
                } else {
                    f32x2 diff = sub2(px[q][0], c[0]);
                    d = mul2(diff, diff);
#pragma unroll
                    for (int k = 1; k < D; ++k) {
                        diff = sub2(px[q][k], c[k]);
                        d = fma2(diff, diff, d);
                    }
                }
                float lo, hi;
                unpack2(d, lo, hi);
                rowmin[q] = min3(rowmin[q], lo, hi);
            }
        }
    }
    if (EXPAND) {
        const unsigned int bits = __reduce_max_sync(0xffffffffu, unbounded ? 0x7f800000u : __float_as_uint(extent));
        if ((tid & 31) == 0) atomicMax(&state->extent, bits);
    }
#pragma unroll
    for (int q = 0; q < F::PM; ++q) {
        const long long c = mt * F::ROWS + q * kFThreads + tid;
        if (c >= rows) continue;
        const float v = EXPAND ? fmaxf(rowmin[q] + xsq[q], 0.f) : rowmin[q];
        float *dst = P.rowmins + pair * P.M1 + c;     // a listed row's minimum lies where its number in the list says
        if (splits == 1) *dst = v;
        else atomicMin(reinterpret_cast<unsigned int *>(dst), __float_as_uint(v));   // non-negative: bits order like values
    }
}

// One CTA per set pair: decode the winning m, recompute its row, pick the first visited n.
template <int D>
__global__ void __launch_bounds__(kThreads)
hausdorff_finish_kernel(const HdParams P) {
    __shared__ unsigned long long best;
    __shared__ long long mstar_s;
    const int tid = threadIdx.x;
    const long long pair = blockIdx.x;
    const long long j = pair % P.N2;
    const long long bi = pair / P.N2;
    const long long b = bi / P.N1;
    const float *x1 = reinterpret_cast<const float *>(P.x1) + bi * P.M1 * D;
    const float *x2 = reinterpret_cast<const float *>(P.x2) + (b * P.N2 + j) * P.M2 * D;
    const unsigned long long key = P.keys[pair];
    const unsigned int pos = (unsigned int)(key & 0xffffffffull);
    if (tid == 0) {
        best = ~0ull;
        mstar_s = P.order1 ? -1 : (long long)pos;
    }
    __syncthreads();
    if (P.order1) {
        for (long long m = tid; m < P.M1; m += kThreads)
            if ((unsigned int)P.order1[b * P.M1 + m] == pos) mstar_s = m;
        __syncthreads();
    }
    const long long mstar = mstar_s;
    float a[D];
#pragma unroll
    for (int k = 0; k < D; ++k) a[k] = (mstar >= 0 && mstar < P.M1) ? x1[mstar * D + k] : 0.f;
    unsigned long long mine = ~0ull;
    for (long long n = tid; n < P.M2; n += kThreads) {
        float c[D];
#pragma unroll
        for (int k = 0; k < D; ++k) c[k] = x2[n * D + k];
        const float d = sqdist_exact(a, c, D);
        const unsigned long long p2 = (unsigned long long)(P.order2 ? P.order2[b * P.M2 + n] : n);
        const unsigned long long kq = ((unsigned long long)__float_as_uint(d) << 32) | (p2 & 0xffffffffull);
        mine = kq < mine ? kq : mine;
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        const unsigned long long other = __shfl_xor_sync(0xffffffffu, mine, off);
        mine = other < mine ? other : mine;
    }
    if ((tid & 31) == 0) atomicMin(&best, mine);
    __syncthreads();
    const unsigned int npos = (unsigned int)(best & 0xffffffffull);
    if (P.order2) {
        for (long long n = tid; n < P.M2; n += kThreads)
            if ((unsigned int)P.order2[b * P.M2 + n] == npos) P.idx2[pair] = n;
    } else if (tid == 0) {
        P.idx2[pair] = P.M2 > 0 ? (long long)npos : 0;
    }
    if (tid == 0) {
        const float cmax = __uint_as_float((unsigned int)(key >> 32));
        reinterpret_cast<float *>(P.out)[pair] = sqrtf(cmax);
        P.idx1[pair] = mstar >= 0 ? mstar : 0;
    }
}

// Fused path: one CTA per set pair.  Every row whose approximate minimum could be the exact maximum is re-evaluated with
// the separately rounded arithmetic (first visited n on ties); the largest exact minimum wins, the last visited m on ties.
// Up to kMaxCandidates rows are evaluated one after another by the whole CTA (one warp to a row had seven warps waiting for
// it: 56 -> 10 us at 64 pairs of 8192-point clouds), more of them a warp to a row.
template <int D, bool EXPAND>
__global__ void __launch_bounds__(kThreads)
hausdorff_refine_kernel(const HdParams P) {
    constexpr int kWarps = kThreads / 32;
    __shared__ unsigned long long s_row[kWarps], s_n[kWarps];
    __shared__ long long s_m[kWarps];
    __shared__ long long s_nstar;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const long long pair = blockIdx.x;
    const long long j = pair % P.N2;
    const long long bi = pair / P.N2;
    const long long b = bi / P.N1;
    const float *x1 = reinterpret_cast<const float *>(P.x1) + bi * P.M1 * D;
    const float *x2 = reinterpret_cast<const float *>(P.x2) + (b * P.N2 + j) * P.M2 * D;
    float *rm = P.rowmins + pair * P.M1;
    PairState *state = reinterpret_cast<PairState *>(P.keys) + pair;
    const unsigned int handed = EXPAND || P.handed_over ? state->direct : kAllRows;
    if (EXPAND ? handed != 0 : handed == 0) return;
    unsigned int *list = P.list + pair * P.M1;
    const bool listed = !EXPAND && handed != kAllRows;
    const long long rows = listed ? (long long)handed : P.M1;
    auto row_of = [&](long long c) -> long long { return listed ? (long long)list[c] : c; };
    auto position = [&](long long m) -> unsigned int { return (unsigned int)(P.order1 ? P.order1[b * P.M1 + m] : m); };
    // the largest approximate minimum, the last visited row on ties
    unsigned long long key = 0ull;
    for (long long c = tid; c < rows; c += kThreads) {
        const unsigned long long kq = ((unsigned long long)__float_as_uint(rm[c]) << 32) | position(row_of(c));
        key = kq > key ? kq : key;
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        const unsigned long long other = __shfl_xor_sync(0xffffffffu, key, off);
        key = other > key ? other : key;
    }
    if (lane == 0) s_row[warp] = key;
    __syncthreads();
#pragma unroll
    for (int w = 0; w < kWarps; ++w) key = s_row[w] > key ? s_row[w] : key;
    __syncthreads();
    const float amax = __uint_as_float((unsigned int)(key >> 32));
    const unsigned int pos_max = (unsigned int)(key & 0xffffffffull);
    // An approximate minimum of exactly 0 means every difference squared to 0, in either arithmetic: all rows then
    // tie at 0 and the last visited one, which the key already names, wins.  Otherwise a row can hold the exact
    // maximum only if its approximate minimum is within the rounding slack of the largest approximate minimum.
    const bool all_zero = !EXPAND && amax == 0.f;
    float lower = amax * (1.f - fused_slack<D>()) - kTiny;
    if (EXPAND) lower -= expanded_slack<D>(__uint_as_float(state->extent));

    // the rows to look at; their order does not matter
    __shared__ unsigned int s_count;
    __shared__ unsigned int s_cand[kMaxCandidates];
    if (tid == 0) s_count = 0;
    __syncthreads();
    for (long long c = tid; c < rows; c += kThreads) {
        const bool cand = all_zero ? position(row_of(c)) == pos_max : rm[c] >= lower;
        if (cand) {
            const unsigned int at = atomicAdd(&s_count, 1u);
            if (at < kMaxCandidates) s_cand[at] = (unsigned int)row_of(c);
        }
    }
    __syncthreads();
    const unsigned int count = s_count;
    if (EXPAND) {
        const bool bounded = __uint_as_float(state->extent) < kExtentMax;
        if (!bounded || count > kMaxExpanded) {
            // hand those rows over, or all of them; the direct form starts from untouched minima
            __syncthreads();
            if (tid == 0) s_count = 0;
            __syncthreads();
            if (bounded)
                for (long long m = tid; m < P.M1; m += kThreads)
                    if (rm[m] >= lower) list[atomicAdd(&s_count, 1u)] = (unsigned int)m;
            __syncthreads();
            for (long long c = tid; c < (bounded ? (long long)count : P.M1); c += kThreads) rm[c] = __uint_as_float(0xffffffffu);
            if (tid == 0) state->direct = bounded ? count : kAllRows;
            return;
        }
    }
    if (count <= kMaxCandidates) {
        unsigned long long row_key = 0ull, n_key = ~0ull;    // best (bits(min) << 32 | position(m)) and its n key, the same in all threads
        long long row = -1;
        for (unsigned int c = 0; c < count; ++c) {
            const long long m = s_cand[c];
            const unsigned int pos = position(m);
            float a[D];
#pragma unroll
            for (int k = 0; k < D; ++k) a[k] = x1[m * D + k];
            unsigned long long mine = ~0ull;
#pragma unroll 4
            for (long long n = tid; n < P.M2; n += kThreads) {
                float v[D];
#pragma unroll
                for (int k = 0; k < D; ++k) v[k] = x2[n * D + k];
                const float d = sqdist_exact(a, v, D);
                const unsigned long long p2 = (unsigned long long)(P.order2 ? P.order2[b * P.M2 + n] : n);
                const unsigned long long kq = ((unsigned long long)__float_as_uint(d) << 32) | (p2 & 0xffffffffull);
                if (d == d && kq < mine) mine = kq;   // a NaN distance never lowers a minimum
            }
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) {
                const unsigned long long other = __shfl_xor_sync(0xffffffffu, mine, off);
                mine = other < mine ? other : mine;
            }
            if (lane == 0) s_n[warp] = mine;
            __syncthreads();
#pragma unroll
            for (int w = 0; w < kWarps; ++w) mine = s_n[w] < mine ? s_n[w] : mine;
            __syncthreads();
            // a row without any comparable distance has the minimum +inf, as in the streaming kernel
            const unsigned int vbits = mine == ~0ull ? 0x7f800000u : (unsigned int)(mine >> 32);
            const unsigned long long rkey = ((unsigned long long)vbits << 32) | pos;
            if (row < 0 || rkey > row_key) { row_key = rkey; n_key = mine; row = m; }
        }
        const unsigned int npos = (unsigned int)(n_key & 0xffffffffull);
        if (tid == 0) s_nstar = (P.order2 || n_key == ~0ull) ? 0 : (long long)npos;
        __syncthreads();
        if (P.order2 && n_key != ~0ull) {
            for (long long n = tid; n < P.M2; n += kThreads)
                if ((unsigned int)P.order2[b * P.M2 + n] == npos) s_nstar = n;
            __syncthreads();
        }
        if (tid == 0) {
            reinterpret_cast<float *>(P.out)[pair] = sqrtf(__uint_as_float((unsigned int)(row_key >> 32)));
            P.idx1[pair] = row < 0 ? 0 : row;
            P.idx2[pair] = s_nstar;
        }
        return;
    }

    unsigned long long wrow = 0ull, wn = ~0ull;   // best (bits(min) << 32 | position(m)) of this warp, its n key
    long long wm = -1;
    for (long long base = (long long)warp * 32; base < rows; base += kThreads) {
        unsigned int pos = 0;
        bool cand = false;
        if (base + lane < rows) {
            pos = position(row_of(base + lane));
            cand = all_zero ? (pos == pos_max) : (rm[base + lane] >= lower);
        }
        unsigned int todo = __ballot_sync(0xffffffffu, cand);
        while (todo) {
            const int src = __ffs(todo) - 1;
            todo &= todo - 1;
            const long long mc = row_of(base + src);
            const unsigned int posc = __shfl_sync(0xffffffffu, pos, src);
            float a[D];
#pragma unroll
            for (int k = 0; k < D; ++k) a[k] = x1[mc * D + k];
            unsigned long long mine = ~0ull;
            for (long long n = lane; n < P.M2; n += 32) {
                float c[D];
#pragma unroll
                for (int k = 0; k < D; ++k) c[k] = x2[n * D + k];
                const float d = sqdist_exact(a, c, D);
                if (d == d) {   // a NaN distance never lowers a minimum
                    const unsigned long long p2 = (unsigned long long)(P.order2 ? P.order2[b * P.M2 + n] : n);
                    const unsigned long long kq = ((unsigned long long)__float_as_uint(d) << 32) | (p2 & 0xffffffffull);
                    mine = kq < mine ? kq : mine;
                }
            }
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) {
                const unsigned long long other = __shfl_xor_sync(0xffffffffu, mine, off);
                mine = other < mine ? other : mine;
            }
            // a row without any comparable distance has the minimum +inf, as in the streaming kernel
            const unsigned int vbits = mine == ~0ull ? 0x7f800000u : (unsigned int)(mine >> 32);
            const unsigned long long rkey = ((unsigned long long)vbits << 32) | posc;
            if (wm < 0 || rkey > wrow) { wrow = rkey; wn = mine; wm = mc; }
        }
    }
    if (lane == 0) { s_row[warp] = wrow; s_n[warp] = wn; s_m[warp] = wm; }
    __syncthreads();
    int bw = -1;
    for (int w = 0; w < kWarps; ++w)
        if (s_m[w] >= 0 && (bw < 0 || s_row[w] > s_row[bw])) bw = w;
    if (bw < 0) {   // cannot happen for M1 > 0: the row the key names is always a candidate
        if (tid == 0) { reinterpret_cast<float *>(P.out)[pair] = sqrtf(amax); P.idx1[pair] = 0; P.idx2[pair] = 0; }
        return;
    }
    const unsigned int npos = (unsigned int)(s_n[bw] & 0xffffffffull);
    if (tid == 0) s_nstar = (P.order2 || s_n[bw] == ~0ull) ? 0 : (long long)npos;
    __syncthreads();
    if (P.order2 && s_n[bw] != ~0ull) {
        for (long long n = tid; n < P.M2; n += kThreads)
            if ((unsigned int)P.order2[b * P.M2 + n] == npos) s_nstar = n;
        __syncthreads();
    }
    if (tid == 0) {
        reinterpret_cast<float *>(P.out)[pair] = sqrtf(__uint_as_float((unsigned int)(s_row[bw] >> 32)));
        P.idx1[pair] = s_m[bw];
        P.idx2[pair] = s_nstar;
    }
}

// ---- float64, D <= 16: the same streaming design ------------------------------------------------------------------------
// A 64-bit distance leaves no room for the visiting position in a 64-bit key, so every row's exact minimum is stored
// (8 bytes per x1 point in the caller's scratch) and one CTA per set pair then scans them: largest minimum, last
// visited row on ties, and for that row the first visited x2 point that attains it.  Products and sums are rounded
// separately, as in the reference's CPU loop, so values and indices equal the one-CTA-per-pair kernel's bit for bit.
constexpr int PMD = 2;             // x1 points per thread
constexpr int CHUNK_D = 4096;      // doubles staged per pass (32 KB)

template <int D>
__global__ void __launch_bounds__(kThreads)
hausdorff_rowmin_f64_kernel(const HdParams P) {
    constexpr int CHUNK = CHUNK_D / D;
    __shared__ double pts[CHUNK_D];
    const int tid = threadIdx.x;
    long long blk = blockIdx.x;
    const long long mt = blk % P.mtiles;
    const long long pair = blk / P.mtiles;
    const long long j = pair % P.N2;
    const long long bi = pair / P.N2;
    const long long b = bi / P.N1;
    const double *x1 = reinterpret_cast<const double *>(P.x1) + bi * P.M1 * D;
    const double *x2 = reinterpret_cast<const double *>(P.x2) + (b * P.N2 + j) * P.M2 * D;
    double px[PMD][D], rowmin[PMD];
    long long mm[PMD];
#pragma unroll
    for (int q = 0; q < PMD; ++q) {
        mm[q] = mt * (kThreads * PMD) + q * kThreads + tid;
        rowmin[q] = INFINITY;
#pragma unroll
        for (int k = 0; k < D; ++k) px[q][k] = mm[q] < P.M1 ? x1[mm[q] * D + k] : 0.0;
    }
    for (long long n0 = 0; n0 < P.M2; n0 += CHUNK) {
        const int cnt = (int)((P.M2 - n0) < CHUNK ? (P.M2 - n0) : CHUNK);
        __syncthreads();
        for (int e = tid; e < cnt * D; e += kThreads) pts[e] = x2[n0 * D + e];
        __syncthreads();
#pragma unroll 2
        for (int e = 0; e < cnt; ++e) {
            double c[D];
#pragma unroll
            for (int k = 0; k < D; ++k) c[k] = pts[e * D + k];
#pragma unroll
            for (int q = 0; q < PMD; ++q) rowmin[q] = fmin(rowmin[q], sqdist_exact(px[q], c, D));
        }
    }
    double *rm = reinterpret_cast<double *>(P.rowmins) + pair * P.M1;
#pragma unroll
    for (int q = 0; q < PMD; ++q)
        if (mm[q] < P.M1) rm[mm[q]] = rowmin[q];
}

template <int D>
__global__ void __launch_bounds__(kThreads)
hausdorff_finish_f64_kernel(const HdParams P) {
    __shared__ double s_val[kThreads];
    __shared__ long long s_pos[kThreads], s_m[kThreads];
    __shared__ unsigned long long s_npos[kThreads];
    __shared__ long long s_nstar;
    const int tid = threadIdx.x;
    const long long pair = blockIdx.x;
    const long long j = pair % P.N2;
    const long long bi = pair / P.N2;
    const long long b = bi / P.N1;
    const double *x1 = reinterpret_cast<const double *>(P.x1) + bi * P.M1 * D;
    const double *x2 = reinterpret_cast<const double *>(P.x2) + (b * P.N2 + j) * P.M2 * D;
    const double *rm = reinterpret_cast<const double *>(P.rowmins) + pair * P.M1;
    // largest row minimum, the last visited row on ties
    double best = -1.0;
    long long best_pos = -1, best_m = 0;
    for (long long m = tid; m < P.M1; m += kThreads) {
        const double v = rm[m];
        const long long p1 = P.order1 ? P.order1[b * P.M1 + m] : m;
        if (v > best || (v == best && p1 > best_pos)) { best = v; best_pos = p1; best_m = m; }
    }
    s_val[tid] = best; s_pos[tid] = best_pos; s_m[tid] = best_m;
    __syncthreads();
    for (int off = kThreads / 2; off > 0; off >>= 1) {
        if (tid < off) {
            const double v = s_val[tid + off];
            const long long p = s_pos[tid + off];
            if (v > s_val[tid] || (v == s_val[tid] && p > s_pos[tid])) { s_val[tid] = v; s_pos[tid] = p; s_m[tid] = s_m[tid + off]; }
        }
        __syncthreads();
    }
    const long long mstar = s_m[0];
    const double cmax = s_pos[0] >= 0 ? s_val[0] : 0.0;
    // the first visited x2 point at the row's minimum distance
    double a[D];
#pragma unroll
    for (int k = 0; k < D; ++k) a[k] = x1[mstar * D + k];
    unsigned long long mine = ~0ull;     // visiting position of the best candidate of this thread
    long long mine_n = 0;
    for (long long n = tid; n < P.M2; n += kThreads) {
        double c[D];
#pragma unroll
        for (int k = 0; k < D; ++k) c[k] = x2[n * D + k];
        if (sqdist_exact(a, c, D) == cmax) {
            const unsigned long long p2 = (unsigned long long)(P.order2 ? P.order2[b * P.M2 + n] : n);
            if (p2 < mine) { mine = p2; mine_n = n; }
        }
    }
    s_npos[tid] = mine; s_pos[tid] = mine_n;
    __syncthreads();
    for (int off = kThreads / 2; off > 0; off >>= 1) {
        if (tid < off && s_npos[tid + off] < s_npos[tid]) { s_npos[tid] = s_npos[tid + off]; s_pos[tid] = s_pos[tid + off]; }
        __syncthreads();
    }
    if (tid == 0) {
        s_nstar = s_npos[0] == ~0ull ? 0 : s_pos[0];
        reinterpret_cast<double *>(P.out)[pair] = sqrt(cmax);
        P.idx1[pair] = mstar;
        P.idx2[pair] = s_nstar;
    }
}

template <int D>
int launch_f64(HdParams P, cudaStream_t s) {
    const long long pairs = P.B * P.N1 * P.N2;
    P.mtiles = (P.M1 + kThreads * PMD - 1) / (kThreads * PMD);
    const long long blocks = pairs * P.mtiles;
    TPW_CHECK_ARG(blocks < (1ll << 31), "hausdorff: too many blocks");
    hausdorff_rowmin_f64_kernel<D><<<(unsigned)blocks, kThreads, 0, s>>>(P);
    TPW_LAUNCH_OK("hausdorff_rowmin_f64_kernel");
    hausdorff_finish_f64_kernel<D><<<(unsigned)pairs, kThreads, 0, s>>>(P);
    TPW_LAUNCH_OK("hausdorff_finish_f64_kernel");
    return TPW_OK;
}

// Plain path: any dtype, any D.  One CTA per set pair; thread t scans rows m = t, t+256, ...
template <typename T>
__global__ void __launch_bounds__(kThreads)
hausdorff_plain_kernel(const HdParams P) {
    __shared__ T s_val[kThreads];
    __shared__ long long s_pos[kThreads], s_m[kThreads], s_n[kThreads];
    const int tid = threadIdx.x;
    const long long pair = blockIdx.x;
    const long long j = pair % P.N2;
    const long long bi = pair / P.N2;
    const long long b = bi / P.N1;
    const int D = (int)P.D;
    const T *x1 = reinterpret_cast<const T *>(P.x1) + bi * P.M1 * D;
    const T *x2 = reinterpret_cast<const T *>(P.x2) + (b * P.N2 + j) * P.M2 * D;

    T best = T(-1);
    long long best_pos = -1, best_m = 0, best_n = 0;
    for (long long m = tid; m < P.M1; m += kThreads) {
        T rowmin = T(INFINITY);
        long long rn = 0, rpos = 0x7fffffffffffffffll;
        for (long long n = 0; n < P.M2; ++n) {
            const T d = sqdist_exact(x1 + m * D, x2 + n * D, D);
            const long long p2 = P.order2 ? P.order2[b * P.M2 + n] : n;
            if (d < rowmin || (d == rowmin && p2 < rpos)) { rowmin = d; rn = n; rpos = p2; }
        }
        const long long p1 = P.order1 ? P.order1[b * P.M1 + m] : m;
        if (rowmin > best || (rowmin == best && p1 > best_pos)) { best = rowmin; best_pos = p1; best_m = m; best_n = rn; }
    }
    s_val[tid] = best; s_pos[tid] = best_pos; s_m[tid] = best_m; s_n[tid] = best_n;
    __syncthreads();
    for (int off = kThreads / 2; off > 0; off >>= 1) {
        if (tid < off) {
            const T v = s_val[tid + off];
            const long long p = s_pos[tid + off];
            if (v > s_val[tid] || (v == s_val[tid] && p > s_pos[tid])) {
                s_val[tid] = v; s_pos[tid] = p; s_m[tid] = s_m[tid + off]; s_n[tid] = s_n[tid + off];
            }
        }
        __syncthreads();
    }
    if (tid == 0) {
        const T cmax = s_pos[0] >= 0 ? s_val[0] : T(0);
        reinterpret_cast<T *>(P.out)[pair] = (T)sqrt((double)cmax);
        P.idx1[pair] = s_m[0];
        P.idx2[pair] = s_n[0];
    }
}

// grad_x1[b,i,m*,k] += g * (x1[m*] - x2[n*]) / out, one thread per (b,i,k), ascending j.
template <typename T, bool SIDE2>
__global__ void hausdorff_backward_kernel(const T *grad, const T *out, const long long *idx1, const long long *idx2,
                                          const T *x1, const T *x2, T *gx,
                                          long long B, long long N1, long long N2, long long M1, long long M2, long long D) {
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long NO = SIDE2 ? N2 : N1; // sets on the side that owns the gradient
    if (idx >= B * NO * D) return;
    const long long k = idx % D, s = (idx / D) % NO, b = idx / (D * NO);
    const long long NI = SIDE2 ? N1 : N2;
    for (long long t = 0; t < NI; ++t) {
        const long long i = SIDE2 ? t : s, j = SIDE2 ? s : t;
        const long long pair = (b * N1 + i) * N2 + j;
        const long long m = idx1[pair], n = idx2[pair];
        const T a = x1[((b * N1 + i) * M1 + m) * D + k];
        const T c = x2[((b * N2 + j) * M2 + n) * D + k];
        const T diff = SIDE2 ? c - a : a - c;
        T *dst = SIDE2 ? gx + ((b * N2 + j) * M2 + n) * D + k : gx + ((b * N1 + i) * M1 + m) * D + k;
        *dst += grad[pair] * diff / out[pair];
    }
}

// P.rowmins != NULL selects the fused hot loop with the refining kernel, NULL the exact hot loop.
template <int D>
int launch_fast(HdParams P, cudaStream_t s) {
    const long long pairs = P.B * P.N1 * P.N2;
    if (P.rowmins) {
        P.mtiles = (P.M1 + Fused<D>::ROWS - 1) / Fused<D>::ROWS;
        // fewer row blocks than four CTAs per SM: share the x2 points, at least 256 of them to a CTA
        const long long want = 4ll * sm_count() / (pairs * P.mtiles), most = P.M2 / 256;
        P.splits = (int)(want < most ? want : most);
        if (P.splits < 1) P.splits = 1;
        const long long blocks = pairs * P.mtiles * P.splits;
        TPW_CHECK_ARG(blocks < (1ll << 31), "hausdorff: too many blocks");
        if (P.splits > 1) TPW_CUDA_OK(cudaMemsetAsync(P.rowmins, 0xff, (size_t)(pairs * P.M1) * sizeof(float), s));
        P.list = reinterpret_cast<unsigned int *>(P.rowmins + pairs * P.M1);
        // From 2^27 point pairs on: below, the sample and the two launches that serve handed-over rows cost what the expanded form
        // saves, and more where rows are handed over (200 pairs of 700 and 800 points: 51 to 99 us, 74 before any expanded form).
        if ((double)pairs * (double)P.M1 * (double)P.M2 >= 134217728.0) {
            // sampling CTAs: 1024 x2 points to one, no more than fill the GPU or than a pair's list has room for
            const long long fill = 4ll * sm_count() / pairs, samples = P.M2 / 1024 < fill ? P.M2 / 1024 : fill;
            if (P.M1 > 8 * kSampleWords) P.samples = (int)(samples < 1 ? 1 : samples < P.M1 / kSampleWords ? samples : P.M1 / kSampleWords);
            if (P.samples > 0) {
                TPW_CHECK_ARG(pairs * P.samples < (1ll << 31), "hausdorff: too many blocks");
                hausdorff_sample_kernel<D><<<(unsigned)(pairs * P.samples), kThreads, 0, s>>>(P);
                TPW_LAUNCH_OK("hausdorff_sample_kernel");
            } else {
                TPW_CUDA_OK(cudaMemsetAsync(P.keys, 0, (size_t)pairs * sizeof(PairState), s));
            }
            hausdorff_rowmin_fused_kernel<D, true><<<(unsigned)blocks, kFThreads, 0, s>>>(P);
            TPW_LAUNCH_OK("hausdorff_rowmin_fused_kernel");
            hausdorff_refine_kernel<D, true><<<(unsigned)pairs, kThreads, 0, s>>>(P);
            TPW_LAUNCH_OK("hausdorff_refine_kernel");
            P.handed_over = 1;
        }
        hausdorff_rowmin_fused_kernel<D, false><<<(unsigned)blocks, kFThreads, 0, s>>>(P);
        TPW_LAUNCH_OK("hausdorff_rowmin_fused_kernel");
        hausdorff_refine_kernel<D, false><<<(unsigned)pairs, kThreads, 0, s>>>(P);
        TPW_LAUNCH_OK("hausdorff_refine_kernel");
        return TPW_OK;
    }
    P.mtiles = (P.M1 + kThreads * PM - 1) / (kThreads * PM);
    const long long blocks = pairs * P.mtiles;
    TPW_CHECK_ARG(blocks < (1ll << 31), "hausdorff: too many blocks");
    TPW_CUDA_OK(cudaMemsetAsync(P.keys, 0, (size_t)pairs * sizeof(unsigned long long), s));
    hausdorff_rowmin_kernel<D><<<(unsigned)blocks, kThreads, 0, s>>>(P);
    TPW_LAUNCH_OK("hausdorff_rowmin_kernel");
    hausdorff_finish_kernel<D><<<(unsigned)pairs, kThreads, 0, s>>>(P);
    TPW_LAUNCH_OK("hausdorff_finish_kernel");
    return TPW_OK;
}

} // namespace
} // namespace tpw

using namespace tpw;

// one 8-byte key per set pair, then 8 bytes per x1 point of every set pair (the row minima: approximate float32 values
// for the fused float32 loop, exact float64 values for the float64 path; the query does not know the dtype)
extern "C" int64_t tpw_hausdorff_scratch_bytes(int64_t B, int64_t N1, int64_t N2, int64_t M1) {
    if (B <= 0 || N1 <= 0 || N2 <= 0) return 0;
    const int64_t pairs = B * N1 * N2;
    return pairs * (int64_t)sizeof(unsigned long long) + (M1 > 0 ? pairs * M1 * 8 : 0);
}

extern "C" int tpw_hausdorff_forward(int dtype, const void *x1, const void *x2,
                                     const int64_t *order1, const int64_t *order2,
                                     void *out, int64_t *idx1, int64_t *idx2, void *scratch,
                                     int64_t B, int64_t N1, int64_t N2, int64_t M1, int64_t M2, int64_t D,
                                     tpw_stream_t stream) {
    clear_error();
    TPW_CHECK_ARG(dtype == TPW_F32 || dtype == TPW_F64, "tpw_hausdorff_forward: dtype must be TPW_F32 or TPW_F64");
    TPW_CHECK_ARG(B >= 0 && N1 >= 0 && N2 >= 0 && M1 >= 0 && M2 >= 0 && D >= 0, "tpw_hausdorff_forward: negative size");
    const long long pairs = B * N1 * N2;
    if (pairs == 0) return TPW_OK;
    TPW_CHECK_ARG(M1 > 0 && M2 > 0 && D > 0, "tpw_hausdorff_forward: empty point sets (M1=%lld, M2=%lld, D=%lld)",
                  (long long)M1, (long long)M2, (long long)D);
    TPW_CHECK_ARG(M1 < (1ll << 32) && M2 < (1ll << 32), "tpw_hausdorff_forward: more than 2^32 points per set");
    TPW_CHECK_ARG(x1 && x2 && out && idx1 && idx2, "tpw_hausdorff_forward: NULL pointer");
    TPW_CHECK_ARG(pairs < (1ll << 31), "tpw_hausdorff_forward: too many set pairs");
    HdParams P;
    memset(&P, 0, sizeof(P));
    P.x1 = x1; P.x2 = x2;
    P.order1 = reinterpret_cast<const long long *>(order1);
    P.order2 = reinterpret_cast<const long long *>(order2);
    P.out = out;
    P.idx1 = reinterpret_cast<long long *>(idx1);
    P.idx2 = reinterpret_cast<long long *>(idx2);
    P.keys = reinterpret_cast<unsigned long long *>(scratch);
    P.B = B; P.N1 = N1; P.N2 = N2; P.M1 = M1; P.M2 = M2; P.D = D;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (dtype == TPW_F32 && D <= kMaxFastD) {
        TPW_CHECK_ARG(scratch != nullptr, "tpw_hausdorff_forward: scratch is NULL");
        TPW_CHECK_ARG((reinterpret_cast<uintptr_t>(scratch) & 7u) == 0, "tpw_hausdorff_forward: scratch must be 8-byte aligned");
        if (!getenv("TPW_HAUSDORFF_EXACT_LOOP")) P.rowmins = reinterpret_cast<float *>(P.keys + pairs);
        switch (D) {
            case 1: return launch_fast<1>(P, s);
            case 2: return launch_fast<2>(P, s);
            case 3: return launch_fast<3>(P, s);
            case 4: return launch_fast<4>(P, s);
            case 5: return launch_fast<5>(P, s);
            case 6: return launch_fast<6>(P, s);
            case 7: return launch_fast<7>(P, s);
            case 8: return launch_fast<8>(P, s);
            case 9: return launch_fast<9>(P, s);
            case 10: return launch_fast<10>(P, s);
            case 11: return launch_fast<11>(P, s);
            case 12: return launch_fast<12>(P, s);
            case 13: return launch_fast<13>(P, s);
            case 14: return launch_fast<14>(P, s);
            case 15: return launch_fast<15>(P, s);
            default: return launch_fast<16>(P, s);
        }
    }
    if (dtype == TPW_F64 && D <= kMaxFastD && scratch != nullptr && (reinterpret_cast<uintptr_t>(scratch) & 7u) == 0 &&
        !getenv("TPW_HAUSDORFF_PLAIN_F64")) {
        P.rowmins = reinterpret_cast<float *>(P.keys + pairs);   // used as double[pairs * M1]
        switch (D) {
            case 1: return launch_f64<1>(P, s);
            case 2: return launch_f64<2>(P, s);
            case 3: return launch_f64<3>(P, s);
            case 4: return launch_f64<4>(P, s);
            case 5: return launch_f64<5>(P, s);
            case 6: return launch_f64<6>(P, s);
            case 7: return launch_f64<7>(P, s);
            case 8: return launch_f64<8>(P, s);
            case 9: return launch_f64<9>(P, s);
            case 10: return launch_f64<10>(P, s);
            case 11: return launch_f64<11>(P, s);
            case 12: return launch_f64<12>(P, s);
            case 13: return launch_f64<13>(P, s);
            case 14: return launch_f64<14>(P, s);
            case 15: return launch_f64<15>(P, s);
            default: return launch_f64<16>(P, s);
        }
    }
    if (dtype == TPW_F32) hausdorff_plain_kernel<float><<<(unsigned)pairs, kThreads, 0, s>>>(P);
    else hausdorff_plain_kernel<double><<<(unsigned)pairs, kThreads, 0, s>>>(P);
    TPW_LAUNCH_OK("hausdorff_plain_kernel");
    return TPW_OK;
}

extern "C" int tpw_hausdorff_backward(int dtype, const void *grad, const void *out,
                                      const int64_t *idx1, const int64_t *idx2,
                                      const void *x1, const void *x2, void *grad_x1, void *grad_x2,
                                      int64_t B, int64_t N1, int64_t N2, int64_t M1, int64_t M2, int64_t D,
                                      tpw_stream_t stream) {
    clear_error();
    TPW_CHECK_ARG(dtype == TPW_F32 || dtype == TPW_F64, "tpw_hausdorff_backward: dtype must be TPW_F32 or TPW_F64");
    TPW_CHECK_ARG(B >= 0 && N1 >= 0 && N2 >= 0 && M1 >= 0 && M2 >= 0 && D >= 0, "tpw_hausdorff_backward: negative size");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const size_t es = dtype == TPW_F32 ? 4 : 8;
    if (grad_x1 && B * N1 * M1 * D > 0) TPW_CUDA_OK(cudaMemsetAsync(grad_x1, 0, (size_t)(B * N1 * M1 * D) * es, s));
    if (grad_x2 && B * N2 * M2 * D > 0) TPW_CUDA_OK(cudaMemsetAsync(grad_x2, 0, (size_t)(B * N2 * M2 * D) * es, s));
    if (B * N1 * N2 == 0 || M1 == 0 || M2 == 0 || D == 0) return TPW_OK;
    TPW_CHECK_ARG(grad && out && idx1 && idx2 && x1 && x2, "tpw_hausdorff_backward: NULL pointer");
    const int threads = 128;
    const long long *i1 = reinterpret_cast<const long long *>(idx1), *i2 = reinterpret_cast<const long long *>(idx2);
#define TPW_HD_BWD(T)                                                                                                   \
    do {                                                                                                                \
        if (grad_x1) {                                                                                                  \
            const long long n = B * N1 * D;                                                                             \
            hausdorff_backward_kernel<T, false><<<(unsigned)((n + threads - 1) / threads), threads, 0, s>>>(            \
                (const T *)grad, (const T *)out, i1, i2, (const T *)x1, (const T *)x2, (T *)grad_x1, B, N1, N2, M1, M2, D); \
        }                                                                                                               \
        if (grad_x2) {                                                                                                  \
            const long long n = B * N2 * D;                                                                             \
            hausdorff_backward_kernel<T, true><<<(unsigned)((n + threads - 1) / threads), threads, 0, s>>>(             \
                (const T *)grad, (const T *)out, i1, i2, (const T *)x1, (const T *)x2, (T *)grad_x2, B, N1, N2, M1, M2, D); \
        }                                                                                                               \
    } while (0)
    if (dtype == TPW_F32) TPW_HD_BWD(float); else TPW_HD_BWD(double);
#undef TPW_HD_BWD
    TPW_LAUNCH_OK("hausdorff_backward_kernel");
    return TPW_OK;
}


// ---- allocation-free variant ----------------------------------------------------------------------
// Some hosts of this library are not allowed to obtain device memory at call time: a serving
// process that hands the whole GPU to its own pool when it starts, a plug-in host that forbids
// allocation inside its compute callback, or a latency-critical loop that cannot afford the
// device-wide synchronisation cudaMalloc may imply.  tpw_hausdorff_forward needs 8 bytes of scratch
// per set pair from such a caller; this variant brings its own instead, in a fixed array that
// lives in the library's device image (every GPU that loads the library holds it until exit).
namespace tpw {
namespace {

constexpr long long kStaticMaxPairs = 65536; // 512 KiB of keys

static __device__ __align__(256) unsigned long long g_hausdorff_static_keys[kStaticMaxPairs];

// `g_hausdorff_static_keys` names a host-side shadow here, not device memory; the device address
// has to be asked for, once per device, while that device is current.  That first lookup may make the
// runtime load this library's device image on the device (memory for the image, the 512 KiB array
// included, and an implicit synchronisation): it belongs in the host's start-up, before the region in
// which nothing may allocate.  The slots are atomic (any host thread may be first; all store the same
// address).  A cudaDeviceReset invalidates the address: a host that resets a device must not call into
// this library on it again in the same process.
int resolve_static_keys(unsigned long long **ptr) {
    static std::atomic<unsigned long long *> cache[64];
    int dev = 0;
    TPW_CUDA_OK(cudaGetDevice(&dev));
    TPW_CHECK_ARG(dev >= 0 && dev < 64, "tpw_hausdorff_forward_static: device ordinal %d is out of range", dev);
    unsigned long long *cached = cache[dev].load(std::memory_order_acquire);
    if (!cached) {
        void *p = nullptr;
        TPW_CUDA_OK(cudaGetSymbolAddress(&p, g_hausdorff_static_keys));
        TPW_CHECK_ARG(p != nullptr, "tpw_hausdorff_forward_static: the scratch symbol resolved to NULL");
        cached = static_cast<unsigned long long *>(p);
        cache[dev].store(cached, std::memory_order_release);
    }
    *ptr = cached;
    return TPW_OK;
}

} // namespace
} // namespace tpw

extern "C" int64_t tpw_hausdorff_static_max_pairs(void) { return tpw::kStaticMaxPairs; }

extern "C" int tpw_hausdorff_forward_static(int dtype, const void *x1, const void *x2,
                                            const int64_t *order1, const int64_t *order2,
                                            void *out, int64_t *idx1, int64_t *idx2,
                                            int64_t B, int64_t N1, int64_t N2, int64_t M1, int64_t M2, int64_t D,
                                            tpw_stream_t stream) {
    clear_error();
    TPW_CHECK_ARG(dtype == TPW_F32 || dtype == TPW_F64, "tpw_hausdorff_forward_static: dtype must be TPW_F32 or TPW_F64");
    TPW_CHECK_ARG(B >= 0 && N1 >= 0 && N2 >= 0 && M1 >= 0 && M2 >= 0 && D >= 0, "tpw_hausdorff_forward_static: negative size");
    const long long pairs = B * N1 * N2;
    if (pairs == 0) return TPW_OK;
    TPW_CHECK_ARG(pairs <= kStaticMaxPairs,
                  "tpw_hausdorff_forward_static: %lld set pairs exceed the built-in scratch of %lld; "
                  "use tpw_hausdorff_forward with caller-provided scratch", pairs, kStaticMaxPairs);
    TPW_CHECK_ARG(M1 > 0 && M2 > 0 && D > 0, "tpw_hausdorff_forward_static: empty point sets (M1=%lld, M2=%lld, D=%lld)",
                  (long long)M1, (long long)M2, (long long)D);
    TPW_CHECK_ARG(M1 < (1ll << 32) && M2 < (1ll << 32), "tpw_hausdorff_forward_static: more than 2^32 points per set");
    TPW_CHECK_ARG(x1 && x2 && out && idx1 && idx2, "tpw_hausdorff_forward_static: NULL pointer");
    HdParams P;
    memset(&P, 0, sizeof(P));
    P.x1 = x1; P.x2 = x2;
    P.order1 = reinterpret_cast<const long long *>(order1);
    P.order2 = reinterpret_cast<const long long *>(order2);
    P.out = out;
    P.idx1 = reinterpret_cast<long long *>(idx1);
    P.idx2 = reinterpret_cast<long long *>(idx2);
    P.B = B; P.N1 = N1; P.N2 = N2; P.M1 = M1; P.M2 = M2; P.D = D;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (dtype == TPW_F32 && D <= kMaxFastD) {
        int st = resolve_static_keys(&P.keys);
        if (st != TPW_OK) return st;
        // launch_fast clears the first `pairs` keys on the stream before the kernels use them; without room for
        // the approximate row minima (P.rowmins stays NULL) it evaluates every point pair in the exact arithmetic
        switch (D) {
            case 1: return launch_fast<1>(P, s);
            case 2: return launch_fast<2>(P, s);
            case 3: return launch_fast<3>(P, s);
            case 4: return launch_fast<4>(P, s);
            case 5: return launch_fast<5>(P, s);
            case 6: return launch_fast<6>(P, s);
            case 7: return launch_fast<7>(P, s);
            case 8: return launch_fast<8>(P, s);
            case 9: return launch_fast<9>(P, s);
            case 10: return launch_fast<10>(P, s);
            case 11: return launch_fast<11>(P, s);
            case 12: return launch_fast<12>(P, s);
            case 13: return launch_fast<13>(P, s);
            case 14: return launch_fast<14>(P, s);
            case 15: return launch_fast<15>(P, s);
            default: return launch_fast<16>(P, s);
        }
    }
    // the one-CTA-per-pair kernel keeps its state in shared memory and needs no scratch at all
    if (dtype == TPW_F32) hausdorff_plain_kernel<float><<<(unsigned)pairs, kThreads, 0, s>>>(P);
    else hausdorff_plain_kernel<double><<<(unsigned)pairs, kThreads, 0, s>>>(P);
    TPW_LAUNCH_OK("hausdorff_plain_kernel");
    return TPW_OK;
}
