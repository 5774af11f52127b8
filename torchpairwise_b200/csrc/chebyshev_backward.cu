// Backward of the Chebyshev distance (cdist with p = +inf) for float32, in three kernels.
//
//   out[b,i,j] = max_k |x1[b,i,k] - x2[b,j,k]|
//   grad_x1[b,i,k] = sum_j g[b,i,j] * sgn(d) * [|d| == out]      (d = x1[b,i,k] - x2[b,j,k]; nothing where out == 0)
//   grad_x2[b,j,k] = -sum_i (same term)
//
// (ATen's cdist backward under OPS/pairwise_metrics.cpp:305: every coordinate that attains the maximum
// receives the gradient.)  The dense form evaluates the test for every (i, j, k) once per gradient.
// Here the attaining coordinate is found once per pair and both gradients are then scattered:
//
//   1. chebyshev_match_kernel: the forward tile (x1 / x2 chunks staged by TMA, 8 x 4 pairs per thread) re-forms d, takes
//      the largest |d| of every group of four features and compares it with the saved output; a match adds
//      65536 + group to the pair's sum, so that sum >> 16 counts the attaining groups.  One group: its four differences
//      are formed once more, and one attaining coordinate makes the pair's code k | sign << 31.  None (out == 0, NaN,
//      padding): the pair is skipped.  Several (a tied maximum): the pair is marked and counted in a device counter.
//      Bound: issue and both arithmetic pipes; six instructions per four features (packed subtract, three-operand
//      maximum) where a compare and two multiply-adds for every feature took sixteen.  [16, 4096, 4096, 256]: 12.0 -> 6.9 ms.
//   2. chebyshev_scatter_kernel (once per gradient): one thread per x1 row (x2 row) walks over the row's pairs in
//      order and adds +-g into its row of a shared-memory gradient block at the coded coordinate; for a marked pair
//      it walks over the features itself.  Every gradient element has one owner and a fixed order of additions:
//      deterministic, no atomics.
//   3. Exact ties are rare in continuous data (a few hundred among the 2.7e8 pairs of 256 normal features) but
//      the rule in lattice-valued data.  When more than one pair in 32768 is marked, the scatter kernels return
//      at once and the dense kernel of lp_backward.cu, which otherwise returns at once, writes both gradients.
#include "common.cuh"
#include "packed_f32x2.cuh"

namespace tpw {
namespace {

constexpr int kThreads = 128;                // four CTAs per SM: while one resolves its groups the others compute
constexpr int kStages = 3;
constexpr int RI = 8, RJ = 4;               // pairs per thread: 8 x1 rows by 4 x2 rows (two registers per pair)
constexpr int TS = kThreads / 16;           // x1 rows between a thread's rows
constexpr int TI = TS * RI, TJ = 16 * RJ;   // 64 x 64 pairs per CTA
constexpr int KC = 32;                      // features per staged chunk (128 bytes per row)
constexpr int XB = TI * 128, YB = TJ * 128; // bytes of one stage's x1 and x2 tiles
constexpr int STAGE = XB + YB;
constexpr int OFF_BAR = kStages * STAGE;
constexpr int MATCH_SMEM = OFF_BAR + kStages * 8 + 1024;
constexpr uint32_t kSkip = 0xffffffffu;   // no gradient from this pair
constexpr uint32_t kTied = 0xfffffffeu;   // several coordinates attain the maximum

// more marked pairs than this and the dense kernel takes over (the same rule on both sides of the hand-over)
__host__ __device__ inline unsigned long long tie_limit(long long pairs) { return (unsigned long long)(pairs >> 15) + 64ull; }

struct MatchParams {
    const float *x1, *x2, *out;
    uint32_t *code;
    unsigned long long *ties;
    long long B, N1, N2, D, tiles_i, tiles_j;
    int *status;
};

__device__ __forceinline__ float match_mask(float d, float o) {   // 1.0 where |d| == o, else 0.0
    float m;
    asm("set.eq.f32.f32 %0, %1, %2;" : "=f"(m) : "f"(fabsf(d)), "f"(o));
    return m;
}

template <int ROWS>
__device__ __forceinline__ void stage_rows_plain(unsigned char *tile, const float *base, long long row0, long long nrows,
                                                 long long D, long long k0) {
    for (int e = threadIdx.x; e < ROWS * KC; e += kThreads) {
        const int r = e / KC, kk = e % KC;
        const long long row = row0 + r, k = k0 + kk;
        const float v = (row < nrows && k < D) ? base[row * D + k] : 0.f;
        *reinterpret_cast<float *>(tile + swz128(r, kk / 4) + (kk % 4) * 4) = v;
    }
}

template <bool USE_TMA>
__global__ void __launch_bounds__(kThreads, 4)
chebyshev_match_kernel(const __grid_constant__ CUtensorMap map1, const __grid_constant__ CUtensorMap map2, const MatchParams P) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char *smem = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t *full = reinterpret_cast<uint64_t *>(smem + OFF_BAR);

    const int tid = threadIdx.x;
    const int ti = tid >> 4, tj = tid & 15;
    long long tile = blockIdx.x;
    const long long tjx = tile % P.tiles_j;
    tile /= P.tiles_j;
    const long long tix = tile % P.tiles_i;
    const long long b = tile / P.tiles_i;
    const long long i0 = tix * TI, j0 = tjx * TJ;

    const float *x1 = P.x1 + b * P.N1 * P.D;
    const float *x2 = P.x2 + b * P.N2 * P.D;
    const float *out = P.out + b * P.N1 * P.N2;
    const int nchunks = (int)((P.D + KC - 1) / KC);

    if (USE_TMA) {
        if (tid == 0) {
#pragma unroll
            for (int s = 0; s < kStages; ++s) mbar_init(&full[s], 1);
            mbar_init_fence();
            tma_prefetch_descriptor(&map1);
            tma_prefetch_descriptor(&map2);
        }
        __syncthreads();
        if (tid == 0) {
            for (int c = 0; c < kStages - 1 && c < nchunks; ++c) {
                mbar_expect_tx(&full[c], STAGE);
                tma_load_3d(smem + c * STAGE, &map1, &full[c], c * KC, (int)i0, (int)b);
                tma_load_3d(smem + c * STAGE + XB, &map2, &full[c], c * KC, (int)j0, (int)b);
            }
        }
    }

    // the saved maximum of every pair; -1 (never equal to an absolute value) where the pair does not exist or
    // the maximum is 0, in which case the gradient is defined as 0
    float o[RI][RJ];
    float acc[RI][RJ];   // sum of (65536 + group) over the attaining groups: exact in float32 up to 255 of them
#pragma unroll
    for (int ri = 0; ri < RI; ++ri) {
        const long long i = i0 + ti + TS * ri;
#pragma unroll
        for (int rj = 0; rj < RJ; ++rj) {
            const long long j = j0 + tj + 16 * rj;
            float v = -1.f;
            if (i < P.N1 && j < P.N2) {
                v = out[i * P.N2 + j];
                if (v == 0.f) v = -1.f;
            }
            o[ri][rj] = v;
            acc[ri][rj] = 0.f;
        }
    }

    int failed = 0;
    for (int t = 0; t < nchunks; ++t) {
        int stage;
        if (USE_TMA) {
            if (__syncthreads_or(failed)) {
                if (tid == 0) {
                    if (P.status) atomicCAS(P.status, 0, (9 << 16) | 1);
                    // the chunks issued earlier may still be landing: the CTA stays (bounded) until they have
                    for (int c = t; c < t + kStages - 1 && c < nchunks; ++c) mbar_wait_bounded(&full[c % kStages], (uint32_t)((c / kStages) & 1));
                }
                return;
            }
            const int nxt = t + kStages - 1;
            if (nxt < nchunks && tid == 0) {
                const int ns = nxt % kStages;
                mbar_expect_tx(&full[ns], STAGE);
                tma_load_3d(smem + ns * STAGE, &map1, &full[ns], nxt * KC, (int)i0, (int)b);
                tma_load_3d(smem + ns * STAGE + XB, &map2, &full[ns], nxt * KC, (int)j0, (int)b);
            }
            stage = t % kStages;
            if (!mbar_wait_bounded(&full[stage], (uint32_t)((t / kStages) & 1))) failed = 1;
        } else {
            stage = 0;
            __syncthreads();
            stage_rows_plain<TI>(smem, x1, i0, P.N1, P.D, (long long)t * KC);
            stage_rows_plain<TJ>(smem + XB, x2, j0, P.N2, P.D, (long long)t * KC);
            __syncthreads();
        }
        const unsigned char *xs = smem + stage * STAGE;
        const unsigned char *ys = xs + XB;
        const uint32_t xrow = ti, yrow = tj;      // rows 8 or 16 apart share row & 7
        const long long kleft = P.D - (long long)t * KC;
        const int cmax = kleft < KC ? (int)((kleft + 3) / 4) : 8;
#pragma unroll 1
        for (int c = 0; c < cmax; ++c) {
            const float group = (float)(0x10000 + t * (KC / 4) + c);
            float4 yb[RJ];
#pragma unroll
            for (int r = 0; r < RJ; ++r)
                yb[r] = *reinterpret_cast<const float4 *>(ys + (yrow + 16 * r) * 128u + ((c ^ (yrow & 7u)) << 4));
#pragma unroll
            for (int ri = 0; ri < RI; ++ri) {
                const float4 xa = *reinterpret_cast<const float4 *>(xs + (xrow + TS * ri) * 128u + ((c ^ (xrow & 7u)) << 4));
#pragma unroll
                for (int rj = 0; rj < RJ; ++rj) {
                    // six instructions per four features: two packed subtracts, the largest |difference| of the group in
                    // two, one compare into 1.0 / 0.0 and one fused multiply-add that takes the match as a factor.
                    // Features past D are zero on both sides: |0| never equals a positive maximum.
                    float d0, d1, d2, d3;
                    unpack2(sub2(pack2(xa.x, xa.y), pack2(yb[rj].x, yb[rj].y)), d0, d1);
                    unpack2(sub2(pack2(xa.z, xa.w), pack2(yb[rj].z, yb[rj].w)), d2, d3);
                    const float m = match_mask(fmaxf(max3_abs(d0, d1, d2), fabsf(d3)), o[ri][rj]);
                    acc[ri][rj] = fmaf(m, group, acc[ri][rj]);
                }
            }
        }
    }
    if (USE_TMA) {
        if (__syncthreads_or(failed)) {
            if (tid == 0 && P.status) atomicCAS(P.status, 0, (9 << 16) | 2);
            return;
        }
    }

    // One attaining group: its four differences are formed again from the rows in global memory (32 bytes per pair, read
    // through L1 and L2) to see which coordinates attain the maximum.  The register tile is parked in the operand stages
    // first, every thread in its own words, so that this loop is not unrolled 32 times.
    uint32_t *code = P.code + b * P.N1 * P.N2;
    float2 *park = reinterpret_cast<float2 *>(smem) + tid;
    static_assert(RI * RJ * kThreads * 8 <= OFF_BAR, "the parked register tile must fit in the operand stages");
    if (!USE_TMA) __syncthreads();
#pragma unroll
    for (int ri = 0; ri < RI; ++ri)
#pragma unroll
        for (int rj = 0; rj < RJ; ++rj) park[(ri * RJ + rj) * kThreads] = make_float2(acc[ri][rj], o[ri][rj]);
    int tied = 0;
#pragma unroll 4
    for (int e = 0; e < RI * RJ; ++e) {
        const long long i = i0 + ti + TS * (e / RJ), j = j0 + tj + 16 * (e % RJ);
        const float2 v = park[e * kThreads];
        const uint32_t a = (uint32_t)v.x;
        uint32_t cd = kSkip;
        if ((a >> 16) == 1u) {
            const long long k = (long long)(a & 0xffffu) * 4;
            const float *xp = x1 + i * P.D + k, *yp = x2 + j * P.D + k;
            float d[4];
            if (USE_TMA) {   // D is a multiple of 4 and both bases are 16-byte aligned
                const float4 xv = __ldg(reinterpret_cast<const float4 *>(xp)), yv = __ldg(reinterpret_cast<const float4 *>(yp));
                d[0] = xv.x - yv.x; d[1] = xv.y - yv.y; d[2] = xv.z - yv.z; d[3] = xv.w - yv.w;
            } else {
#pragma unroll
                for (int u = 0; u < 4; ++u) d[u] = k + u < P.D ? __ldg(xp + u) - __ldg(yp + u) : 0.f;
            }
            int hits = 0;
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (fabsf(d[u]) == v.y) {
                    ++hits;
                    cd = (uint32_t)(k + u) | (d[u] < 0.f ? 0x80000000u : 0u);
                }
            if (hits > 1) { cd = kTied; ++tied; }
        } else if (a != 0u) {
            cd = kTied;
            ++tied;
        }
        if (i < P.N1 && j < P.N2) code[i * P.N2 + j] = cd;
    }
    const int total = __syncthreads_count(tied != 0) ? 1 : 0;
    if (total) {   // rare: let every thread with marked pairs add its own count
        if (tied) atomicAdd(P.ties, (unsigned long long)tied);
    }
}

// ---- scatter ---------------------------------------------------------------------------------------------------------
constexpr int SR = 64;           // gradient rows per CTA, each walked by one thread of the first two warps; two CTAs per SM
constexpr int STHR = 256;        // all eight warps stage the pairs
constexpr int SD = 256;          // most features per CTA
constexpr int SP = 32;           // pairs per gradient row staged at a time
constexpr int SB = 4;            // pairs a walker applies together
constexpr int SPITCH = SP + 4;   // words per staged row of pairs: 16-byte aligned, eight lanes of a 128-bit load in eight bank groups
constexpr int STAGE_WORDS = SR * SPITCH;                      // one array (g or codes) of one stage
// words per row of the accumulators: the CTA's features and one word that takes what belongs elsewhere; odd, so that
// the 32 rows of a warp start in 32 different banks
__host__ __device__ inline int acc_stride(int features) { return (features + 1) | 1; }
__host__ __device__ inline int scatter_smem(int features) { return SR * acc_stride(features) * 4 + 4 * STAGE_WORDS * 4; }

struct ScatterParams {
    const float *grad;
    const uint32_t *code;
    const unsigned long long *ties;
    const float *x1, *x2, *fwd;   // read for marked pairs only
    float *out;                   // [B, NR, D]
    long long B, N1, N2, D, NR, tiles_r, tiles_k;
};

// A pair whose maximum is attained by several coordinates: each of the CTA's kn features among them receives +-g (ascending k).
__device__ __noinline__ void scatter_tied(float *row, const float *a, const float *c, float o, float g, int k0, int kn,
                                          bool negate) {
    for (int k = 0; k < kn; ++k) {
        const float d = a[k0 + k] - c[k0 + k];
        if (fabsf(d) == o) row[k] += (d < 0.f) != negate ? -g : g;
    }
}

// COLS = false: grad_x1.  Thread r of the first 64 walks over the pairs of x1 row r0 + r, j ascending, and adds +-g into
// its row of a shared-memory gradient block.  COLS = true: grad_x2, the same with x2 row r0 + r, i ascending and the sign
// flipped.  The pairs are staged 32 per gradient row at a time by all 256 threads (whole 128-byte segments of g and of
// the codes from global memory, held in registers while the walkers apply the tile before) into one of two buffers.
//
// The bound is the latency of the chain load accumulator -> add -> store.  A walker takes four pairs into registers,
// loads their four accumulators together, adds in order (a pair whose coordinate occurred earlier in the four continues
// from that sum) and stores in order: the additions and their order are those of one pair at a time.  Pairs that do
// not concern the CTA's features go to a spare word beside the row, so that no lane of the warp branches.
// Measured on [16, 4096, 4096] pairs, 256 features: 1.50 -> 0.77 ms per gradient against one pair at a time by four
// walkers a row, each looking at all pairs for those in its quarter of the features; 0.33 ms to read g and the codes.
template <bool COLS>
__global__ void __launch_bounds__(STHR, 2) chebyshev_scatter_kernel(const ScatterParams P) {
    if (*P.ties > tie_limit(P.B * P.N1 * P.N2)) return;   // tied maxima everywhere: the dense kernel that follows writes this gradient
    extern __shared__ float sm[];
    const int tid = threadIdx.x;
    long long tile = blockIdx.x;
    const long long tk = tile % P.tiles_k;
    tile /= P.tiles_k;
    const long long tr = tile % P.tiles_r;
    const long long b = tile / P.tiles_r;
    const long long r0 = tr * SR;
    const int k0 = (int)(tk * SD);
    const int kn = (int)((P.D - k0) < SD ? (P.D - k0) : SD);
    const int stride = acc_stride(P.D < SD ? (int)P.D : SD);
    float *stage = sm;                                    // [2 buffers][g, codes][SR][SPITCH] (COLS: [SP][SR])
    float *accs = sm + 4 * STAGE_WORDS;
    for (int e = tid; e < SR * stride; e += STHR) accs[e] = 0.f;
    const float *grad = P.grad + b * P.N1 * P.N2;
    const uint32_t *code = P.code + b * P.N1 * P.N2;
    const long long NS = COLS ? P.N1 : P.N2;     // length of the walk

    // staging: element e = tid + u * STHR of a tile is (row e / SP, step e % SP) for rows and (step e / SR, column
    // e % SR) for columns, so that consecutive threads read consecutive addresses of g and code.  Everything that does
    // not depend on the tile is worked out once: a thread's step (column) is fixed, its rows (steps) advance by a
    // constant, so a tile costs it one pointer bump and one predicate per element.
    constexpr int PER = SR * SP / STHR;          // 8 elements of each array per thread
    constexpr int UR = COLS ? STHR / SR : STHR / SP;      // rows (steps) between a thread's consecutive elements
    const int fix = COLS ? tid % SR : tid % SP;           // column of the gradient row block / step inside the tile
    const int var0 = COLS ? tid / SR : tid / SP;          // first step / first row
    // offset of element u = 0 of tile s0 = 0, then per element and per tile
    const long long off0 = COLS ? (long long)var0 * P.N2 + r0 + fix : (r0 + var0) * P.N2 + fix;
    const long long off_u = (long long)UR * P.N2;
    const long long off_tile = COLS ? (long long)SP * P.N2 : (long long)SP;
    const bool fix_ok = COLS ? (r0 + fix < P.N2) : true;
    const long long var_end = COLS ? P.N1 : P.N1 - r0;    // rows: row index below this; columns: step s0 + step below this
    const int sm0 = COLS ? var0 * SR + fix : var0 * SPITCH + fix;
    constexpr int sm_u = COLS ? UR * SR : UR * SPITCH;
    float gr[PER];
    uint32_t cr[PER];
    auto fetch = [&](long long s0) {
        const float *gp = grad + off0 + (s0 / SP) * off_tile;
        const uint32_t *cp = code + off0 + (s0 / SP) * off_tile;
        const bool tile_ok = COLS ? fix_ok : (s0 + fix < P.N2);
        const long long first = COLS ? s0 + var0 : (long long)var0;
#pragma unroll
        for (int u = 0; u < PER; ++u) {
            const bool ok = tile_ok && first + (long long)u * UR < var_end;
            gr[u] = ok ? __ldg(gp) : 0.f;
            cr[u] = ok ? __ldg(cp) : kSkip;
            gp += off_u;
            cp += off_u;
        }
    };
    fetch(0);
    int buf = 0;
    for (long long s0 = 0; s0 < NS; s0 += SP, buf ^= 1) {
        // the walkers may still be on the other buffer; this one was last read before the previous barrier
        float *gs = stage + buf * 2 * STAGE_WORDS;
        uint32_t *cs = reinterpret_cast<uint32_t *>(gs + STAGE_WORDS);
#pragma unroll
        for (int u = 0; u < PER; ++u) {
            gs[sm0 + u * sm_u] = gr[u];
            cs[sm0 + u * sm_u] = cr[u];
        }
        __syncthreads();
        if (s0 + SP < NS) fetch(s0 + SP);
        if (tid < SR) {
            float *mine = accs + tid * stride;
#pragma unroll 1
            for (int ss = 0; ss < SP; ss += SB) {
                uint32_t cd[SB];
                float g[SB], v[SB];
                int k[SB];
                if (COLS) {
#pragma unroll
                    for (int u = 0; u < SB; ++u) {
                        cd[u] = cs[(ss + u) * SR + tid];
                        g[u] = gs[(ss + u) * SR + tid];
                    }
                } else {
                    const uint4 cv = *reinterpret_cast<const uint4 *>(cs + tid * SPITCH + ss);
                    const float4 gv = *reinterpret_cast<const float4 *>(gs + tid * SPITCH + ss);
                    cd[0] = cv.x; cd[1] = cv.y; cd[2] = cv.z; cd[3] = cv.w;
                    g[0] = gv.x; g[1] = gv.y; g[2] = gv.z; g[3] = gv.w;
                }
                bool any_tied = false;
#pragma unroll
                for (int u = 0; u < SB; ++u) any_tied |= cd[u] == kTied;
                if (any_tied) {
#pragma unroll 1
                    for (int u = 0; u < SB; ++u) {
                        const uint32_t c1 = u == 0 ? cd[0] : u == 1 ? cd[1] : u == 2 ? cd[2] : cd[3];
                        const float g1 = u == 0 ? g[0] : u == 1 ? g[1] : u == 2 ? g[2] : g[3];
                        if (c1 == kTied) {
                            const long long i = COLS ? s0 + ss + u : r0 + tid, j = COLS ? r0 + tid : s0 + ss + u;
                            scatter_tied(mine, P.x1 + (b * P.N1 + i) * P.D, P.x2 + (b * P.N2 + j) * P.D, P.fwd[(b * P.N1 + i) * P.N2 + j],
                                         g1, k0, kn, COLS);
                        } else if (c1 != kSkip) {
                            const int kk = (int)(c1 & 0xffffu) - k0;
                            if ((unsigned)kk < (unsigned)kn)
                                mine[kk] += __uint_as_float(__float_as_uint(g1) ^ ((c1 ^ (COLS ? 0x80000000u : 0u)) & 0x80000000u));
                        }
                    }
                    continue;
                }
#pragma unroll
                for (int u = 0; u < SB; ++u) {
                    // kSkip's low half is 65535, which is no feature (D < 65536): it lands in the spare word too
                    const unsigned kk = (cd[u] & 0xffffu) - (unsigned)k0;
                    k[u] = (int)min(kk, (unsigned)kn);
                    g[u] = __uint_as_float(__float_as_uint(g[u]) ^ ((cd[u] ^ (COLS ? 0x80000000u : 0u)) & 0x80000000u));
                    v[u] = mine[k[u]];
                }
#pragma unroll
                for (int u = 0; u < SB; ++u) {
#pragma unroll
                    for (int w = 0; w < u; ++w)
                        if (k[w] == k[u]) v[u] = v[w];
                    v[u] += g[u];
                }
#pragma unroll
                for (int u = 0; u < SB; ++u) mine[k[u]] = v[u];
            }
        }
    }
    __syncthreads();
    float *out = P.out + b * P.NR * P.D;
    for (int rr = tid / 32; rr < SR; rr += STHR / 32) {
        const long long row = r0 + rr;
        if (row >= P.NR) break;
        for (int k = tid % 32; k < kn; k += 32) out[row * P.D + k0 + k] = accs[rr * stride + k];
    }
}

constexpr long long kHeader = 256;   // the counter of marked pairs, padded so that the codes start on an aligned address

} // namespace
} // namespace tpw

using namespace tpw;

extern "C" int64_t tpw_chebyshev_backward_scratch_bytes(int dtype, int64_t B, int64_t N1, int64_t N2, int64_t D) {
    if (dtype != TPW_F32 || B <= 0 || N1 <= 0 || N2 <= 0 || D < 16 || D >= 65536) return 0;
    if (N1 >= (1ll << 31) || N2 >= (1ll << 31) || B >= (1ll << 31)) return 0;
    return kHeader + 4 * B * N1 * N2;
}

extern "C" int tpw_chebyshev_backward_ws(const void *grad, const void *out, const void *x1, const void *x2,
                                         void *grad_x1, void *grad_x2, void *scratch, int64_t scratch_bytes,
                                         int64_t B, int64_t N1, int64_t N2, int64_t D, tpw_stream_t stream) {
    clear_error();
    const int64_t need = tpw_chebyshev_backward_scratch_bytes(TPW_F32, B, N1, N2, D);
    TPW_CHECK_ARG(need > 0, "tpw_chebyshev_backward_ws: this problem is served by tpw_lp_backward (scratch query returned 0)");
    TPW_CHECK_ARG(scratch != nullptr && scratch_bytes >= need, "tpw_chebyshev_backward_ws: scratch too small (%lld < %lld)",
                  (long long)scratch_bytes, (long long)need);
    TPW_CHECK_ARG(aligned16(scratch), "tpw_chebyshev_backward_ws: scratch must be 16-byte aligned");
    TPW_CHECK_ARG(grad && out && x1 && x2, "tpw_chebyshev_backward_ws: NULL input");
    if (!grad_x1 && !grad_x2) return TPW_OK;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    unsigned long long *ties = static_cast<unsigned long long *>(scratch);
    uint32_t *code = reinterpret_cast<uint32_t *>(static_cast<unsigned char *>(scratch) + kHeader);
    TPW_CUDA_OK(cudaMemsetAsync(ties, 0, kHeader, s));

    MatchParams M;
    memset(&M, 0, sizeof(M));
    M.x1 = static_cast<const float *>(x1); M.x2 = static_cast<const float *>(x2); M.out = static_cast<const float *>(out);
    M.code = code; M.ties = ties;
    M.B = B; M.N1 = N1; M.N2 = N2; M.D = D;
    M.tiles_i = (N1 + TI - 1) / TI; M.tiles_j = (N2 + TJ - 1) / TJ;
    M.status = device_status_ptr();
    const long long tiles = B * M.tiles_i * M.tiles_j;
    TPW_CHECK_ARG(tiles < (1ll << 31), "tpw_chebyshev_backward_ws: too many tiles (%lld)", tiles);
    const bool tma_ok = !tma_disabled() && aligned16(x1) && aligned16(x2) && (D * 4) % 16 == 0;
    CUtensorMap m1, m2;
    memset(&m1, 0, sizeof(m1));
    memset(&m2, 0, sizeof(m2));
    if (tma_ok) {
        int st = make_tensor_map_3d(&m1, x1, 4, D, N1, B, KC, TI, true);
        if (st != TPW_OK) return st;
        st = make_tensor_map_3d(&m2, x2, 4, D, N2, B, KC, TJ, true);
        if (st != TPW_OK) return st;
        TPW_CUDA_OK(cudaFuncSetAttribute(chebyshev_match_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, MATCH_SMEM));
        chebyshev_match_kernel<true><<<(unsigned)tiles, kThreads, MATCH_SMEM, s>>>(m1, m2, M);
    } else {
        TPW_CUDA_OK(cudaFuncSetAttribute(chebyshev_match_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, MATCH_SMEM));
        chebyshev_match_kernel<false><<<(unsigned)tiles, kThreads, MATCH_SMEM, s>>>(m1, m2, M);
    }
    TPW_LAUNCH_OK("chebyshev_match_kernel");

    ScatterParams S;
    memset(&S, 0, sizeof(S));
    S.grad = static_cast<const float *>(grad); S.code = code; S.ties = ties;
    S.x1 = M.x1; S.x2 = M.x2; S.fwd = M.out;
    S.B = B; S.N1 = N1; S.N2 = N2; S.D = D;
    S.tiles_k = (D + SD - 1) / SD;
    // the limit belongs to the kernel, not to the call: always the largest, so that threads with other feature counts may launch
    const int smem = scatter_smem(D < SD ? (int)D : SD);
    if (grad_x1) {
        S.out = static_cast<float *>(grad_x1); S.NR = N1; S.tiles_r = (N1 + SR - 1) / SR;
        const long long n = B * S.tiles_r * S.tiles_k;
        TPW_CHECK_ARG(n < (1ll << 31), "tpw_chebyshev_backward_ws: too many row blocks");
        TPW_CUDA_OK(cudaFuncSetAttribute(chebyshev_scatter_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, scatter_smem(SD)));
        chebyshev_scatter_kernel<false><<<(unsigned)n, STHR, smem, s>>>(S);
        TPW_LAUNCH_OK("chebyshev_scatter_kernel (grad_x1)");
    }
    if (grad_x2) {
        S.out = static_cast<float *>(grad_x2); S.NR = N2; S.tiles_r = (N2 + SR - 1) / SR;
        const long long n = B * S.tiles_r * S.tiles_k;
        TPW_CHECK_ARG(n < (1ll << 31), "tpw_chebyshev_backward_ws: too many row blocks");
        TPW_CUDA_OK(cudaFuncSetAttribute(chebyshev_scatter_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, scatter_smem(SD)));
        chebyshev_scatter_kernel<true><<<(unsigned)n, STHR, smem, s>>>(S);
        TPW_LAUNCH_OK("chebyshev_scatter_kernel (grad_x2)");
    }
    // tied maxima everywhere: the dense kernel writes both gradients; otherwise it returns at once
    return lp_backward_cdist_inf_if(ties, tie_limit(B * N1 * N2), grad, out, x1, x2, grad_x1, grad_x2, B, N1, N2, D, s);
}
