// Backward of the pairwise L_p reductions in ONE pass over the pairs (float32, CUDA cores).
//
//   grad_x1[b,i,k] =  post * w[b,k] * sum_j coef[b,i,j] * phi(x1[b,i,k] - x2[b,j,k])
//   grad_x2[b,j,k] = -post * w[b,k] * sum_i coef[b,i,j] * phi(x1[b,i,k] - x2[b,j,k])          (phi is odd)
//
// The two-launch form (lp_backward.cu) evaluates the difference and phi once per gradient, 3 operations per pair and
// feature in each launch.  Here a pair's term coef * phi is formed once and added to both sums: 4 operations.
//
// A pass ahead of it (onepass_coef_kernel) turns the upstream gradient and the auxiliary matrix into the coefficients,
// transposed: coefT[b][j][i], rows padded with zeros to a multiple of 4.  The coefficients of two adjacent rows i for one j
// are then one 8-byte word of a tile as TMA delivers it, whatever N2 is, and they are formed once instead of once per
// feature tile: 12 bytes of traffic per pair (0.5 ms at 16 x 4096 x 4096) against a division, a transposition through
// shared memory and a second CTA-wide barrier in every stage of every feature tile.
//
// A CTA of 16 warps owns 256 rows i and 64 features k and walks over all rows j, 32 per stage (TMA, four-stage mbarrier
// ring: the x2 rows and the [32 rows j][256 rows i] coefficient tile).  The warps only meet through the ring: a warp waits
// for a stage to land and reports when it has read it; the stage is refilled two stages behind the slowest warp.  A warp
// owns four features; a thread holds 8 rows i (4 lane, 4 lane + 1, ..., and the same 128 rows further on) x 4 features of
// x1 and of the grad_x1 sums in registers for the whole walk, as packed pairs of adjacent ROWS, so the packed subtract and
// fused multiply-adds take their coefficient pair straight from the tile, and grad_x1 needs no exchange at all.  For
// grad_x2 a thread has the sum over its own 8 rows; it parks the four sums of each row j in a per-warp exchange
// buffer, per four rows j the 32 lanes' contributions to one (j, k) are added in a fixed order, and the CTA's sum over
// its 256 rows goes to a scratch array [B][row blocks][N2][D].  A third kernel adds the row blocks in ascending
// order: no float atomics, every sum in a fixed order, bit-reproducible from run to run.
//
// A CTA's walk is long and there is one CTA per SM, so few blocks, or a last wave of a few, leave SMs idle: the walk is then
// cut into ranges of stages (walk_splits), whose grad_x1 sums go to scratch as well and are added in ascending order.
#include "common.cuh"
#include "lp_backward_phi.cuh"
#include "tcgen05.cuh"

#include <stdlib.h>
#include <string.h>

namespace tpw {
namespace {

constexpr int OP_THREADS = 512;
constexpr int OP_R = 8;           // rows i per thread
constexpr int OP_ROWS = 256;      // rows i per CTA (32 lanes x 8)
constexpr int OP_FEAT = 64;       // features per CTA (16 warps x 4)
constexpr int OP_JT = 32;         // rows j per stage: one 128-byte row of the gradient tile
constexpr int OP_STAGES = 4;
constexpr int OP_AHEAD = 2;       // stages requested ahead of the one in use
constexpr int OP_C_BYTES = OP_JT * OP_ROWS * 4;        // 32 KB of coefficients
constexpr int OP_Y_BYTES = OP_JT * OP_FEAT * 4;        // 8 KB of x2
constexpr int OP_STAGE_BYTES = OP_C_BYTES + OP_Y_BYTES;
constexpr int OP_RED_PITCH = 20;                        // floats per lane in the exchange buffer (16 + 4: conflict-free 16-byte stores)
constexpr int OP_RED_BYTES = 32 * OP_RED_PITCH * 4;    // per warp
constexpr int OP_OFF_RED = OP_STAGES * OP_STAGE_BYTES;
constexpr int OP_OFF_BAR = OP_OFF_RED + (OP_THREADS / 32) * OP_RED_BYTES;   // full[4], empty[4], abort flag
constexpr int OP_SMEM = OP_OFF_BAR + 2 * OP_STAGES * 8 + 8;
constexpr int OP_ALLOC = OP_SMEM + 128;                 // TMA destinations on 128-byte boundaries

struct OnePassParams {
    const float *x1, *x2, *w;
    float *g1, *partial;
    long long B, N1, N2, D;
    long long b0, ib0;           // first batch and first row block of this launch
    long long nib, tiles_k;      // row blocks and feature tiles per batch in this launch
    float *partial1;             // splits > 1: [B][splits][N1][D] sums of grad_x1
    int splits;                  // ranges of stages that share a block's walk
    float q;
    int pow_spec;
    float post;
    int *status;
};

// coefT[lb][j][i - i0] = coefficient of pair (b0 + lb, i, j) for rows i of [i0, i0 + pitch); zero past N1.  64 x 64 pairs per
// CTA through shared memory, whole rows of g and of the auxiliary matrix in, 256-byte row segments out: HBM-bound.
struct CoefParams {
    const float *grad, *aux;
    float *coef;
    long long N1, N2, b0, i0, pitch;
    int vec;                     // N2 % 4 == 0 and 16-byte aligned inputs
    double qd;
};

// COEF: how the coefficient of a pair is formed from the gradient and the auxiliary matrix (COEF_G: the gradient itself)
template <int COEF>
__global__ void __launch_bounds__(256)
onepass_coef_kernel(const CoefParams P) {
    __shared__ float sm[64][65];
    const long long j0 = (long long)blockIdx.x * 64, il0 = (long long)blockIdx.y * 64, b = P.b0 + blockIdx.z;
    const int tid = threadIdx.x;
    const float *grad = P.grad + b * P.N1 * P.N2;
    const float *aux = P.aux + (COEF != COEF_G ? b * P.N1 * P.N2 : 0);
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        const int r = u * 16 + (tid >> 4), c = (tid & 15) * 4;
        const long long i = P.i0 + il0 + r, j = j0 + c;
        float g[4] = {0.f, 0.f, 0.f, 0.f}, o[4] = {0.f, 0.f, 0.f, 0.f};
        if (i < P.N1) {
            if (P.vec) {
                if (j < P.N2) {
                    load4(g, grad + i * P.N2 + j);
                    if (COEF != COEF_G) load4(o, aux + i * P.N2 + j);
                }
            } else {
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (j + e < P.N2) {
                        g[e] = __ldg(grad + i * P.N2 + j + e);
                        if (COEF != COEF_G) o[e] = __ldg(aux + i * P.N2 + j + e);
                    }
            }
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) sm[c + e][r] = COEF != COEF_G ? bwd_coefficient<float>(COEF, g[e], o[e], P.qd) : g[e];
    }
    __syncthreads();
    float *out = P.coef + ((long long)blockIdx.z * P.N2 + j0) * P.pitch + il0;
#pragma unroll
    for (int u = 0; u < 16; ++u) {
        const int jr = u * 4 + (tid >> 6), ir = tid & 63;
        if (j0 + jr < P.N2 && il0 + ir < P.pitch) out[jr * P.pitch + ir] = sm[jr][ir];
    }
}

// coef * phi(x - y) for the metrics whose phi has no packed form
template <int PHI>
__device__ __forceinline__ float onepass_term(float x, float y, float c, float q, int pspec) {
    const float d = x - y;
    if (PHI == PHI_SGN) return d != 0.f ? b_copysign_of(c, d) : 0.f;
    if (PHI == PHI_SGNPOW) return c * b_copysign(pow_abs_spec(fabsf(d), q, pspec), d);
    if (PHI == PHI_D) return c * d;
    return c * (d * fabsf(d));
}

template <int PHI>
__global__ void __launch_bounds__(OP_THREADS, 1)
lp_backward_onepass_kernel(const __grid_constant__ CUtensorMap map_x2, const __grid_constant__ CUtensorMap map_coef,
                           const OnePassParams P) {
    constexpr bool PACKED = (PHI == PHI_DABS || PHI == PHI_D);
    extern __shared__ unsigned char smem_raw[];
    unsigned char *smem = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~uintptr_t(127));
    uint64_t *full = reinterpret_cast<uint64_t *>(smem + OP_OFF_BAR);
    uint64_t *empty = full + OP_STAGES;
    volatile int *abort_flag = reinterpret_cast<volatile int *>(empty + OP_STAGES);

    const int tid = threadIdx.x;
    const int warp = tid >> 5, lane = tid & 31;
    const int kofs = warp * 4;                           // this warp's four features inside the CTA's 64
    float *red = reinterpret_cast<float *>(smem + OP_OFF_RED + warp * OP_RED_BYTES);

    long long tile = blockIdx.x;
    const int sp = (int)(tile % P.splits);
    tile /= P.splits;
    const long long tkx = tile % P.tiles_k;
    tile /= P.tiles_k;
    const long long lib = tile % P.nib, lb = tile / P.nib;   // row block and batch inside this launch (the scratch slot)
    const long long ib = P.ib0 + lib, b = P.b0 + lb;
    const long long i0 = ib * OP_ROWS, k0 = tkx * OP_FEAT;
    const long long kk = k0 + kofs;
    const bool k_ok = kk < P.D;                          // D is a multiple of 4: four features are in or out together

    // x1 rows {i0 + 128 h + 4 lane + e} (h < 2, e < 4) and their sums, resident for the whole walk.  The packed form
    // pairs rows 2m and 2m + 1 of one feature: a pair's two coefficients then lie side by side in the coefficient tile.
    float xr[OP_R][4], acc[OP_R][4];
#pragma unroll
    for (int a = 0; a < OP_R; ++a) {
        const long long row = i0 + (a >> 2) * 128 + lane * 4 + (a & 3);
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (row < P.N1 && k_ok) v = *reinterpret_cast<const float4 *>(P.x1 + (b * P.N1 + row) * P.D + kk);
        xr[a][0] = v.x; xr[a][1] = v.y; xr[a][2] = v.z; xr[a][3] = v.w;
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[a][c] = 0.f;
    }
    f32x2 xr2[PACKED ? OP_R / 2 : 1][4], acc2[PACKED ? OP_R / 2 : 1][4];
    if constexpr (PACKED) {
#pragma unroll
        for (int m = 0; m < OP_R / 2; ++m)
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                xr2[m][c] = pack2(xr[2 * m][c], xr[2 * m + 1][c]);
                acc2[m][c] = 0ull;
            }
    }

    // this CTA's stages [first, first + nchunks) of the walk
    const int all = (int)((P.N2 + OP_JT - 1) / OP_JT), per = (all + P.splits - 1) / P.splits, first = sp * per;
    const int nchunks = first >= all ? 0 : (all - first < per ? all - first : per);
    auto issue = [&](int chunk) {
        unsigned char *base = smem + (chunk % OP_STAGES) * OP_STAGE_BYTES;
        uint64_t *bar = &full[chunk % OP_STAGES];
        mbar_expect_tx(bar, OP_STAGE_BYTES);
        tma_load_3d(base, &map_coef, bar, (int)(lib * OP_ROWS), (first + chunk) * OP_JT, (int)lb);
        tma_load_3d(base + OP_C_BYTES, &map_x2, bar, (int)k0, (first + chunk) * OP_JT, (int)b);
    };
    if (tid == 0) {
#pragma unroll
        for (int s = 0; s < OP_STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], OP_THREADS / 32); }
        *abort_flag = 0;
        mbar_init_fence();
        tma_prefetch_descriptor(&map_x2);
        tma_prefetch_descriptor(&map_coef);
    }
    __syncthreads();
    int issued = 0;                                      // thread 0: chunks requested so far
    if (tid == 0)
        for (; issued < OP_AHEAD && issued < nchunks; ++issued) issue(issued);

    float *part = P.partial + ((lb * P.nib + lib) * P.N2) * P.D;   // this CTA's [N2][D] slab of the scratch
    // after the exchange lanes 0-15 hold the sums of (row j, feature) = (lane >> 2, lane & 3)
    const int o_u = (lane >> 2) & 3;
    const long long okk = kk + (lane & 3);
    for (int t = 0; t < nchunks; ++t) {
        const int stage = t % OP_STAGES;
        if (tid == 0 && issued < nchunks) {
            // the stage to refill held chunk t - (OP_STAGES - OP_AHEAD), which every warp reports when it has read it
            const int use = issued / OP_STAGES;
            if (use > 0 && !wait_or_abort(&empty[issued % OP_STAGES], (uint32_t)((use - 1) & 1), abort_flag)) *abort_flag = 1;
            else { issue(issued); ++issued; }
        }
        __syncwarp();
        const bool landed = wait_or_abort(&full[stage], (uint32_t)((t / OP_STAGES) & 1), abort_flag);
        if (__any_sync(0xffffffffu, !landed)) {
            *abort_flag = 1;
            break;
        }
        const float *ct = reinterpret_cast<const float *>(smem + stage * OP_STAGE_BYTES);
        const float *ys = ct + OP_C_BYTES / 4;

#pragma unroll 1
        for (int jg = 0; jg < OP_JT / 4; ++jg) {
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                float sj[4];
                const int j = jg * 4 + u;
                const float4 yv = *reinterpret_cast<const float4 *>(ys + j * OP_FEAT + kofs);
                const float y[4] = {yv.x, yv.y, yv.z, yv.w};
                if constexpr (PACKED) {
                    f32x2 y2[4], sj2[4];
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        y2[c] = pack2(y[c], y[c]);
                        sj2[c] = 0ull;
                    }
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const float4 cv = *reinterpret_cast<const float4 *>(ct + j * OP_ROWS + h * 128 + lane * 4);
                        const f32x2 c2[2] = {pack2(cv.x, cv.y), pack2(cv.z, cv.w)};
#pragma unroll
                        for (int r = 0; r < 2; ++r)
#pragma unroll
                            for (int c = 0; c < 4; ++c) {
                                f32x2 t2 = sub2(xr2[h * 2 + r][c], y2[c]);
                                if (PHI == PHI_DABS) {
                                    float lo, hi;
                                    unpack2(t2, lo, hi);
                                    t2 = pack2(lo * fabsf(lo), hi * fabsf(hi));
                                }
                                acc2[h * 2 + r][c] = fma2(c2[r], t2, acc2[h * 2 + r][c]);
                                sj2[c] = fma2(c2[r], t2, sj2[c]);
                            }
                    }
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        float lo, hi;
                        unpack2(sj2[c], lo, hi);
                        sj[c] = lo + hi;
                    }
                } else {
#pragma unroll
                    for (int c = 0; c < 4; ++c) sj[c] = 0.f;
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const float4 cv = *reinterpret_cast<const float4 *>(ct + j * OP_ROWS + h * 128 + lane * 4);
                        const float cs[4] = {cv.x, cv.y, cv.z, cv.w};
#pragma unroll
                        for (int r = 0; r < 4; ++r)
#pragma unroll
                            for (int c = 0; c < 4; ++c) {
                                const float term = onepass_term<PHI>(xr[h * 4 + r][c], y[c], cs[r], P.q, P.pow_spec);
                                acc[h * 4 + r][c] += term;
                                sj[c] += term;
                            }
                    }
                }
                // parked in the exchange buffer right away (the previous group's reads ended with a warp barrier)
                *reinterpret_cast<float4 *>(red + lane * OP_RED_PITCH + u * 4) = make_float4(sj[0], sj[1], sj[2], sj[3]);
            }
            // exchange: every lane has written its sums of (4 rows j) x (4 features); lanes l and l + 16 then add the even
            // and the odd lanes' contributions to one (j, feature) in ascending order, and the two are added
            __syncwarp();
            float tot = 0.f;
            const float *src = red + (lane >> 4) * OP_RED_PITCH + (lane & 15);
#pragma unroll
            for (int g = 0; g < 16; ++g) tot += src[2 * g * OP_RED_PITCH];
            tot += __shfl_down_sync(0xffffffffu, tot, 16);
            __syncwarp();
            const long long j = (long long)(first + t) * OP_JT + jg * 4 + o_u;
            if (lane < 16 && j < P.N2 && okk < P.D) part[j * P.D + okk] = tot;
        }
        if (lane == 0) mbar_arrive(&empty[stage]);       // after the warp barrier that ended the last exchange: all lanes have read it
    }
    __syncthreads();
    if (*abort_flag) {
        if (tid == 0) {
            if (P.status) atomicCAS(P.status, 0, (2 << 16) | 3);
            // the last copies may still be landing: the CTA stays (bounded) until they have, so that none of them
            // writes into shared memory the CTA has given back
            for (int c = issued > OP_STAGES ? issued - OP_STAGES : 0; c < issued; ++c)
                mbar_wait_bounded(&full[c % OP_STAGES], (uint32_t)((c / OP_STAGES) & 1));
        }
        return;
    }

    if constexpr (PACKED) {
#pragma unroll
        for (int m = 0; m < OP_R / 2; ++m)
#pragma unroll
            for (int c = 0; c < 4; ++c) unpack2(acc2[m][c], acc[2 * m][c], acc[2 * m + 1][c]);
    }
    if (P.splits > 1) {
        if (!k_ok) return;
        float *dst = P.partial1 + (b * P.splits + sp) * P.N1 * P.D + kk;
#pragma unroll
        for (int a = 0; a < OP_R; ++a) {
            const long long row = i0 + (a >> 2) * 128 + lane * 4 + (a & 3);
            if (row < P.N1) *reinterpret_cast<float4 *>(dst + row * P.D) = make_float4(acc[a][0], acc[a][1], acc[a][2], acc[a][3]);
        }
        return;
    }
    if (k_ok) {
        float4 wv = make_float4(P.post, P.post, P.post, P.post);
        if (P.w) {
            const float4 ww = *reinterpret_cast<const float4 *>(P.w + b * P.D + kk);
            wv.x *= ww.x; wv.y *= ww.y; wv.z *= ww.z; wv.w *= ww.w;
        }
#pragma unroll
        for (int a = 0; a < OP_R; ++a) {
            const long long row = i0 + (a >> 2) * 128 + lane * 4 + (a & 3);
            if (row >= P.N1) continue;
            *reinterpret_cast<float4 *>(P.g1 + (b * P.N1 + row) * P.D + kk) =
                make_float4(acc[a][0] * wv.x, acc[a][1] * wv.y, acc[a][2] * wv.z, acc[a][3] * wv.w);
        }
    }
}

// grad_x2[b,j,k] (+)= -post * w[b,k] * sum over the launch's row blocks, ascending; four features per thread.  grad_x1 of a
// split walk: the same over the splits, with -post for post.
__global__ void __launch_bounds__(256)
lp_backward_onepass_sum_kernel(const float *partial, float *g2, const float *w, long long nb, long long nib, long long b0,
                               long long N2, long long D, float post, int accumulate) {
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long per_batch = N2 * D / 4;
    if (idx >= nb * per_batch) return;
    const long long lb = idx / per_batch, e = idx % per_batch;
    const float4 *src = reinterpret_cast<const float4 *>(partial) + lb * nib * per_batch + e;
    float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
    for (long long ib = 0; ib < nib; ++ib) {
        const float4 v = src[ib * per_batch];
        s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
    }
    const long long b = b0 + lb;
    const long long k = (e * 4) % D;
    s.x *= -post; s.y *= -post; s.z *= -post; s.w *= -post;
    if (w) {
        const float4 ww = *reinterpret_cast<const float4 *>(w + b * D + k);
        s.x *= ww.x; s.y *= ww.y; s.z *= ww.z; s.w *= ww.w;
    }
    float4 *dst = reinterpret_cast<float4 *>(g2) + b * per_batch + e;
    if (accumulate) {
        const float4 o = *dst;
        s.x += o.x; s.y += o.y; s.z += o.z; s.w += o.w;
    }
    *dst = s;
}

constexpr long long kScratchCap = 2ll << 30;
constexpr long long kMaxRows = 65535ll * 64;   // rows of the coefficient pass's grid

// Scratch of one launch over nb batches and nib row blocks: the transposed coefficients, then the grad_x2 slabs.
inline long long coef_pitch(long long N1, long long nib) {
    const long long rows = (N1 + 3) / 4 * 4;
    return nib * OP_ROWS < rows ? nib * OP_ROWS : rows;
}
inline long long unit_bytes(long long N1, long long N2, long long D, long long nib) {
    return N2 * coef_pitch(N1, nib) * 4 + nib * N2 * D * 4;
}

// Ranges of stages the walk is cut into.  One CTA per SM runs ceil(blocks x splits / SMs) waves of walks, each with about two
// stages' worth of time to start and to finish; at least four stages to a range.  The p = 1 backward of
// [1024, 2048, 128] (8 blocks): two launches of one thread per gradient element 290 us, 8 blocks in 16 ranges 90 us.
inline long long walk_splits(long long blocks, long long N2) {
    const long long stages = (N2 + OP_JT - 1) / OP_JT, sms = sm_count();
    long long best = 1, cost = ((blocks + sms - 1) / sms) * (stages + 2);
    for (long long s = 2; s * 4 <= stages && s <= 32; ++s) {
        const long long c = ((blocks * s + sms - 1) / sms) * ((stages + s - 1) / s + 2);
        if (c < cost) { best = s; cost = c; }
    }
    return best;
}
// scratch of the split sums, 0 where the walk is not split: only problems that run as one launch split it
inline long long split_bytes(long long B, long long N1, long long N2, long long D, long long splits) {
    return splits > 1 ? splits * B * N1 * D * 4 : 0;
}

template <int PHI, int COEF>
int launch_onepass(OnePassParams P, double qd, const void *grad, const void *aux, float *g2, void *scratch, long long scratch_bytes,
                   cudaStream_t stream) {
    CUtensorMap mx, mc;
    int st = make_tensor_map_3d(&mx, P.x2, 4, P.D, P.N2, P.B, OP_FEAT, OP_JT, false);
    if (st != TPW_OK) return st;
    auto kern = lp_backward_onepass_kernel<PHI>;
    TPW_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, OP_ALLOC));
    const long long nblk = (P.N1 + OP_ROWS - 1) / OP_ROWS;
    // batches and row blocks per launch: whole batches where one fits, else as many row blocks of one batch as do
    long long bpl = scratch_bytes / unit_bytes(P.N1, P.N2, P.D, nblk), ipl = nblk;
    if (bpl > P.B) bpl = P.B;
    if (bpl > 65535) bpl = 65535;
    if (bpl < 1) {
        bpl = 1;
        ipl = scratch_bytes / unit_bytes(P.N1, P.N2, P.D, 1);
        TPW_CHECK_ARG(ipl >= 1, "lp backward: the scratch holds no row block");
    }
    P.tiles_k = (P.D + OP_FEAT - 1) / OP_FEAT;
    P.status = device_status_ptr();
    P.splits = 1;
    if (bpl == P.B && ipl == nblk) {
        const long long sp = walk_splits(P.B * nblk * P.tiles_k, P.N2), used = P.B * unit_bytes(P.N1, P.N2, P.D, nblk);
        if (used + split_bytes(P.B, P.N1, P.N2, P.D, sp) <= scratch_bytes) P.splits = (int)sp;
        P.partial1 = reinterpret_cast<float *>(static_cast<unsigned char *>(scratch) + used);
    }
    CoefParams C;
    memset(&C, 0, sizeof(C));
    C.grad = reinterpret_cast<const float *>(grad);
    C.aux = reinterpret_cast<const float *>(aux);
    C.coef = reinterpret_cast<float *>(scratch);
    C.N1 = P.N1; C.N2 = P.N2; C.qd = qd;
    C.vec = P.N2 % 4 == 0 && aligned16(grad) && (COEF == COEF_G || aligned16(aux)) ? 1 : 0;
    for (long long b0 = 0; b0 < P.B; b0 += bpl) {
        const long long nb = P.B - b0 < bpl ? P.B - b0 : bpl;
        for (long long ib0 = 0; ib0 < nblk; ib0 += ipl) {
            P.b0 = b0; P.ib0 = ib0;
            P.nib = nblk - ib0 < ipl ? nblk - ib0 : ipl;
            C.b0 = b0; C.i0 = ib0 * OP_ROWS;
            C.pitch = coef_pitch(P.N1 - C.i0, P.nib);
            P.partial = C.coef + nb * P.N2 * C.pitch;
            st = make_tensor_map_3d(&mc, C.coef, 4, C.pitch, P.N2, nb, OP_ROWS, OP_JT, false);
            if (st != TPW_OK) return st;
            const long long gx = (P.N2 + 63) / 64, gy = (C.pitch + 63) / 64;
            TPW_CHECK_ARG(gx < (1ll << 31) && gy <= 65535, "lp backward: too many pairs");
            onepass_coef_kernel<COEF><<<dim3((unsigned)gx, (unsigned)gy, (unsigned)nb), 256, 0, stream>>>(C);
            TPW_LAUNCH_OK("onepass_coef_kernel");
            const long long ctas = nb * P.nib * P.tiles_k * P.splits;
            TPW_CHECK_ARG(ctas < (1ll << 31), "lp backward: too many tiles (%lld)", ctas);
            kern<<<(unsigned)ctas, OP_THREADS, OP_ALLOC, stream>>>(mx, mc, P);
            TPW_LAUNCH_OK("lp_backward_onepass_kernel");
            const long long n4 = nb * P.N2 * P.D / 4;
            lp_backward_onepass_sum_kernel<<<(unsigned)((n4 + 255) / 256), 256, 0, stream>>>(
                P.partial, g2, P.w, nb, P.nib, b0, P.N2, P.D, P.post, ib0 > 0 ? 1 : 0);
            if (P.splits > 1) {
                const long long m4 = P.B * P.N1 * P.D / 4;
                lp_backward_onepass_sum_kernel<<<(unsigned)((m4 + 255) / 256), 256, 0, stream>>>(
                    P.partial1, P.g1, P.w, P.B, P.splits, 0, P.N1, P.D, -P.post, 0);
            }
            TPW_LAUNCH_OK("lp_backward_onepass_sum_kernel");
        }
    }
    return TPW_OK;
}

} // namespace

// 0 where the one-pass kernel does not apply; otherwise the scratch it wants (at most 2 GiB: larger problems run as
// several launches over batch or row-block ranges)
long long lp_backward_onepass_scratch_bytes(int mode, long long B, long long N1, long long N2, long long D, double p) {
    if (getenv("TPW_DISABLE_ONEPASS_BWD") || tma_disabled()) return 0;
    if (mode != TPW_LP_BWD_CDIST && mode != TPW_LP_BWD_PPMINKOWSKI && mode != TPW_LP_BWD_WMINKOWSKI) return 0;
    if (!(p > 0) || isinf(p) || isnan(p)) return 0;
    if (B <= 0 || N1 < OP_ROWS || N2 < OP_JT || D < 16 || D % 4 != 0) return 0;
    if (B >= (1ll << 31) || N1 >= kMaxRows || N2 >= (1ll << 31) || D >= (1ll << 31)) return 0;
    const long long nblk = (N1 + OP_ROWS - 1) / OP_ROWS, tiles_k = (D + OP_FEAT - 1) / OP_FEAT;
    // The two-launch tile has 128 rows and 128 features, so features idle in this tile's 64 idle there too; rows may be idle up
    // to the half of them by which the second launch costs more.  minkowski p = 3, forward and backward: [5, 2910, 1602, 100]
    // 2860 -> 998 us, [6, 384, 663, 192] 318 -> 146 us.
    if (nblk * OP_ROWS * 2 > N1 * 3) return 0;
    // four launches instead of two, and one CTA per SM: from 2^26 terms on, on at least half of the SMs
    if ((double)B * (double)N1 * (double)N2 * (double)D < 67108864.0) return 0;
    const long long splits = walk_splits(B * nblk * tiles_k, N2);
    if (B * nblk * tiles_k * splits * 2 < sm_count()) return 0;
    const long long one = unit_bytes(N1, N2, D, 1), batch = unit_bytes(N1, N2, D, nblk);
    if (one > kScratchCap) return 0;
    if (batch > kScratchCap) return kScratchCap / one * one;
    if (B * batch > kScratchCap) return kScratchCap / batch * batch;
    const long long split = split_bytes(B, N1, N2, D, splits);
    return B * batch + (B * batch + split <= kScratchCap ? split : 0);
}

// the least scratch lp_backward_onepass runs with: one row block of one batch
long long lp_backward_onepass_min_bytes(long long N1, long long N2, long long D) { return unit_bytes(N1, N2, D, 1); }

int lp_backward_onepass(int mode, const void *grad, const void *aux, const void *x1, const void *x2, const void *w,
                        void *grad_x1, void *grad_x2, long long B, long long N1, long long N2, long long D, double p,
                        void *scratch, long long scratch_bytes, cudaStream_t stream) {
    OnePassParams P;
    memset(&P, 0, sizeof(P));
    P.x1 = reinterpret_cast<const float *>(x1);
    P.x2 = reinterpret_cast<const float *>(x2);
    P.g1 = reinterpret_cast<float *>(grad_x1);
    P.B = B; P.N1 = N1; P.N2 = N2; P.D = D;
    const double qd = p - 1.0;
    P.q = (float)(p - 1.0);
    P.pow_spec = make_pow_spec(p - 1.0);
    P.post = 1.f;
    float *g2 = reinterpret_cast<float *>(grad_x2);
    switch (mode) {
        case TPW_LP_BWD_CDIST:
            if (p == 1.0) return launch_onepass<PHI_SGN, COEF_G>(P, qd, grad, nullptr, g2, scratch, scratch_bytes, stream);
            if (p == 2.0) return launch_onepass<PHI_D, COEF_DIV_O>(P, qd, grad, aux, g2, scratch, scratch_bytes, stream);
            if (p == 3.0) return launch_onepass<PHI_DABS, COEF_DIV_O2>(P, qd, grad, aux, g2, scratch, scratch_bytes, stream);
            return launch_onepass<PHI_SGNPOW, COEF_DIV_POW>(P, qd, grad, aux, g2, scratch, scratch_bytes, stream);
        case TPW_LP_BWD_PPMINKOWSKI:
            P.post = (float)p;
            if (p == 1.0) return launch_onepass<PHI_SGN, COEF_G>(P, qd, grad, nullptr, g2, scratch, scratch_bytes, stream);
            if (p == 2.0) return launch_onepass<PHI_D, COEF_G>(P, qd, grad, nullptr, g2, scratch, scratch_bytes, stream);
            if (p == 3.0) return launch_onepass<PHI_DABS, COEF_G>(P, qd, grad, nullptr, g2, scratch, scratch_bytes, stream);
            return launch_onepass<PHI_SGNPOW, COEF_G>(P, qd, grad, nullptr, g2, scratch, scratch_bytes, stream);
        case TPW_LP_BWD_WMINKOWSKI:
            P.w = reinterpret_cast<const float *>(w);
            if (p == 1.0) return launch_onepass<PHI_SGN, COEF_MUL>(P, qd, grad, aux, g2, scratch, scratch_bytes, stream);
            if (p == 2.0) return launch_onepass<PHI_D, COEF_MUL>(P, qd, grad, aux, g2, scratch, scratch_bytes, stream);
            if (p == 3.0) return launch_onepass<PHI_DABS, COEF_MUL>(P, qd, grad, aux, g2, scratch, scratch_bytes, stream);
            return launch_onepass<PHI_SGNPOW, COEF_MUL>(P, qd, grad, aux, g2, scratch, scratch_bytes, stream);
        default:
            return fail(TPW_ERR_INVALID, "lp backward: unknown mode %d", mode);
    }
}

} // namespace tpw
