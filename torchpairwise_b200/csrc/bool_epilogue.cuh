// Contingency-table epilogue of the boolean metrics, shared by the popcount kernels (bool_popcount.cu) and the
// tensor-core count kernel (bool_tcgen05.cu): from the exact integers n11 = |x & y|, |x|, |y| and D to the requested
// metric with the float32 operation order of the reference's tensor compositions (OPS/pairwise_metrics.cpp:206-399),
// every *, +, -, / rounded separately, so that the float32 output is bit-identical whichever kernel counted.
#pragma once
#include "common.cuh"
#include "packed_f32x2.cuh"

namespace tpw {
namespace {

// int -> float for 0 <= v < 2^23.  The conversion instruction issues at a quarter of the arithmetic rate; placing
// the integer in the mantissa of 2^23 and subtracting 2^23 gives the same exact value with one logic operation and
// one add.  FAST is set by the few-words kernel, where the conversions are a large share of the work per pair.
template <bool FAST>
__device__ __forceinline__ float count_to_float(int v) {
    return FAST ? __int_as_float(0x4B000000 | v) - 8388608.f : (float)v;
}

// x / y rounded to nearest for integers 0 <= x, 0 < y < 2^18 with the quotient at most 1, given an approximate reciprocal r of
// y (2 ulp): one Newton step on the quotient with an exact residual (P. Markstein, "Computation of elementary functions on the
// IBM RISC System/6000 processor", 1990).  q = x r is within a few ulp of x / y, x - q y is exact in a fused multiply-add, and the sum
// q + (x - q y) r is, before its one rounding, within 2^-20 ulp of x / y.  A quotient of integers below 2^18 that is not
// itself a float lies at least 2^-19 ulp from every rounding boundary, so the rounding is that of x / y.  Four instructions
// without a branch: jaccard [65536, 16384, 1024] 1.62 -> 1.41 ms.
__device__ __forceinline__ float quotient_of_counts(float x, float y, float r) {
    const float q = __fmul_rn(x, r);
    return __fmaf_rn(__fmaf_rn(-q, y, x), r, q);
}
constexpr int kQuotientMax = 1 << 18;
__device__ __forceinline__ float approximate_reciprocal(float y) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(y));
    return r;
}

// INV: -1 = decide per call from inv_d, 1 = D is a power of two and inv_d its reciprocal, 0 = divide, 2 = D is below kQuotientMax
// and inv_d an approximate reciprocal of it (the means), or any value (jaccard): quotients as above.  A caller that
// knows which holds for a whole tile passes it as a constant: decided per element, the division sequence is
// if-converted and executed next to the multiplication for every element.
template <bool FAST = false, int INV = -1>
__device__ __forceinline__ float bool_epilogue(int metric, int n11, int a, int b, int D, float inv_d) {
    const int nxor_i = a + b - 2 * n11;
    const int nor_i = a + b - n11;
    const float fand = count_to_float<FAST>(n11), fxor = count_to_float<FAST>(nxor_i), f_or = count_to_float<FAST>(nor_i);
    const float feq = count_to_float<FAST>(D - nxor_i), fD = count_to_float<FAST>(D);
    switch (metric) {
        case TPW_BOOL_AND_SUM: return fand;
        case TPW_BOOL_OR_SUM: return f_or;
        case TPW_BOOL_XOR_SUM:
        case TPW_BOOL_NE_SUM: return fxor;
        case TPW_BOOL_EQ_SUM: return feq;
        // dividing by a power of two is exact, and so is multiplying by its reciprocal
        case TPW_BOOL_EQ_MEAN:
            if (INV == 1) return __fmul_rn(feq, inv_d);
            if (INV == 0) return __fdiv_rn(feq, fD);
            if (INV == 2) return quotient_of_counts(feq, fD, inv_d);
            return inv_d != 0.f ? __fmul_rn(feq, inv_d) : __fdiv_rn(feq, fD);
        case TPW_BOOL_NE_MEAN:
            if (INV == 1) return __fmul_rn(fxor, inv_d);
            if (INV == 0) return __fdiv_rn(fxor, fD);
            if (INV == 2) return quotient_of_counts(fxor, fD, inv_d);
            return inv_d != 0.f ? __fmul_rn(fxor, inv_d) : __fdiv_rn(fxor, fD);
        case TPW_BOOL_JACCARD:
            if (INV == 2) return f_or != 0.f ? quotient_of_counts(fxor, f_or, approximate_reciprocal(f_or)) : 0.f;
            return f_or != 0.f ? __fdiv_rn(fxor, f_or) : 0.f;
        case TPW_BOOL_KULSINSKI: return __fdiv_rn(__fadd_rn(__fsub_rn(fxor, fand), fD), __fadd_rn(fxor, fD));
        case TPW_BOOL_KULCZYNSKI1: return __fdiv_rn(fand, fxor);
        case TPW_BOOL_YULE: {
            const float half_r = __fmul_rn(count_to_float<FAST>(a - n11), count_to_float<FAST>(b - n11));
            const float den = __fadd_rn(__fmul_rn(fand, count_to_float<FAST>(D - nor_i)), half_r);
            return den != 0.f ? __fdiv_rn(__fmul_rn(2.f, half_r), den) : 0.f;
        }
        case TPW_BOOL_DICE: return __fdiv_rn(fxor, __fadd_rn(__fmul_rn(2.f, fand), fxor));
        case TPW_BOOL_ROGERSTANIMOTO:
        case TPW_BOOL_SOKALMICHENER: {
            const float r2 = __fmul_rn(2.f, fxor);
            return __fdiv_rn(r2, __fadd_rn(feq, r2));
        }
        case TPW_BOOL_RUSSELLRAO: return __fdiv_rn(__fsub_rn(fD, fand), fD);
        case TPW_BOOL_SOKALSNEATH: {
            const float r2 = __fmul_rn(2.f, fxor);
            return __fdiv_rn(r2, __fadd_rn(fand, r2));
        }
        default: return 0.f;
    }
}

// The same values for two pairs at a time, two lanes to an instruction, with every count held as a float: for the metrics that
// need no more than |x & y|, |x| + |y| and one quotient, and D < 2^18.  All sums are integers below 2^24 and therefore exact, and
// the quotient is quotient_of_counts, so the results are bool_epilogue's bit for bit; 6.5 arithmetic instructions per jaccard
// distance where the integer form takes 14, and 4 for a mean where D is no power of two.
// n0, n1: the two counts as integers; a2: |x| in both lanes; b2: |y| of the two columns.
constexpr bool has_packed_epilogue(int metric) {
    return metric == TPW_BOOL_AND_SUM || metric == TPW_BOOL_OR_SUM || metric == TPW_BOOL_XOR_SUM || metric == TPW_BOOL_NE_SUM ||
           metric == TPW_BOOL_EQ_SUM || metric == TPW_BOOL_EQ_MEAN || metric == TPW_BOOL_NE_MEAN || metric == TPW_BOOL_JACCARD;
}
template <int METRIC>
constexpr bool kPackedEpilogue = has_packed_epilogue(METRIC);
template <int METRIC, int INV>
__device__ __forceinline__ f32x2 bool_epilogue_packed(uint32_t n0, uint32_t n1, f32x2 a2, f32x2 b2, float D, float inv_d) {
    const float kMagic = 8388608.f;   // 2^23: its mantissa takes a count as it is
    const f32x2 magic = pack2(kMagic, kMagic);
    const f32x2 m = pack2(__uint_as_float(0x4B000000u | n0), __uint_as_float(0x4B000000u | n1));   // 2^23 + n
    const f32x2 D2 = pack2(D, D), inv2 = pack2(inv_d, inv_d);
    if (METRIC == TPW_BOOL_AND_SUM) return sub2(m, magic);
    if (METRIC == TPW_BOOL_OR_SUM) return sub2(add2(add2(a2, magic), b2), m);
    if (METRIC == TPW_BOOL_JACCARD) {
        // - (|x| + |y| - n), as the residual below takes it, and 2 (|x| + |y| - n) - |x| - |y|
        const f32x2 nor = sub2(m, add2(add2(a2, magic), b2));
        const f32x2 fxor = sub2(fma2(nor, pack2(-2.f, -2.f), sub2(pack2(0.f, 0.f), a2)), b2);
        float y0, y1;
        unpack2(nor, y0, y1);
        y0 = fminf(y0, -1.f);   // two empty rows: 0 / 1 in the place of 0 / 0, which the metric defines as 0
        y1 = fminf(y1, -1.f);
        const f32x2 r = pack2(approximate_reciprocal(-y0), approximate_reciprocal(-y1));
        const f32x2 qt = mul2(fxor, r);
        return fma2(fma2(qt, pack2(y0, y1), fxor), r, qt);
    }
    // |x| + |y| - 2 n
    const f32x2 fxor = fma2(sub2(m, magic), pack2(-2.f, -2.f), add2(a2, b2));
    if (METRIC == TPW_BOOL_XOR_SUM || METRIC == TPW_BOOL_NE_SUM) return fxor;
    const f32x2 x = METRIC == TPW_BOOL_EQ_SUM || METRIC == TPW_BOOL_EQ_MEAN ? sub2(D2, fxor) : fxor;
    if (METRIC == TPW_BOOL_EQ_SUM) return x;
    const f32x2 qt = mul2(x, inv2);
    if (INV == 1) return qt;
    return fma2(fma2(qt, pack2(-D, -D), x), inv2, qt);
}

} // namespace
} // namespace tpw
