// Host interface and device tables of the FP64 path on the tensor cores (okg_split64.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <vector>

#define OKG_SPLIT_PK 16     // columns of an operand panel: one MMA K-step
#define OKG_SPLIT_EXP 2048  // entries of the exponential's table

namespace okg {

// A primitive for the radial sums: alpha log2(e) = A 2^ea, w, -2 alpha w, 4 alpha^2 w.
struct alignas(16) SplitPrim {
    uint64_t A;
    int ea, unused;
    double w, w1, w2, neg_alpha;
};

struct SplitDev {
    const int4* shell;      // nshell, panel by panel: {atom, L | first column << 8 | panel << 16, first primitive, primitives}
    const int* panel;       // npanel + 1: first entry of each panel in shell
    const int* col_cart;    // npanel x 16: listed Cartesian row of each column, or -1
    const double* col_g;    // npanel x 16: angular norm of each column times its 2^shift
    const float4* prim_lg;  // nprim: {alpha log2(e), log2 |w|, alpha, 0}, ascending alpha per shell
    const SplitPrim* prim;  // nprim, ascending alpha per shell
    const int* prim_place;  // nprim: place of each sorted primitive in the caller's order
    const uint64_t* exp_tab;  // 2^(63 - j / 2048), rounded
    const int* flags;       // non-zero: a parameter or position out of the tables' range
    int npanel;
};

// One primitive (alpha, w) as the FP64 tensor-core path's bounds and radial sums read it; false
// if it is out of their range, 1e-9 <= alpha <= 1e37 and finite w (such a basis takes the DFMA
// kernels).  With |positions| < 2^29 and alpha >= 1e-9 every AO is exactly zero at
// |coordinate| >= 2^30; above 1e37 alpha log2(e) leaves the range of a float.
__device__ __forceinline__ bool split_prim(double2 p, float4& lg, SplitPrim& o)
{
    // log2 |w| from exponent field and mantissa (|w| beyond the range of a float keeps its size)
    const long long wb = __double_as_longlong(p.y);
    const int we = (int)((wb >> 52) & 0x7FF);
    const float lw = we == 0 ? -3.0e38f
                             : (float)(we - 1023) + log2f((float)__longlong_as_double((wb & 0xFFFFFFFFFFFFFll) | 0x3FF0000000000000ll));
    lg = make_float4((float)(p.x * 1.4426950408889634), lw, (float)p.x, 0.f);
    // alpha log2(e) = A 2^ea with a 64-bit mantissa
    const long long bits = __double_as_longlong(p.x);
    const int ex = (int)((bits >> 52) & 0x7FF);
    const uint64_t m = (((uint64_t)bits & 0xFFFFFFFFFFFFFull) | 0x10000000000000ull) << 11;
    const uint64_t l2e = 0xB8AA3B295C17F0BCull;  // log2(e) 2^63
    uint64_t h = __umul64hi(m, l2e);
    o.ea = ex - 1086 + 1;
    if (!(h >> 63)) {
        h = (h << 1) | ((m * l2e) >> 63);
        --o.ea;
    }
    o.A = h;
    o.unused = 0;
    o.w = p.y;
    o.w1 = -2.0 * p.x * p.y;
    o.w2 = 4.0 * p.x * p.x * p.y;
    o.neg_alpha = -p.x;
    return p.x >= 1.0e-9 && p.x <= 1.0e37 && isfinite(p.y);
}
// e^(-alpha rr) as an FP64 value in integer arithmetic (the FP64 pipe bounds the
// kernels that use it, and an FP64 exponential takes 9 to 18 of its operations, this one
// none).  mr 2^er = rr with a 64-bit mantissa; A 2^ea = alpha log2(e) likewise.
//   u = alpha log2(e) rr from the upper half of mr A, as a fixed-point number with 53
//   fraction bits: integer part k, 11 bits j, remainder f (42 bits);
//   e = 2^-k 2^(-j/2048) 2^-f, 2^(-j/2048) from a table of 64-bit fixed-point numbers
//   (table-driven exponential after P. T. P. Tang, ACM TOMS 15 (1989)) and
//   2^-f = 1 - f (c1 - f (c2 - f (c3 - f c4))), c_n = (ln 2)^n / n! (f < 2^-11: the first
//   term left out is below 2^-65), the inner terms in 32 bits.
// Error before the final rounding: 0.7 2^-53 relative (the truncation of u).
__device__ __forceinline__ double exp_neg(uint64_t mr, int er, uint64_t A, int ea, const uint64_t* __restrict__ tab)
{
    int s = -(er + ea) - 117;
    const uint64_t Y = __umul64hi(mr, A) >> (s > 63 ? 63 : s < 0 ? 0 : s);
    const int k = (int)(Y >> 53);
    const uint64_t T = tab[(unsigned)(Y >> 42) & (OKG_SPLIT_EXP - 1)];
    const uint64_t F = Y << 22;
    const unsigned fh = (unsigned)(F >> 32);
    const unsigned r3 = 3814213304u - (__umulhi(fh, 2643811198u) >> 13);
    const unsigned r2 = 4127059964u - (__umulhi(fh, r3) >> 13);
    const uint64_t c = 0xB17217F7D1CF79ACull - (((uint64_t)fh * r2) >> 13);
    const uint64_t E = T - (__umul64hi(T, __umul64hi(F, c)) >> 11);
    const int lz = __clz((int)(E >> 32));
    const uint64_t n = E << lz;
    const uint64_t m = (n >> 11) + ((n >> 10) & 1);
    const uint64_t bits = m + ((uint64_t)(unsigned)(1022 - lz - k) << 52);
    return (s < 0 || k > 1000) ? 0.0 : __longlong_as_double((long long)bits);
}

// rr >= 0 as mr 2^er, mr with its top bit set (rr = 0: a value far below any exponent's range).
__device__ __forceinline__ void split_mantissa(double rr, uint64_t& mr, int& er)
{
    const unsigned rh = (unsigned)__double2hiint(rr), rl = (unsigned)__double2loint(rr);
    er = (int)(rh >> 20) - 1086;
    mr = ((uint64_t)__funnelshift_l(rl, (rh & 0xFFFFFu) | 0x100000u, 11) << 32) | (uint64_t)(rl << 11);
}
}  // namespace okg
