// FP64-accurate products on the FP16 tensor cores: operands as 55-bit block-fixed-point
// numbers of 7 balanced base-256 digits, digit products summed exactly in FP32 accumulators
// (see okg_split64.cu).  The pieces shared by the kernels that use them.
#pragma once
#include <cuda_fp16.h>

#include "okg_split64.cuh"
#include "okg_tc.cuh"

namespace okg {
namespace sp {

using namespace mx;

constexpr int ND = 7;                   // digits of an operand
constexpr int PK = OKG_SPLIT_PK;        // columns of a panel: one MMA K-step
constexpr int DT = 128 * PK * 2;        // bytes of one digit of one 128-row operand tile
constexpr int ROW_NAN = 30000, ROW_ZERO = 30001;  // row exponents of points without finite values
constexpr int MO_NAN = 200000;                    // exponent of a column with coefficients out of range

// v = t 2^(E - 55), t rounded to an integer of 7 balanced base-256 digits; returned
// biased by 128 per digit (byte b holds digit + 128), rs0 = E + 1030.  Integer
// instructions only; |v| < 0.99 2^E.
__device__ __forceinline__ uint64_t digits7(double v, int rs0)
{
    const int hi = __double2hiint(v);
    const unsigned lo = (unsigned)__double2loint(v);
    const int ex = (hi >> 20) & 0x7FF;
    const unsigned mh = ((unsigned)hi & 0xFFFFFu) | 0x100000u;
    const uint64_t m = ((uint64_t)__funnelshift_l(lo, mh, 10) << 32) | (uint64_t)(lo << 10);
    int s = rs0 - 1 - ex;
    s = s < 7 ? 7 : s > 63 ? 63 : s;
    const uint64_t q = ((m >> s) + 1) >> 1;
    const uint64_t neg = (uint64_t)(long long)(hi >> 31);
    return ((q ^ neg) - neg) + 0x0080808080808080ull;
}

// Two biased digit bytes (byte b of two values) -> two FP16 digits.
__device__ __forceinline__ uint32_t digit_pair(uint32_t w0, uint32_t w1, int b)
{
    const uint32_t r = (__byte_perm(w0, w1, (uint32_t)(b | (b << 4) | ((4 + b) << 8) | (b << 12))) & 0x00FF00FFu) | 0x64006400u;
    const __half2 h = __hsub2(*reinterpret_cast<const __half2*>(&r), __half2(__ushort_as_half(0x6480), __ushort_as_half(0x6480)));
    return *reinterpret_cast<const uint32_t*>(&h);
}

// byte offset of (row m, column k) in a 128 x 16 FP16 digit tile: M-major, 128-byte
// swizzle (64 rows per 128-byte line, lines of 8 columns per atom)
__device__ __forceinline__ uint32_t a_off(int m, int k)
{
    return (uint32_t)((m >> 6) * 1024 + (k >> 3) * 2048 + (k & 7) * 128 + ((((m >> 3) ^ k) & 7) << 4) + ((m & 7) << 1));
}

// byte offset of (row n, column k) of the coefficient digits: K-major, 32-byte rows,
// 32-byte swizzle
__host__ __device__ __forceinline__ uint32_t b_off(int n, int k)
{
    return (uint32_t)((n >> 3) * 256 + (n & 7) * 32 + ((((k >> 3) ^ (n >> 2)) & 1) << 4) + ((k & 7) << 1));
}

__device__ __forceinline__ uint64_t a_desc(uint32_t addr)
{
    return (uint64_t)((addr >> 4) & 0x3FFF) | ((uint64_t)(1024 >> 4) << 16) | ((uint64_t)(2048 >> 4) << 32) |
           ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}
__device__ __forceinline__ uint64_t b_desc(uint32_t addr)
{
    return (uint64_t)((addr >> 4) & 0x3FFF) | ((uint64_t)1 << 16) | ((uint64_t)(256 >> 4) << 32) | ((uint64_t)1 << 46) |
           ((uint64_t)6 << 61);
}
// kind::f16, A = B = FP16, D = FP32, M-major A, K-major B, M = 128
__host__ __device__ constexpr uint32_t idesc(int n) { return (1u << 4) | (1u << 15) | ((uint32_t)(n >> 3) << 17) | (8u << 24); }

__device__ __forceinline__ void mma_f16(uint32_t d, uint64_t a, uint64_t b, uint32_t id, uint32_t acc)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d),
        "l"(a), "l"(b), "r"(id), "r"(acc));
}

__device__ __forceinline__ void sts16(uint32_t a, unsigned v) { asm volatile("st.shared.u16 [%0], %1;" ::"r"(a), "h"((unsigned short)v) : "memory"); }

// Digits of one column value (value channel alone) into the 7 digit tiles.  A call, like
// put4: the digit code appears once instead of once per component and angular momentum
// (inlined, the kernel's hot code was far beyond the instruction cache: 30 % of its
// instruction requests missed).
static __device__ __noinline__ void put1(double v, int rs, uint32_t a)
{
    const uint64_t t = digits7(v, rs);
    const uint32_t lo = (uint32_t)t, hi = (uint32_t)(t >> 32);
    // digit 0 is the most significant byte (byte 6)
    const uint32_t h20 = digit_pair(hi, hi >> 16, 0), h1 = digit_pair(hi, hi, 1);
    const uint32_t h64 = digit_pair(lo, lo >> 16, 0), h53 = digit_pair(lo, lo >> 16, 1);
    sts16(a + 0 * DT, h20 >> 16);
    sts16(a + 1 * DT, h1);
    sts16(a + 2 * DT, h20);
    sts16(a + 3 * DT, h53 >> 16);
    sts16(a + 4 * DT, h64 >> 16);
    sts16(a + 5 * DT, h53);
    sts16(a + 6 * DT, h64);
}

// Seven accumulators of four MOs (columns n0 .. n0 + 3) of this lane's row.
struct Acc4 {
    uint32_t r[7][4];
};
__device__ __forceinline__ void acc_load(Acc4& a, uint32_t taddr, int np)
{
#pragma unroll
    for (int w = 0; w < 7; ++w)
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
                     : "=r"(a.r[w][0]), "=r"(a.r[w][1]), "=r"(a.r[w][2]), "=r"(a.r[w][3])
                     : "r"(taddr + (uint32_t)(w * np)));
}
// (the loaded registers are operands: no use of them moves before the wait)
__device__ __forceinline__ void acc_wait(Acc4& a)
{
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(a.r[0][0]), "+r"(a.r[0][1]), "+r"(a.r[0][2]), "+r"(a.r[0][3]), "+r"(a.r[1][0]), "+r"(a.r[1][1]), "+r"(a.r[1][2]), "+r"(a.r[1][3]), "+r"(a.r[2][0]), "+r"(a.r[2][1]), "+r"(a.r[2][2]), "+r"(a.r[2][3]), "+r"(a.r[3][0]), "+r"(a.r[3][1]), "+r"(a.r[3][2]), "+r"(a.r[3][3]), "+r"(a.r[4][0]), "+r"(a.r[4][1]), "+r"(a.r[4][2]), "+r"(a.r[4][3]), "+r"(a.r[5][0]), "+r"(a.r[5][1]), "+r"(a.r[5][2]), "+r"(a.r[5][3]), "+r"(a.r[6][0]), "+r"(a.r[6][1]), "+r"(a.r[6][2]), "+r"(a.r[6][3]));
}

__device__ __forceinline__ int f2i(uint32_t r) { return __float2int_rn(__uint_as_float(r)); }

// sum_w acc_w 2^(-8 w) 2^x as an FP64 value, rounded once, in integer arithmetic (a
// conversion on the FP64 pipe would cost its bound): t = sum acc_w 2^(40 - 8 w) in 64
// bits, x = scale - 40 included by the caller.
__device__ __forceinline__ double combine7(const int (&a)[7], int x)
{
    const long long lo = (long long)a[4] * 256 + a[5] + ((a[6] + 128) >> 8);
    const long long t = (((long long)(a[0] * 256 + a[1])) << 32) + ((long long)(a[2] * 256 + a[3]) << 16) + lo;
    const unsigned long long neg = (unsigned long long)(t >> 63);
    const unsigned long long u = ((unsigned long long)t ^ neg) - neg;
    const int lz = __clzll((long long)u);
    const unsigned long long n = u << (lz & 63);
    const unsigned long long m = (n >> 11) + ((n >> 10) & 1);  // 53 bits, rounded
    const int e = 1023 + 63 - lz + x;                          // biased exponent of the leading bit
    if (u == 0 || e <= 0) return 0.0;
    if (e >= 0x7FF) return __hiloint2double((int)(0x7FF00000u | (unsigned)(neg & 0x80000000u)), 0);
    const unsigned long long bits = ((unsigned long long)(unsigned)(e - 1) << 52) + m;
    return __longlong_as_double((long long)(bits | (neg & 0x8000000000000000ull)));
}

// Accumulators of four MOs -> FP64 values of this lane's row.
__device__ __forceinline__ void acc_values(const Acc4& a, int rowx, const int4& f4, double (&v)[4])
{
    const int f[4] = {f4.x, f4.y, f4.z, f4.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int t[7] = {f2i(a.r[0][i]), f2i(a.r[1][i]), f2i(a.r[2][i]), f2i(a.r[3][i]), f2i(a.r[4][i]), f2i(a.r[5][i]), f2i(a.r[6][i])};
        // a = t 2^(E - 55), c = s 2^(F - 55); leading digits weigh 2^48: products 2^(E + F - 14)
        v[i] = combine7(t, rowx + f[i] - 54);
    }
}

__device__ __forceinline__ double shfl_d(double v, int src)
{
    return __hiloint2double(__shfl_sync(0xffffffffu, __double2hiint(v), src),
                            __shfl_sync(0xffffffffu, __double2loint(v), src));
}

// The same for two MOs (half the registers).
struct Acc2 {
    uint32_t r[7][2];
};
__device__ __forceinline__ void acc2_load(Acc2& a, uint32_t taddr, int np)
{
#pragma unroll
    for (int w = 0; w < 7; ++w)
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x2.b32 {%0,%1}, [%2];" : "=r"(a.r[w][0]), "=r"(a.r[w][1]) : "r"(taddr + (uint32_t)(w * np)));
}
__device__ __forceinline__ void acc2_wait(Acc2& a)
{
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(a.r[0][0]), "+r"(a.r[0][1]), "+r"(a.r[1][0]), "+r"(a.r[1][1]), "+r"(a.r[2][0]), "+r"(a.r[2][1]), "+r"(a.r[3][0]), "+r"(a.r[3][1]), "+r"(a.r[4][0]), "+r"(a.r[4][1]), "+r"(a.r[5][0]), "+r"(a.r[5][1]), "+r"(a.r[6][0]), "+r"(a.r[6][1]));
}
__device__ __forceinline__ void acc2_values(const Acc2& a, int rowx, const int2& f2, double (&v)[2])
{
    const int f[2] = {f2.x, f2.y};
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int t[7] = {f2i(a.r[0][i]), f2i(a.r[1][i]), f2i(a.r[2][i]), f2i(a.r[3][i]), f2i(a.r[4][i]), f2i(a.r[5][i]), f2i(a.r[6][i])};
        v[i] = combine7(t, rowx + f[i] - 54);
        if (rowx >= ROW_NAN) v[i] = rowx == ROW_ZERO ? 0.0 : __longlong_as_double(0x7FF8000000000000ll);
    }
}

// Magnitude bits of a largest |v| too large for sums of digit products (a partial sum may
// overflow, or it is not finite), or (vanishing) too small for all digits.
__device__ __forceinline__ bool too_large(unsigned long long top) { return (top >> 52) >= 2023; }
__device__ __forceinline__ bool vanishing(unsigned long long top) { return top != 0 && (top >> 52) < 123; }

// Exponent F with |v| < 0.99 2^F for the magnitude bits `top` of the largest |v| (finite).
__device__ __forceinline__ int scale_of(unsigned long long top)
{
    const int ex = (int)(top >> 52);
    int F = ex == 0 ? -1022 : ex - 1022;
    if (((top >> 44) & 0xFF) >= 0xFA) ++F;
    return F < -900 ? -900 : F;
}

}  // namespace sp
}  // namespace okg
