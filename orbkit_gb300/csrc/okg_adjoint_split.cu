// The adjoint of the density (okg_rho_backward) for up to 64 MOs, as a pipeline over runs of
// grid points with its intermediates in global memory.  Why: a point needs 8 NMO NAO FMAs
// (MOs, A, B, dC below) and the FP64 pipe runs 2 per clock and SM, so the one-kernel form
// (okg_adjoint.cu) is bound by it, while a double written to and read back from HBM costs as
// much as three FP64 operations.  Notation as in okg_adjoint.cu:
//   1. W_i, V_i (cotangents of the MOs) from the tensor-core density kernel (okg_split64.cu);
//   2. A_k = sum_i C_ik W_i, B_k = sum_i C_ik V_i: exact digit products on the tensor cores;
//   3. shell_kernel: one warp per shell and run of points; radial sums and polynomials once,
//      chi_k and G_k = sum_d g_d d_d chi_k written for step 4, the exponent, coefficient and
//      nuclear terms summed over the points in registers:
//        Pa = sum_k A_k g_k P_k, Pb = sum_k B_k g_k P_k, F = Pa + g . grad Pb, T = (g . X) Pb,
//        dL/dR_u    = -sum_r R0 (d_u Pa + sum_d H_ud g_d) + S1 (F X_u + (g.X) d_u Pb + Pb g_u) + S2 X_u T,
//                     H = Hessian of Pb, S1 = -2 R1, S2 = 4 R2,
//        dL/dalpha  = w' U0 - w U1 - 2 w U2,  dL/dc = N U0,  with y = F - 2 alpha T and
//        U0 = sum_r e y, U1 = sum_r r^2 e y, U2 = sum_r e T   (e = exp(-alpha r^2));
//   4. dC_ik = sum_r W_i chi_k + V_i G_k: digit products with the points as the summed index,
//      64 points per accumulation, FP64 sums of those;
//   5. partial sums added in a fixed order.
// What the digits cannot hold (values that are not finite, a call that step 1 gives up), and a
// wait that expires, raises the call's redo word, and the one-kernel form, launched at the end, computes the call.
// FP32 precision: W, V, A, B, chi and G are floats, the products of steps 2 and 4 take 4
// digits (31 bits), step 3 computes in FP32.
//
// Measured (12 atoms, 51 shells, 40 MOs), us per step, FP64 at 64^3 points | FP32 at 104 x 96 x 101
// (two runs): 1: 815 | 3910, 2: 492 | 850, 3: 3080 | 1870, 4: 695 | 1840, 5: 22 | 36.  Forward
// and backward together: 28.0 -> 5.9 ms | 13.1 -> 9.1 ms with the one-kernel form -> this.
// FP64 is bound by step 3 and that by the FP64 pipe (85 % busy; 116 instructions per shell
// and 32 points at 16 cycles each are 2.7 ms); FP32 by step 1, which is the FP64 density kernel
// with the results as floats.
#include "okg_digits.cuh"
#include "okg_internal.cuh"

namespace okg {
namespace adjs {

using namespace sp;

constexpr int NMO_MAX = 64;

// Which calls take this pipeline: bases within the tables of step 1, up to 64 MOs (one
// accumulator set of the column kernel), and in FP32 at least 2048 points.  Backward pass, one-kernel form | pipeline, us, FP64: 3 atoms, 5 MOs
// and 50 points 215 | 158, 20 atoms, 60 MOs and 50 points 1679 | 333; FP32: 3 atoms and 500
// points 106 | 152, 3000 points 225 | 156; 12 atoms, 40 MOs and 500 points 198 | 275, 3000 points
// 315 | 282; 20 atoms and 500 points 457 | 397, 3000 points 574 | 412.
static bool takes(const okg_basis* b, long long npts, int nmo, int precision)
{
    return split_basis(b) && nmo <= NMO_MAX && npts >= (precision == 32 ? 2048 : 1);
}

// Digit operands of the intermediates: doubles as 7 digits (55 bits), floats as 4 (31 bits,
// 10 digit products instead of 28), both with the leading digit of weight 2^(E - 7).
template <typename T>
struct Dg;

template <>
struct Dg<double> {
    static constexpr int D = 7;
    using U = unsigned long long;
    static __device__ __forceinline__ U magnitude(double v) { return (U)__double_as_longlong(v) & 0x7FFFFFFFFFFFFFFFull; }
    static __device__ __forceinline__ bool special(U m) { return too_large(m); }
    static __device__ __forceinline__ int scale(U m) { return scale_of(m); }
    static __device__ __forceinline__ U shfl_max(U m, int o)
    {
        const U u = __shfl_xor_sync(0xffffffffu, m, o);
        return u > m ? u : m;
    }
    // digits at a, a + stride, ...
    static __device__ __forceinline__ void put(double v, int E, uint32_t a, uint32_t stride)
    {
        const uint64_t t = digits7(v, E + 1030);
        const uint32_t lo = (uint32_t)t, hi = (uint32_t)(t >> 32);
        const uint32_t h20 = digit_pair(hi, hi >> 16, 0), h1 = digit_pair(hi, hi, 1);
        const uint32_t h64 = digit_pair(lo, lo >> 16, 0), h53 = digit_pair(lo, lo >> 16, 1);
        sts16(a, h20 >> 16);
        sts16(a + stride, h1);
        sts16(a + 2 * stride, h20);
        sts16(a + 3 * stride, h53 >> 16);
        sts16(a + 4 * stride, h64 >> 16);
        sts16(a + 5 * stride, h53);
        sts16(a + 6 * stride, h64);
    }
};

template <>
struct Dg<float> {
    static constexpr int D = 4;
    using U = unsigned;
    static __device__ __forceinline__ U magnitude(float v) { return __float_as_uint(v) & 0x7FFFFFFFu; }
    static __device__ __forceinline__ bool special(U m) { return (m >> 23) >= 0xF8; }
    static __device__ __forceinline__ int scale(U m)
    {
        const int ex = (int)(m >> 23);
        return ex == 0 ? -126 : ex - 126 + (((m >> 15) & 0xFF) >= 0xFA ? 1 : 0);
    }
    static __device__ __forceinline__ U shfl_max(U m, int o) { return max(m, __shfl_xor_sync(0xffffffffu, m, o)); }
    // v = t 2^(E - 31), t rounded, 4 balanced base-256 digits
    static __device__ __forceinline__ void put(float v, int E, uint32_t a, uint32_t stride)
    {
        const unsigned u = __float_as_uint(v);
        const int s = E + 126 - (int)((u >> 23) & 0xFF);
        const unsigned m = (u << 8) | 0x80000000u;
        // (from s = 32 on v is below half a unit: the mantissa's leading bit is gone too)
        const unsigned q = s > 31 ? 0u : ((m >> (s < 0 ? 0 : s)) + 1) >> 1;
        const unsigned neg = (unsigned)((int)u >> 31);
        const unsigned t = ((u & 0x7F800000u) ? ((q ^ neg) - neg) : 0u) + 0x80808080u;
        const uint32_t h20 = digit_pair(t, t >> 16, 1), h31 = digit_pair(t, t >> 16, 0);  // bytes 1 | 3, 0 | 2
        sts16(a, h20 >> 16);
        sts16(a + stride, h31 >> 16);
        sts16(a + 2 * stride, h20);
        sts16(a + 3 * stride, h31);
    }
};

// Accumulators of four columns (D weights) -> FP64 values of this lane's row.
template <int D>
struct AccN {
    uint32_t r[D][4];
};
template <int D>
__device__ __forceinline__ void acc_get(AccN<D>& a, uint32_t taddr, int np)
{
#pragma unroll
    for (int w = 0; w < D; ++w)
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
                     : "=r"(a.r[w][0]), "=r"(a.r[w][1]), "=r"(a.r[w][2]), "=r"(a.r[w][3])
                     : "r"(taddr + (uint32_t)(w * np)));
    // (the loaded registers are operands of the wait: no use of them moves before it)
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int w = 0; w < D; ++w)
        asm volatile("" : "+r"(a.r[w][0]), "+r"(a.r[w][1]), "+r"(a.r[w][2]), "+r"(a.r[w][3]));
}
template <int D>
__device__ __forceinline__ void acc_doubles(const AccN<D>& a, int rowx, const int4& f4, double (&v)[4])
{
    const int f[4] = {f4.x, f4.y, f4.z, f4.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        int t[7];
#pragma unroll
        for (int w = 0; w < 7; ++w) t[w] = w < D ? f2i(a.r[w < D ? w : 0][i]) : 0;
        v[i] = combine7(t, rowx + f[i] - 54);
    }
}
// ... as floats: 4 weights, sums below 2^22, so the upper and lower pair are exact in 32 bits
__device__ __forceinline__ void acc_floats(const AccN<4>& a, int rowx, const int4& f4, float (&v)[4])
{
    const int f[4] = {f4.x, f4.y, f4.z, f4.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int hi = f2i(a.r[0][i]) * 256 + f2i(a.r[1][i]), lo = f2i(a.r[2][i]) * 256 + f2i(a.r[3][i]);
        const float t = fmaf((float)hi, 65536.0f, (float)lo);
        // t 2^(E + F - 38) in two exact steps (either alone may leave the exponent range)
        int x = rowx + f[i] - 38;
        x = x < -250 ? -250 : x > 250 ? 250 : x;
        const int x1 = x / 2, x2 = x - x1;
        v[i] = t * __int_as_float((127 + x1) << 23) * __int_as_float((127 + x2) << 23);
    }
}

// Double to float without the FP64 pipe (round to nearest, results below 2^-126 to zero).
__device__ __forceinline__ float narrow(double d)
{
    const unsigned long long u = (unsigned long long)__double_as_longlong(d) + 0x10000000ull;
    const unsigned hi = (unsigned)(u >> 32), lo = (unsigned)u, e = (hi >> 20) & 0x7FF;
    const unsigned long long m = (unsigned long long)__double_as_longlong(d) & 0x7FFFFFFFFFFFFFFFull;
    if (m > 0x7FF0000000000000ull) return __uint_as_float(0x7FC00000u);
    if (e >= 1151u) return __uint_as_float((hi & 0x80000000u) | 0x7F800000u);
    if (e <= 896u) return 0.0f;
    return __uint_as_float((hi & 0x80000000u) | ((e - 896u) << 23) | ((hi & 0xFFFFFu) << 3) | (lo >> 29));
}
template <typename T>
__device__ __forceinline__ T as(double d);
template <>
__device__ __forceinline__ double as<double>(double d) { return d; }
template <>
__device__ __forceinline__ float as<float>(double d) { return narrow(d); }

// ------------------------------------------------------------------ step 2
// out[z][n][p] = sum_a C[a][n] X[z][a][p]  (z: W -> A, V -> B); a < nmo <= 64, n in passes of
// NP columns.  A CTA keeps the digits of its pass's coefficients in shared memory and walks
// tiles of 128 points, G threads per point; the next tile's MO cotangents are loaded before
// the accumulators are read.
template <typename T>
struct ColArgs {
    long long npts, ld;
    const T* X;        // 2 x nmo x ld
    const double* C;   // nmo x ncart
    int nmo, ncart, kp;
    T* out;            // 2 x ncart x ld
    int* redo;         // raised where a value is not finite or a wait expires
    long long limit;   // polls of a wait
};

template <typename T>
struct ColCfg {
    static constexpr int NP = 64, D = Dg<T>::D;
    // floats: 4 x 64 accumulator columns, two CTAs of 256 threads per SM
    static constexpr int G = D == 4 ? 2 : 4, CTAS = D == 4 ? 2 : 1, TM = D == 4 ? 256 : 512;
    static size_t smem(int kp) { return 1024 + (size_t)kp * (D * DT + D * NP * 32) + G * 128 * 8 + NP * 4 + 64; }
};

template <typename T>
__global__ void __launch_bounds__(128 * ColCfg<T>::G, ColCfg<T>::CTAS) column_kernel(const __grid_constant__ ColArgs<T> A)
{
    using DG = Dg<T>;
    using U = typename DG::U;
    constexpr int D = DG::D, np = ColCfg<T>::NP, G = ColCfg<T>::G, bpanel = D * np * 32;
    constexpr unsigned TM = ColCfg<T>::TM;
    extern __shared__ unsigned char raw[];
    unsigned char* base = (unsigned char*)(((uintptr_t)raw + 1023) & ~(uintptr_t)1023);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, KP = A.kp;
    const int n_first = blockIdx.y * np, ncol = A.ncart - n_first < np ? A.ncart - n_first : np;
    const T* X = A.X + (long long)blockIdx.z * A.nmo * A.ld;
    T* out = A.out + ((long long)blockIdx.z * A.ncart + n_first) * A.ld;
    unsigned char* Bs = base + (size_t)KP * D * DT;
    U* tops = (U*)(Bs + (size_t)KP * bpanel);  // G x 128
    int* fexp = (int*)(Bs + (size_t)KP * bpanel + G * 128 * 8);
    uint64_t* bar = (uint64_t*)(fexp + np);
    uint32_t* tmem_slot = (uint32_t*)(bar + 1);
    const uint32_t bar_a = smem_u32(bar);
    for (int b = warp; b < np; b += 4 * G) {
        U m = 0;
        for (int a = lane; a < A.nmo && b < ncol; a += 32) {
            const U u = DG::magnitude(as<T>(A.C[(long long)a * A.ncart + n_first + b]));
            m = u > m ? u : m;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) m = DG::shfl_max(m, o);
        const int F = DG::scale(m);
        if (DG::special(m)) *(volatile int*)A.redo = 1;
        if (lane == 0) fexp[b] = F;
        for (int a = lane; a < KP * 16; a += 32)
            DG::put((a < A.nmo && b < ncol) ? as<T>(A.C[(long long)a * A.ncart + n_first + b]) : T(0), F,
                    smem_u32(Bs) + (a >> 4) * bpanel + b_off(b, a & 15), np * 32);
    }
    if (tid == 0) {
        mbar_init(bar_a, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(TM));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    fence_proxy_async();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    const int r = tid & 127, grp = tid >> 7, per = KP * (16 / G), h0 = grp * per;
    const long long ntiles = (A.npts + 127) / 128;
    constexpr int HOLD = 8;  // values of the next tile held in registers (more MOs: read again)
    T hold[HOLD];
    auto fetch = [&](long long tile) {
        const long long p = tile * 128 + r < A.npts ? tile * 128 + r : A.npts - 1;
#pragma unroll
        for (int q = 0; q < HOLD; ++q) hold[q] = q < per && h0 + q < A.nmo ? X[(long long)(h0 + q) * A.ld + p] : T(0);
    };
    if (blockIdx.x < ntiles) fetch(blockIdx.x);
    uint32_t parity = 0;
    for (long long tile = blockIdx.x; tile < ntiles; tile += gridDim.x, parity ^= 1) {
        const long long p = tile * 128 + r < A.npts ? tile * 128 + r : A.npts - 1;
        U m = 0;
#pragma unroll
        for (int q = 0; q < HOLD; ++q) m = max(m, DG::magnitude(hold[q]));
        for (int q = HOLD; q < per; ++q)
            if (h0 + q < A.nmo) m = max(m, DG::magnitude(X[(long long)(h0 + q) * A.ld + p]));
        tops[grp * 128 + r] = m;
        __syncthreads();
#pragma unroll
        for (int g = 0; g < G; ++g) m = max(m, tops[g * 128 + r]);
        const int E = DG::scale(m);
#pragma unroll
        for (int q = 0; q < HOLD; ++q)
            if (q < per) DG::put(hold[q], E, smem_u32(base) + ((h0 + q) >> 4) * (D * DT) + a_off(r, (h0 + q) & 15), DT);
        for (int q = HOLD; q < per; ++q)
            DG::put(h0 + q < A.nmo ? X[(long long)(h0 + q) * A.ld + p] : T(0), E,
                    smem_u32(base) + ((h0 + q) >> 4) * (D * DT) + a_off(r, (h0 + q) & 15), DT);
        fence_proxy_async();
        __syncthreads();
        if (tid == 0) {
            tc_fence_after();
#pragma unroll 1
            for (int k = 0; k < KP; ++k)
#pragma unroll 1
                for (int i = 0; i < D; ++i)
#pragma unroll 1
                    for (int j = 0; j < D - i; j += 256 / np) {
                        const int nd = D - i - j < 256 / np ? D - i - j : 256 / np;
                        mma_f16(tmem + (uint32_t)((i + j) * np), a_desc(smem_u32(base) + (uint32_t)(k * D + i) * DT),
                                b_desc(smem_u32(Bs) + (uint32_t)(k * bpanel + j * np * 32)), idesc(nd * np), (k > 0 || i > 0) ? 1u : 0u);
                    }
            mma_commit(bar_a);
        }
        if (tile + gridDim.x < ntiles) fetch(tile + gridDim.x);
        const bool ok = mbar_wait(bar_a, parity, A.redo, A.limit);
        if (!__syncthreads_and(ok)) {
            parity ^= 1;
            break;
        }
        tc_fence_after();
        const int quad = warp & 3, row = quad * 32 + lane;
        const long long q = tile * 128 + row;
        U mr = 0;
#pragma unroll
        for (int g = 0; g < G; ++g) mr = max(mr, tops[g * 128 + row]);
        if (DG::special(mr)) *(volatile int*)A.redo = 1;
        const int rowx = DG::scale(mr);
#pragma unroll 1
        for (int n0 = 4 * (warp >> 2); n0 < ncol; n0 += 4 * G) {
            AccN<D> va;
            acc_get(va, tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)n0, np);
            const int4 f4 = *(const int4*)(fexp + n0);
            T t[4];
            if constexpr (D == 4) acc_floats(va, rowx, f4, t);
            else acc_doubles(va, rowx, f4, t);
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (n0 + i < ncol && q < A.npts) out[(long long)(n0 + i) * A.ld + q] = t[i];
        }
        tc_fence_before();
        __syncthreads();
    }
    if (tid == 0 && blockIdx.x < ntiles) mbar_drain(bar_a, parity ^ 1);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TM));
}

// ------------------------------------------------------------------ step 4
// part[slot][k][i] = sum over the slot's points of W_i chi_k + V_i G_k.  Rows of the operand:
// 128 AO columns k, summed index: points in blocks of 64 (4 panels), each block's rows and
// MOs with scales of their own; W chi and V G one after the other through the accumulators.
// Both operands K-major (points contiguous in memory): a lane's value lands beside its
// neighbours'.
template <typename T>
struct RowArgs {
    long long npts, ld;
    const T* X;       // W, V: 2 x nmo x ld
    const T* Y;       // chi, G: 2 x ncart x ld
    int nmo, ncart, np;
    double* part;     // gridDim.x x ncart x nmo: sums of a block's points, over all runs
    bool first;       // first run: written, else added to
    int* redo;        // raised where a value is not finite or a wait expires
    long long limit;  // polls of a wait
    unsigned tm_cols;
};

constexpr int RB = 4;  // panels (64 points) per accumulation

template <typename T>
static size_t row_smem(int np)
{
    return 1024 + (size_t)RB * Dg<T>::D * (DT + np * 32) + 128 * 4 + 64 * 4 + 64;
}

// A row's two points of this lane.
template <typename T>
struct Pair {
    T v[2];
};
template <typename T>
__device__ __forceinline__ Pair<T> load_row(const T* __restrict__ src, long long p0, long long npts, int lane, bool live)
{
    Pair<T> o;
#pragma unroll
    for (int h = 0; h < 2; ++h) o.v[h] = live && p0 + h * 32 + lane < npts ? src[p0 + h * 32 + lane] : T(0);
    return o;
}
// Their digits into the K-major tiles (row `row` of panels panel_bytes apart, digits
// digit_bytes apart); the row's scale.
template <typename T>
__device__ __forceinline__ int put_row(const Pair<T>& x, int lane, uint32_t base, uint32_t panel_bytes, uint32_t digit_bytes, int row,
                                       int* redo)
{
    using DG = Dg<T>;
    typename DG::U m = max(DG::magnitude(x.v[0]), DG::magnitude(x.v[1]));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = DG::shfl_max(m, o);
    const int E = DG::scale(m);
#pragma unroll
    for (int h = 0; h < 2; ++h)
        DG::put(x.v[h], E, base + (uint32_t)(2 * h + (lane >> 4)) * panel_bytes + b_off(row, lane & 15), digit_bytes);
    if (DG::special(m)) *(volatile int*)redo = 1;
    return E;
}

template <typename T>
__global__ void __launch_bounds__(512, 1) row_kernel(const __grid_constant__ RowArgs<T> A)
{
    extern __shared__ unsigned char raw[];
    unsigned char* base = (unsigned char*)(((uintptr_t)raw + 1023) & ~(uintptr_t)1023);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, np = A.np;
    constexpr int D = Dg<T>::D;
    const int bpanel = D * np * 32;
    unsigned char* Bs = base + (size_t)RB * D * DT;
    int* rexp = (int*)(Bs + (size_t)RB * bpanel);  // 128
    int* fexp = rexp + 128;
    uint64_t* bar = (uint64_t*)(fexp + 64);
    uint32_t* tmem_slot = (uint32_t*)(bar + 1);
    const uint32_t bar_a = smem_u32(bar);
    for (int i = tid; i < RB * D * (DT + np * 32) / 16; i += 512) ((uint4*)base)[i] = make_uint4(0, 0, 0, 0);
    if (tid < 128) rexp[tid] = 0;
    if (tid < 64) fexp[tid] = 0;
    if (tid == 0) {
        mbar_init(bar_a, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(A.tm_cols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    const int k0 = blockIdx.y * 128, nrow = A.ncart - k0 < 128 ? A.ncart - k0 : 128;
    const long long nblk = (A.npts + 63) / 64;
    const int quad = warp & 3, row = quad * 32 + lane, hf = warp >> 2, dmax = 256 / np;
    double acc[4][4];
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[j][i] = 0.0;
    uint32_t parity = 0;
    bool good = true, issued = false;
    for (long long blk = blockIdx.x; good && blk < nblk; blk += gridDim.x)
        for (int z = 0; good && z < 2; ++z, parity ^= 1) {
            const T* Y = A.Y + ((long long)z * A.ncart + k0) * A.ld;
            const T* X = A.X + (long long)z * A.nmo * A.ld;
            // live rows only (the others' digits stay zero), four loaded ahead of their use
            const int total = nrow + A.nmo;
            Pair<T> x[4];
#pragma unroll 1
            for (int kb = warp; kb < total; kb += 64) {
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const int k = kb + 16 * u;
                    const bool live = k < total;
                    x[u] = load_row(k < nrow ? Y + (long long)k * A.ld : X + (long long)(live ? k - nrow : 0) * A.ld, blk * 64, A.npts, lane, live);
                }
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const int k = kb + 16 * u;
                    if (k >= total) break;
                    const bool left = k < nrow;
                    const int rw = left ? k : k - nrow;
                    const int e = put_row(x[u], lane, left ? smem_u32(base) : smem_u32(Bs), left ? (uint32_t)(D * DT) : (uint32_t)bpanel,
                                          left ? (uint32_t)DT : (uint32_t)(np * 32), rw, A.redo);
                    if (lane == 0) {
                        if (left) rexp[rw] = e;
                        else fexp[rw] = e;
                    }
                }
            }
            fence_proxy_async();
            __syncthreads();
            if (tid == 0) {
                tc_fence_after();
#pragma unroll 1
                for (int k = 0; k < RB; ++k)
#pragma unroll 1
                    for (int i = 0; i < D; ++i)
#pragma unroll 1
                        for (int j = 0; j < D - i; j += dmax) {
                            const int nd = D - i - j < dmax ? D - i - j : dmax;
                            // (K-major rows on both sides: the M-major bit off)
                            mma_f16(tmem + (uint32_t)((i + j) * np), b_desc(smem_u32(base) + (uint32_t)(k * D + i) * DT),
                                    b_desc(smem_u32(Bs) + (uint32_t)(k * bpanel + j * np * 32)), idesc(nd * np) & ~(1u << 15),
                                    (k > 0 || i > 0) ? 1u : 0u);
                        }
                mma_commit(bar_a);
            }
            issued = true;
            const bool ok = mbar_wait(bar_a, parity, A.redo, A.limit);
            good = __syncthreads_and(ok);
            if (!good) continue;
            tc_fence_after();
            const int rx = rexp[row];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int n0 = 4 * hf + 16 * j;
                if (n0 >= np) continue;
                AccN<D> va;
                double t[4];
                acc_get(va, tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)n0, np);
                const int4 f4 = *(const int4*)(fexp + n0);
                acc_doubles(va, rx, f4, t);
#pragma unroll
                for (int i = 0; i < 4; ++i) acc[j][i] += t[i];
            }
            tc_fence_before();
            __syncthreads();
        }
    if (tid == 0 && issued) mbar_drain(bar_a, parity ^ 1);
    double* part = A.part + ((long long)blockIdx.x * A.ncart + k0 + row) * A.nmo;
    if (row < nrow)
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int n = 4 * hf + 16 * j + i;
                if (n < A.nmo) part[n] = A.first ? acc[j][i] : part[n] + acc[j][i];
            }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(A.tm_cols));
}

// dC[i][k]: 8 threads per element sum every eighth slot in order, then their sums in order.
__global__ void __launch_bounds__(256) dcoeff_kernel(const double* __restrict__ part, int nslot, int nmo, int ncart, double* __restrict__ dC)
{
    __shared__ double sums[8][32];
    const int j = blockIdx.x * 32 + threadIdx.x;
    double s = 0.0;
    if (j < nmo * ncart)
        for (int b = threadIdx.y; b < nslot; b += 8) s += part[(long long)b * nmo * ncart + j];
    sums[threadIdx.y][threadIdx.x] = s;
    __syncthreads();
    if (threadIdx.y || j >= nmo * ncart) return;
    for (int y = 1; y < 8; ++y) s += sums[y][threadIdx.x];
    dC[(long long)(j % nmo) * ncart + j / nmo] = s;
}

// ------------------------------------------------------------------ step 3
constexpr int QB = 8;  // primitives whose sums a warp holds

template <typename T>
struct ShellArgs {
    BasisDev B;
    SplitDev S;
    Grid g;
    const double* g_grad;  // 3 x g_ld, or null
    long long g_ld, ld;
    const T* AB;           // A, B: 2 x ncart x ld
    T* Y;                  // chi, G: 2 x ncart x ld
    double* part_p;        // nslot x nprim x 3: U0, U1, U2, over all runs
    double* part_g;        // nslot x nshell x 3
    bool first;            // first run: written, else added to
    long long per;         // points of a slot (multiple of 32)
    int* redo;             // raised where a cotangent is not finite
};

// Coordinates of points visited in ascending order, 32 or fewer apart: the indices of a
// regular grid advance instead of being divided out at every point.
struct Walk {
    long long at;
    int i, j, k;
    __device__ __forceinline__ void start(const Grid& g, long long p)
    {
        at = p;
        if (!g.regular) return;
        const long long q = p + g.offset, nyz = (long long)g.ny * g.nz, r = q % nyz;
        i = (int)(q / nyz);
        j = (int)(r / g.nz);
        k = (int)(r - (long long)j * g.nz);
    }
    __device__ __forceinline__ void point(const Grid& g, long long p, double& x, double& y, double& z)
    {
        if (!g.regular) {
            x = __ldg(g.x + p);
            y = __ldg(g.y + p);
            z = __ldg(g.z + p);
            return;
        }
        k += (int)(p - at);
        at = p;
        while (k >= g.nz) {
            k -= g.nz;
            if (++j == g.ny) {
                j = 0;
                ++i;
            }
        }
        x = __ldg(g.x + i);
        y = __ldg(g.y + j);
        z = __ldg(g.z + k);
    }
};

template <typename T>
__device__ __forceinline__ T warp_total(T v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Value, gradient and Hessian monomials of a component as compile-time factors of px, py, pz.
template <int a, int b, int c, typename T>
__device__ __forceinline__ T mono(const T* px, const T* py, const T* pz)
{
    if constexpr (a < 0 || b < 0 || c < 0) return T(0);
    else return px[a] * py[b] * pz[c];
}

template <typename T>
struct PolySums {
    T Pa, Pb, dA[3], dB[3], H[6];  // H: xx, yy, zz, xy, xz, yz
};

// What the components of a shell contribute at one point: chi and G (written), and the
// polynomial sums of A and B.  off[J]: the component's offset in the arrays (its row), norm[J]
// its angular norm; a component that the shell does not list has norm 0 and is not written.
template <int L, typename T>
__device__ __forceinline__ void shell_polynomials(const T (&Av)[(L + 1) * (L + 2) / 2], const T (&Bv)[(L + 1) * (L + 2) / 2],
                                                  T* __restrict__ Yp, unsigned nb, const unsigned (&off)[(L + 1) * (L + 2) / 2], const T (&norm)[(L + 1) * (L + 2) / 2],
                                                  bool full, bool valid, T X, T Y, T Z, T gx, T gy, T gz, T R0, T q, PolySums<T>& o)
{
    T px[L + 1], py[L + 1], pz[L + 1];
    px[0] = py[0] = pz[0] = T(1);
#pragma unroll
    for (int i = 1; i <= L; ++i) {
        px[i] = px[i - 1] * X;
        py[i] = py[i - 1] * Y;
        pz[i] = pz[i - 1] * Z;
    }
    [&]<int... J>(std::integer_sequence<int, J...>) {
        (
            [&] {
                constexpr int a = canon_l(L, J, 0), b = canon_l(L, J, 1), c = canon_l(L, J, 2);
                const T g = norm[J];
                if (!full && off[J] == 0xFFFFFFFFu) return;
                const T Ak = Av[J] * g, Bk = Bv[J] * g;
                const T P = mono<a, b, c>(px, py, pz);
                const T Px = T(a) * mono<a - 1, b, c>(px, py, pz), Py = T(b) * mono<a, b - 1, c>(px, py, pz),
                        Pz = T(c) * mono<a, b, c - 1>(px, py, pz);
                o.Pa += Ak * P;
                o.Pb += Bk * P;
                if constexpr (a > 0) { o.dA[0] += Ak * Px; o.dB[0] += Bk * Px; }
                if constexpr (b > 0) { o.dA[1] += Ak * Py; o.dB[1] += Bk * Py; }
                if constexpr (c > 0) { o.dA[2] += Ak * Pz; o.dB[2] += Bk * Pz; }
                if constexpr (a > 1) o.H[0] += Bk * (T(a * (a - 1)) * mono<a - 2, b, c>(px, py, pz));
                if constexpr (b > 1) o.H[1] += Bk * (T(b * (b - 1)) * mono<a, b - 2, c>(px, py, pz));
                if constexpr (c > 1) o.H[2] += Bk * (T(c * (c - 1)) * mono<a, b, c - 2>(px, py, pz));
                if constexpr (a > 0 && b > 0) o.H[3] += Bk * (T(a * b) * mono<a - 1, b - 1, c>(px, py, pz));
                if constexpr (a > 0 && c > 0) o.H[4] += Bk * (T(a * c) * mono<a - 1, b, c - 1>(px, py, pz));
                if constexpr (b > 0 && c > 0) o.H[5] += Bk * (T(b * c) * mono<a, b - 1, c - 1>(px, py, pz));
                if (valid) {
                    T D = T(0);  // g . grad P
                    if constexpr (a > 0) D += gx * Px;
                    if constexpr (b > 0) D += gy * Py;
                    if constexpr (c > 0) D += gz * Pz;
                    Yp[off[J]] = g * (P * R0);
                    Yp[nb + off[J]] = g * (D * R0 + P * q);  // q = (g . X) S1
                }
            }(),
            ...);
    }(std::make_integer_sequence<int, ncanon(L)>{});
}

// e^(-alpha rr)
__device__ __forceinline__ double gauss(double, uint64_t mr, int er, const SplitPrim* pr, double, const uint64_t* tab)
{
    return exp_neg(mr, er, pr->A, pr->ea, tab);
}
__device__ __forceinline__ float gauss(float rr, uint64_t, int, const SplitPrim*, float alpha, const uint64_t*) { return expf(-alpha * rr); }

// e^(-alpha rr) is certainly zero (alpha > 0); doubles: alpha rr >= 2^10, from the exponents
__device__ __forceinline__ bool underflows(double alpha, double rr)
{
    const int ea = __double2hiint(alpha) >> 20, er = __double2hiint(rr) >> 20;
    return er < 0x7FF && ea < 0x7FF && ea + er >= 2 * 1023 + 10;
}
__device__ __forceinline__ bool underflows(float alpha, float rr) { return alpha * rr > 104.0f; }

// Why a warp per shell and run of points: the sums of the shell's parameters stay in registers
// over the run, which a block over all shells of a tile (the one-kernel form) sums through shared
// memory per tile.  Primitives whose exponential is zero at all 32 points are passed over
// (FP32 1.56 -> 1.08 ms per run).  f and g shells have their own kernel: with them in one the
// registers of all were those of a g shell (FP64 3.5 -> 3.1 ms).
// One shell and one run of points; everything that does not change along the run in registers.
template <int L, typename T>
__device__ __forceinline__ void run_shell(const ShellArgs<T>& A, const Shell& sh, int s, int slot, int lane)
{
    constexpr int N = ncanon(L);
    const long long i0 = slot * A.per, i1 = i0 + A.per < A.g.npts ? i0 + A.per : A.g.npts;
    const double ax = A.B.atoms[4 * sh.atom], ay = A.B.atoms[4 * sh.atom + 1], az = A.B.atoms[4 * sh.atom + 2];
    const unsigned nb = (unsigned)(A.B.ncart * A.ld);
    unsigned off[N];
    T norm[N];
    bool full = true;
#pragma unroll
    for (int j = 0; j < N; ++j) {
        const int row = A.B.comp_row[sh.comp0 + j];
        off[j] = row < 0 ? 0xFFFFFFFFu : (unsigned)((sh.cart0 + row) * A.ld);
        norm[j] = row < 0 ? T(0) : as<T>(A.B.comp_g[sh.comp0 + j]);
        full = full && row >= 0;
    }
    T dR[3] = {T(0), T(0), T(0)};
    for (int q0 = 0; q0 < sh.nprim; q0 += QB) {
        const int nq = sh.nprim - q0 < QB ? sh.nprim - q0 : QB;
        const SplitPrim* prims = A.S.prim + sh.prim0 + q0;
        // exponents and coefficients: floats in registers, doubles (whose sums take those) read again
        constexpr bool HELD = sizeof(T) == 4;
        T U0[QB], U1[QB], U2[QB], al_[HELD ? QB : 1], w_[HELD ? QB : 1];
#pragma unroll
        for (int q = 0; q < QB; ++q) {
            U0[q] = U1[q] = U2[q] = T(0);
            if (q >= nq) continue;
            if constexpr (HELD) {
                al_[q] = as<T>(-prims[q].neg_alpha);
                w_[q] = as<T>(prims[q].w);
            }
        }
        auto al = [&](int q) -> T {
            if constexpr (HELD) return al_[q];
            else return as<T>(-prims[q].neg_alpha);
        };
        auto w = [&](int q) -> T {
            if constexpr (HELD) return w_[q];
            else return as<T>(prims[q].w);
        };
        Walk walk;
        if (i0 < i1) walk.start(A.g, i0 + lane < i1 ? i0 + lane : i1 - 1);
#pragma unroll 1
        for (long long i = i0; i < i1; i += 32) {
            const bool valid = i + lane < i1;
            const long long p = valid ? i + lane : i1 - 1;
            // (all of a point's loads first: they are under way during the exponentials)
            T Av[N], Bv[N];
#pragma unroll
            for (int j = 0; j < N; ++j) {
                const bool on = valid && off[j] != 0xFFFFFFFFu;
                Av[j] = on ? A.AB[p + off[j]] : T(0);
                Bv[j] = on ? A.AB[p + nb + off[j]] : T(0);
            }
            double xd, yd, zd;
            walk.point(A.g, p, xd, yd, zd);
            xd -= ax;
            yd -= ay;
            zd -= az;
            const double rd = xd * xd + yd * yd + zd * zd;
            uint64_t mr = 0;
            int er = 0;
            if constexpr (sizeof(T) == 8) split_mantissa(rd, mr, er);
            const T X = as<T>(xd), Y = as<T>(yd), Z = as<T>(zd), rr = as<T>(rd);
            const bool gg = valid && A.g_grad;
            const T gx = gg ? as<T>(A.g_grad[p]) : T(0), gy = gg ? as<T>(A.g_grad[A.g_ld + p]) : T(0),
                    gz = gg ? as<T>(A.g_grad[2 * A.g_ld + p]) : T(0);
            T R0 = T(0), R1 = T(0), R2 = T(0), e[QB];
            unsigned live = 0;  // primitives whose exponential is not zero at all of the warp's points
#pragma unroll
            for (int q = 0; q < QB; ++q) {
                e[q] = T(0);
                if (q >= nq) continue;
                const T aq = al(q);
                if (!__any_sync(0xffffffffu, !underflows(aq, rr))) continue;
                live |= 1u << q;
                e[q] = gauss(rr, mr, er, prims + q, aq, A.S.exp_tab);
                const T we = w(q) * e[q];
                R0 += we;
                R1 += aq * we;
                R2 += aq * (aq * we);
            }
            // (more primitives than the warp holds: the others' part of the radial sums)
#pragma unroll 1
            for (int q = 0; q < sh.nprim; ++q) {
                if (q >= q0 && q < q0 + nq) {
                    q = q0 + nq - 1;
                    continue;
                }
                const SplitPrim* pr = A.S.prim + sh.prim0 + q;
                const T a = as<T>(-pr->neg_alpha), we = as<T>(pr->w) * gauss(rr, mr, er, pr, a, A.S.exp_tab);
                R0 += we;
                R1 += a * we;
                R2 += a * (a * we);
            }
            const T S1 = T(-2) * R1, S2 = T(4) * R2, gX = gx * X + gy * Y + gz * Z;
            PolySums<T> o;
            o.Pa = o.Pb = T(0);
#pragma unroll
            for (int u = 0; u < 3; ++u) o.dA[u] = o.dB[u] = T(0);
#pragma unroll
            for (int u = 0; u < 6; ++u) o.H[u] = T(0);
            shell_polynomials<L, T>(Av, Bv, A.Y + p, nb, off, norm, full, valid, X, Y, Z, gx, gy, gz, R0, gX * S1, o);
            T F = o.Pa;
            if constexpr (L > 0) F += gx * o.dB[0] + gy * o.dB[1] + gz * o.dB[2];
            const T Tt = gX * o.Pb, T2 = T(2) * Tt;
            // (a cotangent that is not finite would reach every primitive, as 0 times it is not 0)
            if (!(F - F == T(0) && Tt - Tt == T(0))) *(volatile int*)A.redo = 1;
            if (q0 == 0) {
                const T s1F = S1 * F + S2 * Tt, s1b = S1 * o.Pb;
                dR[0] += s1F * X + s1b * gx;
                dR[1] += s1F * Y + s1b * gy;
                dR[2] += s1F * Z + s1b * gz;
                if constexpr (L > 0) {
                    const T s1g = S1 * gX;
                    T h[3] = {o.dA[0], o.dA[1], o.dA[2]};
                    if constexpr (L > 1) {
                        h[0] += o.H[0] * gx + o.H[3] * gy + o.H[4] * gz;
                        h[1] += o.H[3] * gx + o.H[1] * gy + o.H[5] * gz;
                        h[2] += o.H[4] * gx + o.H[5] * gy + o.H[2] * gz;
                    }
#pragma unroll
                    for (int u = 0; u < 3; ++u) dR[u] += R0 * h[u] + s1g * o.dB[u];
                }
            }
#pragma unroll
            for (int q = 0; q < QB; ++q) {
                if (q >= nq || !(live >> q & 1)) continue;
                const T y = F - al(q) * T2, ey = e[q] * y;
                U0[q] += ey;
                U1[q] += rr * ey;
                U2[q] += e[q] * Tt;
            }
        }
#pragma unroll
        for (int q = 0; q < QB; ++q) {
            if (q >= nq) continue;
            const T a = warp_total(U0[q]), b = warp_total(U1[q]), c = warp_total(U2[q]);
            if (lane == 0) {
                double* o = A.part_p + ((long long)slot * A.B.nprim + sh.prim0 + q0 + q) * 3;
                o[0] = A.first ? (double)a : o[0] + (double)a;
                o[1] = A.first ? (double)b : o[1] + (double)b;
                o[2] = A.first ? (double)c : o[2] + (double)c;
            }
        }
    }
#pragma unroll
    for (int u = 0; u < 3; ++u) {
        const T v = warp_total(dR[u]);
        double* o = A.part_g + ((long long)slot * A.B.nshell + s) * 3 + u;
        if (lane == 0) *o = A.first ? (double)v : *o + (double)v;
    }
}

// A block: one shell, 4 warps with a run of points each.
template <typename T, bool HIGH>
__global__ void __launch_bounds__(128, HIGH ? 1 : sizeof(T) == 4 ? 5 : 2) shell_kernel(const __grid_constant__ ShellArgs<T> A)
{
    const int lane = threadIdx.x & 31, s = blockIdx.x, slot = blockIdx.y * 4 + (threadIdx.x >> 5);
    const Shell sh = A.B.shells[s];
    if ((sh.L > 2) != HIGH) return;
    if constexpr (HIGH) {
        if (sh.L == 3) run_shell<3, T>(A, sh, s, slot, lane);
        else run_shell<4, T>(A, sh, s, slot, lane);
    } else {
        switch (sh.L) {
        case 0: run_shell<0, T>(A, sh, s, slot, lane); break;
        case 1: run_shell<1, T>(A, sh, s, slot, lane); break;
        default: run_shell<2, T>(A, sh, s, slot, lane); break;
        }
    }
}

// dL/d(alpha, c) of every primitive in the caller's order (the shell kernel's primitives are
// sorted by exponent, prim_place[] their original places), dL/dR per atom over its shells: a
// warp per primitive or atom, the lanes' slots in order, then the lanes in a fixed tree.
__global__ void __launch_bounds__(128) finish_kernel(BasisDev B, SplitDev S, const double* __restrict__ part_p,
                                                     const double* __restrict__ part_g, int nslot, double* __restrict__ dprim,
                                                     double* __restrict__ dgeo)
{
    const int j = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    double u[3] = {0.0, 0.0, 0.0};
    if (j < B.nprim) {
        for (int b = lane; b < nslot; b += 32)
            for (int c = 0; c < 3; ++c) u[c] += part_p[((long long)b * B.nprim + j) * 3 + c];
    } else if (j < B.nprim + B.natom) {
        const int a = j - B.nprim;
        for (int b = lane; b < nslot; b += 32)
            for (int k = B.atom_shell_ptr[a]; k < B.atom_shell_ptr[a + 1]; ++k)
                for (int c = 0; c < 3; ++c) u[c] += part_g[((long long)b * B.nshell + B.atom_shells[k]) * 3 + c];
    } else {
        return;
    }
    for (int c = 0; c < 3; ++c) u[c] = warp_total(u[c]);
    if (lane) return;
    if (j < B.nprim) {
        const int i = S.prim_place[j];
        const double w = B.prim[2 * i + 1];
        dprim[2 * i] = B.prim_adj[2 * i] * u[0] - w * u[1] - 2.0 * w * u[2];
        dprim[2 * i + 1] = B.prim_adj[2 * i + 1] * u[0];
    } else {
        for (int c = 0; c < 3; ++c) dgeo[3 * (j - B.nprim) + c] = -u[c];
    }
}

// ------------------------------------------------------------------ host side
struct Plan {
    long long run;     // points of a run
    int nruns, nchunk; // runs; slots of the shell kernel (multiple of 4)
    int nbx;           // point slots of the row kernel
    size_t o_x, o_ab, o_y, o_pc, o_pp, o_pg, bytes;
};

static size_t up256(size_t v) { return (v + 255) & ~(size_t)255; }

template <typename T>
static Plan make_plan(const okg_basis* b, long long npts, int nmo, int sms)
{
    Plan P;
    // intermediates of a run: at most about 1 GB
    const size_t per_point = sizeof(T) * (2 * (size_t)nmo + 4 * (size_t)b->ncart);
    const long long most_run = (long long)((1ull << 30) / per_point) / 128 * 128;
    P.nruns = (int)((npts + most_run - 1) / most_run);
    P.run = P.nruns == 1 ? npts : ((npts + P.nruns - 1) / P.nruns + 127) / 128 * 128;
    P.nruns = (int)((npts + P.run - 1) / P.run);
    int want = (sms * 64 + b->nshell - 1) / b->nshell;  // warps to fill the chip, over the shells
    const long long most = (P.run + 31) / 32;
    if (want > 256) want = 256;
    if (want > most) want = (int)most;
    P.nchunk = (want + 3) / 4 * 4;
    const int tiles = (b->ncart + 127) / 128;
    const long long blocks = (P.run + 63) / 64;
    P.nbx = (sms + tiles - 1) / tiles;
    if (P.nbx > blocks) P.nbx = (int)blocks;
    const size_t ld = (size_t)P.run;
    P.o_x = 0;
    P.o_ab = P.o_x + up256(2 * (size_t)nmo * ld * sizeof(T));
    P.o_y = P.o_ab + up256(2 * (size_t)b->ncart * ld * sizeof(T));
    P.o_pc = P.o_y + up256(2 * (size_t)b->ncart * ld * sizeof(T));
    // (the runs follow one another on the stream and add to the same partial sums)
    P.o_pp = P.o_pc + up256((size_t)P.nbx * b->ncart * nmo * 8);
    P.o_pg = P.o_pp + up256((size_t)P.nchunk * b->nprim * 3 * 8);
    P.bytes = P.o_pg + up256((size_t)P.nchunk * b->nshell * 3 * 8);
    return P;
}

static int sm_count()
{
    int dev = 0, n = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    return n > 0 ? n : 1;
}

template <typename T>
static int run(const okg_basis* b, const Grid& g, int nmo, const double* C, const double* occ, const double* grho, const double* ggrad,
               long long ld, double* dC, double* dprim, double* dgeo, char* work, const Plan& P, int* redo, cudaStream_t st, bool& done)
{
    const long long limit = split_wait_limit();
    T* X = (T*)(work + P.o_x);
    T* AB = (T*)(work + P.o_ab);
    T* Y = (T*)(work + P.o_y);
    double *pc = (double*)(work + P.o_pc), *pp = (double*)(work + P.o_pp), *pg = (double*)(work + P.o_pg);
    const int kp = (nmo + 15) / 16, np = kp * 16;
    const size_t cs = ColCfg<T>::smem(kp), rs = row_smem<T>(np);
    // (the attributes are set to what the kernels take at most: other host threads launch under them)
    cudaError_t e = cudaFuncSetAttribute(column_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ColCfg<T>::smem(NMO_MAX / 16));
    if (e == cudaSuccess) e = cudaFuncSetAttribute(row_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)row_smem<T>(NMO_MAX));
    if (e != cudaSuccess) return cuda_status(e, "okg_rho_backward: shared memory");
    e = cudaMemsetAsync(redo, 0, sizeof(int), st);
    if (e != cudaSuccess) return cuda_status(e, "okg_rho_backward: memset");
    const int passes = (b->ncart + 63) / 64, sms = sm_count();
    for (int r = 0; r < P.nruns; ++r) {
        const long long i0 = r * P.run, n = g.npts - i0 < P.run ? g.npts - i0 : P.run;
        Grid gr = g;
        gr.npts = n;
        if (g.regular) {
            gr.offset = g.offset + i0;
        } else {
            gr.x += i0;
            gr.y += i0;
            gr.z += i0;
        }
        SplitCall c{nmo, C, occ, DrvList{}, 0xFu, false, (double*)X, nullptr, nullptr, P.run};
        c.wv_float = sizeof(T) == 4;
        c.g_rho = grho + i0;
        c.g_grad = ggrad ? ggrad + i0 : nullptr;
        c.g_ld = ld;
        c.redo = redo;
        bool wv = false;
        int s = split_run(b, gr, c, SplitGeneral{}, st, wv);
        if (s || !wv) return s;
        const long long tiles = (n + 127) / 128;
        int gx = (sms * ColCfg<T>::CTAS + 2 * passes - 1) / (2 * passes);
        if (gx > tiles) gx = (int)tiles;
        column_kernel<T><<<dim3(gx, passes, 2), 128 * ColCfg<T>::G, cs, st>>>(ColArgs<T>{n, P.run, X, C, nmo, b->ncart, kp, AB, redo, limit});
        long long per = ((n + P.nchunk - 1) / P.nchunk + 31) / 32 * 32;
        const ShellArgs<T> sa{b->dev, b->split, gr, c.g_grad, ld, P.run, AB, Y, pp, pg, r == 0, per, redo};
        shell_kernel<T, false><<<dim3(b->nshell, P.nchunk / 4), 128, 0, st>>>(sa);
        if (b->max_l > 2) shell_kernel<T, true><<<dim3(b->nshell, P.nchunk / 4), 128, 0, st>>>(sa);
        unsigned tm = 32;
        while ((int)tm < Dg<T>::D * np) tm *= 2;
        row_kernel<T><<<dim3(P.nbx, (b->ncart + 127) / 128), 512, rs, st>>>(
            RowArgs<T>{n, P.run, X, Y, nmo, b->ncart, np, pc, r == 0, redo, limit, tm});
    }
    dcoeff_kernel<<<(nmo * b->ncart + 31) / 32, dim3(32, 8), 0, st>>>(pc, P.nbx, nmo, b->ncart, dC);
    finish_kernel<<<(b->nprim + b->natom + 3) / 4, 128, 0, st>>>(b->dev, b->split, pp, pg, P.nchunk, dprim, dgeo);
    done = true;
    return cuda_status(cudaGetLastError(), "okg_rho_backward launch");
}

}  // namespace adjs

size_t adjoint_split_bytes(const okg_basis* b, long long npts, int nmo, int precision)
{
    if (!adjs::takes(b, npts, nmo, precision)) return 0;
    const int sms = adjs::sm_count();
    return precision == 32 ? adjs::make_plan<float>(b, npts, nmo, sms).bytes : adjs::make_plan<double>(b, npts, nmo, sms).bytes;
}

int adjoint_split_run(const okg_basis* b, const Grid& g, int nmo, const double* C, const double* occ, const double* grho,
                      const double* ggrad, long long ld, int precision, double* dC, double* dprim, double* dgeo, void* work,
                      int* redo, cudaStream_t st, bool& done)
{
    done = false;
    if (!adjs::takes(b, g.npts, nmo, precision)) return OKG_OK;
    const int sms = adjs::sm_count();
    if (precision == 32)
        return adjs::run<float>(b, g, nmo, C, occ, grho, ggrad, ld, dC, dprim, dgeo, (char*)work,
                                adjs::make_plan<float>(b, g.npts, nmo, sms), redo, st, done);
    return adjs::run<double>(b, g, nmo, C, occ, grho, ggrad, ld, dC, dprim, dgeo, (char*)work,
                             adjs::make_plan<double>(b, g.npts, nmo, sms), redo, st, done);
}
}  // namespace okg
