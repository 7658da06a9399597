// CI (transition) densities and flux densities on a grid from MO grids: the grid
// loops of orbkit's detCI module (orbkit/detci/cy_ci.pyx:70-96 get_rho,
// :152-178 get_jab, :203-229 get_a_nabla_b; drivers orbkit/detci/ci_core.py:84-267).
//
// Inputs are the MO grids (nmo x ld, points contiguous, as orbkit's molist) and the
// determinant-comparison terms of orbkit/detci/occ_check.py: "zero" terms
// (coefficient, orbital) contribute c MO_s^2, "single" terms (coefficient, orbital
// pair a, b) contribute c MO_a MO_b.  One thread per grid point walks the terms in
// the given order with each product and sum rounded as orbkit writes it (no FMA
// contraction), so for the same MO grids the results are orbkit's to the bit.
// Term tables are read by every thread of a warp at the same address (broadcast
// through L1); MO values are read coalesced.
#include "okg_digits.cuh"
#include "okg_internal.cuh"

namespace okg {

__global__ void ci_rho_kernel(long long npts, const double* __restrict__ mo, long long ld, int nz,
                              const double* __restrict__ zc, const int* __restrict__ zi, int ns,
                              const double* __restrict__ sc, const int* __restrict__ sp, double* __restrict__ rho)
{
    const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= npts) return;
    double r = 0.0;
    for (int t = 0; t < nz; ++t) {
        const double m = mo[(long long)__ldg(zi + t) * ld + p];
        r = __dadd_rn(r, __dmul_rn(__dmul_rn(__ldg(zc + t), m), m));
    }
    for (int t = 0; t < ns; ++t) {
        const double ma = mo[(long long)__ldg(sp + 2 * t) * ld + p];
        const double mb = mo[(long long)__ldg(sp + 2 * t + 1) * ld + p];
        r = __dadd_rn(r, __dmul_rn(__dmul_rn(__ldg(sc + t), ma), mb));
    }
    rho[p] = r;
}

// ANTISYM: j_d -= 0.5 (c (MO_a dMO_b - MO_b dMO_a))  (get_jab)
// else:    j_d += c (MO_a dMO_b)                       (get_a_nabla_b)
template <bool ANTISYM>
__global__ void ci_flux_kernel(long long npts, const double* __restrict__ mo, const double* __restrict__ drv,
                               long long ld, int nmo, int ns, const double* __restrict__ sc,
                               const int* __restrict__ sp, double* __restrict__ j)
{
    const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= npts) return;
    const long long dstride = (long long)nmo * ld;
    double acc[3] = {0.0, 0.0, 0.0};
    for (int t = 0; t < ns; ++t) {
        const int a = __ldg(sp + 2 * t), b = __ldg(sp + 2 * t + 1);
        const double c = __ldg(sc + t);
        const double ma = mo[(long long)a * ld + p];
        const double mb = mo[(long long)b * ld + p];
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const double db = drv[d * dstride + (long long)b * ld + p];
            if (ANTISYM) {
                const double da = drv[d * dstride + (long long)a * ld + p];
                const double t2 = __dmul_rn(0.5, __dmul_rn(c, __dsub_rn(__dmul_rn(ma, db), __dmul_rn(mb, da))));
                acc[d] = __dsub_rn(acc[d], t2);
            } else {
                acc[d] = __dadd_rn(acc[d], __dmul_rn(c, __dmul_rn(ma, db)));
            }
        }
    }
#pragma unroll
    for (int d = 0; d < 3; ++d) j[(long long)d * npts + p] = acc[d];
}

// Quadratic-form evaluation of the same sums.  The terms collapse into NMO x NMO
// coefficient matrices (host side): rho = sum_ab M_ab MO_a MO_b and
// j_d = scale sum_ab Q_ab MO_a dMO_b, so a point costs NMO^2 FMAs instead of work
// proportional to the number of terms.  Each thread owns one point and walks the
// bra orbitals in chunks of CI_CH held in registers; per ket orbital b it forms
// t_b = sum_{a in chunk} Q^T[b][a] MO_a (coefficients read as broadcasts through
// L1) and adds t_b MO_b (rho) or t_b dMO_b for the three directions (flux), so the
// flux shares one matrix-vector product between x, y and z.  For rho the matrix is
// symmetrised and only a <= b is visited (lower triangle of Q^T, zero above).
// FP64 FMAs; the sum order differs from orbkit's term order.
#define CI_CH 16

template <bool FLUX>
__device__ __forceinline__ void quad_point(long long npts, const double* __restrict__ mo, const double* __restrict__ drv,
                                           long long ld, int nmo, const double* __restrict__ qt, double scale,
                                           double* __restrict__ out, long long p)
{
    const long long dstride = (long long)nmo * ld;
    double acc0 = 0.0, acc1 = 0.0, acc2 = 0.0;
    for (int a0 = 0; a0 < nmo; a0 += CI_CH) {
        double pa[CI_CH];
#pragma unroll
        for (int i = 0; i < CI_CH; ++i) pa[i] = (a0 + i < nmo) ? mo[(long long)(a0 + i) * ld + p] : 0.0;
        // rho: rows b < a0 of the lower-triangular Q^T hold zeros for this chunk
        for (int b = FLUX ? 0 : a0; b < nmo; ++b) {
            const double2* q = reinterpret_cast<const double2*>(qt + (long long)b * ((nmo + CI_CH - 1) / CI_CH * CI_CH) + a0);
            double t = 0.0;
#pragma unroll
            for (int i = 0; i < CI_CH / 2; ++i) {
                const double2 c = __ldg(q + i);
                t = fma(c.x, pa[2 * i], t);
                t = fma(c.y, pa[2 * i + 1], t);
            }
            if (FLUX) {
                acc0 = fma(t, drv[(long long)b * ld + p], acc0);
                acc1 = fma(t, drv[dstride + (long long)b * ld + p], acc1);
                acc2 = fma(t, drv[2 * dstride + (long long)b * ld + p], acc2);
            } else {
                acc0 = fma(t, mo[(long long)b * ld + p], acc0);
            }
        }
    }
    if (FLUX) {
        out[p] = scale * acc0;
        out[npts + p] = scale * acc1;
        out[2 * npts + p] = scale * acc2;
    } else {
        out[p] = scale * acc0;
    }
}

template <bool FLUX>
__global__ void __launch_bounds__(128) ci_quad_kernel(long long npts, const double* __restrict__ mo,
                                                      const double* __restrict__ drv, long long ld, int nmo,
                                                      const double* __restrict__ qt, double scale,
                                                      double* __restrict__ out)
{
    const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (p < npts) quad_point<FLUX>(npts, mo, drv, ld, nmo, qt, scale, out, p);
}

// The same quadratic forms with the matrix-vector product on the tensor cores: per 128 points
// the MO values become exact digit operands (okg_digits.cuh), t_b = sum_a Q^T[b][a] MO_a comes
// back as FP64 values, and the FP64 pipe is left with t_b MO_b (NMO FMAs per point) or
// t_b dMO_b (3 NMO) of the NMO^2 (+ 3 NMO).  The coefficient digits are made by every CTA for
// itself (at most 64 x 64 values) and stay in shared memory; the MO values are read twice
// (scale, then digits: the second time from L1).  Points and coefficients beyond the digits'
// range, and what a block has left when a wait expires, are evaluated as in ci_quad_kernel.
struct CiSplit {
    long long npts, ld;
    const double* mo;
    const double* drv;
    const double* qt;
    int nmo, ldq, np;  // np: nmo rounded up to 16 (= ldq)
    double scale;
    double* out;
    long long limit;  // polls of a wait
    unsigned tm_cols;
};

// The block's tiles [first, ntiles): points beyond the digits' range before tile `left`, every
// point from there on.  One call behind the loop over the tiles (a call inside it took 36
// registers and spilled: 24 MOs, 200 K points, density and flux 2.5 % slower as whole calls).
template <bool FLUX>
__device__ __noinline__ void direct_points(const CiSplit& A, long long first, long long left)
{
    for (long long tile = first; tile * 128 < A.npts; tile += gridDim.x) {
        const long long p = tile * 128 + threadIdx.x;
        if (threadIdx.x >= 128 || p >= A.npts) continue;
        bool on = tile >= left;
        for (int a = 0; !on && a < A.nmo; ++a)
            on = sp::too_large((unsigned long long)__double_as_longlong(A.mo[a * A.ld + p]) & 0x7FFFFFFFFFFFFFFFull);
        if (on) quad_point<FLUX>(A.npts, A.mo, A.drv, A.ld, A.nmo, A.qt, A.scale, A.out, p);
    }
}

constexpr int CI_SPLIT_MAX = 64;  // MOs: 7 accumulators per MO in 512 TMEM columns

static size_t ci_split_smem(int np)
{
    return 1024 + (size_t)(np / 16) * (sp::ND * sp::DT + sp::ND * np * 32) + 3 * 3 * 128 * 8 + 4 * 128 * 8 + 64 * 4 + 64;
}

template <int G>
__device__ __forceinline__ unsigned long long largest(const unsigned long long* tops, int r)
{
    unsigned long long m = tops[r];
#pragma unroll
    for (int g = 1; g < G; ++g) m = tops[g * 128 + r] > m ? tops[g * 128 + r] : m;
    return m;
}

// G threads per point (G warps per 32 accumulator rows).  Phases alternate in a CTA (digits,
// MMAs, accumulators), so their latency shows: with more than 32 MOs one CTA of 512 threads
// per SM (42 MOs, 2^20 points: rho 2.26 ms with the DFMA kernel, 0.92 with G = 2, 0.72 with
// G = 4; flux 4.07, 1.09, 0.88), up to 32 MOs two CTAs of 256 (24 MOs: rho 0.93, 0.35 with
// G = 2, 0.48 with G = 4; 8 MOs: 0.24, 0.16, 0.27).
template <bool FLUX, int G>
__global__ void __launch_bounds__(128 * G, 4 / G) ci_split_kernel(const __grid_constant__ CiSplit A)
{
    using namespace sp;
    extern __shared__ unsigned char raw[];
    unsigned char* base = (unsigned char*)(((uintptr_t)raw + 1023) & ~(uintptr_t)1023);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int np = A.np, KP = np / 16, bpanel = ND * np * 32;
    unsigned char* Bs = base + (size_t)KP * ND * DT;
    double* part = (double*)(Bs + (size_t)KP * bpanel);            // 3 x 3 x 128
    unsigned long long* tops = (unsigned long long*)(part + 9 * 128);  // 4 x 128
    int* fexp = (int*)(tops + 512);
    uint64_t* bar = (uint64_t*)(fexp + CI_SPLIT_MAX);
    uint32_t* tmem_slot = (uint32_t*)(bar + 1);
    const uint32_t bar_a = smem_u32(bar);
    // coefficient digits
    bool direct = false;
    for (int b = warp; b < np; b += 4 * G) {
        unsigned long long m = 0;
        for (int a = lane; a < A.nmo && b < A.nmo; a += 32) {
            const unsigned long long u = (unsigned long long)__double_as_longlong(A.qt[(long long)b * A.ldq + a]) & 0x7FFFFFFFFFFFFFFFull;
            m = u > m ? u : m;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const unsigned long long u = __shfl_xor_sync(0xffffffffu, m, o);
            m = u > m ? u : m;
        }
        direct |= too_large(m) || vanishing(m);
        const int F = scale_of(m);
        if (lane == 0) fexp[b] = F;
        for (int a = lane; a < np; a += 32) {
            const double v = (a < A.nmo && b < A.nmo) ? A.qt[(long long)b * A.ldq + a] : 0.0;
            const uint64_t t = digits7(v, F + 1030);
#pragma unroll
            for (int j = 0; j < ND; ++j)
                *(__half*)(Bs + (a >> 4) * bpanel + b_off(j * np + b, a & 15)) = __int2half_rn((int)((t >> (8 * (6 - j))) & 0xFF) - 128);
        }
    }
    if (tid == 0) {
        mbar_init(bar_a, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(A.tm_cols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    fence_proxy_async();
    tc_fence_before();
    direct = __syncthreads_or(direct);
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    const int r = tid & 127, part4 = tid >> 7;
    const long long ntiles = (A.npts + 127) / 128, dstride = (long long)A.nmo * A.ld;
    const int h0 = part4 * KP * (16 / G), h1 = h0 + KP * (16 / G);  // this thread's MOs
    uint32_t parity = 0;
    bool issued = false, late = false;  // late: points beyond the digits' range
    long long tile = blockIdx.x;
    for (; !direct && tile < ntiles; tile += gridDim.x, parity ^= 1) {
        const long long p = tile * 128 + r < A.npts ? tile * 128 + r : A.npts - 1;
        unsigned long long m = 0;
#pragma unroll 8
        for (int a = h0; a < h1; ++a) {
            const unsigned long long u = a < A.nmo ? (unsigned long long)__double_as_longlong(A.mo[(long long)a * A.ld + p]) & 0x7FFFFFFFFFFFFFFFull : 0ull;
            m = u > m ? u : m;
        }
        tops[part4 * 128 + r] = m;
        __syncthreads();
        m = largest<G>(tops, r);
        const int E = scale_of(m), rs = E + 1030;
#pragma unroll 4
        for (int a = h0; a < h1; ++a)
            put1(a < A.nmo ? A.mo[(long long)a * A.ld + p] : 0.0, rs, smem_u32(base) + (a >> 4) * (ND * DT) + a_off(r, a & 15));
        fence_proxy_async();
        __syncthreads();
        if (tid == 0) {
            tc_fence_after();
            const int dmax = 256 / np;
#pragma unroll 1
            for (int k = 0; k < KP; ++k)
#pragma unroll 1
                for (int i = 0; i < ND; ++i) {
                    const uint64_t ad = a_desc(smem_u32(base) + (uint32_t)(k * ND + i) * DT);
#pragma unroll 1
                    for (int j = 0; j < ND - i; j += dmax) {
                        const int nd = ND - i - j < dmax ? ND - i - j : dmax;
                        mma_f16(tmem + (uint32_t)((i + j) * np), ad, b_desc(smem_u32(Bs) + (uint32_t)(k * bpanel + j * np * 32)),
                                idesc(nd * np), (k > 0 || i > 0) ? 1u : 0u);
                    }
                }
            mma_commit(bar_a);
        }
        issued = true;
        direct = __syncthreads_or(!mbar_try_for(bar_a, parity, A.limit));
        if (direct) {
            parity ^= 1;
            break;
        }
        tc_fence_after();
        // accumulators: warps w, w + 4, ... share 32 rows, every G-th group of 4 MOs each
        const int quad = warp & 3, row = quad * 32 + lane, hf = warp >> 2;
        const long long q = tile * 128 + row;
        const bool valid = q < A.npts;
        const long long pr = valid ? q : A.npts - 1;
        const unsigned long long mr = largest<G>(tops, row);
        const int rowx = scale_of(mr);
        double acc[3] = {0.0, 0.0, 0.0};
#pragma unroll 1
        for (int n0 = 4 * hf; n0 < A.nmo; n0 += 4 * G) {
            Acc4 va;
            double t[4];
            acc_load(va, tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)n0, np);
            const int4 f4 = *(const int4*)(fexp + n0);
            double x[FLUX ? 3 : 1][4];
            const double* src = FLUX ? A.drv : A.mo;
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int d = 0; d < (FLUX ? 3 : 1); ++d)
                    x[d][i] = n0 + i < A.nmo ? src[d * dstride + (long long)(n0 + i) * A.ld + pr] : 0.0;
            acc_wait(va);
            acc_values(va, rowx, f4, t);
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int d = 0; d < (FLUX ? 3 : 1); ++d)
                    if (n0 + i < A.nmo) acc[d] = fma(t[i], x[d][i], acc[d]);
        }
        if (hf > 0)
            for (int d = 0; d < (FLUX ? 3 : 1); ++d) part[((hf - 1) * 3 + d) * 128 + row] = acc[d];
        tc_fence_before();
        __syncthreads();
        late |= too_large(mr);
        if (hf == 0 && valid)
            for (int d = 0; d < (FLUX ? 3 : 1); ++d) {
                double t = acc[d];
                for (int h = 0; h < G - 1; ++h) t += part[(h * 3 + d) * 128 + row];
                A.out[d * A.npts + q] = A.scale * t;
            }
    }
    // (after an expired wait: the MMAs issued last complete before the CTA leaves)
    if (tid == 0 && issued) mbar_drain(bar_a, parity ^ 1);
    late = __syncthreads_or(late);
    if (late || tile < ntiles) direct_points<FLUX>(A, late ? blockIdx.x : tile, tile);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(A.tm_cols));
}

// Runs the quadratic form on the tensor cores where it is one for them.
template <bool FLUX>
static int ci_split(long long npts, const double* mo, const double* drv, long long ld, int nmo, const double* qt, double scale,
                    double* out, cudaStream_t st, bool& done)
{
    done = false;
    if (nmo > CI_SPLIT_MAX) return OKG_OK;
    CiSplit A{npts, ld, mo, drv, qt, nmo, (nmo + 15) / 16 * 16, (nmo + 15) / 16 * 16, scale, out, split_wait_limit(), 32};
    while ((int)A.tm_cols < sp::ND * A.np) A.tm_cols *= 2;
    const size_t smem = ci_split_smem(A.np);
    int dev = 0, sms = 1;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int per = A.np <= 32 ? 2 : 1;  // CTAs per SM
    const long long ntiles = (npts + 127) / 128, cap = (long long)sms * per;
    const unsigned nblk = (unsigned)(ntiles < cap ? ntiles : cap);
    // (the attribute is set to what the kernel takes at most: other host threads launch under it)
    auto go = [&](auto kernel, int threads, int np_max) -> int {
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ci_split_smem(np_max));
        if (e != cudaSuccess) return cuda_status(e, "detCI quadratic form: shared memory");
        kernel<<<nblk, threads, smem, st>>>(A);
        return OKG_OK;
    };
    const int s = per == 2 ? go(ci_split_kernel<FLUX, 2>, 256, 32) : go(ci_split_kernel<FLUX, 4>, 512, CI_SPLIT_MAX);
    if (s) return s;
    done = true;
    return cuda_status(cudaGetLastError(), "detCI quadratic form launch");
}

}  // namespace okg

using namespace okg;

static int ci_check_terms(int n, const double* c, const int* idx, const char* what)
{
    if (n < 0 || (n > 0 && (!c || !idx))) return set_error(OKG_ERR_ARG, what);
    return OKG_OK;
}

extern "C" int okg_ci_rho(int64_t npts, const double* d_mo, int64_t ld, int nz, const double* d_zcoef,
                          const int* d_zidx, int ns, const double* d_scoef, const int* d_spair, double* d_rho,
                          okg_stream stream)
{
    if (npts < 0 || !d_rho || (npts > 0 && !d_mo) || ld < npts)
        return set_error(OKG_ERR_ARG, "okg_ci_rho: NULL MO grid / output, npts < 0 or ld < npts");
    int st = ci_check_terms(nz, d_zcoef, d_zidx, "okg_ci_rho: zero-term table NULL or nz < 0");
    if (st) return st;
    if ((st = ci_check_terms(ns, d_scoef, d_spair, "okg_ci_rho: single-term table NULL or ns < 0"))) return st;
    if (npts == 0) return OKG_OK;
    const unsigned nblk = (unsigned)((npts + 127) / 128);
    ci_rho_kernel<<<nblk, 128, 0, (cudaStream_t)stream>>>(npts, d_mo, ld, nz, d_zcoef, d_zidx, ns, d_scoef, d_spair,
                                                          d_rho);
    return cuda_status(cudaGetLastError(), "okg_ci_rho launch");
}

static int ci_flux(bool antisym, int64_t npts, const double* d_mo, const double* d_drv, int64_t ld, int nmo, int ns,
                   const double* d_scoef, const int* d_spair, double* d_j, cudaStream_t st, const char* name)
{
    if (npts < 0 || !d_j || (npts > 0 && (!d_mo || !d_drv)) || ld < npts || nmo <= 0)
        return set_error(OKG_ERR_ARG, name);
    int s = ci_check_terms(ns, d_scoef, d_spair, name);
    if (s) return s;
    if (npts == 0) return OKG_OK;
    const unsigned nblk = (unsigned)((npts + 127) / 128);
    if (antisym)
        ci_flux_kernel<true><<<nblk, 128, 0, st>>>(npts, d_mo, d_drv, ld, nmo, ns, d_scoef, d_spair, d_j);
    else
        ci_flux_kernel<false><<<nblk, 128, 0, st>>>(npts, d_mo, d_drv, ld, nmo, ns, d_scoef, d_spair, d_j);
    return cuda_status(cudaGetLastError(), name);
}

extern "C" int okg_ci_jab(int64_t npts, const double* d_mo, const double* d_drv, int64_t ld, int nmo, int ns,
                          const double* d_scoef, const int* d_spair, double* d_j, okg_stream stream)
{
    return ci_flux(true, npts, d_mo, d_drv, ld, nmo, ns, d_scoef, d_spair, d_j, (cudaStream_t)stream,
                   "okg_ci_jab: bad argument (NULL pointer, npts < 0, ld < npts, nmo <= 0 or ns < 0)");
}

extern "C" int okg_ci_a_nabla_b(int64_t npts, const double* d_mo, const double* d_drv, int64_t ld, int nmo, int ns,
                                const double* d_scoef, const int* d_spair, double* d_j, okg_stream stream)
{
    return ci_flux(false, npts, d_mo, d_drv, ld, nmo, ns, d_scoef, d_spair, d_j, (cudaStream_t)stream,
                   "okg_ci_a_nabla_b: bad argument (NULL pointer, npts < 0, ld < npts, nmo <= 0 or ns < 0)");
}

// Q^T is nmo rows of ldq = nmo rounded up to a multiple of 16 doubles (zero padded;
// 16-byte aligned rows).
extern "C" int okg_ci_rho_matrix(int64_t npts, const double* d_mo, int64_t ld, int nmo, const double* d_qt,
                                 double* d_rho, okg_stream stream)
{
    if (npts < 0 || !d_rho || (npts > 0 && (!d_mo || !d_qt)) || ld < npts || nmo <= 0)
        return set_error(OKG_ERR_ARG, "okg_ci_rho_matrix: bad argument (NULL pointer, npts < 0, ld < npts, nmo <= 0)");
    if (((uintptr_t)d_qt & 15) != 0) return set_error(OKG_ERR_ARG, "okg_ci_rho_matrix: d_qt not 16-byte aligned");
    if (npts == 0) return OKG_OK;
    bool done = false;
    const int s = ci_split<false>(npts, d_mo, nullptr, ld, nmo, d_qt, 1.0, d_rho, (cudaStream_t)stream, done);
    if (s || done) return s;
    const unsigned nblk = (unsigned)((npts + 127) / 128);
    ci_quad_kernel<false><<<nblk, 128, 0, (cudaStream_t)stream>>>(npts, d_mo, nullptr, ld, nmo, d_qt, 1.0, d_rho);
    return cuda_status(cudaGetLastError(), "okg_ci_rho_matrix launch");
}

extern "C" int okg_ci_flux_matrix(int64_t npts, const double* d_mo, const double* d_drv, int64_t ld, int nmo,
                                  const double* d_qt, double scale, double* d_j, okg_stream stream)
{
    if (npts < 0 || !d_j || (npts > 0 && (!d_mo || !d_drv || !d_qt)) || ld < npts || nmo <= 0)
        return set_error(OKG_ERR_ARG, "okg_ci_flux_matrix: bad argument (NULL pointer, npts < 0, ld < npts, nmo <= 0)");
    if (((uintptr_t)d_qt & 15) != 0) return set_error(OKG_ERR_ARG, "okg_ci_flux_matrix: d_qt not 16-byte aligned");
    if (npts == 0) return OKG_OK;
    bool done = false;
    const int s = ci_split<true>(npts, d_mo, d_drv, ld, nmo, d_qt, scale, d_j, (cudaStream_t)stream, done);
    if (s || done) return s;
    const unsigned nblk = (unsigned)((npts + 127) / 128);
    ci_quad_kernel<true><<<nblk, 128, 0, (cudaStream_t)stream>>>(npts, d_mo, d_drv, ld, nmo, d_qt, scale, d_j);
    return cuda_status(cudaGetLastError(), "okg_ci_flux_matrix launch");
}
