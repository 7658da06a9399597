// Analytic overlap of contracted Cartesian Gaussians between a bra basis at one
// geometry and a ket basis at another, with an optional first derivative of the ket
// and optional ket exponents: orbkit's get_ao_overlap
// (orbkit/analytical_integrals.py:37-116) over cy_overlap.aooverlap
// (orbkit/cy_overlap.pyx:78-163) and get_overlap (orbkit/c_non-grid-based.c:9-52).
//
// Per call, a table holds what a primitive pair shares across all component pairs of
// its two shells (1/(2p), the prefactor, P - A; ov_pairs_kernel).  Then one thread per
// bra row and ket shell (ao_overlap_shell_kernel; kets in the canonical component order), or
// per output Cartesian pair (I, J) (any other ket).  It walks the primitives of I (outer)
// and of J (inner), which is the order orbkit's flattened primitive loop adds them
// to aoom[I, J].  The 1D factors are evaluated with orbkit's operations and
// rounding (IEEE divisions, no FMA contraction): the two terms of a derivative can
// cancel to a small fraction of their size, and only this keeps such elements
// within 1e-12 of orbkit's.  The factors common to all terms of a primitive pair,
// exp(-mu R^2) and (pi/p)^(3/2), use one reciprocal of p and a square root (a few
// units in the last place from orbkit's exp/pow values).  The 1D factors follow the recursion of
// M. Ho and J. M. Hernandez-Perez, "Evaluation of Gaussian Molecular Integrals",
// Mathematica Journal 14 (2012), doi:10.3888/tmj.14-3, that orbkit uses:
//   s(0,0) = 1,  s(1,0) = P - A,
//   s(a,0) = (P - A) s(a-1,0) + (a-1)/(2p) s(a-2,0),
//   s(a,b) = s(a+1,b-1) + (A - B) s(a,b-1),
// evaluated bottom-up in a small table instead of recursively (same values).
//
// A derivative d/dx_d of the ket (drv = d + 1) replaces its 1D factor along d by
// l s(l_a, l_b - 1) - 2 beta s(l_a, l_b + 1) (only the second term when l_b = 0),
// the two terms added to the element separately as orbkit does.
//
// The plan holds the basis tables on the device: per listed Cartesian row its
// primitive range, atom and packed exponents (bra from ao_spec, ket optionally
// overridden), the primitive (alpha, c) pairs and the primitive norms
// ao_norm(l, m, n, alpha) of orbkit/c_support.c:177-188 per (row, primitive),
// computed on the host once with the same formula.  The per-AO 'N' factor and the
// spherical transform (orbkit/analytical_integrals.py:109-116, 118-182) are applied
// by a second kernel: out[r, s] = sum_a sum_b k_a k_b (N_a N_b S[a, b]).
#include <math.h>

#include <algorithm>
#include <vector>

#include "okg_internal.cuh"

#define OKG_OV_MAXV 24  // longest vertical recursion: max l_bra + max l_ket + 2
#define OV_PAIR_TABLE_MAX (2ull << 30)  // bytes of the primitive-pair table a plan may hold

namespace okg {

struct OvRow {
    int prim0;  // first primitive (into prim)
    int nprim;
    int atom;
    int rp0;    // first (row, primitive) norm
    int la;     // bra exponents packed lx | ly << 8 | lz << 16
    int lb;     // ket exponents, same packing
};

__device__ __forceinline__ int lcomp(int packed, int d) { return (packed >> (8 * d)) & 0xff; }

// (n / 2p) rounded once, n = a - 1 >= 1: multiples of the pair's 1/(2p) and 3/(2p) by a power
// of two are exact, so the IEEE division is left for n = 5, 7, 9, ...
__device__ __forceinline__ double recur(int n, double h1, double h3, double p)
{
    switch (n) {
    case 1: return h1;
    case 2: return 2.0 * h1;
    case 3: return h3;
    case 4: return 4.0 * h1;
    case 6: return 2.0 * h3;
    case 8: return 8.0 * h1;
    default: return (double)n / (2.0 * p);
    }
}

// s(la, lb) along one axis (and, for the derivative axis, s(la, lb - 1) and
// s(la, lb + 1)).  v holds s(a, k) for a >= la after transfer round k.
__device__ __forceinline__ void os_axis(double xpa, double ab, double p, int la, int lb, bool deriv, double* v,
                                        double& s0, double& sm, double& sp)
{
    const int top = la + lb + (deriv ? 1 : 0);
    v[0] = 1.0;
    if (top >= 1) v[1] = xpa;
    for (int a = 2; a <= top; ++a)
        v[a] = __dadd_rn(__dmul_rn(xpa, v[a - 1]), __dmul_rn((double)(a - 1) / (2.0 * p), v[a - 2]));
    s0 = v[la];
    sm = 0.0;
    const int rounds = lb + (deriv ? 1 : 0);
    for (int k = 1; k <= rounds; ++k) {
        if (deriv && k == lb) sm = v[la];  // s(la, lb - 1) is v[la] after round lb - 1
        for (int a = la; a <= top - k; ++a) v[a] = __dadd_rn(v[a + 1], __dmul_rn(ab, v[a]));
        if (k == lb) s0 = v[la];
    }
    sp = v[la];
}

// Quantities of a primitive pair (bra primitive i at its atom in geo_a, ket primitive j
// at its atom in geo_b) shared by every Cartesian component pair of the two shells:
// 1/(2p) and 3/(2p) of p = alpha + beta, pref = exp(-mu R^2) (pi/p)^(3/2) (0 where the
// exponential underflows) and P - A per axis.  Evaluated once per call into a table of
// nprim x nprim entries when the plan holds one, with the same operations as the
// element kernel's own evaluation.
struct alignas(16) OvPair {
    double pref, h1, xpa[3], h3;  // h1 = 1 / (2p), h3 = 3 / (2p)
};

// n / p rounded once, y = 1/p rounded once: two Newton corrections of the quotient with exact
// remainders (P. W. Markstein, IBM J. Res. Dev. 34 (1990) 111); p and n far from the ends of
// the exponent range.
__device__ __forceinline__ double quotient(double n, double p, double y)
{
    double q = n * y;
    q = fma(fma(-q, p, n), y, q);
    return fma(fma(-q, p, n), y, q);
}

// Per call about 100 FP64 operations per entry were 0.23 ms for 1128 primitives (87 % of the
// FP64 pipe), a third of a matrix: the exponential in integers, corrected quotients instead
// of four IEEE divisions and half the entries leave about a third of that.
// SYM: bra and ket at the same positions; entries (i, j) and (j, i) share everything but
// which atom P - A refers to, so the threads below the diagonal leave and the others write
// both (bit for bit what two threads would).
template <bool SYM>
__global__ void ov_pairs_kernel(int nprim, const double2* __restrict__ prim, const int* __restrict__ prim_atom,
                                const double* __restrict__ geo_a, const double* __restrict__ geo_b,
                                const uint64_t* __restrict__ tab, OvPair* __restrict__ pairs)
{
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    const int i = blockIdx.y * blockDim.y + threadIdx.y;
    if (i >= nprim || j >= nprim || (SYM && j < i)) return;
    const double al = prim[i].x, be = prim[j].x;
    double A[3], B[3];
    double rr = 0.0;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        A[d] = geo_a[3 * prim_atom[i] + d];
        B[d] = geo_b[3 * prim_atom[j] + d];
        const double ab = A[d] - B[d];
        rr = fma(ab, ab, rr);
    }
    OvPair e;
    const double p = al + be, inv_p = 1.0 / p;
    const bool plain = p > 1.0e-100 && p < 1.0e100;  // (and finite)
    e.h1 = 0.5 * inv_p;
    e.h3 = plain ? quotient(1.5, p, inv_p) : 3.0 / (2.0 * p);
    const double arg = al * be * inv_p * rr;
    if (arg > 746.0) {
        e.pref = 0.0;  // exp(-arg) is 0 in double
    } else {
        uint64_t m;
        int x;
        split_mantissa(arg, m, x);
        const double t = M_PI * inv_p;
        // (negative or non-finite arguments: alpha or beta out of their usual range)
        const double ex = arg >= 0.0 ? exp_neg(m, x, 0xB8AA3B295C17F0BCull, -63, tab) : exp(-arg);
        e.pref = ex * t * sqrt(t);
    }
    double P[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const double n = __dadd_rn(__dmul_rn(al, A[d]), __dmul_rn(be, B[d]));
        P[d] = plain && fabs(n) < 1.0e100 && (fabs(n) > 1.0e-100 || n == 0.0) ? quotient(n, p, inv_p) : n / p;
        e.xpa[d] = -(A[d] - P[d]);
    }
    pairs[(long long)i * nprim + j] = e;
    if (SYM && j != i) {
#pragma unroll
        for (int d = 0; d < 3; ++d) e.xpa[d] = -(B[d] - P[d]);
        pairs[(long long)j * nprim + i] = e;
    }
}

// Elements of one bra row with every component of a ket shell in the canonical (Molden)
// order, the common case: a warp takes one bra row I and 32 ket shells of one (L, primitive
// count), so the loops are uniform.  Per primitive pair the one-dimensional factors
// s(la, 0 .. L (+ 1)) are built once per axis and shared by the shell's components, with the
// operations and the rounding of the one-element kernel below (the elements are the same
// bits): for a d shell 6 components share them, for f 10.  Bound by the FP64 pipe (62-74 %
// active).  120 atoms, 1560 Cartesian rows, one matrix with its pair table and transform:
// 0.95 ms with the one-element kernel, 0.46 ms with this one (a derivative matrix).
struct OvKet {
    int prim0, nprim, atom, rp0, row0;  // first primitive, count, atom, first norm, first row
};

template <int LB, bool DRV>
__device__ __forceinline__ void axis_factors(double xpa, double ab, double h1, double h3, double p, int la,
                                             double (&sb)[LB + 2])
{
    constexpr int N = LB + (DRV ? 2 : 1);
    double w[N];
    // s(0), s(1), ... up to s(la), then the window s(la) .. s(la + N - 1)
    double prev = 0.0, cur = 1.0;
    for (int a = 1; a <= la; ++a) {
        const double nxt = a == 1 ? xpa : __dadd_rn(__dmul_rn(xpa, cur), __dmul_rn(recur(a - 1, h1, h3, p), prev));
        prev = cur;
        cur = nxt;
    }
    w[0] = cur;
#pragma unroll
    for (int i = 1; i < N; ++i) {
        const int a = la + i;
        const double nxt = a == 1 ? xpa : __dadd_rn(__dmul_rn(xpa, cur), __dmul_rn(recur(a - 1, h1, h3, p), prev));
        prev = cur;
        cur = nxt;
        w[i] = cur;
    }
    sb[0] = w[0];
#pragma unroll
    for (int k = 1; k < N; ++k) {
#pragma unroll
        for (int i = 0; i < N - k; ++i) w[i] = __dadd_rn(w[i + 1], __dmul_rn(ab, w[i]));
        sb[k] = w[0];
    }
}

struct OvShellArgs {
    int nrow;
    const OvRow* rows;
    const OvKet* kets;
    int shell0[OKG_MAX_L + 2];   // ket shells of each L
    int block0[OKG_MAX_L + 2];   // first block column of each L, highest L first
    const double2* prim;
    const double* pnorm;
    const double* geo_a;
    const double* geo_b;
    const OvPair* pairs;
    int nprim;
    double* out;
    long long ld;
};

template <int LB, int DD>  // DD: derivative axis, or -1
__device__ __forceinline__ void shell_elements(const OvShellArgs& G, int bx)
{
    const int nrow = G.nrow, nprim = G.nprim, nket = G.shell0[LB + 1] - G.shell0[LB];
    const OvRow* __restrict__ rows = G.rows;
    const OvKet* __restrict__ kets = G.kets + G.shell0[LB];
    const double2* __restrict__ prim = G.prim;
    const double* __restrict__ pnorm = G.pnorm;
    const double* __restrict__ geo_a = G.geo_a;
    const double* __restrict__ geo_b = G.geo_b;
    const OvPair* __restrict__ pairs = G.pairs;
    double* __restrict__ out = G.out;
    const long long ld = G.ld;
    constexpr int NC = (LB + 1) * (LB + 2) / 2;
    const int jk = bx * 32 + threadIdx.x;
    const int I = blockIdx.y * blockDim.y + threadIdx.y;
    if (I >= nrow) return;
    const bool live = jk < nket;
    const OvRow ri = rows[I];
    const OvKet kt = kets[live ? jk : nket - 1];
    double AB[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) AB[d] = geo_a[3 * ri.atom + d] - geo_b[3 * kt.atom + d];
    const int la[3] = {lcomp(ri.la, 0), lcomp(ri.la, 1), lcomp(ri.la, 2)};
    double acc[NC];
#pragma unroll
    for (int c = 0; c < NC; ++c) acc[c] = 0.0;
    // (the lanes of a warp may differ in the primitive count at the end of a group)
    const int np = __reduce_max_sync(0xffffffffu, kt.nprim);
    for (int ip = 0; ip < ri.nprim; ++ip) {
        const double2 pa = prim[ri.prim0 + ip];
        const double na = pnorm[ri.rp0 + ip];
        for (int jp = 0; jp < np; ++jp) {
            const bool on = jp < kt.nprim;
            const double2* e = reinterpret_cast<const double2*>(pairs + (long long)(ri.prim0 + ip) * nprim + kt.prim0 +
                                                               (on ? jp : 0));
            const double2 e0 = e[0], e1 = e[1], e2 = e[2];
            if (__all_sync(0xffffffffu, !on || e0.x == 0.0)) continue;  // the pair adds exactly 0
            if (!on) continue;
            const double2 pb = prim[kt.prim0 + jp];
            const double p = pa.x + pb.x;
            double s[3][LB + 2];
            axis_factors<LB, DD == 0>(e1.x, AB[0], e0.y, e2.y, p, la[0], s[0]);
            axis_factors<LB, DD == 1>(e1.y, AB[1], e0.y, e2.y, p, la[1], s[1]);
            axis_factors<LB, DD == 2>(e2.x, AB[2], e0.y, e2.y, p, la[2], s[2]);
            [&]<int... J>(std::integer_sequence<int, J...>) {
                (
                    [&] {
                        constexpr int b[3] = {canon_l(LB, J, 0), canon_l(LB, J, 1), canon_l(LB, J, 2)};
                        const double nb = pnorm[kt.rp0 + J * kt.nprim + jp];
                        if constexpr (DD < 0) {
                            const double v = __dmul_rn(__dmul_rn(__dmul_rn(e0.x, s[0][b[0]]), s[1][b[1]]), s[2][b[2]]);
                            acc[J] = __dadd_rn(acc[J], __dmul_rn(__dmul_rn(__dmul_rn(__dmul_rn(pa.y, pb.y), na), nb), v));
                        } else {
                            constexpr int lbd = b[DD < 0 ? 0 : DD];
                            if constexpr (lbd > 0) {
                                const double v = __dmul_rn(__dmul_rn(__dmul_rn(e0.x, s[0][b[0] - (DD == 0)]), s[1][b[1] - (DD == 1)]),
                                                           s[2][b[2] - (DD == 2)]);
                                const double t = __dmul_rn(__dmul_rn(__dmul_rn((double)lbd * pa.y, pb.y), na), nb);
                                acc[J] = __dadd_rn(acc[J], __dmul_rn(t, v));
                            }
                            const double v = __dmul_rn(__dmul_rn(__dmul_rn(e0.x, s[0][b[0] + (DD == 0)]), s[1][b[1] + (DD == 1)]),
                                                       s[2][b[2] + (DD == 2)]);
                            const double t = __dmul_rn(__dmul_rn(__dmul_rn(__dmul_rn(-2.0 * pb.x, pa.y), pb.y), na), nb);
                            acc[J] = __dadd_rn(acc[J], __dmul_rn(t, v));
                        }
                    }(),
                    ...);
            }(std::make_integer_sequence<int, NC>{});
        }
    }
    if (live) {
        double* o = out + (long long)I * ld + kt.row0;
#pragma unroll
        for (int c = 0; c < NC; ++c) o[c] = acc[c];
    }
}

// All ket shells in one launch (separate launches per L left a partly filled last wave each).
template <int DD>
__global__ void __launch_bounds__(128, 4) ao_overlap_shell_kernel(const __grid_constant__ OvShellArgs G)
{
    const int bx = blockIdx.x;
    if (bx >= G.block0[0]) shell_elements<0, DD>(G, bx - G.block0[0]);
    else if (bx >= G.block0[1]) shell_elements<1, DD>(G, bx - G.block0[1]);
    else if (bx >= G.block0[2]) shell_elements<2, DD>(G, bx - G.block0[2]);
    else if (bx >= G.block0[3]) shell_elements<3, DD>(G, bx - G.block0[3]);
    else shell_elements<4, DD>(G, bx - G.block0[4]);
}

// A warp computes 32 elements of one bra row I.  Its kets are consecutive in the
// plan's ket order (sorted by primitive count, then exponents), so the lanes run
// the same primitive loops and recursion lengths; a primitive pair is skipped only
// when exp(-mu R^2) underflows for every lane (it contributes exactly 0 to the
// others as well).
template <bool TABLE>
__global__ void __launch_bounds__(256) ao_overlap_kernel(int nrow, const OvRow* __restrict__ rows,
                                                         const int* __restrict__ ket_order,
                                                         const double2* __restrict__ prim,
                                                         const double* __restrict__ pnorm,
                                                         const double* __restrict__ geo_a,
                                                         const double* __restrict__ geo_b,
                                                         const OvPair* __restrict__ pairs, int nprim, int drv,
                                                         double* __restrict__ out, long long ld)
{
    const int Jo = blockIdx.x * blockDim.x + threadIdx.x;
    const int I = blockIdx.y * blockDim.y + threadIdx.y;
    if (I >= nrow || Jo >= nrow) return;
    const int J = ket_order[Jo];
    const OvRow ri = rows[I], rj = rows[J];
    double A[3], B[3], AB[3];
    double rr = 0.0;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        A[d] = geo_a[3 * ri.atom + d];
        B[d] = geo_b[3 * rj.atom + d];
        AB[d] = A[d] - B[d];
        rr = fma(AB[d], AB[d], rr);
    }
    const int dd = drv - 1;  // derivative axis or -1
    double v[OKG_OV_MAXV];
    double acc = 0.0;
    for (int ip = 0; ip < ri.nprim; ++ip) {
        const double2 pa = prim[ri.prim0 + ip];
        const double na = pnorm[ri.rp0 + ip];
        for (int jp = 0; jp < rj.nprim; ++jp) {
            const double2 pb = prim[rj.prim0 + jp];
            const double nb = pnorm[rj.rp0 + jp];
            const double al = pa.x, be = pb.x;
            double pref, p, xpa_t[3];
            if (TABLE) {
                const double2* e = reinterpret_cast<const double2*>(pairs + (long long)(ri.prim0 + ip) * nprim +
                                                                   rj.prim0 + jp);
                const double2 e0 = e[0], e1 = e[1], e2 = e[2];
                pref = e0.x;
                p = al + be;
                xpa_t[0] = e1.x;
                xpa_t[1] = e1.y;
                xpa_t[2] = e2.x;
                if (__all_sync(__activemask(), pref == 0.0)) continue;  // the pair adds exactly 0
            } else {
                const double inv_p = 1.0 / (al + be);
                const double arg = al * be * inv_p * rr;
                if (__all_sync(__activemask(), arg > 746.0)) continue;  // exp(-arg) is 0 in double: adds exactly 0
                const double eab = exp(-arg);
                const double t = M_PI * inv_p;
                pref = eab * t * sqrt(t);
                p = al + be;
            }
            // product of the 1D factors of the non-derivative axes, in axis order;
            // along the derivative axis the two shifted factors are kept apart
            double s_plain = pref, s_minus = pref, s_plus = pref;
            int lbd = 0;
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                double xpa;
                if (TABLE) {
                    xpa = xpa_t[d];
                } else {
                    const double P = __dadd_rn(__dmul_rn(al, A[d]), __dmul_rn(be, B[d])) / p;
                    xpa = -(A[d] - P);
                }
                const int la = lcomp(ri.la, d), lb = lcomp(rj.lb, d);
                const bool deriv = (d == dd);
                double s0, sm, sp;
                os_axis(xpa, AB[d], p, la, lb, deriv, v, s0, sm, sp);
                if (deriv) {
                    lbd = lb;
                    s_minus = __dmul_rn(s_minus, sm);
                    s_plus = __dmul_rn(s_plus, sp);
                    s_plain = __dmul_rn(s_plain, s0);
                } else {
                    s_plain = __dmul_rn(s_plain, s0);
                    s_minus = __dmul_rn(s_minus, s0);
                    s_plus = __dmul_rn(s_plus, s0);
                }
            }
            const double cc = __dmul_rn(pa.y, pb.y);
            if (dd < 0) {
                acc = __dadd_rn(acc, __dmul_rn(__dmul_rn(__dmul_rn(cc, na), nb), s_plain));
            } else {
                if (lbd > 0) {
                    const double t = __dmul_rn(__dmul_rn(__dmul_rn((double)lbd * pa.y, pb.y), na), nb);
                    acc = __dadd_rn(acc, __dmul_rn(t, s_minus));
                }
                const double t = __dmul_rn(__dmul_rn(__dmul_rn(__dmul_rn(-2.0 * be, pa.y), pb.y), na), nb);
                acc = __dadd_rn(acc, __dmul_rn(t, s_plus));
            }
        }
    }
    out[(long long)I * ld + J] = acc;
}

// out[r, s] = sum_{a in r} sum_{b in s} (k_a k_b) (N_a N_b S[a, b]); for a Cartesian
// output (nsph = 0) the rows are the Cartesian rows with k = 1.
__global__ void aoom_transform_kernel(int nout, const int* __restrict__ ptr, const int* __restrict__ cart,
                                      const double* __restrict__ coef, const double* __restrict__ renorm,
                                      const double* __restrict__ S, long long lds, double* __restrict__ out,
                                      long long ld)
{
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    const int r = blockIdx.y * blockDim.y + threadIdx.y;
    if (r >= nout || s >= nout) return;
    const int i0 = ptr[r], i1 = ptr[r + 1], j0 = ptr[s], j1 = ptr[s + 1];
    // (most rows are one Cartesian row with coefficient 1: its element as it is)
    if (!renorm && i1 - i0 == 1 && j1 - j0 == 1 && coef[i0] == 1.0 && coef[j0] == 1.0) {
        out[(long long)r * ld + s] = S[(long long)cart[i0] * lds + cart[j0]] + 0.0;
        return;
    }
    double acc = 0.0;
    for (int i = i0; i < i1; ++i) {
        const int a = cart[i];
        const double ka = coef[i];
        const double na = renorm ? renorm[a] : 1.0;
        for (int j = j0; j < j1; ++j) {
            const int b = cart[j];
            double sab = S[(long long)a * lds + b];
            if (renorm) sab = __dmul_rn(__dmul_rn(na, renorm[b]), sab);
            acc = __dadd_rn(acc, __dmul_rn(__dmul_rn(ka, coef[j]), sab));
        }
    }
    out[(long long)r * ld + s] = acc;
}

}  // namespace okg

using namespace okg;

struct okg_overlap_plan {
    // ket shells whose rows are the canonical components in order, sorted by (L, primitives):
    // [shell0[L], shell0[L + 1]) per L; all kets of the plan, or none (canonical = 0)
    OvKet* kets = nullptr;
    uint64_t* exp_tab = nullptr;  // 2^(63 - j/2048), for the pair table
    int shell0[OKG_MAX_L + 2] = {};
    int canonical = 0;
    std::vector<int> h_shell_ncart;
    int* ket_order = nullptr;  // kets sorted by (primitive count, exponents): the kernel's column order
    int* prim_atom = nullptr;  // atom of every primitive
    OvPair* pairs = nullptr;   // nprim x nprim primitive-pair table (NULL above OV_PAIR_TABLE_MAX bytes)
    int natom, nshell, ncart, nprim, nout;
    int max_la;
    int spherical, has_renorm;
    std::vector<OvRow> h_rows;
    std::vector<int> h_lxa;  // ncart x 3 (bra)
    OvRow* rows = nullptr;
    double2* prim = nullptr;
    double* pnorm = nullptr;
    double* renorm = nullptr;
    int* tptr = nullptr;    // transform rows (nout + 1)
    int* tcart = nullptr;
    double* tcoef = nullptr;
    double* work = nullptr; // ncart x ncart Cartesian matrix before the transform
    int max_lb;             // of the current ket exponents
    int device;
};

static double ov_dfact(int n) { return n <= 0 ? 1.0 : n * ov_dfact(n - 2); }

// orbkit/c_support.c:177-188 (ao_norm), evaluated on the host as orbkit does.
static double ov_ao_norm(int l, int m, int n, double alpha, int is_normalized)
{
    if (is_normalized > 0) return 1.0;
    return pow(2. / M_PI, 3. / 4.) * (pow(2., l + m + n) * pow(alpha, (2. * l + 2. * m + 2. * n + 3.) / 4.)) /
           pow(ov_dfact(2 * l - 1) * ov_dfact(2 * m - 1) * ov_dfact(2 * n - 1), 0.5);
}

static int ov_pack(const int* l) { return l[0] | (l[1] << 8) | (l[2] << 16); }

// Kets sorted by (primitive count, packed ket exponents, row): rows a warp handles
// together then run the same loops.
static std::vector<int> ov_ket_order(const std::vector<OvRow>& rows)
{
    std::vector<int> o(rows.size());
    for (size_t i = 0; i < o.size(); ++i) o[i] = (int)i;
    std::stable_sort(o.begin(), o.end(), [&](int a, int b) {
        if (rows[a].nprim != rows[b].nprim) return rows[a].nprim < rows[b].nprim;
        return rows[a].lb < rows[b].lb;
    });
    return o;
}

// The plan's ket shells for the shell kernel; empty if a shell's listed rows are not the
// canonical components of one L in order (explicit component lists, shifted exponents).
static std::vector<OvKet> ov_canonical_kets(const std::vector<OvRow>& rows, const std::vector<int>& ncart, int (&shell0)[OKG_MAX_L + 2])
{
    std::vector<OvKet> k;
    std::vector<int> ls;
    int r0 = 0;
    for (size_t s = 0; s < ncart.size(); r0 += ncart[s], ++s) {
        int L = -1;
        for (int l = 0; l <= OKG_MAX_L; ++l)
            if (ncart[s] == ncanon(l)) L = l;
        if (L < 0) return {};
        for (int c = 0; c < ncart[s]; ++c)
            for (int d = 0; d < 3; ++d)
                if (((rows[r0 + c].lb >> (8 * d)) & 0xff) != canon_l(L, c, d)) return {};
        k.push_back(OvKet{rows[r0].prim0, rows[r0].nprim, rows[r0].atom, rows[r0].rp0, r0});
        ls.push_back(L);
    }
    std::vector<int> o(k.size());
    for (size_t i = 0; i < o.size(); ++i) o[i] = (int)i;
    std::stable_sort(o.begin(), o.end(), [&](int a, int b) {
        return ls[a] != ls[b] ? ls[a] < ls[b] : k[a].nprim < k[b].nprim;
    });
    std::vector<OvKet> sorted;
    for (int l = 0; l <= OKG_MAX_L + 1; ++l) shell0[l] = 0;
    for (int i : o) {
        sorted.push_back(k[i]);
        ++shell0[ls[i] + 1];
    }
    for (int l = 1; l <= OKG_MAX_L + 1; ++l) shell0[l] += shell0[l - 1];
    return sorted;
}

static void ov_free(okg_overlap_plan* p)
{
    if (!p) return;
    cudaFree(p->rows);
    cudaFree(p->prim);
    cudaFree(p->pnorm);
    cudaFree(p->renorm);
    cudaFree(p->tptr);
    cudaFree(p->tcart);
    cudaFree(p->tcoef);
    cudaFree(p->work);
    cudaFree(p->ket_order);
    cudaFree(p->prim_atom);
    cudaFree(p->pairs);
    cudaFree(p->kets);
    cudaFree(p->exp_tab);
    delete p;
}

template <class T>
static int ov_upload(T** dst, const T* src, size_t n, const char* what)
{
    if (n == 0) return OKG_OK;
    cudaError_t e = cudaMalloc((void**)dst, n * sizeof(T));
    if (e != cudaSuccess) return cuda_status(e, what);
    return cuda_status(cudaMemcpy(*dst, src, n * sizeof(T), cudaMemcpyHostToDevice), what);
}

extern "C" int okg_overlap_plan_create(int natom, int nshell, const int* h_shell_atom, const int* h_shell_ncart,
                                       const int* h_shell_nprim, const int* h_lxlylz, int is_normalized,
                                       const double* h_prim, const double* h_renorm, int nsph, const int* h_sph_ptr,
                                       const int* h_sph_cart, const double* h_sph_coef, okg_overlap_plan** out)
{
    if (!out) return set_error(OKG_ERR_ARG, "okg_overlap_plan_create: out is NULL");
    *out = nullptr;
    if (natom <= 0 || nshell <= 0 || !h_shell_atom || !h_shell_ncart || !h_shell_nprim || !h_lxlylz || !h_prim)
        return set_error(OKG_ERR_ARG, "okg_overlap_plan_create: empty basis or NULL array");
    if (nsph < 0 || (nsph > 0 && (!h_sph_ptr || !h_sph_cart || !h_sph_coef)))
        return set_error(OKG_ERR_ARG, "okg_overlap_plan_create: spherical transform arrays missing");
    okg_overlap_plan* P = new okg_overlap_plan();
    P->natom = natom;
    P->nshell = nshell;
    int ncart = 0, nprim = 0, nrp = 0, max_l = 0;
    for (int s = 0; s < nshell; ++s) {
        const int nc = h_shell_ncart[s], np = h_shell_nprim[s], at = h_shell_atom[s];
        if (nc <= 0 || np <= 0 || at < 0 || at >= natom) {
            delete P;
            return set_error(OKG_ERR_ARG, "okg_overlap_plan_create: shell with no components/primitives or bad atom");
        }
        for (int r = 0; r < nc; ++r) {
            const int* l = h_lxlylz + 3 * (ncart + r);
            for (int d = 0; d < 3; ++d) {
                if (l[d] < 0 || l[d] > 64) {
                    delete P;
                    return set_error(OKG_ERR_L, "okg_overlap_plan_create: Cartesian exponent outside 0..64");
                }
                max_l = l[d] > max_l ? l[d] : max_l;
            }
            OvRow row;
            row.prim0 = nprim;
            row.nprim = np;
            row.atom = at;
            row.rp0 = nrp;
            row.la = row.lb = ov_pack(l);
            P->h_rows.push_back(row);
            P->h_lxa.insert(P->h_lxa.end(), l, l + 3);
            nrp += np;
        }
        P->h_shell_ncart.push_back(nc);
        ncart += nc;
        nprim += np;
    }
    if (2 * max_l + 2 > OKG_OV_MAXV - 1) {
        delete P;
        return set_error(OKG_ERR_L, "okg_overlap_plan_create: Cartesian exponent too large for the overlap tables");
    }
    std::vector<double2> prim(nprim);
    for (int i = 0; i < nprim; ++i) prim[i] = make_double2(h_prim[2 * i], h_prim[2 * i + 1]);
    std::vector<double> pnorm(nrp);
    for (int r = 0; r < ncart; ++r) {
        const OvRow& row = P->h_rows[r];
        const int* l = &P->h_lxa[3 * r];
        for (int q = 0; q < row.nprim; ++q)
            pnorm[row.rp0 + q] = ov_ao_norm(l[0], l[1], l[2], prim[row.prim0 + q].x, is_normalized);
    }
    // transform rows: spherical rows from the tables, else one Cartesian row each
    std::vector<int> tptr, tcart;
    std::vector<double> tcoef;
    if (nsph > 0) {
        if (h_sph_ptr[0] != 0) {
            delete P;
            return set_error(OKG_ERR_ARG, "okg_overlap_plan_create: sph_ptr[0] must be 0");
        }
        for (int r = 0; r <= nsph; ++r) tptr.push_back(h_sph_ptr[r]);
        for (int r = 0; r < nsph; ++r)
            if (h_sph_ptr[r + 1] < h_sph_ptr[r]) {
                delete P;
                return set_error(OKG_ERR_ARG, "okg_overlap_plan_create: sph_ptr not ascending");
            }
        for (int i = 0; i < h_sph_ptr[nsph]; ++i) {
            if (h_sph_cart[i] < 0 || h_sph_cart[i] >= ncart) {
                delete P;
                return set_error(OKG_ERR_ARG, "okg_overlap_plan_create: spherical component outside the Cartesian rows");
            }
            tcart.push_back(h_sph_cart[i]);
            tcoef.push_back(h_sph_coef[i]);
        }
    } else {
        for (int r = 0; r <= ncart; ++r) tptr.push_back(r);
        for (int r = 0; r < ncart; ++r) {
            tcart.push_back(r);
            tcoef.push_back(1.0);
        }
    }
    cudaGetDevice(&P->device);
    P->ncart = ncart;
    P->nprim = nprim;
    P->nout = nsph > 0 ? nsph : ncart;
    P->spherical = nsph > 0;
    P->has_renorm = h_renorm != nullptr;
    P->max_la = max_l;
    P->max_lb = max_l;
    int st = OKG_OK;
    if ((st = ov_upload(&P->rows, P->h_rows.data(), P->h_rows.size(), "okg_overlap_plan_create")) ||
        (st = ov_upload(&P->prim, prim.data(), prim.size(), "okg_overlap_plan_create")) ||
        (st = ov_upload(&P->pnorm, pnorm.data(), pnorm.size(), "okg_overlap_plan_create")) ||
        (h_renorm && (st = ov_upload(&P->renorm, h_renorm, (size_t)ncart, "okg_overlap_plan_create"))) ||
        (st = ov_upload(&P->tptr, tptr.data(), tptr.size(), "okg_overlap_plan_create")) ||
        (st = ov_upload(&P->tcart, tcart.data(), tcart.size(), "okg_overlap_plan_create")) ||
        (st = ov_upload(&P->tcoef, tcoef.data(), tcoef.size(), "okg_overlap_plan_create")) ||
        (st = ov_upload(&P->ket_order, ov_ket_order(P->h_rows).data(), (size_t)ncart, "okg_overlap_plan_create"))) {
        ov_free(P);
        return st;
    }
    cudaError_t e = cudaMalloc((void**)&P->work, (size_t)ncart * ncart * sizeof(double));
    if (e != cudaSuccess) {
        ov_free(P);
        return cuda_status(e, "okg_overlap_plan_create: workspace");
    }
    // primitive-pair table (geometry-dependent, filled by every okg_ao_overlap call)
    const size_t pair_bytes = (size_t)nprim * nprim * sizeof(OvPair);
    if (pair_bytes <= OV_PAIR_TABLE_MAX) {
        std::vector<int> prim_atom;
        prim_atom.reserve(nprim);
        for (int sh = 0; sh < nshell; ++sh)
            for (int q = 0; q < h_shell_nprim[sh]; ++q) prim_atom.push_back(h_shell_atom[sh]);
        if ((st = ov_upload(&P->prim_atom, prim_atom.data(), prim_atom.size(), "okg_overlap_plan_create")) ||
            (st = ov_upload(&P->exp_tab, split_exp_table(), (size_t)OKG_SPLIT_EXP, "okg_overlap_plan_create"))) {
            ov_free(P);
            return st;
        }
        e = cudaMalloc((void**)&P->pairs, pair_bytes);
        if (e != cudaSuccess) {
            ov_free(P);
            return cuda_status(e, "okg_overlap_plan_create: primitive-pair table");
        }
    }
    const std::vector<OvKet> kets = ov_canonical_kets(P->h_rows, P->h_shell_ncart, P->shell0);
    P->canonical = !kets.empty();
    e = cudaMalloc((void**)&P->kets, sizeof(OvKet) * nshell);
    if (e == cudaSuccess && P->canonical)
        e = cudaMemcpy(P->kets, kets.data(), sizeof(OvKet) * kets.size(), cudaMemcpyHostToDevice);
    if (e != cudaSuccess) {
        ov_free(P);
        return cuda_status(e, "okg_overlap_plan_create: ket shells");
    }
    *out = P;
    return OKG_OK;
}

extern "C" int okg_overlap_plan_destroy(okg_overlap_plan* plan)
{
    ov_free(plan);
    return OKG_OK;
}

extern "C" int okg_overlap_plan_info(const okg_overlap_plan* plan, int* ncart, int* nao)
{
    if (!plan) return set_error(OKG_ERR_ARG, "okg_overlap_plan_info: NULL plan");
    if (ncart) *ncart = plan->ncart;
    if (nao) *nao = plan->nout;
    return OKG_OK;
}

extern "C" int okg_overlap_plan_set_ket(okg_overlap_plan* plan, const int* h_lxlylz_b)
{
    if (!plan) return set_error(OKG_ERR_ARG, "okg_overlap_plan_set_ket: NULL plan");
    int max_lb = 0;
    for (int r = 0; r < plan->ncart; ++r) {
        const int* l = h_lxlylz_b ? h_lxlylz_b + 3 * r : &plan->h_lxa[3 * r];
        for (int d = 0; d < 3; ++d) {
            if (l[d] < 0 || l[d] > 64) return set_error(OKG_ERR_L, "okg_overlap_plan_set_ket: exponent outside 0..64");
            max_lb = l[d] > max_lb ? l[d] : max_lb;
        }
    }
    if (plan->max_la + max_lb + 2 > OKG_OV_MAXV - 1)
        return set_error(OKG_ERR_L, "okg_overlap_plan_set_ket: exponents too large for the overlap tables");
    for (int r = 0; r < plan->ncart; ++r) {
        const int* l = h_lxlylz_b ? h_lxlylz_b + 3 * r : &plan->h_lxa[3 * r];
        plan->h_rows[r].lb = ov_pack(l);
    }
    plan->max_lb = max_lb;
    int st = cuda_status(cudaMemcpy(plan->rows, plan->h_rows.data(), plan->h_rows.size() * sizeof(OvRow),
                                    cudaMemcpyHostToDevice),
                         "okg_overlap_plan_set_ket");
    if (st) return st;
    const std::vector<OvKet> kets = ov_canonical_kets(plan->h_rows, plan->h_shell_ncart, plan->shell0);
    plan->canonical = !kets.empty();
    if (plan->canonical) {
        st = cuda_status(cudaMemcpy(plan->kets, kets.data(), sizeof(OvKet) * kets.size(), cudaMemcpyHostToDevice),
                         "okg_overlap_plan_set_ket");
        if (st) return st;
    }
    const std::vector<int> order = ov_ket_order(plan->h_rows);
    return cuda_status(cudaMemcpy(plan->ket_order, order.data(), order.size() * sizeof(int), cudaMemcpyHostToDevice),
                       "okg_overlap_plan_set_ket");
}

static void ov_shells(const okg_overlap_plan* P, const double* ga, const double* gb, int drv, double* S, long long lds,
                      cudaStream_t st)
{
    OvShellArgs G;
    G.nrow = P->ncart;
    G.rows = P->rows;
    G.kets = P->kets;
    int nb = 0;
    for (int l = 0; l <= OKG_MAX_L + 1; ++l) G.shell0[l] = P->shell0[l];
    for (int l = OKG_MAX_L; l >= 0; --l) {
        G.block0[l] = nb;
        nb += (P->shell0[l + 1] - P->shell0[l] + 31) / 32;
    }
    G.block0[OKG_MAX_L + 1] = 0;
    G.prim = P->prim;
    G.pnorm = P->pnorm;
    G.geo_a = ga;
    G.geo_b = gb;
    G.pairs = P->pairs;
    G.nprim = P->nprim;
    G.out = S;
    G.ld = lds;
    const dim3 blk(32, 4), grd(nb, (P->ncart + 3) / 4);
    switch (drv) {
    case 0: ao_overlap_shell_kernel<-1><<<grd, blk, 0, st>>>(G); break;
    case 1: ao_overlap_shell_kernel<0><<<grd, blk, 0, st>>>(G); break;
    case 2: ao_overlap_shell_kernel<1><<<grd, blk, 0, st>>>(G); break;
    default: ao_overlap_shell_kernel<2><<<grd, blk, 0, st>>>(G); break;
    }
}

extern "C" int okg_ao_overlap(okg_overlap_plan* plan, const double* d_geo_a, const double* d_geo_b, int drv,
                              int raw, double* d_out, int64_t ld, okg_stream stream)
{
    if (!plan || !d_geo_a || !d_geo_b || !d_out)
        return set_error(OKG_ERR_ARG, "okg_ao_overlap: NULL plan, geometry or output");
    if (drv < 0 || drv > 3)
        return set_error(OKG_ERR_DRV, "okg_ao_overlap: only drv 0 (none) and 1..3 (d/dx, d/dy, d/dz) are supported");
    const int nout = raw ? plan->ncart : plan->nout;
    if (ld < nout) return set_error(OKG_ERR_ARG, "okg_ao_overlap: ld smaller than the matrix");
    cudaStream_t st = (cudaStream_t)stream;
    const bool direct = raw || (!plan->spherical && !plan->has_renorm);
    double* S = direct ? d_out : plan->work;
    const long long lds = direct ? ld : plan->ncart;
    const dim3 blk(32, 8);
    const dim3 grd((plan->ncart + 31) / 32, (plan->ncart + 7) / 8);
    if (plan->pairs) {
        const dim3 gpp((plan->nprim + 31) / 32, (plan->nprim + 7) / 8);
        if (d_geo_a == d_geo_b)
            ov_pairs_kernel<true><<<gpp, blk, 0, st>>>(plan->nprim, plan->prim, plan->prim_atom, d_geo_a, d_geo_b,
                                                       plan->exp_tab, plan->pairs);
        else
            ov_pairs_kernel<false><<<gpp, blk, 0, st>>>(plan->nprim, plan->prim, plan->prim_atom, d_geo_a, d_geo_b,
                                                        plan->exp_tab, plan->pairs);
        if (plan->canonical)
            ov_shells(plan, d_geo_a, d_geo_b, drv, S, lds, st);
        else
            ao_overlap_kernel<true><<<grd, blk, 0, st>>>(plan->ncart, plan->rows, plan->ket_order, plan->prim,
                                                        plan->pnorm, d_geo_a, d_geo_b, plan->pairs, plan->nprim, drv,
                                                        S, lds);
    } else {
        ao_overlap_kernel<false><<<grd, blk, 0, st>>>(plan->ncart, plan->rows, plan->ket_order, plan->prim,
                                                     plan->pnorm, d_geo_a, d_geo_b, nullptr, 0, drv, S, lds);
    }
    int s = cuda_status(cudaGetLastError(), "okg_ao_overlap launch");
    if (s || direct) return s;
    const dim3 tblk(16, 16);
    const dim3 grt((plan->nout + 15) / 16, (plan->nout + 15) / 16);
    aoom_transform_kernel<<<grt, tblk, 0, st>>>(plan->nout, plan->tptr, plan->tcart, plan->tcoef, plan->renorm, S,
                                               lds, d_out, ld);
    return cuda_status(cudaGetLastError(), "okg_ao_overlap transform launch");
}
