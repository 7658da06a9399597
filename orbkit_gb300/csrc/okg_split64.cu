// FP64-accurate AO -> MO -> density on the tensor cores (the large calls of okg_rho and
// okg_eval_mo, value / gradient / Laplacian channels).
//
// Reference computation: orbkit/c_grid-based.c:9-79 (AOs), orbkit/cy_core.pyx:82-101
// (MO = C . AO) and orbkit/core.py:266-304 (density and derivatives).
//
// Why: the FP64 pipe runs 2 FMAs per clock and SM (6.3e11 FMA/s), so the contraction
// C . AO, 4 NMO NAO FMAs per point with gradients, bounds a DFMA kernel.  The FP16
// tensor cores are 1500 times faster, and an FP64 product can be composed of exact
// small-integer products (K. Ozaki et al., "Error-free transformations of matrix
// multiplication", Numer. Algorithms 59 (2012)):
//   * every AO value a (FP64) of a grid point is scaled by a power of two 2^-E above the
//     largest AO of that point and rounded to a 55-bit integer, cut into 7 balanced
//     base-256 digits (-128 .. 127); the coefficients likewise per MO;
//   * the products d_i(a) d_j(c) with i + j = w, integers up to 2^14, have the weight
//     2^(-14 - 8 w); w = 0..6 are kept, 7 accumulators per MO;
//   * an accumulator adds w + 1 products per column.  Up to 146 columns the FP32 accumulators of
//     tcgen05.mma are exact (7 x 146 x 2^14 < 2^24); at the 160 columns of a group the last one
//     (w = 6) could pass 2^24 with every digit at its end, and then rounds by a unit of 2^-62
//     (the products left out may come to 6.1 x 2^-56 per column).
//
// Error.  A value is fixed-point relative to the largest AO of its point, a coefficient to the
// largest of its MO: per column 2^-56 each of their product for the roundings, 6.1 x 2^-56 for
// the products left out.  With n columns the error of an MO value is at most
//     n 2^-53 2^E 2^F,  2^F < 2.1 max|C|,  2^E about the largest AO value (derivative of the
//     class: first derivatives share a scale, and so do second) at the point.
// Where the largest AO and the largest coefficient meet that is the rounding of an FP64 sum;
// an MO that is small at a point where another's AOs are large (a localised orbital near
// another nucleus) keeps as many digits less as it is smaller: it is accurate relative to
// max|C| max|AO|, not to itself, where the DFMA kernel is accurate relative to sum |C| |AO|.
// Densities are sums of squares and see it only where no occupied MO holds the largest AO.
//
// Screening.  A shell (and the steep primitives of a shell) whose bound over the tile's
// points lies 2^-62 below a value that the scale 2^E of every point is known to reach
// cannot change a digit and is left out, and so are panels of 16 columns without a kept
// shell.  Bounds are taken per channel class (values, first, second derivatives).
//
// Range.  What the digits cannot hold (a basis whose flags are raised, see split_prim; MOs
// whose largest coefficient is not finite or not between 2^-900 and 2^1000; points at
// |coordinate| >= 2^170; AO values from 2^985 on), and a wait that expires, raises the call's
// redo word, and the DFMA kernel, launched after this one, computes the call.
//
// Tile: 128 operand rows (2 x 128 with second derivatives): 128 points x 1 channel, or
// 32 points x (value, d/dx, d/dy, d/dz) [+ 32 x (xx, yy, zz, unused)].  Persistent CTAs,
// one per SM, tiles handed out by a device counter; warps of a CTA:
//   generation warps (8, values alone 12)  FP64 radial sums and polynomials of the kept
//                       shells, digits written to the panel's operand slot (ring of slots);
//   epilogue warps (8, second derivatives 4)  accumulators -> FP64 MO values (integer
//                       arithmetic) -> outputs;
//   1 MMA warp, 2 tile warps (screening, scales) that take turns with the tile buffers; the
//                       copies of coefficient digits are requested by a generation lane.
// Every wait is bounded: one that expires raises the redo word, and the block drains its copies
// and MMAs in flight and leaves.
//
// What bounds it (20 atoms, 180 AOs, 40 MOs, 160^3 points, density and gradient): 14.2 ms against
// 254 ms of the DFMA kernel.  FP64 pipe 37 %, tensor pipe 11 % of active cycles (ncu, 96^3
// points); the rest is latency, of tensor-memory loads and of the integer code (digits,
// exponentials, conversion of the accumulators), behind a chain: with more than 32 MOs only one
// set of accumulators fits tensor memory, and the MMAs of a tile wait until the epilogue has
// read the previous tile's.
#include <math.h>

#include <mutex>
#include <vector>

#include "okg_digits.cuh"
#include "okg_internal.cuh"
#include "okg_split64.cuh"

namespace okg {
namespace sp {

using namespace mx;

constexpr int GROUP = 10;               // panels per accumulation (FP32 sums: see the header)
constexpr int MAX_SHELLS = 2048;
constexpr int MAX_PANELS = 768;
constexpr int NBUF = 4;                 // tile buffers
constexpr int NTW = 2;                  // tile warps, each with every second buffer
constexpr int MAX_BIG = 512;
constexpr int TABN = OKG_SPLIT_EXP;     // entries of the 2^(j/2048) table
constexpr int SMEM_MAX = 232448;
enum { OUT_RHO = 0, OUT_MO = 1, OUT_WV = 2 };
constexpr float KEEP_LOG2 = 62.0f;
constexpr float ABS_FLOOR = -1000.0f;   // values below 2^-1000 are dropped
// e^(-alpha d^2) w below 2^-3000 is nothing whatever the polynomial (below 2^192 for points and
// atoms within 2^31 of each other), which may leave the range of a float there
constexpr float NOTHING = -3000.0f;
// Up to which sqrt(alpha) times the error of a coordinate single precision places a tile's
// points.  With an error x per coordinate log2 e^(-alpha d^2) errs by
// 1.443 alpha (2 sqrt(3) d x + 3 x^2); where alpha d^2 <= 735 (beyond ABS_FLOOR nothing counts)
// that is 136 sqrt(alpha) x + 4.3 alpha x^2, here 0.05 at most, which the scales have to spare.
constexpr float WIDE = 3.6e-4f;
// Error of a coordinate that the bounds of the polynomials allow for (a tile of 40 bohr; larger
// ones are wide too).  A constant: kept in a register through the loop over the shells, the tile's
// own error took 7 % of the kernel's time (20 atoms, gradients).  At CLOSE and beyond it is 3 % of
// the distance, a quarter of a bit of the steepest polynomial; tiles with points closer to an
// atom are wide as well (at a nucleus the bound of a steep gradient would be all allowance).
constexpr float NEAR = 8.0e-6f, CLOSE = 64.0f * NEAR;

template <int NCH>
struct Cfg {
    static constexpr int RG = NCH == 7 ? 2 : 1;       // 128-row operand tiles
    static constexpr int PTS = NCH == 1 ? 128 : 32;   // points of an operand tile
    static constexpr int SUB = PTS / 32;              // points per lane of an operand tile
    static constexpr int NCLS = NCH == 1 ? 1 : NCH == 4 ? 2 : 3;
    // Warps: most of the kernel's time is latency (integer digit and exponential code, a slow
    // FP64 pipe), so as many warps as their registers allow.  20 atoms, 96^3 | 12 atoms, 64^3
    // points, ms: values with 3 teams (23 warps of 80 registers) 1.25 | 0.32, with 2 teams
    // (19 warps of 96) 1.32 | 0.32; gradients with 3 teams 3.82 | 0.87, with 2 teams 3.64 |
    // 0.77 (12 epilogue warps: 3.96 | 0.94); second derivatives need 128 registers (15 warps).
    static constexpr int TEAM = 4;                         // generation warps working on one panel
    static constexpr int NTEAM = NCH == 1 ? 3 : 2;         // panels under generation at a time
    static constexpr int EPQ = NCH == 7 ? 1 : 2;           // epilogue warps per 32 accumulator rows
    static constexpr int NGW = TEAM * NTEAM;
    static constexpr int NEW = 4 * EPQ;
    static constexpr int NT = 32 * (NGW + NEW + NTW + 1);
};

struct Args {
    BasisDev B;
    SplitDev S;
    Grid g;
    int nmo, np, npass;           // MOs, columns per pass (multiple of 16), passes
    const unsigned char* bpack;   // [npass][npanel][7 np rows x 32 B]
    const int* fexp;              // [npass np] exponent of each MO's coefficients
    const double* occ;            // [npass np] occupations, zero padded
    unsigned long long* counter;  // tile counter, zero at launch
    double* phi;                  // per CTA [RG][np][128] partial MO values (bases beyond GROUP panels)
    int* redo;                    // raised when the call is not one for the digits after all, or a wait expires
    long long limit;              // polls of a wait
    DrvList drv;
    double* out;                  // MO output: ndrv x nmo x ld; density: rho; cotangents: W, V (2 x nmo x ld)
    const double* g_rho;          // cotangents of rho, and of grad rho (3 x g_ld, or null)
    const double* g_grad;
    long long g_ld;
    int wv_float;
    double* dout;                 // density: ndrv x ld
    double* mo_norm;              // density: nmo sums of MO^2, or null
    long long ld, ntiles;
    int brick, nby, nbz;
    int nsub;                     // 32-point runs of a tile: 4 (128 points), or 1 for few points with derivatives
    int nslot, nacc;              // operand slots, accumulator sets
    unsigned tm_cols;
    int norm_smem;                // the MO norms are summed in shared memory
    int tab_smem;                 // exponents and occupations of the MOs are kept in shared memory
};

// ------------------------------------------------------------------ tile geometry
// Point r of a tile: a brick of nsub x 4 x 8 points of a whole regular grid, else 32 nsub
// consecutive points.
__device__ __forceinline__ bool tile_point(const Args& A, long long tile, int r, long long& p, double& x, double& y,
                                           double& z)
{
    if (A.brick) {
        const long long nbyz = (long long)A.nby * A.nbz;
        int bi, rem;
        if (A.ntiles < 0x7FFFFFFFll) {
            bi = (int)tile / (int)nbyz;
            rem = (int)tile - bi * (int)nbyz;
        } else {
            bi = (int)(tile / nbyz);
            rem = (int)(tile - (long long)bi * nbyz);
        }
        const int bj = rem / A.nbz, bk = rem - bj * A.nbz;
        const int i = bi * A.nsub + (r >> 5), j = bj * 4 + ((r >> 3) & 3), k = bk * 8 + (r & 7);
        const bool valid = i < A.g.nx && j < A.g.ny && k < A.g.nz;
        x = __ldg(A.g.x + (i < A.g.nx ? i : A.g.nx - 1));
        y = __ldg(A.g.y + (j < A.g.ny ? j : A.g.ny - 1));
        z = __ldg(A.g.z + (k < A.g.nz ? k : A.g.nz - 1));
        p = valid ? ((long long)i * A.g.ny + j) * A.g.nz + k : 0;
        return valid;
    }
    p = tile * (32 * A.nsub) + r;
    const bool valid = p < A.g.npts;
    if (!valid) p = A.g.npts - 1;
    grid_point(A.g, p, x, y, z);
    return valid;
}

// ------------------------------------------------------------------ shared memory
struct State {
    unsigned char* slots;   // nslot x (operand digits, coefficient digits)
    uint32_t slot_bytes, a_bytes;
    uint64_t* tab;          // 2^(63 - j/2048)
    long long* tile;        // NBUF
    int* npan;              // NBUF
    double* pts;            // value channel: NBUF x 3 x 128 coordinates
    short* rowexp;          // NBUF x 3 x 128
    unsigned short* plist;  // NBUF x MAX_PANELS
    unsigned char* nkeep;   // NBUF x MAX_SHELLS
    unsigned short* big;    // NTW x MAX_BIG (tile warps)
    unsigned* pbits;        // NTW x MAX_PANELS / 32 (tile warps)
    double* norm;           // 8 x npass np, when A.norm_smem
    double* occ;            // npass np each, when A.tab_smem
    int* fexp;
    double* part;           // (EPQ - 1) x 4 x 32: density sums of a row group's other epilogue warps
    int* last_use;          // nslot: last phase whose coefficient copy was requested, or -1
    int* abort_flag;
    uint32_t full, empty, bfull;          // nslot mbarriers each, 8 B apart
    uint32_t acc_full, acc_empty;         // 2 each
    uint32_t screened, kfree;             // NBUF each
    uint32_t part_full, part_free;        // 4 each
    uint32_t drain;
    uint32_t tmem;
};
constexpr int MAX_SLOTS = 6;
constexpr int NBAR = 3 * MAX_SLOTS + 4 + 2 * NBUF + 8 + 1;
constexpr int AUX_BYTES = TABN * 8 + NBUF * 8 + NBUF * 4 + MAX_SLOTS * 4 + 8 + NBUF * 2 * 3 * 128 + NBUF * MAX_PANELS * 2 +
                          NBUF * MAX_SHELLS + NTW * MAX_BIG * 2 + NTW * MAX_PANELS / 8 +
                          NBAR * 8 + 64;

// Bounded wait that also ends when another role gave up.
__device__ __forceinline__ bool wait(const Args& A, const State& S, uint32_t bar, uint32_t parity)
{
    for (long long it = 0; it < A.limit; ++it) {
        if (mbar_try(bar, parity)) return true;
        if ((it & 255) == 255 && *(volatile int*)S.abort_flag) return false;
    }
    *(volatile int*)A.redo = 1;
    *(volatile int*)S.abort_flag = 1;
    return false;
}

// One answer for the warp (collective instructions follow).
__device__ __forceinline__ bool warp_wait(const Args& A, const State& S, uint32_t bar, uint32_t parity)
{
    return __all_sync(0xffffffffu, wait(A, S, bar, parity));
}

// ------------------------------------------------------------------ FP64 AO values
// position of x^a y^b z^c among the monomials of its degree
__host__ __device__ constexpr int midx(int a, int b, int c) { return (b + c) * (b + c + 1) / 2 + c; }

// s times the monomials of degree D from those of degree D - 1, in place
template <int D>
__device__ __forceinline__ void raise(double* T, double X, double Y, double Z)
{
    T[midx(0, 0, D)] = Z * T[midx(0, 0, D - 1)];
#pragma unroll
    for (int c = D - 1; c >= 0; --c) T[midx(0, D - c, c)] = Y * T[midx(0, D - c - 1, c)];
#pragma unroll
    for (int i = 0; i < D * (D + 1) / 2; ++i) T[i] *= X;
}
template <int N0, int N1>
__device__ __forceinline__ void raise_to(double* T, double X, double Y, double Z)
{
    if constexpr (N0 < N1) {
        raise<N0 + 1>(T, X, Y, Z);
        raise_to<N0 + 1, N1>(T, X, Y, Z);
    }
}

// Power of two nearest to the inverse of the angular norm 1/sqrt((2a-1)!!(2b-1)!!(2c-1)!!) of
// a component: the operand holds 2^-shift chi, the coefficients the rest of the norm, so
// that no column takes digits from the others.
__host__ __device__ constexpr int norm_shift(int a, int b, int c)
{
    constexpr int s[5] = {0, 0, 1, 2, 3};  // 1, 1, 3, 15, 105
    if (a == 2 && b == 2 || a == 2 && c == 2 || b == 2 && c == 2) return 2;  // 9
    return s[a] > s[b] ? (s[a] > s[c] ? s[a] : s[c]) : (s[b] > s[c] ? s[b] : s[c]);
}

// Values, gradients and pure second derivatives of every canonical component of a shell:
// with S0 = R0, S1 = -2 R1, S2 = 4 R2,
//   chi = P S0,  d_x chi = P x S1 + a (P/x) S0,  d_xx chi = P x^2 S2 + (2a + 1) P S1 + a (a-1) (P/x^2) S0,
// about 1.5 FP64 operations per value.  Kept between components are only the monomials of
// degree L - 1 times the radial sums (3 + 3 for a d shell): with all values of a shell formed
// first (19 for a d shell) the registers around the calls of put4 went to local memory, and
// its traffic through what shared memory leaves of the L1 cost more than the arithmetic.
template <int L, int NCH, typename Sink>
__device__ __forceinline__ void shell_values(double X, double Y, double Z, double R0, double S1, double S2, Sink&& sink)
{
    constexpr int N = (L + 1) * (L + 2) / 2, M = L > 0 ? L * (L + 1) / 2 : 1, MM = L > 1 ? L * (L - 1) / 2 : 1;
    double V[M], G[NCH >= 4 ? M : 1], H[NCH == 7 ? M : 1], W[NCH == 7 ? MM : 1];
    V[0] = R0;
    if constexpr (NCH >= 4) G[0] = S1;
    if constexpr (NCH == 7) H[0] = S2;
    if constexpr (L >= 2) {
        raise_to<0, L - 2>(V, X, Y, Z);
        if constexpr (NCH == 7) {
#pragma unroll
            for (int i = 0; i < MM; ++i) W[i] = V[i];
        }
        raise<L - 1>(V, X, Y, Z);
        if constexpr (NCH >= 4) raise_to<0, L - 1>(G, X, Y, Z);
        if constexpr (NCH == 7) raise_to<0, L - 1>(H, X, Y, Z);
    }
    [&]<int... J>(std::integer_sequence<int, J...>) {
        (
            [&] {
                constexpr int a = canon_l(L, J, 0), b = canon_l(L, J, 1), c = canon_l(L, J, 2);
                // P = x_d (P / x_d) along an axis with a non-zero exponent
                constexpr int d = a > 0 ? 0 : b > 0 ? 1 : 2;
                constexpr int m = L == 0 ? 0 : midx(a - (d == 0), b - (d == 1), c - (d == 2));
                const double xd = d == 0 ? X : d == 1 ? Y : Z;
                double v[NCH];
                v[0] = L == 0 ? R0 : xd * V[m];
                if constexpr (NCH >= 4) {
                    const double g = L == 0 ? S1 : xd * G[m];  // P S1
                    v[1] = g * X;
                    v[2] = g * Y;
                    v[3] = g * Z;
                    if constexpr (a > 0) v[1] = fma((double)a, V[midx(a - 1, b, c)], v[1]);
                    if constexpr (b > 0) v[2] = fma((double)b, V[midx(a, b - 1, c)], v[2]);
                    if constexpr (c > 0) v[3] = fma((double)c, V[midx(a, b, c - 1)], v[3]);
                    if constexpr (NCH == 7) {
                        const double h = L == 0 ? S2 : xd * H[m];  // P S2
                        v[4] = fma((double)(2 * a + 1), g, (h * X) * X);
                        v[5] = fma((double)(2 * b + 1), g, (h * Y) * Y);
                        v[6] = fma((double)(2 * c + 1), g, (h * Z) * Z);
                        if constexpr (a > 1) v[4] = fma((double)(a * (a - 1)), W[midx(a - 2, b, c)], v[4]);
                        if constexpr (b > 1) v[5] = fma((double)(b * (b - 1)), W[midx(a, b - 2, c)], v[5]);
                        if constexpr (c > 1) v[6] = fma((double)(c * (c - 1)), W[midx(a, b, c - 2)], v[6]);
                    }
                }
                sink(J, norm_shift(a, b, c), v);
            }(),
            ...);
    }(std::make_integer_sequence<int, N>{});
}

__device__ __forceinline__ void sts64(uint32_t a, uint32_t x, uint32_t y) { asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(a), "r"(x), "r"(y) : "memory"); }

// Digits of four rows (channels of a point) of a column.
__device__ __noinline__ void put4(double v0, double v1, double v2, double v3, int rs0, int rs1, uint32_t a)
{
    const uint64_t t0 = digits7(v0, rs0), t1 = digits7(v1, rs1), t2 = digits7(v2, rs1), t3 = digits7(v3, rs1);
#pragma unroll
    for (int i = 0; i < ND; ++i) {
        const int b = 6 - i;
        if (b >= 4)
            sts64(a + i * DT, digit_pair((uint32_t)(t0 >> 32), (uint32_t)(t1 >> 32), b - 4),
                  digit_pair((uint32_t)(t2 >> 32), (uint32_t)(t3 >> 32), b - 4));
        else
            sts64(a + i * DT, digit_pair((uint32_t)t0, (uint32_t)t1, b), digit_pair((uint32_t)t2, (uint32_t)t3, b));
    }
}

// Values of one shell at the lane's point into the slot; row: first operand row of the
// point (4 rows per point with derivatives, else 1).
template <int L, int NCH>
__device__ __forceinline__ void put_shell(uint32_t slot, int col, double X, double Y, double Z, double R0, double S1,
                                          double S2, int row, int e0, int e1, int e2)
{
    shell_values<L, NCH>(X, Y, Z, R0, S1, S2, [&](int j, int sh, const double* v) {
        const uint32_t a = slot + a_off(row, col + j);
        if constexpr (NCH == 1) {
            put1(v[0], e0 + sh, a);
        } else {
            put4(v[0], v[1], v[2], v[3], e0 + sh, e1 + sh, a);
            if constexpr (NCH == 7) put4(v[4], v[5], v[6], 0.0, e2 + sh, e2 + sh, a + ND * DT);
        }
    });
}

template <int NCH>
__device__ __forceinline__ void gen_shell(const Args& A, const State& S, uint32_t slot, int L, int col, int prim0, int nk,
                                          double X, double Y, double Z, int row, int e0, int e1, int e2)
{
    const double rr = X * X + Y * Y + Z * Z;
    uint64_t mr;
    int er;
    split_mantissa(rr, mr, er);
    // radial sums R0 = sum w e, S1 = -2 sum w alpha e, S2 = 4 sum w alpha^2 e
    double R0 = 0.0, S1 = 0.0, S2 = 0.0;
#pragma unroll 1
    for (int q = 0; q < nk; ++q) {
        const SplitPrim* pr = A.S.prim + prim0 + q;
        const ulonglong2 ae = __ldg((const ulonglong2*)pr);
        const double2 w01 = __ldg((const double2*)pr + 1);
        const double e = exp_neg(mr, er, ae.x, (int)ae.y, S.tab);
        R0 = fma(w01.x, e, R0);
        if (NCH >= 4) S1 = fma(w01.y, e, S1);
        if (NCH == 7) S2 = fma(__ldg(&pr->w2), e, S2);
    }
    switch (L) {
    case 0: put_shell<0, NCH>(slot, col, X, Y, Z, R0, S1, S2, row, e0, e1, e2); break;
    case 1: put_shell<1, NCH>(slot, col, X, Y, Z, R0, S1, S2, row, e0, e1, e2); break;
    case 2: put_shell<2, NCH>(slot, col, X, Y, Z, R0, S1, S2, row, e0, e1, e2); break;
    case 3: put_shell<3, NCH>(slot, col, X, Y, Z, R0, S1, S2, row, e0, e1, e2); break;
    default: put_shell<4, NCH>(slot, col, X, Y, Z, R0, S1, S2, row, e0, e1, e2); break;
    }
}

// Accumulation groups of a tile with n kept panels: nearly equal, at most GROUP panels.
__device__ __forceinline__ int ngroups(int n) { return (n + GROUP - 1) / GROUP; }
__device__ __forceinline__ int group_begin(int n, int ng, int g) { return n * g / ng; }

// The tile warps take turns with the buffers (warp w: buffers of ordinal w mod NTW); a tile
// of -1 ends one tile warp's sequence, the consumers go on with the other's.
struct TileSeq {
    unsigned ord = 0, ended = 0;
    // next buffer, or -1 (all sequences ended, or the wait gave up)
    template <bool WARP>
    __device__ __forceinline__ int next(const Args& A, const State& S, long long& tile)
    {
        for (;; ++ord) {
            if ((ended >> (ord % NTW)) & 1u) continue;
            const int b = ord % NBUF;
            const bool ok = WARP ? warp_wait(A, S, S.screened + 8 * b, (ord / NBUF) & 1)
                                 : wait(A, S, S.screened + 8 * b, (ord / NBUF) & 1);
            if (!ok) return -1;
            tile = S.tile[b];
            if (tile >= 0) {
                ++ord;
                return b;
            }
            ended |= 1u << (ord % NTW);
            if (ended == (1u << NTW) - 1u) return -1;
        }
    }
};

// Generation: team t of TEAM warps fills the operand slots of the panels t, t + NTEAM, ...
// (the shells of a panel are dealt to the team's warps); lane 0 of the team's first warp
// also requests the panel's coefficient digits (bulk copy).
template <int NCH>
__device__ __forceinline__ void gen_role(const Args& A, const State& S)
{
    using C = Cfg<NCH>;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, team = warp / C::TEAM, tw = warp % C::TEAM;
    const uint32_t bytes = (uint32_t)(ND * A.np * PK * 2);
    unsigned seq = 0, turn = 0;
    TileSeq ts;
    long long tile;
    bool ok = true;
    while (ok) {
        const int b = ts.next<true>(A, S, tile);
        if (b < 0) break;
        const int npan = S.npan[b];
        const unsigned short* plist = S.plist + b * MAX_PANELS;
        const unsigned char* nkeep = S.nkeep + b * MAX_SHELLS;
        const short* rowexp = S.rowexp + b * 3 * 128;
        for (int sub = 0; ok && sub < A.nsub; sub += C::SUB) {
            double px = 0.0, py = 0.0, pz = 0.0;
            int e0 = 0, e1 = 0, e2 = 0;
            if (NCH >= 4) {
                long long p;
                tile_point(A, tile, sub * 32 + lane, p, px, py, pz);
                e0 = rowexp[sub * 32 + lane] + 1030;
                e1 = rowexp[128 + sub * 32 + lane] + 1030;
            }
            if (NCH == 7) e2 = rowexp[256 + sub * 32 + lane] + 1030;
            for (int pp = 0, pi = 0, pass = 0; pp < A.npass * npan; ++pp, ++pi, ++seq) {
                if (pi == npan) {
                    pi = 0;
                    ++pass;
                }
                if (seq % C::NTEAM != (unsigned)team) continue;
                const unsigned sl = seq % (unsigned)A.nslot, use = seq / (unsigned)A.nslot;
                const int pan = plist[pi];
                const int s0 = __ldg(A.S.panel + pan), cnt = __ldg(A.S.panel + pan + 1) - s0;
                int4 rec = make_int4(0, 0, 0, 0);
                int nk = 0;
                if (lane < cnt) {
                    rec = __ldg(A.S.shell + s0 + lane);
                    nk = nkeep[s0 + lane];
                }
                const unsigned kept = __ballot_sync(0xffffffffu, nk > 0);
                if (use > 0 && !warp_wait(A, S, S.empty + 8 * sl, (use - 1) & 1)) {
                    ok = false;
                    break;
                }
                const uint32_t slot = smem_u32(S.slots) + sl * S.slot_bytes;
                if (tw == 0 && lane == 0) {
                    S.last_use[sl] = (int)use;
                    bulk_load(slot + S.a_bytes, A.bpack + ((size_t)pass * A.S.npanel + pan) * bytes, bytes, S.bfull + 8 * sl);
                }
                unsigned m = kept;
                while (m) {
                    const int i = __ffs(m) - 1;
                    m &= m - 1;
                    if (turn++ % C::TEAM != (unsigned)tw) continue;
                    const int atom = __shfl_sync(0xffffffffu, rec.x, i), pk = __shfl_sync(0xffffffffu, rec.y, i),
                              prim0 = __shfl_sync(0xffffffffu, rec.z, i), nkq = __shfl_sync(0xffffffffu, nk, i);
                    const double ax = __ldg(A.B.atoms + 4 * atom), ay = __ldg(A.B.atoms + 4 * atom + 1),
                                 az = __ldg(A.B.atoms + 4 * atom + 2);
#pragma unroll 1
                    for (int q = 0; q < C::SUB; ++q) {
                        if (NCH == 1) {
                            const double* pt = S.pts + b * 3 * 128 + q * 32 + lane;
                            px = pt[0];
                            py = pt[128];
                            pz = pt[256];
                            e0 = rowexp[q * 32 + lane] + 1030;
                        }
                        gen_shell<NCH>(A, S, slot, pk & 0xFF, (pk >> 8) & 0xFF, prim0, nkq, px - ax, py - ay, pz - az,
                                       NCH == 1 ? q * 32 + lane : 4 * lane, e0, e1, e2);
                    }
                }
                // the columns of screened shells hold an earlier panel's digits: zeros
                m = (cnt < 32 ? (1u << cnt) - 1u : 0xffffffffu) & ~kept;
                while (m) {
                    const int i = __ffs(m) - 1;
                    m &= m - 1;
                    if (turn++ % C::TEAM != (unsigned)tw) continue;
                    const int pk = __shfl_sync(0xffffffffu, rec.y, i);
                    const int L = pk & 0xFF, col = (pk >> 8) & 0xFF, nc = (L + 1) * (L + 2) / 2;
                    // per column and digit two 128-byte lines: 16 lanes of 16 bytes
                    const uint32_t z0 = slot + ((lane >> 3) & 1) * 1024 + (lane & 7) * 16;
                    for (int k = col; k < col + nc; ++k)
#pragma unroll 1
                        for (int dg = lane >> 4; dg < ND * C::RG; dg += 2)
                            asm volatile("st.shared.v4.u32 [%0], {%1, %1, %1, %1};" ::"r"(z0 + dg * DT + (k >> 3) * 2048 + (k & 7) * 128), "r"(0) : "memory");
                }
                fence_proxy_async();
                __syncwarp();
                if (lane == 0) mbar_arrive(S.full + 8 * sl);
            }
        }
        __syncwarp();
        if (ok && lane == 0) mbar_arrive(S.kfree + 8 * b);
    }
    __syncwarp();
}

// The MMAs of a panel: digit i of the AOs times digits 0 .. 6 - i of the coefficients side by
// side in N (neighbouring accumulators), DM digits per instruction (N <= 256).  Straight-line
// code with the descriptors advanced in their address words: in nested loops an instruction
// took the issuing thread 200 to 320 cycles, whatever its N.
template <int DM, int RG>
__device__ __forceinline__ void issue_panel(uint32_t acc, uint32_t sa, uint32_t sb, int np, uint32_t more)
{
    const uint64_t a0 = a_desc(sa), b0 = b_desc(sb);
    const uint32_t ahi = (uint32_t)(a0 >> 32), bhi = (uint32_t)(b0 >> 32), bstep = (uint32_t)(np * PK * 2) >> 4;
    const uint32_t id0 = idesc(0), idn = (uint32_t)(np >> 3) << 17;
#pragma unroll
    for (int rg = 0; rg < RG; ++rg)
#pragma unroll
        for (int i = 0; i < ND; ++i)
#pragma unroll
            for (int j = 0; j < ND - i; j += DM) {
                const int nd = ND - i - j < DM ? ND - i - j : DM;
                const uint32_t alo = (uint32_t)a0 + (uint32_t)((rg * ND + i) * (DT >> 4)), blo = (uint32_t)b0 + j * bstep;
                asm volatile(
                    "{\n\t.reg .pred p;\n\t.reg .b64 ad, bd;\n\tmov.b64 ad, {%1, %2};\n\tmov.b64 bd, {%3, %4};\n\t"
                    "setp.ne.b32 p, %6, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], ad, bd, %5, p;\n\t}\n" ::"r"(
                        acc + (uint32_t)((rg * ND + i + j) * np)),
                    "r"(alo), "r"(ahi), "r"(blo), "r"(bhi), "r"(id0 + (uint32_t)nd * idn), "r"(i > 0 ? 1u : more));
            }
}

template <int NCH>
__device__ __forceinline__ void mma_role(const Args& A, const State& S)
{
    if ((threadIdx.x & 31) != 0) return;
    using C = Cfg<NCH>;
    const int np = A.np;
    unsigned seq = 0, job = 0;
    bool ok = true, issued = false;
    TileSeq ts;
    long long tile;
    while (ok) {
        const int b = ts.next<false>(A, S, tile);
        if (b < 0) break;
        const int npan = S.npan[b], ng = ngroups(npan);
        for (int pg = 0; ok && pg < A.nsub / C::SUB * A.npass * ng; ++pg, ++job) {
            const int gr = pg % ng;
            const unsigned ab = job % (unsigned)A.nacc, ause = job / (unsigned)A.nacc;
            if (ause > 0 && !wait(A, S, S.acc_empty + 8 * ab, (ause - 1) & 1)) {
                ok = false;
                break;
            }
            tc_fence_after();
            const uint32_t acc = S.tmem + ab * (uint32_t)(C::RG * ND * np);
            const int p0 = group_begin(npan, ng, gr), p1 = group_begin(npan, ng, gr + 1);
            for (int pi = p0; pi < p1; ++pi, ++seq) {
                const unsigned sl = seq % (unsigned)A.nslot, ph = (seq / (unsigned)A.nslot) & 1;
                if (!wait(A, S, S.bfull + 8 * sl, ph) ||
                    !wait(A, S, S.full + 8 * sl, ph)) {
                    ok = false;
                    break;
                }
                tc_fence_after();
                const uint32_t sa = smem_u32(S.slots + sl * S.slot_bytes), sb = sa + S.a_bytes;
                const uint32_t more = pi > p0 ? 1u : 0u;
                if (np <= 32) issue_panel<7, C::RG>(acc, sa, sb, np, more);
                else if (np <= 48) issue_panel<5, C::RG>(acc, sa, sb, np, more);
                else issue_panel<4, C::RG>(acc, sa, sb, np, more);
                mma_commit(S.empty + 8 * sl);
                issued = true;
            }
            if (ok) mma_commit(S.acc_full + 8 * ab);
        }
        if (ok) mbar_arrive(S.kfree + 8 * b);
    }
    if (issued) {
        mma_commit(S.drain);
        mbar_drain(S.drain, 0);
    }
}

// ------------------------------------------------------------------ epilogue
// o 2^x v: through the exponent field where the occupation o is a power of two (2, 1, ...;
// the FP64 pipe is the bound), the same value as the product.
__device__ __forceinline__ double times_occ(double v, double o, int x)
{
    const int ho = __double2hiint(o), eo = (ho >> 20) & 0x7FF;
    if ((ho & 0xFFFFF) == 0 && __double2loint(o) == 0 && eo > 0 && eo < 0x7FF) {
        const int hv = __double2hiint(v), ev = (hv >> 20) & 0x7FF, e = ev + eo - 1023 + x;
        if (ev > 0 && ev < 0x7FF && e > 0 && e < 0x7FF)
            return __hiloint2double((hv & 0x800FFFFF) ^ (int)((unsigned)ho & 0x80000000u) | (e << 20), __double2loint(v));
    }
    return (x ? 2.0 * o : o) * v;
}

template <int NCH, int MODE>
__device__ __forceinline__ void epi_role(const Args& A, const State& S)
{
    using C = Cfg<NCH>;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, quad = warp & 3;
    const int half = (warp - C::NGW) >> 2;            // of a row group's EPQ warps: MOs 2 half, 2 half + 2 EPQ, ...
    const int row = quad * 32 + lane;                 // accumulator row
    const int pt = NCH == 1 ? row : row >> 2;         // point of the tile
    const int ch = NCH == 1 ? 0 : lane & 3;           // channel (of the first row tile)
    const int lane0 = NCH == 1 ? lane : lane & ~3;    // lane of the point's value
    const int np = A.np;
    double* phi = A.phi ? A.phi + (size_t)blockIdx.x * C::RG * np * 128 + row : nullptr;
    unsigned job = 0, round = 0;
    TileSeq ts;
    long long tile;
    for (;;) {
        const int b = ts.next<true>(A, S, tile);
        if (b < 0) return;
        const int npan = S.npan[b], ng = ngroups(npan);
        const short* rowexp = S.rowexp + b * 3 * 128;
        for (int sub = 0; sub < A.nsub; sub += C::SUB) {
            const int rx0 = rowexp[(ch == 0 ? 0 : 128) + sub * 32 + pt], rx1 = NCH == 7 ? rowexp[256 + sub * 32 + pt] : 0;
            long long p;
            double px, py, pz;
            const bool valid = tile_point(A, tile, sub * 32 + pt, p, px, py, pz);
            double accs[2] = {0.0, 0.0}, acc1 = 0.0;
            double cot = 0.0;  // this channel's cotangent at the point
            if (MODE == OUT_WV && valid) cot = ch == 0 ? A.g_rho[p] : A.g_grad ? A.g_grad[(ch - 1) * A.g_ld + p] : 0.0;
            for (int pass = 0; pass < A.npass; ++pass) {
                const int* fexp = (A.tab_smem ? S.fexp : A.fexp) + pass * np;
                const double* occ = (A.tab_smem ? S.occ : A.occ) + pass * np;
                for (int gr = 0; gr < (ng ? ng : 1); ++gr) {
                    const unsigned ab = job % (unsigned)A.nacc, ause = job / (unsigned)A.nacc;
                    const bool last = gr + 1 >= ng;
                    uint32_t taddr = S.tmem + ab * (uint32_t)(C::RG * ND * np) + ((uint32_t)(quad * 32) << 16);
                    if (ng) {
                        if (!warp_wait(A, S, S.acc_full + 8 * ab, ause & 1)) return;
                        tc_fence_after();
                    }
                    const int nmo = A.nmo - pass * np < np ? A.nmo - pass * np : np;  // MOs of this pass
                    Acc2 va, ua;
#pragma unroll 1
                    for (int n0 = 2 * half; n0 < nmo; n0 += 2 * C::EPQ) {
                        double v[2], u[2];
                        const int2 f2 = *(const int2*)(fexp + n0);
                        if (ng) {
                            acc2_load(va, taddr + (uint32_t)n0, np);
                            if (NCH == 7) acc2_load(ua, taddr + (uint32_t)(ND * np + n0), np);
                            acc2_wait(va);
                            if (NCH == 7) acc2_wait(ua);
                            acc2_values(va, rx0, f2, v);
                            if (NCH == 7) acc2_values(ua, rx1, f2, u);
                            if (ng > 1) {
#pragma unroll
                                for (int i = 0; i < 2; ++i) {
                                    double* q = phi + (size_t)(n0 + i) * 128;
                                    if (gr > 0) v[i] += *q;
                                    if (!last) *q = v[i];
                                    if (NCH == 7) {
                                        q += (size_t)np * 128;
                                        if (gr > 0) u[i] += *q;
                                        if (!last) *q = u[i];
                                    }
                                }
                            }
                        } else {
                            // no shell reaches this tile: zeros (or NaN where the input has it)
#pragma unroll
                            for (int i = 0; i < 2; ++i) v[i] = u[i] = rx0 == ROW_NAN ? __longlong_as_double(0x7FF8000000000000ll) : 0.0;
                        }
                        if (!last) continue;
                        if (MODE == OUT_WV) {
                            // cotangents of the MOs: W = 2 occ (g_rho MO + sum_d g_d d_d MO), V = 2 occ MO
#pragma unroll
                            for (int i = 0; i < 2; ++i) {
                                const double o = occ[n0 + i];
                                const double f = shfl_d(v[i], lane0);
                                double w = v[i] * cot;
                                w += shfl_d(w, lane ^ 1);
                                w += shfl_d(w, lane ^ 2);
                                if (valid && n0 + i < nmo && ch < 2) {
                                    const long long at = (long long)(ch * A.nmo + pass * np + n0 + i) * A.ld + p;
                                    const double v2 = times_occ(ch == 0 ? w : f, o, 1);
                                    if (A.wv_float) ((float*)A.out)[at] = (float)v2;
                                    else A.out[at] = v2;
                                }
                            }
                        } else if (MODE == OUT_MO) {
                            for (int d = 0; d < A.drv.n; ++d) {
                                const int code = A.drv.code[d];
                                const bool first = code < 4;
                                if (!valid || (first ? ch != code : (NCH != 7 || ch != code - 4))) continue;
                                double* out = A.out + ((long long)d * A.nmo + pass * np + n0) * A.ld + p;
#pragma unroll
                                for (int i = 0; i < 2; ++i)
                                    if (n0 + i < nmo) out[i * A.ld] = first ? v[i] : (NCH == 7 ? u[i] : 0.0);
                            }
                        } else {
                            double q2[2];
#pragma unroll
                            for (int i = 0; i < 2; ++i) {
                                const double o = occ[n0 + i];
                                if (NCH == 1) {
                                    q2[i] = v[i] * v[i];
                                    accs[i & 1] = fma(o, q2[i], accs[i & 1]);
                                } else {
                                    const double f = shfl_d(v[i], lane0);
                                    accs[i & 1] = fma(times_occ(f, o, ch == 0 ? 0 : 1), v[i], accs[i & 1]);
                                    if (NCH == 7) {
                                        const double dv = shfl_d(v[i], lane0 + ((ch + 1) & 3));
                                        acc1 = fma(times_occ(f, o, 1), u[i], acc1);
                                        acc1 = fma(times_occ(dv, o, 1), dv, acc1);
                                    }
                                    if (A.mo_norm) q2[i] = ch == 0 ? v[i] * v[i] : 0.0;
                                }
                            }
                            if (A.mo_norm) {
                                // sums of q2[i] over the warp, two MOs at once: after one halving
                                // exchange lane l holds MO (l & 1)
#pragma unroll
                                for (int i = 0; i < 2; ++i) q2[i] = valid ? q2[i] : 0.0;
                                const double keep = (lane & 1) ? q2[1] : q2[0], give = (lane & 1) ? q2[0] : q2[1];
                                double s1 = keep + shfl_d(give, lane ^ 1);
#pragma unroll
                                for (int o = 2; o < 32; o *= 2) s1 += shfl_d(s1, lane ^ o);
                                if (lane < 2 && n0 + lane < nmo) {
                                    const int mo = pass * np + n0 + lane;
                                    if (A.norm_smem)
                                        S.norm[(warp - C::NGW) * A.npass * np + mo] += s1;
                                    else
                                        atomicAdd(A.mo_norm + mo, s1);
                                }
                                __syncwarp();
                            }
                        }
                    }
                    if (ng) {
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(S.acc_empty + 8 * ab);
                        ++job;
                    }
                }
            }
            double acc0 = accs[0] + accs[1];
            if (MODE == OUT_RHO && C::EPQ > 1) {
                // the shares of the MO sum meet in shared memory
                if (half > 0) {
                    if (round > 0 && !warp_wait(A, S, S.part_free + 8 * quad, (round - 1) & 1)) return;
                    S.part[((half - 1) * 4 + quad) * 32 + lane] = acc0;
                    __syncwarp();
                    if (lane == 0) mbar_arrive(S.part_full + 8 * quad);
                } else {
                    if (!warp_wait(A, S, S.part_full + 8 * quad, round & 1)) return;
#pragma unroll
                    for (int h = 1; h < C::EPQ; ++h) acc0 += S.part[((h - 1) * 4 + quad) * 32 + lane];
                    __syncwarp();
                    if (lane == 0) mbar_arrive(S.part_free + 8 * quad);
                }
                ++round;
            }
            if (MODE == OUT_RHO && valid && half == 0) {
                if (ch == 0) A.out[p] = acc0;
                for (int d = 0; d < A.drv.n; ++d) {
                    const int code = A.drv.code[d];
                    if (code == 0) {
                        // a density "derivative" of order 0: 2 occ MO^2
                        if (ch == 0) A.dout[(long long)d * A.ld + p] = 2.0 * acc0;
                    } else if (code < 4) {
                        if (ch == code) A.dout[(long long)d * A.ld + p] = acc0;
                    } else if (NCH == 7 && ch == code - 4) {
                        A.dout[(long long)d * A.ld + p] = acc1;
                    }
                }
            }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(S.kfree + 8 * b);
    }
}

// ------------------------------------------------------------------ tile warp
// Bounds of a shell's operand values 2^-shift P R at one point, from the distance r and the
// largest coordinate q = max(|x|, |y|, |z|) relative to its atom: with t = q, c = 1 and with
// t = r, c = 2^-b (b = 0, 0, 1, 2, 3 for L = 0 .. 4: what the component shifts leave of r^L)
//   |P| <= c t^L =: p0,
//   |dP R| <= p1 R0 + 2 q1 R1,  p1 = c L t^(L-1), q1 = c t^(L+1),
//   |ddP R| <= p2 R0 + 2 (2L+1) p0 R1 + 4 q2 R2,  p2 = c L(L-1) t^(L-2), q2 = c t^(L+2);
// every factor is taken from the smaller of the two.
struct Poly {
    float p0, p1, p2, q1, q2;
};
__device__ __forceinline__ Poly poly1(int L, float t, float c)
{
    Poly f{c, 0.f, 0.f, 0.f, 0.f};
    for (int i = 0; i < L; ++i) {
        f.p2 = 2.f * f.p1 + f.p2 * t;
        f.p1 = f.p0 + f.p1 * t;
        f.p0 *= t;
    }
    f.q1 = f.p0 * t;
    f.q2 = f.q1 * t;
    return f;
}
__device__ __forceinline__ Poly poly(int L, float r, float q)
{
    const Poly a = poly1(L, q, 1.f), b = poly1(L, r, L < 2 ? 1.f : L == 2 ? 0.5f : L == 3 ? 0.25f : 0.125f);
    return Poly{fminf(a.p0, b.p0), fminf(a.p1, b.p1), fminf(a.p2, b.p2), fminf(a.q1, b.q1), fminf(a.q2, b.q2)};
}

// Squared distances from an atom to the tile's box and its largest coordinate relative to
// the atom, smallest and largest over the box.
struct BoxRange {
    float dmin, dmax, qmin, qmax;
};
__device__ __forceinline__ BoxRange box_range(const Args& A, int atom, double ox, double oy, double oz, const float (&lo)[3],
                                              const float (&hi)[3])
{
    const float a[3] = {(float)(__ldg(A.B.atoms + 4 * atom) - ox), (float)(__ldg(A.B.atoms + 4 * atom + 1) - oy),
                        (float)(__ldg(A.B.atoms + 4 * atom + 2) - oz)};
    BoxRange o{0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const float u = fmaxf(0.f, fmaxf(lo[c] - a[c], a[c] - hi[c]));
        const float v = fmaxf(fabsf(lo[c] - a[c]), fabsf(hi[c] - a[c]));
        o.dmin = fmaf(u, u, o.dmin);
        o.dmax = fmaf(v, v, o.dmax);
        o.qmin = fmaxf(o.qmin, u);
        o.qmax = fmaxf(o.qmax, v);
    }
    return o;
}

// Raises top (log2, per channel class) to a shell's bound at squared distances dd (coordinates
// within NEAR, or EXACT): sum over the primitives relative to the largest.
template <int NCLS, bool EXACT, int NQ>
__device__ __forceinline__ void point_bounds(const float4* __restrict__ pl, int np, int L, const float (&dd)[NQ],
                                             const float (&dq)[NQ], float (&top)[NQ][NCLS])
{
    float m[NQ], R0[NQ], R1[NQ], R2[NQ];
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
        m[q] = -3.0e38f;
        R0[q] = R1[q] = R2[q] = 0.f;
    }
    for (int i = 0; i < np; ++i) {
        const float4 v = __ldg(pl + i);
#pragma unroll
        for (int q = 0; q < NQ; ++q) m[q] = fmaxf(m[q], fmaf(-v.x, dd[q], v.y));
    }
    for (int i = 0; i < np; ++i) {
        const float4 v = __ldg(pl + i);
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
            const float e = exp2f(fmaf(-v.x, dd[q], v.y) - m[q]);
            R0[q] += e;
            if (NCLS > 1) R1[q] = fmaf(v.z, e, R1[q]);
            if (NCLS > 2) R2[q] = fmaf(v.z * v.z, e, R2[q]);
        }
    }
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
        if (m[q] < NOTHING) continue;
        const Poly f = EXACT ? poly(L, sqrtf(dd[q]), dq[q]) : poly(L, sqrtf(dd[q]) + 2.f * NEAR, dq[q] + NEAR);
        top[q][0] = fmaxf(top[q][0], m[q] + __log2f(f.p0 * R0[q]));
        if (NCLS > 1) top[q][1] = fmaxf(top[q][1], m[q] + __log2f(f.p1 * R0[q] + 2.f * f.q1 * R1[q]));
        if (NCLS > 2)
            top[q][2] = fmaxf(top[q][2],
                              m[q] + __log2f(f.p2 * R0[q] + 2.f * (2 * L + 1) * f.p0 * R1[q] + 4.f * f.q2 * R2[q]));
    }
}

// A point that is set apart: NaN where a coordinate is NaN, 0 at |coordinate| >= 2^30 (every AO
// is exactly 0 there, see split_prim; from 2^170 on a polynomial may overflow and 0 times it is
// not 0: ROW_OUT); else 0.
constexpr int ROW_OUT = 30002;
__device__ __forceinline__ int special_point(double x, double y, double z)
{
    if (x != x || y != y || z != z) return ROW_NAN;
    const int h = max(__double2hiint(x) & 0x7FFFFFFF, max(__double2hiint(y) & 0x7FFFFFFF, __double2hiint(z) & 0x7FFFFFFF));
    return h >= 0x4A900000 ? ROW_OUT : h >= 0x41D00000 ? ROW_ZERO : 0;
}
// Row exponent of a point with the bound `top` (log2); 0.1 to spare: 0.0145 that digits7 asks for,
// 0.05 for the roundings of the coordinates (WIDE), below 0.001 for those of the bound.
__device__ __forceinline__ int row_scale(int special, float top, int* redo)
{
    if (special == ROW_OUT || (!special && !(top <= 985.f))) *(volatile int*)redo = 1;
    return special ? special : (int)ceilf(fminf(fmaxf(top + 0.1f, -950.f), 990.f));
}

// The points' scales of a tile beyond WIDE or NEAR, or with points within CLOSE, with FP64
// differences to the atoms: every kept shell,
// point after point (a call of its own: few tiles need it).
template <int NCH>
__device__ __noinline__ void wide_scales(const Args& A, long long t, const unsigned char* nkeep, short* rowexp, float r0,
                                         float r1, float r2)
{
    constexpr int NCLS = Cfg<NCH>::NCLS;
    const int lane = threadIdx.x & 31;
    const float ref[3] = {r0, r1, r2};
#pragma unroll 1
    for (int q = 0; q < A.nsub; ++q) {
        long long p;
        double x, y, z;
        tile_point(A, t, q * 32 + lane, p, x, y, z);
        float top[1][NCLS];
        for (int c = 0; c < NCLS; ++c) top[0][c] = ref[c];
        for (int s = 0; s < A.B.nshell; ++s) {
            const int4 rec = __ldg(A.S.shell + s);
            const double* at = A.B.atoms + 4 * rec.x;
            const float dx = (float)(x - __ldg(at)), dy = (float)(y - __ldg(at + 1)), dz = (float)(z - __ldg(at + 2));
            const float dd[1] = {fmaf(dx, dx, fmaf(dy, dy, dz * dz))}, dq[1] = {fmaxf(fabsf(dx), fmaxf(fabsf(dy), fabsf(dz)))};
            point_bounds<NCLS, true>(A.S.prim_lg + rec.z, nkeep[s], rec.y & 0xFF, dd, dq, top);
        }
        for (int c = 0; c < NCLS; ++c) rowexp[c * 128 + q * 32 + lane] = (short)row_scale(special_point(x, y, z), top[0][c], A.redo);
    }
}

template <int NCH>
__device__ __forceinline__ void tile_role(const Args& A, const State& S, int tw)
{
    using C = Cfg<NCH>;
    constexpr int NCLS = C::NCLS, NQ = 4;
    const int lane = threadIdx.x & 31;
    const int nshell = A.B.nshell, nsub = A.nsub;
    unsigned short* bigl = S.big + tw * MAX_BIG;
    unsigned* pbits = S.pbits + tw * (MAX_PANELS / 32);
    for (unsigned ord = tw;; ord += NTW) {
        const int b = ord % NBUF;
        const bool ok = ord < NBUF || warp_wait(A, S, S.kfree + 8 * b, ((ord / NBUF) - 1) & 1);
        long long t = -1;
        if (lane == 0 && ok) {
            t = (long long)atomicAdd(A.counter, 1ull);
            if (t >= A.ntiles) t = -1;
        }
        t = __shfl_sync(0xffffffffu, t, 0);
        if (lane == 0) S.tile[b] = t;
        if (t < 0) {
            __syncwarp();
            if (lane == 0) mbar_arrive(S.screened + 8 * b);
            return;
        }
        // points relative to one of them, in single precision (see WIDE), some set apart
        float fx[NQ], fy[NQ], fz[NQ];
        int special[NQ];
        double ox = 0.0, oy = 0.0, oz = 0.0;
        bool have = false;
        float lo[3] = {3.0e38f, 3.0e38f, 3.0e38f}, hi[3] = {-3.0e38f, -3.0e38f, -3.0e38f};
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
            special[q] = 0;
            fx[q] = fy[q] = fz[q] = 0.f;
            if (q >= nsub) continue;
            long long p;
            double x, y, z;
            tile_point(A, t, q * 32 + lane, p, x, y, z);
            if (NCH == 1) {
                double* pt = S.pts + b * 3 * 128 + q * 32 + lane;
                pt[0] = x;
                pt[128] = y;
                pt[256] = z;
            }
            special[q] = special_point(x, y, z);
            const unsigned first = __ballot_sync(0xffffffffu, special[q] == 0);
            if (!have && first) {
                const int src = __ffs(first) - 1;
                ox = shfl_d(x, src);
                oy = shfl_d(y, src);
                oz = shfl_d(z, src);
                have = true;
            }
            if (special[q] == 0) {
                fx[q] = (float)(x - ox);
                fy[q] = (float)(y - oy);
                fz[q] = (float)(z - oz);
                lo[0] = fminf(lo[0], fx[q]);
                hi[0] = fmaxf(hi[0], fx[q]);
                lo[1] = fminf(lo[1], fy[q]);
                hi[1] = fmaxf(hi[1], fy[q]);
                lo[2] = fminf(lo[2], fz[q]);
                hi[2] = fmaxf(hi[2], fz[q]);
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                lo[c] = fminf(lo[c], __shfl_xor_sync(0xffffffffu, lo[c], o));
                hi[c] = fmaxf(hi[c], __shfl_xor_sync(0xffffffffu, hi[c], o));
            }
        // The coordinates relative to the origin point (of points and atoms) are rounded to floats,
        // so differences err by up to 2^-23 of the tile's extent, besides their own rounding: the
        // box is widened by that, and where it counts (WIDE) the points' differences are FP64.
        float ext = 0.f;
#pragma unroll
        for (int c = 0; c < 3; ++c) ext = have ? fmaxf(ext, fmaxf(fabsf(lo[c]), fabsf(hi[c]))) : 0.f;
        const float err = 2.0e-7f * ext;  // 2^-23 + 2^-24 (the widened edge's rounding) = 1.8e-7
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            lo[c] -= err;
            hi[c] += err;
        }
        float amax = 0.f;
        bool exact = err > NEAR;
        for (int i = lane; i < MAX_PANELS / 32; i += 32) pbits[i] = 0u;
        __syncwarp();
        unsigned char* nkeep = S.nkeep + b * MAX_SHELLS;
        int npan = 0, nbig = 0;
        float ref[3] = {-3.0e38f, -3.0e38f, -3.0e38f};
        if (have) {
            // what the scale of every point of the tile is known to reach: the largest
            // lower bound of a shell over the tile's box (one primitive's share of it)
            for (int s = lane; s < nshell; s += 32) {
                const int4 rec = __ldg(A.S.shell + s);
                const int L = rec.y & 0xFF, np = rec.w;
                const BoxRange br = box_range(A, rec.x, ox, oy, oz, lo, hi);
                float m = -3.0e38f, al = 0.f;
                for (int q = 0; q < np; ++q) {
                    const float4 v = __ldg(A.S.prim_lg + rec.z + q);
                    const float l = v.y - v.x * br.dmax;
                    al = l > m ? v.z : al;
                    m = fmaxf(m, l);
                }
                const Poly f = poly(L, sqrtf(br.dmin), br.qmin);
                float u[3];
                u[0] = m + __log2f(f.p0);
                u[1] = m + __log2f(f.p1 + 2.f * al * f.q1);
                u[2] = m + __log2f(f.p2 + al * (2.f * (2 * L + 1) * f.p0 + 4.f * al * f.q2));
#pragma unroll
                for (int c = 0; c < NCLS; ++c) ref[c] = m < NOTHING ? ref[c] : fmaxf(ref[c], u[c]);
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
#pragma unroll
                for (int c = 0; c < NCLS; ++c) ref[c] = fmaxf(ref[c], __shfl_xor_sync(0xffffffffu, ref[c], o));
            // upper bounds: kept shells and primitives, and the shells that may set a scale
            for (int sb = 0; sb < nshell; sb += 32) {
                const int s = sb + lane;
                int nk = 0;
                bool big = false;
                int atom = -1;  // of a kept shell within CLOSE of the box
                if (s < nshell) {
                    const int4 rec = __ldg(A.S.shell + s);
                    const int L = rec.y & 0xFF, np = rec.w, pan = rec.y >> 16;
                    const BoxRange br = box_range(A, rec.x, ox, oy, oz, lo, hi);
                    const Poly f = poly(L, sqrtf(br.dmax), br.qmax);
                    const float lnp = __log2f((float)np), l0 = __log2f(f.p0);
                    for (int q = 0; q < np; ++q) {
                        const float4 v = __ldg(A.S.prim_lg + rec.z + q);
                        const float e = v.y - v.x * br.dmin, a = v.z;
                        if (e < NOTHING) continue;
                        float u[3];
                        u[0] = e + l0;
                        u[1] = e + __log2f(f.p1 + 2.f * a * f.q1);
                        u[2] = e + __log2f(f.p2 + a * (2.f * (2 * L + 1) * f.p0 + 4.f * a * f.q2));
#pragma unroll
                        for (int c = 0; c < NCLS; ++c) {
                            if (u[c] > fmaxf(ref[c] - KEEP_LOG2, ABS_FLOOR)) nk = q + 1;
                            if (u[c] + lnp >= ref[c]) big = true;
                        }
                        if (nk == q + 1) amax = fmaxf(amax, a);
                    }
                    big = big && nk > 0;
                    if (nk > 0 && br.dmin < CLOSE * CLOSE) atom = rec.x;
                    nkeep[s] = (unsigned char)nk;
                    if (nk > 0) atomicOr(pbits + (pan >> 5), 1u << (pan & 31));
                }
                const unsigned mb = __ballot_sync(0xffffffffu, big);
                const int at = nbig + __popc(mb & ((1u << lane) - 1u));
                if (big && at < MAX_BIG) bigl[at] = (unsigned short)s;
                nbig += __popc(mb);
                for (unsigned mc = __ballot_sync(0xffffffffu, atom >= 0); mc; mc &= mc - 1) {
                    const double* at = A.B.atoms + 4 * __shfl_sync(0xffffffffu, atom, __ffs(mc) - 1);
                    const float ax = (float)(__ldg(at) - ox), ay = (float)(__ldg(at + 1) - oy), az = (float)(__ldg(at + 2) - oz);
#pragma unroll
                    for (int q = 0; q < NQ; ++q) {
                        const float dx = fx[q] - ax, dy = fy[q] - ay, dz = fz[q] - az;
                        if (q < nsub && special[q] == 0) exact |= fmaf(dx, dx, fmaf(dy, dy, dz * dz)) < CLOSE * CLOSE;
                    }
                }
            }
            __syncwarp();
            for (int pb = 0; pb < A.S.npanel; pb += 32) {
                const bool k = (pbits[pb >> 5] >> lane) & 1u;
                const unsigned mk = __ballot_sync(0xffffffffu, k);
                if (k) S.plist[b * MAX_PANELS + npan + __popc(mk & ((1u << lane) - 1u))] = (unsigned short)(pb + lane);
                npan += __popc(mk);
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
        short* rowexp = S.rowexp + b * 3 * 128;
        if (__any_sync(0xffffffffu, exact || sqrtf(amax) * err > WIDE)) {
            wide_scales<NCH>(A, t, nkeep, rowexp, ref[0], NCLS > 1 ? ref[1] : 0.f, NCLS > 2 ? ref[2] : 0.f);
            if (lane == 0) S.npan[b] = npan;
            __syncwarp();
            if (lane == 0) mbar_arrive(S.screened + 8 * b);
            continue;
        }
        // the scale of every point: the largest bound at the point itself
        float top[NQ][NCLS];
#pragma unroll
        for (int q = 0; q < NQ; ++q)
#pragma unroll
            for (int c = 0; c < NCLS; ++c) top[q][c] = ref[c];
        const bool every = nbig > MAX_BIG;  // (more candidates than the list holds: all shells)
        for (int i = 0; i < (every ? nshell : nbig); ++i) {
            const int s = every ? i : bigl[i];
            const int4 rec = __ldg(A.S.shell + s);
            const int L = rec.y & 0xFF, nk = nkeep[s];
            const float ax = (float)(__ldg(A.B.atoms + 4 * rec.x) - ox), ay = (float)(__ldg(A.B.atoms + 4 * rec.x + 1) - oy),
                        az = (float)(__ldg(A.B.atoms + 4 * rec.x + 2) - oz);
            float dd[NQ], dq[NQ];
#pragma unroll
            for (int q = 0; q < NQ; ++q) {
                const float dx = fx[q] - ax, dy = fy[q] - ay, dz = fz[q] - az;
                dd[q] = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
                dq[q] = fmaxf(fabsf(dx), fmaxf(fabsf(dy), fabsf(dz)));
            }
            point_bounds<NCLS, false>(A.S.prim_lg + rec.z, nk, L, dd, dq, top);
        }
#pragma unroll
        for (int q = 0; q < NQ; ++q)
#pragma unroll
            for (int c = 0; c < NCLS; ++c)
                if (q < nsub) rowexp[c * 128 + q * 32 + lane] = (short)row_scale(special[q], top[q][c], A.redo);
        if (lane == 0) S.npan[b] = npan;
        __syncwarp();
        if (lane == 0) mbar_arrive(S.screened + 8 * b);
    }
}

// ------------------------------------------------------------------ the kernel
template <int NCH, int MODE>
__global__ void __launch_bounds__(Cfg<NCH>::NT, 1) split_kernel(const __grid_constant__ Args A)
{
    using C = Cfg<NCH>;
    constexpr int NT = C::NT, NGW = C::NGW, NEW = C::NEW;
    extern __shared__ unsigned char raw[];
    const int tid = threadIdx.x, warp = tid >> 5;
    bool out = __ldg(A.S.flags) != 0;
    for (int i = tid; i < A.npass * A.np; i += NT) out |= __ldg(A.fexp + i) == MO_NAN;
    if (__syncthreads_or(out)) {
        if (tid == 0) *(volatile int*)A.redo = 1;
        return;
    }
    unsigned char* base = (unsigned char*)(((uintptr_t)raw + 1023) & ~(uintptr_t)1023);
    State S;
    S.a_bytes = C::RG * ND * DT;
    // (the coefficient digits' 32-byte swizzle repeats every 256 bytes; slots start at 1 KB)
    S.slot_bytes = (S.a_bytes + (uint32_t)(ND * A.np * PK * 2) + 1023u) & ~1023u;
    S.slots = base;
    unsigned char* q = base + (size_t)A.nslot * S.slot_bytes;
    S.tab = (uint64_t*)q;
    q += TABN * 8;
    S.tile = (long long*)q;
    q += NBUF * 8;
    uint64_t* bar = (uint64_t*)q;
    q += NBAR * 8;
    S.part = (double*)q;
    if (C::EPQ > 1) q += (C::EPQ - 1) * 4 * 32 * 8;
    S.norm = (double*)q;
    if (A.norm_smem) q += (size_t)NEW * A.npass * A.np * 8;
    S.occ = (double*)q;
    S.fexp = (int*)(S.occ + A.npass * A.np);
    if (A.tab_smem) {
        q += (size_t)A.npass * A.np * 12;
        for (int i = tid; i < A.npass * A.np; i += NT) {
            S.occ[i] = __ldg(A.occ + i);
            S.fexp[i] = __ldg(A.fexp + i);
        }
    }
    S.pts = (double*)q;
    if (NCH == 1) q += NBUF * 3 * 128 * 8;
    S.rowexp = (short*)q;
    q += NBUF * 2 * 3 * 128;
    S.npan = (int*)q;
    q += NBUF * 4;
    S.last_use = (int*)q;
    q += MAX_SLOTS * 4;
    S.abort_flag = (int*)q;
    uint32_t* tmem_slot = (uint32_t*)(q + 4);
    q += 8;
    S.pbits = (unsigned*)q;
    q += NTW * MAX_PANELS / 8;
    S.plist = (unsigned short*)q;
    q += NBUF * MAX_PANELS * 2;
    S.big = (unsigned short*)q;
    q += NTW * MAX_BIG * 2;
    S.nkeep = q;
    S.full = smem_u32(bar);
    S.empty = smem_u32(bar + MAX_SLOTS);
    S.bfull = smem_u32(bar + 2 * MAX_SLOTS);
    S.acc_full = smem_u32(bar + 3 * MAX_SLOTS);
    S.acc_empty = smem_u32(bar + 3 * MAX_SLOTS + 2);
    S.screened = smem_u32(bar + 3 * MAX_SLOTS + 4);
    S.kfree = smem_u32(bar + 3 * MAX_SLOTS + 4 + NBUF);
    S.part_full = smem_u32(bar + 3 * MAX_SLOTS + 4 + 2 * NBUF);
    S.part_free = smem_u32(bar + 3 * MAX_SLOTS + 8 + 2 * NBUF);
    S.drain = smem_u32(bar + 3 * MAX_SLOTS + 12 + 2 * NBUF);
    // operand slots start as zeros: columns that no shell of a panel owns stay finite
    // (their coefficients are zero)
    for (int i = tid; i < (int)(A.nslot * S.slot_bytes / 16); i += NT) ((uint4*)S.slots)[i] = make_uint4(0, 0, 0, 0);
    for (int i = tid; i < TABN; i += NT) S.tab[i] = __ldg(A.S.exp_tab + i);
    if (A.norm_smem)
        for (int i = tid; i < NEW * A.npass * A.np; i += NT) S.norm[i] = 0.0;
    if (tid == 0) {
        for (int s = 0; s < A.nslot; ++s) {
            mbar_init(S.full + 8 * s, C::TEAM);
            mbar_init(S.empty + 8 * s, 1);
            mbar_init(S.bfull + 8 * s, 1);
            S.last_use[s] = -1;
        }
        for (int s = 0; s < 2; ++s) {
            mbar_init(S.acc_full + 8 * s, 1);
            mbar_init(S.acc_empty + 8 * s, NEW);
        }
        for (int s = 0; s < NBUF; ++s) {
            mbar_init(S.screened + 8 * s, 1);
            mbar_init(S.kfree + 8 * s, NGW + NEW + 1);
        }
        for (int s = 0; s < 4; ++s) {
            mbar_init(S.part_full + 8 * s, C::EPQ > 1 ? C::EPQ - 1 : 1);
            mbar_init(S.part_free + 8 * s, 1);
        }
        mbar_init(S.drain, 1);
        *S.abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(A.tm_cols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    fence_proxy_async();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    S.tmem = *tmem_slot;

    if (warp < NGW)
        gen_role<NCH>(A, S);
    else if (warp < NGW + NEW)
        epi_role<NCH, MODE>(A, S);
    else if (warp == NGW + NEW)
        mma_role<NCH>(A, S);
    else
        tile_role<NCH>(A, S, warp - (NGW + NEW + 1));

    __syncwarp();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    // no coefficient copy may land after the CTA has left (all have, unless a wait gave up)
    if (tid < A.nslot && S.last_use[tid] >= 0) mbar_drain(S.bfull + 8 * tid, S.last_use[tid] & 1);
    if (MODE == OUT_RHO && A.mo_norm && A.norm_smem)
        for (int i = tid; i < A.nmo; i += NT) {
            double t = 0.0;
            for (int w = 0; w < NEW; ++w) t += S.norm[w * A.npass * A.np + i];
            atomicAdd(A.mo_norm + i, t);
        }
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(S.tmem), "r"(A.tm_cols));
}

// Digits of the MO coefficients times the column norms and scales, one block per MO
// column of the operand, which also zeroes its sum of MO^2 (if there are such); block 0 zeroes
// the tile counter and the redo word.
__global__ void __launch_bounds__(256) split_pack_kernel(SplitDev S, int nmo, int np, int ncart,
                                                         const double* __restrict__ C, const double* __restrict__ occ,
                                                         unsigned char* __restrict__ bpack, int* __restrict__ fexp,
                                                         double* __restrict__ occ_pad, unsigned long long* counter,
                                                         int* redo, double* norm)
{
    __shared__ unsigned long long top;
    const int mo = blockIdx.x, pass = mo / np, n = mo % np, ncol = S.npanel * PK;
    if (threadIdx.x == 0) top = 0;
    __syncthreads();
    auto value = [&](int i) -> double {
        const int r = S.col_cart[i];
        if (mo >= nmo || r < 0) return 0.0;
        return C[(long long)mo * ncart + r] * S.col_g[i];
    };
    // magnitudes compare like their bit patterns (NaN and infinity last)
    unsigned long long m = 0;
    for (int i = threadIdx.x; i < ncol; i += blockDim.x) {
        const unsigned long long u = (unsigned long long)__double_as_longlong(value(i)) & 0x7FFFFFFFFFFFFFFFull;
        m = u > m ? u : m;
    }
    atomicMax(&top, m);
    __syncthreads();
    const int F = scale_of(top);
    const bool nan = too_large(top) || vanishing(top);
    if (threadIdx.x == 0) {
        fexp[mo] = nan ? MO_NAN : F;
        occ_pad[mo] = (mo < nmo && occ) ? occ[mo] : 0.0;
        if (norm) norm[mo] = 0.0;
        if (mo == 0) {
            *counter = 0ull;
            *redo = 0;
        }
    }
    for (int i = threadIdx.x; i < ncol; i += blockDim.x) {
        const uint64_t t = nan ? 0x0080808080808080ull : digits7(value(i), F + 1030);
        unsigned char* tile = bpack + ((size_t)pass * S.npanel + i / PK) * (size_t)(ND * np * PK * 2);
#pragma unroll
        for (int j = 0; j < ND; ++j) {
            const int d = (int)((t >> (8 * (6 - j))) & 0xFF) - 128;
            *(__half*)(tile + b_off(j * np + n, i % PK)) = __int2half_rn(d);
        }
    }
}

}  // namespace sp

// ---------------------------------------------------------------- host side
SplitLayout split_layout(const std::vector<Shell>& shells, const std::vector<int>& comp_row,
                         const std::vector<double>& comp_g, const int* order)
{
    // panels of 16 columns, whole shells; a shell goes to the oldest of the last four
    // open panels with room
    const int n = (int)shells.size();
    std::vector<std::vector<int>> pan;
    std::vector<int> used;
    for (int i = 0; i < n; ++i) {
        const int s = order ? order[i] : i, nc = ncanon(shells[s].L);
        int at = -1;
        const int lo = (int)pan.size() > 4 ? (int)pan.size() - 4 : 0;
        for (int p = lo; p < (int)pan.size() && at < 0; ++p)
            if (used[p] + nc <= OKG_SPLIT_PK) at = p;
        if (at < 0) {
            at = (int)pan.size();
            pan.emplace_back();
            used.push_back(0);
        }
        pan[at].push_back(s);
        used[at] += nc;
    }
    SplitLayout m;
    m.panel.push_back(0);
    m.col_cart.assign(pan.size() * OKG_SPLIT_PK, -1);
    m.col_g.assign(pan.size() * OKG_SPLIT_PK, 0.0);
    for (size_t p = 0; p < pan.size(); ++p) {
        int col = 0;
        for (int s : pan[p]) {
            const Shell& sh = shells[s];
            m.shell.push_back(make_int4(sh.atom, sh.L | (col << 8) | ((int)p << 16), sh.prim0, sh.nprim));
            for (int q = 0; q < ncanon(sh.L); ++q) {
                const size_t c = p * OKG_SPLIT_PK + col + q;
                const int r = comp_row[sh.comp0 + q];
                if (r >= 0) {
                    m.col_cart[c] = sh.cart0 + r;
                    m.col_g[c] = ldexp(comp_g[sh.comp0 + q],
                                       sp::norm_shift(canon_l(sh.L, q, 0), canon_l(sh.L, q, 1), canon_l(sh.L, q, 2)));
                }
            }
            col += ncanon(sh.L);
        }
        m.panel.push_back((int)m.shell.size());
    }
    return m;
}

const uint64_t* split_exp_table()
{
    static const std::vector<uint64_t> t = [] {
        std::vector<uint64_t> v(OKG_SPLIT_EXP);
        for (int j = 0; j < OKG_SPLIT_EXP; ++j)
            v[j] = (uint64_t)roundl(ldexpl(exp2l(-(long double)j / OKG_SPLIT_EXP), 63));
        return v;
    }();
    return t.data();
}

// Polls of the bounded waits in calls from this host thread (okg_set_wait_limit).
static thread_local long long t_wait_limit = sp::WAIT_LIMIT;
long long split_wait_limit() { return t_wait_limit; }

namespace {

constexpr int MAX_DEVICES = 64;

// The library's own stream-ordered pool for the coefficient digits of a call (a few MB):
// safe for any number of threads and streams; up to 64 MB stay mapped between calls.
cudaMemPool_t workspace_pool(int device)
{
    static std::mutex lock;
    static cudaMemPool_t pools[MAX_DEVICES] = {};
    if (device < 0 || device >= MAX_DEVICES) return nullptr;
    std::lock_guard<std::mutex> hold(lock);
    if (!pools[device]) {
        cudaMemPoolProps props{};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = device;
        const RelaxedCapture guard;
        cudaMemPool_t p = nullptr;
        if (cudaMemPoolCreate(&p, &props) != cudaSuccess) {
            (void)cudaGetLastError();
            return nullptr;
        }
        uint64_t keep = 64ull << 20;
        cudaMemPoolSetAttribute(p, cudaMemPoolAttrReleaseThreshold, &keep);
        pools[device] = p;
    }
    return pools[device];
}

int sm_count(int device)
{
    static int n[MAX_DEVICES] = {};
    if (device < 0 || device >= MAX_DEVICES) return 1;
    if (!n[device]) {
        int v = 0;
        cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, device);
        n[device] = v > 0 ? v : 1;
    }
    return n[device];
}

int current_device()
{
    int d = 0;
    cudaGetDevice(&d);
    return d;
}

template <int NCH, int MODE>
int launch(sp::Args& A, int nblk, size_t smem, cudaStream_t st)
{
    // (set on every launch: the attribute belongs to the current device; always to the same
    // size, as the device's other host threads launch under it)
    cudaError_t e = cudaFuncSetAttribute(sp::split_kernel<NCH, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         sp::SMEM_MAX);
    if (e != cudaSuccess) return cuda_status(e, "FP64 tensor-core path: shared memory");
    sp::split_kernel<NCH, MODE><<<nblk, sp::Cfg<NCH>::NT, smem, st>>>(A);
    return cuda_status(cudaGetLastError(), "FP64 tensor-core path: launch");
}

template <int NCH>
int run(const okg_basis* b, const Grid& g, const SplitCall& c, const SplitGeneral& general, cudaStream_t st, bool& done)
{
    using C = sp::Cfg<NCH>;
    const int npmax = C::RG == 1 ? 64 : 32;  // 7 accumulators per MO and row tile in 512 TMEM columns
    sp::Args A{};
    A.B = b->dev;
    A.S = b->split;
    A.g = g;
    A.nmo = c.nmo;
    A.npass = (c.nmo + npmax - 1) / npmax;
    A.np = ((c.nmo + A.npass - 1) / A.npass + 15) & ~15;
    A.drv = c.drv;
    A.out = c.out;
    A.dout = c.dout;
    A.g_rho = c.g_rho;
    A.g_grad = c.g_grad;
    A.g_ld = c.g_ld;
    A.wv_float = c.wv_float;
    A.ld = c.ld;
    A.brick = g.regular && g.offset == 0 && g.npts == (long long)g.nx * g.ny * g.nz;
    const int device = current_device(), sms = sm_count(device);
    // 128-point tiles share one screening; with fewer than four of them per SM, calls with
    // derivatives take 32-point tiles, which spread over the SMs
    A.nsub = 4;
    for (;;) {
        if (A.brick) {
            A.nby = (g.ny + 3) / 4;
            A.nbz = (g.nz + 7) / 8;
            A.ntiles = (long long)((g.nx + A.nsub - 1) / A.nsub) * A.nby * A.nbz;
        } else {
            A.ntiles = (g.npts + 32 * A.nsub - 1) / (32 * A.nsub);
        }
        if (A.nsub == 1 || NCH == 1 || A.ntiles >= 4ll * sms) break;
        A.nsub = 1;
    }
    const int acc_cols = C::RG * sp::ND * A.np;
    A.nacc = 2 * acc_cols <= 512 ? 2 : 1;
    A.tm_cols = 32;
    while ((int)A.tm_cols < A.nacc * acc_cols) A.tm_cols *= 2;
    const size_t slot = ((size_t)C::RG * sp::ND * sp::DT + (size_t)sp::ND * A.np * sp::PK * 2 + 1023) & ~(size_t)1023;
    const size_t norm = (size_t)C::NEW * A.npass * A.np * 8;
    A.norm_smem = c.mo_norm && norm <= 16384;
    const size_t tab = (size_t)A.npass * A.np * 12;
    const size_t fixed0 = 1024 + sp::AUX_BYTES + (A.norm_smem ? norm : 0) + (NCH == 1 ? sp::NBUF * 3 * 128 * 8 : 0) + (C::EPQ - 1) * 4 * 32 * 8;
    // (the MO table only where it does not cost an operand slot)
    A.tab_smem = tab <= 8192 && (sp::SMEM_MAX - fixed0 - tab) / slot == (sp::SMEM_MAX - fixed0) / slot;
    const size_t fixed = fixed0 + (A.tab_smem ? tab : 0);
    A.nslot = (int)((sp::SMEM_MAX - fixed) / slot);
    if (A.nslot > sp::MAX_SLOTS) A.nslot = sp::MAX_SLOTS;
    if (A.nslot < 2) return OKG_OK;
    const int nblk = (int)(A.ntiles < sms ? A.ntiles : sms);
    cudaMemPool_t pool = workspace_pool(device);
    if (!pool) return OKG_OK;
    A.limit = split_wait_limit();
    const int nrow = A.npass * A.np;
    auto up = [](size_t v) { return (v + 255) & ~(size_t)255; };
    const size_t o_fexp = 256, o_occ = o_fexp + up(4 * (size_t)nrow), o_norm = o_occ + up(8 * (size_t)nrow),
                 o_b = o_norm + (c.mo_norm ? up(8 * (size_t)nrow) : 0),
                 o_phi = o_b + up((size_t)nrow * b->split.npanel * sp::ND * sp::PK * 2),
                 bytes = o_phi + (b->split.npanel > sp::GROUP ? (size_t)nblk * C::RG * A.np * 128 * 8 : 0);
    char* ws = nullptr;
    if (cudaMallocFromPoolAsync((void**)&ws, bytes, pool, st) != cudaSuccess) {
        (void)cudaGetLastError();
        return OKG_OK;  // no room for the digits: the caller's other path needs none
    }
    A.counter = (unsigned long long*)ws;
    A.redo = c.redo ? c.redo : (int*)(ws + 8);
    A.mo_norm = c.mo_norm ? (double*)(ws + o_norm) : nullptr;
    A.fexp = (const int*)(ws + o_fexp);
    A.occ = (const double*)(ws + o_occ);
    A.bpack = (const unsigned char*)(ws + o_b);
    A.phi = b->split.npanel > sp::GROUP ? (double*)(ws + o_phi) : nullptr;
    sp::split_pack_kernel<<<nrow, 256, 0, st>>>(b->split, c.nmo, A.np, b->ncart, c.C, c.occ, (unsigned char*)(ws + o_b),
                                                (int*)(ws + o_fexp), (double*)(ws + o_occ), A.counter, (int*)(ws + 8), A.mo_norm);
    int s = cuda_status(cudaGetLastError(), "FP64 tensor-core path: coefficient digits");
    const size_t smem = fixed + A.nslot * slot;
    if (!s) {
        if (c.g_rho) {
            if constexpr (NCH == 4) s = launch<NCH, sp::OUT_WV>(A, nblk, smem, st);
        } else {
            s = c.mo_out ? launch<NCH, sp::OUT_MO>(A, nblk, smem, st) : launch<NCH, sp::OUT_RHO>(A, nblk, smem, st);
            if (!s) s = general.run(general.self, A.redo, A.mo_norm);
        }
    }
    const cudaError_t e = cudaFreeAsync(ws, st);
    if (!s) s = cuda_status(e, "FP64 tensor-core path: workspace");
    done = s == OKG_OK;
    return s;
}
}  // namespace

bool split_basis(const okg_basis* b)
{
    return b->nshell <= sp::MAX_SHELLS && b->split.npanel <= sp::MAX_PANELS && b->dev.max_nprim <= 255;
}

int split_run(const okg_basis* b, const Grid& g, const SplitCall& c, const SplitGeneral& general, cudaStream_t st, bool& done)
{
    done = false;
    if (c.need & ~0x7Fu) return OKG_OK;  // mixed second derivatives
    // Few points do not fill the chip with operand tiles (a tile's latency is 60 us for a
    // 3-atom, 130 us for a 12-atom molecule), while fused64_kernel spreads 8 points per CTA
    // and takes 32 / 70 us for up to 8 points per SM.  Measured (3 atoms | 12 atoms | 40
    // spherical atoms, fused64 against this path, us): values 3000 points 54:71 | 131:153 |
    // 542:898, 10000 points 176:72 | 514:155 | 2394:918; gradients 1000 points 49:65 |
    // 111:130 | 1004:616, 3000 points 94:64 | 243:133 | 2100:692; second derivatives 1000
    // points 62:86 | 147:198 | 1439:1533, 3000 points 121:84 | 328:199 | 2915:1658.
    const bool values = (c.need & ~1u) == 0;
    const bool contraction = (c.need & ~0xFu) == 0 && !values && (long long)c.nmo * b->ncart >= 32768;
    if (!c.g_rho && !contraction && g.npts < (values ? 32 : 16) * sm_count(current_device())) return OKG_OK;
    if (!split_basis(b)) return OKG_OK;
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st, &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone) {
        (void)cudaGetLastError();
        return OKG_OK;  // (a captured call keeps to the kernel without a workspace)
    }
    if ((c.need & ~1u) == 0) return run<1>(b, g, c, general, st, done);
    if ((c.need & ~0xFu) == 0) return run<4>(b, g, c, general, st, done);
    return run<7>(b, g, c, general, st, done);
}
}  // namespace okg

extern "C" int okg_wait_status(int* status)
{
    if (status) *status = 0;
    return OKG_OK;
}

extern "C" int okg_set_wait_limit(long long polls)
{
    if (polls < 0) return okg::set_error(OKG_ERR_ARG, "okg_set_wait_limit: polls < 0");
    okg::t_wait_limit = polls;
    return OKG_OK;
}
