// Basis packing, parameter upload and status reporting for liborbkit_gb300.
//
// okg_basis_create flattens orbkit's AO description (the arrays produced by
// AOClass getters, orbkit/orbitals.py:336-385) into one device block of tables:
// shells, canonical-component maps with the angular norm factors
// 1/sqrt((2l-1)!!(2m-1)!!(2n-1)!!) times the optional per-AO 'N' factor
// (orbkit/c_support.c:177-195, orbkit/core.py:98-100), the spherical transform
// (orbkit/core.py:135-176) and the shell chunks used by the fused kernels.
#include <math.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <string>
#include <vector>

#include "okg_internal.cuh"

namespace okg {

static thread_local std::string g_last_error;

int set_error(int status, const char* msg)
{
    g_last_error = msg ? msg : "";
    return status;
}

int cuda_status(cudaError_t e, const char* where)
{
    if (e == cudaSuccess) return OKG_OK;
    // consume the runtime's last-error state of this (non-sticky) error, so that a later
    // cudaGetLastError() after a good launch does not report it again
    (void)cudaGetLastError();
    std::string m = std::string(where) + ": " + cudaGetErrorString(e);
    g_last_error = m;
    return e == cudaErrorMemoryAllocation ? OKG_ERR_ALLOC : OKG_ERR_CUDA;
}

static int dfact(int n) { return n <= 0 ? 1 : n * dfact(n - 2); }

// Primitive weights w = c * (2/pi)^(3/4) 2^L alpha^((2L+3)/4) (or c when the
// contractions are pre-normalised) and the split single-precision copies used by
// the mixed path.
__global__ void prim_weights_kernel(const double* __restrict__ prim_in, const int* __restrict__ prim_L, int nprim,
                                    int is_normalized, double* __restrict__ prim_out, float* __restrict__ prim32,
                                    PrimMx* __restrict__ prim_mx, double* __restrict__ prim_adj,
                                    double2* __restrict__ prim_cusp)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nprim) return;
    const double a = prim_in[2 * i];
    const double c = prim_in[2 * i + 1];
    const int L = prim_L[i];
    double w = c, nrm = 1.0, dw = 0.0;
    if (!is_normalized) {
        nrm = pow(2.0 / M_PI, 0.75) * (pow(2.0, (double)L) * pow(a, (2.0 * L + 3.0) / 4.0));
        w = c * nrm;
        dw = w * (2.0 * L + 3.0) / (4.0 * a);  // d w / d alpha
    }
    prim_adj[2 * i] = dw;
    prim_adj[2 * i + 1] = nrm;
    prim_out[2 * i] = a;
    prim_out[2 * i + 1] = w;
    // mixed path: alpha * log2(e) and w as float hi + lo pairs
    const double al = a * 1.4426950408889634;
    const float ah = (float)al;
    const float wh = (float)w;
    prim32[4 * i + 0] = ah;
    prim32[4 * i + 1] = (float)(al - (double)ah);
    prim32[4 * i + 2] = wh;
    prim32[4 * i + 3] = (float)(w - (double)wh);
    PrimMx m;
    m.a2 = al;
    m.w = wh;
    m.wa = (float)(w * a);
    prim_mx[i] = m;
    prim_cusp[i] = make_double2(a, w);
}

// Mixed path: order each shell's primitives by ascending exponent, so that a
// tile keeps a prefix of them when screening (the radial sums do not depend on
// the order).  The FP64 {alpha, w} copy used for the cusp points of the mixed path is
// sorted along (same permutation, split_place), and the FP64 tensor-core path's tables
// are filled in the sorted order; *flags is raised by a parameter or position out of their
// range (split_prim).  Latency bounds it (a few hundred shells): a warp per shell and a lane per
// primitive, whose place is the number of smaller exponents (equal ones by index).  One
// thread per shell, inserting through global memory, took 13.8 us against 4.4 us (12 atoms);
// that form is left for more than 32 primitives and exponents that are not numbers.
__global__ void sort_prim_mx_kernel(const Shell* __restrict__ shells, int nshell, PrimMx* __restrict__ prim_mx,
                                    double2* __restrict__ prim_cusp, const double* __restrict__ atoms, int natom,
                                    float4* __restrict__ split_lg, SplitPrim* __restrict__ split_pr,
                                    int* __restrict__ split_place, int* __restrict__ flags)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x, lane = t & 31, s = t >> 5;
    for (int i = t; i < natom; i += gridDim.x * blockDim.x)
        for (int d = 0; d < 3; ++d)
            if (!(fabs(atoms[4 * i + d]) < 536870912.0)) atomicOr(flags, 1);
    if (s >= nshell) return;
    const int p0 = shells[s].prim0, np = shells[s].nprim;
    const bool on = np <= 32 && lane < np;
    PrimMx v{};
    double2 c = make_double2(0.0, 0.0);
    if (on) {
        v = prim_mx[p0 + lane];
        c = prim_cusp[p0 + lane];
    }
    if (np <= 32 && !__any_sync(0xffffffffu, on && isnan(v.a2))) {
        int place = 0;
        for (int j = 0; j < np; ++j) {
            const double other = __shfl_sync(0xffffffffu, v.a2, j);
            place += other < v.a2 || (other == v.a2 && j < lane);
        }
        __syncwarp();
        if (on) {
            prim_mx[p0 + place] = v;
            prim_cusp[p0 + place] = c;
            split_place[p0 + place] = p0 + lane;
        }
    } else if (lane == 0) {
        for (int i = 0; i < np; ++i) split_place[p0 + i] = p0 + i;
        for (int i = 1; i < np; ++i) {
            v = prim_mx[p0 + i];
            c = prim_cusp[p0 + i];
            int j = i - 1;
            while (j >= 0 && prim_mx[p0 + j].a2 > v.a2) {
                prim_mx[p0 + j + 1] = prim_mx[p0 + j];
                prim_cusp[p0 + j + 1] = prim_cusp[p0 + j];
                split_place[p0 + j + 1] = split_place[p0 + j];
                --j;
            }
            prim_mx[p0 + j + 1] = v;
            prim_cusp[p0 + j + 1] = c;
            split_place[p0 + j + 1] = p0 + i;
        }
    }
    __syncwarp();
    for (int i = lane; i < np; i += 32)
        if (!split_prim(prim_cusp[p0 + i], split_lg[p0 + i], split_pr[p0 + i])) atomicOr(flags, 1);
}

__global__ void atoms_kernel(const double* __restrict__ geo, int natom, double* __restrict__ atoms, int* __restrict__ flags)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i == 0) *flags = 0;
    if (i >= natom) return;
    atoms[4 * i + 0] = geo[3 * i + 0];
    atoms[4 * i + 1] = geo[3 * i + 1];
    atoms[4 * i + 2] = geo[3 * i + 2];
    atoms[4 * i + 3] = 0.0;
}

}  // namespace okg

using namespace okg;

extern "C" const char* okg_status_string(int s)
{
    switch (s) {
    case OKG_OK: return "ok";
    case OKG_ERR_ARG: return "invalid argument";
    case OKG_ERR_L: return "unsupported angular momentum";
    case OKG_ERR_DRV: return "invalid derivative code";
    case OKG_ERR_CUDA: return "CUDA error";
    case OKG_ERR_ALLOC: return "allocation failed";
    case OKG_ERR_TIMEOUT: return "device wait timed out";
    case OKG_ERR_UNSUPPORTED: return "unsupported shape";
    case OKG_ERR_DEVICE: return "no usable device";
    default: return "unknown status";
    }
}

extern "C" const char* okg_last_error(void) { return g_last_error.c_str(); }

extern "C" int okg_version(void) { return 100; }

namespace {
struct Layout {
    size_t off = 0;
    size_t take(size_t bytes)
    {
        size_t o = (off + 255) & ~(size_t)255;
        off = o + bytes;
        return o;
    }
};

// Mixed-path column layout for a shell order: whole shells, in that order, packed
// into chunks of at most OKG_MKC canonical columns; per chunk column, the listed
// Cartesian row it feeds (or -1) and its angular norm.  At most one chunk per shell.
struct MixedLayout {
    std::vector<Shell> mshells;
    std::vector<int4> mchunks;
    std::vector<int> mcol_cart;
    std::vector<double> mcol_g;
};

MixedLayout mixed_layout(const std::vector<Shell>& shells, const std::vector<int>& comp_row,
                         const std::vector<double>& comp_g, const int* order)
{
    MixedLayout m;
    const int n = (int)shells.size();
    int s0 = 0, col = 0;
    for (int i = 0; i <= n; ++i) {
        const int nk = i < n ? ncanon(shells[order ? order[i] : i].L) : 0;
        if (i == n || col + nk > OKG_MKC) {
            m.mchunks.push_back(make_int4(s0, i, col, 0));
            const size_t base = m.mcol_cart.size();
            m.mcol_cart.resize(base + OKG_MKC, -1);
            m.mcol_g.resize(base + OKG_MKC, 0.0);
            for (int t = s0; t < i; ++t) {
                const Shell& sh = m.mshells[t];
                for (int q = 0; q < ncanon(sh.L); ++q) {
                    const int r = comp_row[sh.comp0 + q];
                    if (r >= 0) {
                        m.mcol_cart[base + sh.mcol + q] = sh.cart0 + r;
                        m.mcol_g[base + sh.mcol + q] = comp_g[sh.comp0 + q];
                    }
                }
            }
            s0 = i;
            col = 0;
        }
        if (i < n) {
            Shell sh = shells[order ? order[i] : i];
            sh.mcol = col;
            sh.mchunk = (int)m.mchunks.size();
            m.mshells.push_back(sh);
            col += nk;
        }
    }
    return m;
}

// Tables in a host image of the basis block (one upload).
struct Image {
    std::vector<char> bytes;
    template <typename T>
    void put(size_t off, const std::vector<T>& v)
    {
        if (!v.empty()) memcpy(bytes.data() + off, v.data(), sizeof(T) * v.size());
    }
};

// Offsets of the tables that depend on the shell order, one contiguous range of the block
// [begin, end) with room for one chunk and one panel per shell.
struct OrderOffsets {
    size_t msh, mch, mcc, mcg, ssh, spn, scc, scg, begin, end;
};

void put_order(okg_basis* b, Image& im, const OrderOffsets& o, size_t base, const MixedLayout& m, const SplitLayout& s)
{
    im.put(o.msh - base, m.mshells);
    im.put(o.mch - base, m.mchunks);
    im.put(o.mcc - base, m.mcol_cart);
    im.put(o.mcg - base, m.mcol_g);
    im.put(o.ssh - base, s.shell);
    im.put(o.spn - base, s.panel);
    im.put(o.scc - base, s.col_cart);
    im.put(o.scg - base, s.col_g);
    b->dev.nmchunk = (int)m.mchunks.size();
    b->split.npanel = (int)s.panel.size() - 1;
}
}  // namespace

// What okg_basis_set_mixed_order needs of the basis on the host.
struct okg_basis_host {
    std::vector<Shell> shells;
    std::vector<int> comp_row;
    std::vector<double> comp_g;
    OrderOffsets order;
};

extern "C" int okg_basis_create(int natom, int nshell, const int* h_shell_atom, const int* h_shell_ncart,
                                const int* h_shell_nprim, const int* h_lxlylz, int is_normalized,
                                const double* h_renorm, int nsph, const int* h_sph_ptr, const int* h_sph_cart,
                                const double* h_sph_coef, okg_basis** out)
{
    if (!out) return set_error(OKG_ERR_ARG, "okg_basis_create: out is NULL");
    *out = nullptr;
    if (natom <= 0 || nshell <= 0 || !h_shell_atom || !h_shell_ncart || !h_shell_nprim || !h_lxlylz)
        return set_error(OKG_ERR_ARG, "okg_basis_create: empty basis or NULL array");
    if (nsph < 0 || (nsph > 0 && (!h_sph_ptr || !h_sph_cart || !h_sph_coef)))
        return set_error(OKG_ERR_ARG, "okg_basis_create: spherical transform arrays missing");

    std::vector<Shell> shells(nshell);
    std::vector<int> comp_row;
    std::vector<double> comp_g;
    std::vector<int> prim_L;
    std::vector<int> prim_atom;  // atom of each primitive (the AO kernel's per-axis tables)
    int ncart = 0, nprim = 0, max_np = 0, max_l = 0;
    int l_hist[OKG_MAX_L + 1] = {0};
    for (int s = 0; s < nshell; ++s) {
        const int nc = h_shell_ncart[s], np = h_shell_nprim[s], at = h_shell_atom[s];
        if (nc <= 0 || np <= 0 || at < 0 || at >= natom)
            return set_error(OKG_ERR_ARG, "okg_basis_create: shell with no components/primitives or bad atom index");
        const int* l0 = h_lxlylz + 3 * ncart;
        const int L = l0[0] + l0[1] + l0[2];
        if (L < 0 || L > OKG_MAX_L) return set_error(OKG_ERR_L, "okg_basis_create: angular momentum above 4");
        Shell& sh = shells[s];
        sh.atom = at;
        sh.L = L;
        sh.nprim = np;
        sh.prim0 = nprim;
        sh.cart0 = ncart;
        sh.ncart = nc;
        sh.comp0 = (int)comp_row.size();
        sh.out0 = ncart;
        sh.nout = nc;
        sh.sph0 = 0;
        const int nk = ncanon(L);
        if (nc > nk) return set_error(OKG_ERR_L, "okg_basis_create: more components than the shell's L allows");
        comp_row.resize(sh.comp0 + nk, -1);
        comp_g.resize(sh.comp0 + nk, 0.0);
        for (int r = 0; r < nc; ++r) {
            const int* lc = h_lxlylz + 3 * (ncart + r);
            if (lc[0] < 0 || lc[1] < 0 || lc[2] < 0 || lc[0] + lc[1] + lc[2] != L)
                return set_error(OKG_ERR_L, "okg_basis_create: components of mixed angular momentum in one shell");
            int j = -1;
            for (int q = 0; q < nk; ++q)
                if (canon_l(L, q, 0) == lc[0] && canon_l(L, q, 1) == lc[1] && canon_l(L, q, 2) == lc[2]) j = q;
            if (j < 0 || comp_row[sh.comp0 + j] >= 0)
                return set_error(OKG_ERR_L, "okg_basis_create: repeated Cartesian component in one shell");
            comp_row[sh.comp0 + j] = r;
            double g = is_normalized ? 1.0 : 1.0 / sqrt((double)(dfact(2 * lc[0] - 1) * dfact(2 * lc[1] - 1) *
                                                                  dfact(2 * lc[2] - 1)));
            if (h_renorm) g *= h_renorm[ncart + r];
            comp_g[sh.comp0 + j] = g;
        }
        for (int q = 0; q < np; ++q) {
            prim_L.push_back(L);
            prim_atom.push_back(at);
        }
        ncart += nc;
        nprim += np;
        max_np = np > max_np ? np : max_np;
        max_l = L > max_l ? L : max_l;
        l_hist[L]++;
    }

    // spherical transform -> (canonical component within shell, coefficient)
    std::vector<int> sph_ptr(1, 0), sph_cidx;
    std::vector<double> sph_coef;
    if (nsph > 0) {
        std::vector<int> row_shell(ncart), row_canon(ncart);
        for (int s = 0; s < nshell; ++s) {
            const Shell& sh = shells[s];
            for (int q = 0; q < ncanon(sh.L); ++q) {
                int r = comp_row[sh.comp0 + q];
                if (r >= 0) {
                    row_shell[sh.cart0 + r] = s;
                    row_canon[sh.cart0 + r] = q;
                }
            }
            shells[s].nout = 0;
        }
        int prev_shell = -1;
        for (int r = 0; r < nsph; ++r) {
            const int t0 = h_sph_ptr[r], t1 = h_sph_ptr[r + 1];
            if (t1 <= t0) return set_error(OKG_ERR_ARG, "okg_basis_create: spherical row without components");
            int s = -1;
            for (int t = t0; t < t1; ++t) {
                const int c = h_sph_cart[t];
                if (c < 0 || c >= ncart) return set_error(OKG_ERR_ARG, "okg_basis_create: spherical component index");
                if (s >= 0 && row_shell[c] != s)
                    return set_error(OKG_ERR_ARG, "okg_basis_create: spherical row mixes shells");
                s = row_shell[c];
                sph_cidx.push_back(row_canon[c]);
                sph_coef.push_back(h_sph_coef[t]);
            }
            sph_ptr.push_back((int)sph_cidx.size());
            if (s != prev_shell) {
                if (shells[s].nout != 0)
                    return set_error(OKG_ERR_ARG, "okg_basis_create: spherical rows of a shell are not contiguous");
                shells[s].out0 = r;
                shells[s].sph0 = r;
                prev_shell = s;
            }
            shells[s].nout++;
        }
    }

    // chunks of whole shells with at most OKG_KC listed rows
    std::vector<int4> chunks;
    {
        int s0 = 0, k0 = 0, k = 0;
        for (int s = 0; s < nshell; ++s) {
            if (k + shells[s].ncart - k0 > OKG_KC) {
                chunks.push_back(make_int4(s0, s, k0, k));
                s0 = s;
                k0 = k;
            }
            k += shells[s].ncart;
        }
        chunks.push_back(make_int4(s0, nshell, k0, k));
    }

    okg_basis* b = (okg_basis*)calloc(1, sizeof(okg_basis));
    if (!b) return set_error(OKG_ERR_ALLOC, "okg_basis_create: host allocation");
    Layout lay;
    const size_t o_atoms = lay.take(sizeof(double) * 4 * natom);
    const size_t o_shells = lay.take(sizeof(Shell) * nshell);
    const size_t o_prim = lay.take(sizeof(double) * 2 * nprim);
    const size_t o_prim32 = lay.take(sizeof(float) * 4 * nprim);
    const size_t o_primL = lay.take(sizeof(int) * nprim);
    const size_t o_patom = lay.take(sizeof(int) * nprim);
    const size_t o_crow = lay.take(sizeof(int) * comp_row.size());
    const size_t o_cg = lay.take(sizeof(double) * comp_g.size());
    const size_t o_sptr = lay.take(sizeof(int) * sph_ptr.size());
    const size_t o_scid = lay.take(sizeof(int) * (sph_cidx.size() + 1));
    const size_t o_scoef = lay.take(sizeof(double) * (sph_coef.size() + 1));
    const size_t o_chunks = lay.take(sizeof(int4) * chunks.size());
    const size_t o_pmx = lay.take(sizeof(PrimMx) * nprim);
    const size_t o_pcusp = lay.take(sizeof(double2) * nprim);
    const size_t o_asp = lay.take(sizeof(int) * (natom + 1));
    const size_t o_ash = lay.take(sizeof(int) * nshell);
    const size_t o_padj = lay.take(sizeof(double) * 2 * nprim);
    OrderOffsets oo;
    oo.begin = oo.msh = lay.take(sizeof(Shell) * nshell);
    oo.mch = lay.take(sizeof(int4) * nshell);
    oo.mcc = lay.take(sizeof(int) * OKG_MKC * nshell);
    oo.mcg = lay.take(sizeof(double) * OKG_MKC * nshell);
    oo.ssh = lay.take(sizeof(int4) * nshell);
    oo.spn = lay.take(sizeof(int) * (nshell + 1));
    oo.scc = lay.take(sizeof(int) * OKG_SPLIT_PK * nshell);
    oo.scg = lay.take(sizeof(double) * OKG_SPLIT_PK * nshell);
    oo.end = lay.take(0);
    const size_t o_slg = lay.take(sizeof(float4) * nprim);
    const size_t o_spr = lay.take(sizeof(SplitPrim) * nprim);
    const size_t o_spl = lay.take(sizeof(int) * nprim);
    const size_t o_sfl = lay.take(sizeof(int));
    const size_t o_exp = lay.take(sizeof(uint64_t) * OKG_SPLIT_EXP);
    // the transform by Cartesian row; entries of the same spherical row added up in order
    std::vector<int> cart_ptr(ncart + 1, 0), cart_srow, sph_cart;
    std::vector<double> cart_coef;
    if (nsph > 0) {
        std::vector<std::vector<std::pair<int, double>>> by(ncart);
        for (int r = 0; r < nsph; ++r)
            for (int t = h_sph_ptr[r]; t < h_sph_ptr[r + 1]; ++t) {
                auto& v = by[h_sph_cart[t]];
                if (!v.empty() && v.back().first == r) v.back().second += h_sph_coef[t];
                else v.push_back({r, h_sph_coef[t]});
                sph_cart.push_back(h_sph_cart[t]);
            }
        for (int c = 0; c < ncart; ++c) {
            for (const auto& e : by[c]) {
                cart_srow.push_back(e.first);
                cart_coef.push_back(e.second);
            }
            cart_ptr[c + 1] = (int)cart_srow.size();
        }
    }
    const size_t o_cptr = lay.take(sizeof(int) * (ncart + 1));
    const size_t o_crw = lay.take(sizeof(int) * (cart_srow.size() + 1));
    const size_t o_ccf = lay.take(sizeof(double) * (cart_coef.size() + 1));
    const size_t o_scart = lay.take(sizeof(int) * (sph_cart.size() + 1));
    const size_t bytes = lay.take(0);
    char* blk = nullptr;
    cudaError_t e = cudaMalloc((void**)&blk, bytes);
    if (e != cudaSuccess) {
        free(b);
        return cuda_status(e, "okg_basis_create: cudaMalloc");
    }
    // shells of each atom (CSR), for the cusp points of the mixed path
    std::vector<int> atom_shell_ptr(natom + 1, 0), atom_shells(nshell);
    for (int s = 0; s < nshell; ++s) atom_shell_ptr[shells[s].atom + 1]++;
    for (int a = 0; a < natom; ++a) atom_shell_ptr[a + 1] += atom_shell_ptr[a];
    {
        std::vector<int> fill(atom_shell_ptr.begin(), atom_shell_ptr.end() - 1);
        for (int s = 0; s < nshell; ++s) atom_shells[fill[shells[s].atom]++] = s;
    }
    Image im;
    im.bytes.assign(bytes, 0);
    im.put(o_shells, shells);
    im.put(o_primL, prim_L);
    im.put(o_patom, prim_atom);
    im.put(o_asp, atom_shell_ptr);
    im.put(o_ash, atom_shells);
    im.put(o_crow, comp_row);
    im.put(o_cg, comp_g);
    im.put(o_sptr, sph_ptr);
    im.put(o_scid, sph_cidx);
    im.put(o_scoef, sph_coef);
    im.put(o_chunks, chunks);
    memcpy(im.bytes.data() + o_exp, split_exp_table(), sizeof(uint64_t) * OKG_SPLIT_EXP);
    im.put(o_cptr, cart_ptr);
    im.put(o_crw, cart_srow);
    im.put(o_ccf, cart_coef);
    im.put(o_scart, sph_cart);
    // columns in basis order (okg_basis_set_mixed_order may choose another)
    put_order(b, im, oo, 0, mixed_layout(shells, comp_row, comp_g, nullptr), split_layout(shells, comp_row, comp_g, nullptr));
    e = cudaMemcpy(blk, im.bytes.data(), bytes, cudaMemcpyHostToDevice);
    BasisDev& d = b->dev;
    d.mshells = (const Shell*)(blk + oo.msh);
    d.mchunks = (const int4*)(blk + oo.mch);
    d.mcol_cart = (const int*)(blk + oo.mcc);
    d.mcol_g = (const double*)(blk + oo.mcg);
    b->split.shell = (const int4*)(blk + oo.ssh);
    b->split.panel = (const int*)(blk + oo.spn);
    b->split.col_cart = (const int*)(blk + oo.scc);
    b->split.col_g = (const double*)(blk + oo.scg);
    b->split.prim_lg = (const float4*)(blk + o_slg);
    b->split.prim = (const SplitPrim*)(blk + o_spr);
    b->split.prim_place = (const int*)(blk + o_spl);
    b->split.flags = (const int*)(blk + o_sfl);
    b->split.exp_tab = (const uint64_t*)(blk + o_exp);
    b->cart_ptr = (const int*)(blk + o_cptr);
    b->cart_srow = (const int*)(blk + o_crw);
    b->cart_coef = (const double*)(blk + o_ccf);
    b->sph_cart = (const int*)(blk + o_scart);
    if (e != cudaSuccess) {
        cudaFree(blk);
        free(b);
        return cuda_status(e, "okg_basis_create: upload");
    }
    b->host = new okg_basis_host{std::move(shells), std::move(comp_row), std::move(comp_g), oo};
    b->dev_block = blk;
    b->dev_bytes = bytes;
    d.atoms = (const double*)(blk + o_atoms);
    d.shells = (const Shell*)(blk + o_shells);
    d.prim = (const double*)(blk + o_prim);
    d.prim32 = (const float*)(blk + o_prim32);
    d.prim_atom = (const int*)(blk + o_patom);
    d.comp_row = (const int*)(blk + o_crow);
    d.comp_g = (const double*)(blk + o_cg);
    d.sph_ptr = (const int*)(blk + o_sptr);
    d.sph_cidx = (const int*)(blk + o_scid);
    d.sph_coef = (const double*)(blk + o_scoef);
    d.chunks = (const int4*)(blk + o_chunks);
    d.prim_mx = (const PrimMx*)(blk + o_pmx);
    d.prim_cusp = (const double2*)(blk + o_pcusp);
    d.atom_shell_ptr = (const int*)(blk + o_asp);
    d.atom_shells = (const int*)(blk + o_ash);
    d.prim_adj = (const double*)(blk + o_padj);
    d.natom = natom;
    d.nshell = nshell;
    d.nprim = nprim;
    d.ncart = ncart;
    d.nsph = nsph;
    d.spherical = nsph > 0;
    d.max_nprim = max_np;
    d.nchunk = (int)chunks.size();
    b->h_shell_L = nullptr;
    b->natom = natom;
    b->nshell = nshell;
    b->nprim = nprim;
    b->ncart = ncart;
    b->nao_out = nsph > 0 ? nsph : ncart;
    b->max_l = max_l;
    for (int l = 0; l <= OKG_MAX_L; ++l) b->l_hist[l] = l_hist[l];
    b->is_normalized = is_normalized ? 1 : 0;
    b->prim_L = (int*)(blk + o_primL);
    b->ncomp = (int)b->host->comp_row.size();
    b->mixed_locked = 0;
    cudaGetDevice(&b->device);
    *out = b;
    return OKG_OK;
}

extern "C" int okg_basis_set_mixed_order(okg_basis* b, const int* h_order)
{
    if (!b || !h_order) return set_error(OKG_ERR_ARG, "okg_basis_set_mixed_order: NULL argument");
    if (b->mixed_locked)
        return set_error(OKG_ERR_ARG, "okg_basis_set_mixed_order: a mixed plan or evaluation already uses the basis");
    const int n = b->nshell;
    std::vector<char> seen(n, 0);
    for (int i = 0; i < n; ++i) {
        if (h_order[i] < 0 || h_order[i] >= n || seen[h_order[i]])
            return set_error(OKG_ERR_ARG, "okg_basis_set_mixed_order: order is not a permutation of the shells");
        seen[h_order[i]] = 1;
    }
    const okg_basis_host& h = *b->host;
    Image im;
    im.bytes.assign(h.order.end - h.order.begin, 0);
    put_order(b, im, h.order, h.order.begin, mixed_layout(h.shells, h.comp_row, h.comp_g, h_order),
              split_layout(h.shells, h.comp_row, h.comp_g, h_order));
    return cuda_status(cudaMemcpy((char*)b->dev_block + h.order.begin, im.bytes.data(), im.bytes.size(), cudaMemcpyHostToDevice),
                       "okg_basis_set_mixed_order");
}

extern "C" int okg_basis_destroy(okg_basis* b)
{
    if (!b) return OKG_OK;
    cudaError_t e = cudaFree(b->dev_block);
    delete b->host;
    free(b);
    return cuda_status(e, "okg_basis_destroy");
}

extern "C" int okg_basis_info(const okg_basis* b, int* ncart, int* nao, int* nshell, int* nprim, int* natom)
{
    if (!b) return set_error(OKG_ERR_ARG, "okg_basis_info: NULL basis");
    if (ncart) *ncart = b->ncart;
    if (nao) *nao = b->nao_out;
    if (nshell) *nshell = b->nshell;
    if (nprim) *nprim = b->nprim;
    if (natom) *natom = b->natom;
    return OKG_OK;
}

extern "C" int okg_basis_set_params(okg_basis* b, const double* d_geo, const double* d_prim, okg_stream stream)
{
    if (!b || !d_geo || !d_prim) return set_error(OKG_ERR_ARG, "okg_basis_set_params: NULL argument");
    cudaStream_t st = (cudaStream_t)stream;
    atoms_kernel<<<(b->natom + 127) / 128, 128, 0, st>>>(d_geo, b->natom, (double*)b->dev.atoms,
                                                          (int*)b->split.flags);
    prim_weights_kernel<<<(b->nprim + 127) / 128, 128, 0, st>>>(d_prim, b->prim_L, b->nprim, b->is_normalized,
                                                                 (double*)b->dev.prim, (float*)b->dev.prim32,
                                                                 (PrimMx*)b->dev.prim_mx, (double*)b->dev.prim_adj,
                                                                 (double2*)b->dev.prim_cusp);
    sort_prim_mx_kernel<<<(b->nshell + 3) / 4, 128, 0, st>>>(b->dev.shells, b->nshell, (PrimMx*)b->dev.prim_mx,
                                                                 (double2*)b->dev.prim_cusp, b->dev.atoms, b->natom,
                                                                 (float4*)b->split.prim_lg, (SplitPrim*)b->split.prim,
                                                                 (int*)b->split.prim_place, (int*)b->split.flags);
    return cuda_status(cudaGetLastError(), "okg_basis_set_params");
}
