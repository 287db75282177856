// mps_cluster.cuh -- the small levels of a V-cycle in one thread-block cluster.
//
// Below about 65^3 cells a level's work is smaller than the cost of launching
// it: every red-black pass and transfer is a dependent launch of about 4-6 us
// inside the captured graphs.  k_cluster runs the whole correction-scheme
// V-cycle from a top level down to the coarsest and back in one launch of one
// cluster of up to 16 blocks:
//   * a level's planes are split along z over the blocks; each block holds u of
//     its planes plus one ghost plane on either side in shared memory (x and y
//     ghosts included), and a pass that updates a boundary plane also stores the
//     new values into the neighbour block's ghost plane through distributed
//     shared memory, so every stencil read is local;
//   * one hardware cluster barrier separates the phases; a pass issues its
//     global loads (right-hand side of the top level, row coefficients) before
//     it waits;
//   * the split is chosen on the coarsest split level and inherited upwards
//     (a fine plane belongs to the block of its coarse parent), so restriction
//     and prolongation between split levels need no exchange either;
//   * levels of at most CL_GATHER cells live in the first block alone, where a
//     block barrier separates the phases;
//   * sixteen SMs must issue what the whole chip issued before, so the passes
//     are bound by instructions: a thread keeps one (x pair, y) column of a
//     level, its neighbour offsets and coefficients in registers, and marches
//     along its planes two at a time, without branches, and every phase's code
//     appears once (the instruction cache starts cold).
// Measured (257^3 mixed plasma solve, clock64 phase times): the V-cycle from
// 32^3 down takes about 45 us, against about 95 us for a one-block kernel of
// the levels of 16^3 and below plus the 32^3 level's launches; a 32^3 pass
// takes 1.5 us against 4.5 us for a launch, of which about 0.5 us is the
// barrier that publishes the stores into the neighbours.  FP64 divisions
// replaced by kept reciprocals gave nothing.
// A pass updates in place: the levels it accepts have no odd periodic size, so
// no cell has a neighbour of its own colour, and in place is the same as the
// "Jacobi within a colour" rule of perform_gseidel_smoothing
// (mgridlib/discretepde.f90:202-229).
//
// Operators: uniform coefficient (faces from per-axis tables), or explicit row
// coefficients, eight words per cell (the rows of convection operators, or those
// of a cell coefficient, packed once per solve by k_crows).  The transfers are
// the per-level kernels' own: volume-weighted mean of the children's residuals
// and trilinear prolongation on the geometric hierarchy (its widths),
// restriction / prolongation1 on the reference's (mgridsteps.f90:11-53,
// :170-216).  The coarsest solve is u = A^{-1} f with the precomputed dense
// inverse.
#pragma once

#include "mps_kernels.cuh"

namespace mps {

constexpr int CL_MAXC = 16;               // blocks of a cluster at most
constexpr int CL_MAXL = 12;               // levels of one launch, the coarsest included
constexpr int CL_TPB = 576;               // threads of a block: a column each of a 33 x 33 level, 96 registers
constexpr int CL_GATHER = 1024;           // cells of a level that one block takes alone
constexpr int CL_SMEM_MAX = 224 * 1024;   // shared-memory bytes of a block at most
// Cells of one colour in the largest block's share of the top level at most: beyond it
// one launch per pass on the whole chip is faster.  Explicit rows come from L2, in FP64
// at twice the words, and the launches for row operators (convection) read them with
// less around it than those for a cell coefficient do, so the lines differ.  Below the
// finest level the cluster also takes over the transfers, which FP32 rows repay.  Few
// blocks, of a level with few planes, replace launches that were small themselves.
// us a V-cycle with the level in the cluster / with its own launches, on a B200
// (cells of the share, blocks):
//   uniform    FP64 36^3 (2592, 16) 109 / 119, 33x65x33 (3315, 16) 131 / 122; FP32 97^3 (48^3
//              below: 4608, 12) 147 / 150, 64x64x16 (4096, 8) 103 / 89, 116x116x28 (3364, 7) 127 / 121
//   cell       FP64 33^3 (1683, 16) 111 / 121, 100x83x61 (2050, 15) 210 / 198; FP32 36^3 (2592, 16)
//              87 / 91, 40x33x65 (3300, 16) 104 / 95, 89^3 (44^3 below: 3872, 11) 155 / 160
//   convection FP64 33^3 112 / 103; FP32 50x41x30 (2050, 15) 81 / 87, 36^3 86 / 81, 81^3 (40^3 below:
//              3200, 16) 152 / 164
//   few blocks uniform FP32 64x64x1 (2048, 1) 80 / 59, FP64 45x50x1 (1150, 1) 81 / 84, 100x100x2
//              (50x50x1 below: 1250, 1) 131 / 119, 48x40x6 (1920, 3) 84 / 97, 100x30x8 (3000, 4) FP64
//              108 / 118, FP32 82 / 77
template <class T>
constexpr int cl_max_share(bool rows, bool row_operator, bool below, int blocks)
{
    int most = 3000;
    if (sizeof(T) == 4) most = !rows ? 4700 : below ? 3900 : row_operator ? 2200 : 3250;
    else if (rows) most = row_operator ? 1100 : 1750;
    const int few = sizeof(T) == 4 ? 900 + 340 * blocks : 600 + 640 * blocks;
    return most < few ? most : few;
}

// one fine position along one axis of a transfer: the offsets of two coarse
// cells in the coarse ghosted layout (x, gx y, gp z; z counted from plane 0) and
// their weights.  Geometric: the bracketing coarse centres; reference: the
// coarse neighbours up and down with +-1/8 of the central slope.  A coarse ghost
// across a physical face is folded into the weight of the cell it copies or
// mirrors (the rule of coarse_at); periodic x and y wrap, periodic z reads the
// ghost planes.
template <class T>
struct ClLin {
    int o0, o1;
    T w0, w1;
};

// one cell position along one axis of a level: the offsets of its two
// neighbours in the ghosted layout (periodic x and y faces wrap; along z the
// ghost planes hold the neighbours) and the coefficients of its two faces:
// Lev's face coefficient in the grid and across periodic faces, the Dirichlet
// coefficient dr / dlast or 0 at physical faces, whose ghost cells hold 0.
template <class T>
struct ClAx {
    int om, op;
    T cm, cp;
};

template <class T>
struct ClLev {
    int nx, ny, nz, nh;
    int gx, gp;                  // ghosted row pitch and plane size
    int P;                       // row pitch of the split layout
    int uo, fo;                  // u (ghosted) and f (natural order) in shared memory
    int ax0, lin0[3];            // first axis entry (x, y at +nx, z at +nx+ny); first bracket per axis
    int per;                     // bit a: periodic axis a
    int ncol, pg;                // columns (nh ny) and threads per column
    int rlog;                    // log2 of the lanes per coarse cell of the restriction from this level
    int z[CL_MAXC + 1];          // first plane of each block (split levels)
    FastDiv dcol, dnh, dny, dnx;
    T w[3], wl[3];
    T om0, om1;                  // relaxation of the first pre-smoothing sweep and of the other passes
    const T* rows;               // explicit rows: 8 words of the cell at split offset o of colour c at rows + 8 (c half + o)
    long long half;
};

template <class T>
struct ClPlan {
    int nl, m, nc;               // levels, split levels (the first m), blocks
    int nu1, nu2, geom;
    int only_black;              // the prolongation corrects the black cells only (nu2 >= 1)
    int load_u;                  // the top level starts from the state in uout (else from zero)
    int stage_off, part_off;     // byte offsets: restricted planes of the last split level, coarsest partial sums
    int ax_off, lin_off;         // byte offsets of the tables
    int nax, nlin, zero_vecs;    // table entries; 16-byte words of all u and f (cleared at the start)
    int share;                   // cells of one colour in the largest block of the top level
    T kc, dexc;                  // uniform coefficient / diagonal extra
    ClLev<T> lev[CL_MAXL];
};

__device__ __forceinline__ unsigned cl_rank()
{
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cl_arrive()
{
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");
}
__device__ __forceinline__ void cl_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }
__device__ __forceinline__ unsigned cl_map(unsigned a, unsigned rank)
{
    unsigned r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    return r;
}
__device__ __forceinline__ void cl_st(unsigned a, float v)
{
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
}
__device__ __forceinline__ void cl_st(unsigned a, double v)
{
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}
__device__ __forceinline__ void cl_ld(unsigned a, float& v)
{
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
}
__device__ __forceinline__ void cl_ld(unsigned a, double& v)
{
    asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(a) : "memory");
}

// one block's view of the launch
template <class T>
struct ClMem {
    T* S;                    // fields
    unsigned self;           // mapped field base of this block
    const ClAx<T>* ax;
    const ClLin<T>* lin;
    int rank;
    unsigned lo, hi, zero;   // mapped field bases of the lower / upper neighbour and of block 0
    int rlo, rhi;            // their ranks along z (wrapped; lower == own - 1 unless periodic)
};

// the planes of level s that this block holds: [z0, z0 + nl)
template <class T>
__device__ __forceinline__ void cl_span(const ClPlan<T>& P, int rank, int s, int& z0, int& nl)
{
    const ClLev<T>& G = P.lev[s];
    z0 = s >= P.m ? 0 : G.z[rank];
    nl = (s >= P.m ? G.nz : G.z[rank + 1]) - z0;
}

// the barrier between two phases of level s: blocks of the cluster, or the
// threads of the one block that holds the level
template <class T>
__device__ __forceinline__ void cl_end(const ClPlan<T>& P, int s)
{
    if (s < P.m) cl_arrive();
}
template <class T>
__device__ __forceinline__ void cl_begin(const ClPlan<T>& P, int s)
{
    if (s < P.m) cl_wait();
    else __syncthreads();
}

// where a level's boundary planes are shown: a cell at ghosted index g of local
// plane 0 (nl-1) also goes to lo (hi) + g elements, the upper (lower) ghost plane
// of the block below (above); CL_NOWHERE: to no block.  Each is an address less
// the offset of the cell's own plane, so it may lie below the shared memory or
// wrap: any multiple of the word can occur, 0 among them, an odd number cannot
struct ClPush {
    unsigned lo, hi;
};
constexpr unsigned CL_NOWHERE = 1u;
template <class T>
__device__ __forceinline__ ClPush cl_pushes(const ClPlan<T>& P, const ClMem<T>& M, int s, int z0, int nl)
{
    const ClLev<T>& G = P.lev[s];
    const bool per = (G.per >> 2) & 1, one = s >= P.m;  // one: the first block holds the whole level
    const int nlo = one ? nl : G.z[M.rlo + 1] - G.z[M.rlo];
    ClPush p;
    p.lo = z0 > 0 || per ? (one ? M.self : M.lo) + (unsigned)sizeof(T) * (unsigned)(G.uo + G.gp * nlo) : CL_NOWHERE;
    p.hi = z0 + nl < G.nz || per ? (one ? M.self : M.hi) + (unsigned)sizeof(T) * (unsigned)(G.uo - G.gp * nl) : CL_NOWHERE;
    return p;
}
template <class T>
__device__ __forceinline__ void cl_push(const ClPush& p, int g, int kl, int nl, T v)
{
    if (kl == 0 && p.lo != CL_NOWHERE) cl_st(p.lo + (unsigned)sizeof(T) * (unsigned)g, v);
    if (kl == nl - 1 && p.hi != CL_NOWHERE) cl_st(p.hi + (unsigned)sizeof(T) * (unsigned)g, v);
}

// the explicit row of one cell: diagonal, its reciprocal, x-, x+, y-, y+, z-, z+
template <class T, bool RF>
struct ClCell {
    T a[RF ? 8 : 1];
};
template <class T, bool RF>
__device__ __forceinline__ void cl_load(const T* rows, int o, ClCell<T, RF>& C)
{
    if constexpr (RF) {
        const T* r = rows + 8 * (long long)o;
        constexpr int W = 32 / (int)sizeof(T);
#pragma unroll
        for (int q = 0; q < 8; q += W) {
            const VecW<T, W> v = ldv<T, W>(r + q);
#pragma unroll
            for (int e = 0; e < W; e++) C.a[q + e] = v.v[e];
        }
    }
}

// what a thread keeps of its column: cells (2h, j), (2h+1, j) of every plane.
// Uniform coefficient: face weights (the tables hold coefficient times face
// coefficient), the x/y part of the diagonal and the reciprocal diagonals of the
// two cells for the z part zs.
template <class T, bool RF>
struct ClCol {
    int j, h, g0;          // g0: ghosted index of (2h, j) in the ghost plane below
    int has1;              // 2h+1 is a cell
    int xm[2], xp[2], ym, yp;
    T cxm[2], cxp[2], cym, cyp, d[2];
};
template <class T, bool RF>
__device__ __forceinline__ void cl_col(const ClPlan<T>& P, const ClMem<T>& M, const ClLev<T>& G, int cc,
                                       ClCol<T, RF>& K)
{
    K.j = (int)G.dnh.div((unsigned)cc);
    K.h = cc - K.j * G.nh;
    K.g0 = 2 * K.h + 1 + G.gx * (K.j + 1);
    K.has1 = 2 * K.h + 1 < G.nx;
    const ClAx<T>* ax = M.ax + G.ax0;
    const ClAx<T> Y = ax[G.nx + K.j];
    K.ym = Y.om;
    K.yp = Y.op;
#pragma unroll
    for (int q = 0; q < 2; q++) {
        const ClAx<T> X = ax[2 * K.h + (q && K.has1 ? 1 : 0)];
        K.xm[q] = X.om;
        K.xp[q] = X.op;
        if constexpr (!RF) {
            K.cxm[q] = X.cm;
            K.cxp[q] = X.cp;
            K.d[q] = P.dexc + ((X.cm + X.cp) + (Y.cm + Y.cp));
        }
    }
    if constexpr (!RF) {
        K.cym = Y.cm;
        K.cyp = Y.cp;
    }
}

// the red-black passes of level s before (pre) or after the coarse correction,
// in place.  CL_BATCH planes of a column at a time: their cells are independent
// (one colour), so their loads overlap; the row words of the first batch are in
// flight while the barrier is waited for.
template <class T>
struct ClBatch {
    static constexpr int N = 2;
};
template <class T, bool RF>
__device__ __forceinline__ void cl_smooth(const ClPlan<T>& P, const ClMem<T>& M, int s, bool pre)
{
    constexpr int B = ClBatch<T>::N;
    const ClLev<T>& G = P.lev[s];
    int z0, nl;
    cl_span(P, M.rank, s, z0, nl);
    const ClPush pd = cl_pushes(P, M, s, z0, nl);
    T* u = M.S + G.uo;
    const T* f = M.S + G.fo;
    const int nx = G.nx, gp = G.gp, pg = G.pg, ncol = G.ncol, split = s < P.m;
    const int sn = nx * G.ny, so = G.P * G.ny, pitch = G.P;
    const ClAx<T>* az = M.ax + G.ax0 + nx + G.ny + z0;
    const T om0 = G.om0, om1 = G.om1;
    const T* const rows = G.rows;
    const long long rhalf = 8 * G.half;
    const int p0 = pg > 1 ? (int)G.dcol.div(threadIdx.x) : 0;
    const int c0 = (int)threadIdx.x - p0 * ncol;
    const bool on = p0 < pg && c0 < ncol;
    const bool once = ncol <= CL_TPB;  // one column per thread: kept over the passes
    ClCol<T, RF> K;
    if (on) cl_col<T, RF>(P, M, G, c0, K);
    const int nsw = pre ? P.nu1 : P.nu2;
    for (int ps = 0; ps < 2 * nsw; ps++) {
        const int c = ps & 1, sw = ps >> 1;
        // pass_omega's schedule: plain where the transfers count on it
        T om;
        if (pre) om = c == 1 && sw == nsw - 1 ? T(1) : (sw == 0 ? om0 : om1);
        else om = c == 0 && sw == 0 ? T(1) : om1;
        // the last pass of all stores into no other block (they may have left)
        const bool push = pre || s > 0 || ps < 2 * nsw - 1;
        const unsigned lo = push ? pd.lo : CL_NOWHERE, hi = push ? pd.hi : CL_NOWHERE;
        const T* rc = rows + c * rhalf;
        ClCell<T, RF> w[B];
        // no branches within a batch: a cell that does not exist takes the column's first row
        auto exists = [&](int kl, int q) { return kl < nl && (q == 0 || K.has1); };
        auto fetch = [&](int kb) {  // the row words of planes kb, kb + pg, ... of the column
            if constexpr (RF) {
#pragma unroll
                for (int b = 0; b < B; b++) {
                    const int kl = kb + b * pg;
                    const int at = exists(kl, (K.j + z0 + kl + c) & 1) ? K.h + pitch * K.j + so * (z0 + kl) : 0;
                    cl_load<T, RF>(rc, at, w[b]);
                }
            }
        };
        if (on) {
            if (!once && ps > 0) cl_col<T, RF>(P, M, G, c0, K);
            fetch(p0);
        }
        if (split) cl_wait();
        else __syncthreads();
        for (int cc = c0; on && cc < ncol; cc += CL_TPB) {
            if (cc != c0) {
                cl_col<T, RF>(P, M, G, cc, K);
                fetch(p0);
            }
            for (int kb = p0; kb < nl; kb += B * pg) {
                if (kb != p0) fetch(kb);
                T v[B];
#pragma unroll
                for (int b = 0; b < B; b++) {
                    const int k1 = kb + b * pg, q1 = (K.j + z0 + k1 + c) & 1;
                    const bool ok = exists(k1, q1);
                    const int kl = ok ? k1 : p0, q = ok ? q1 : 0;
                    const int g = K.g0 + q + gp * (kl + 1);
                    const int xm = q ? K.xm[1] : K.xm[0], xp = q ? K.xp[1] : K.xp[0];
                    const T fv = f[2 * K.h + q + nx * K.j + sn * kl];
                    T val;
                    if constexpr (RF) {
                        const T off = ((w[b].a[2] * u[g + xm] + w[b].a[3] * u[g + xp]) +
                                       (w[b].a[4] * u[g + K.ym] + w[b].a[5] * u[g + K.yp])) +
                                      (w[b].a[6] * u[g - gp] + w[b].a[7] * u[g + gp]);
                        val = (fv - off) * w[b].a[1];
                    } else {
                        const T cxm = q ? K.cxm[1] : K.cxm[0], cxp = q ? K.cxp[1] : K.cxp[0];
                        const T zm = az[kl].cm, zp = az[kl].cp;
                        const T sum = ((cxm * u[g + xm] + cxp * u[g + xp]) +
                                       (K.cym * u[g + K.ym] + K.cyp * u[g + K.yp])) +
                                      (zm * u[g - gp] + zp * u[g + gp]);
                        val = gs_value<T>(fv, (q ? K.d[1] : K.d[0]) + (zm + zp), -sum);
                    }
                    v[b] = om == T(1) ? val : relax_to(om, val, u[g]);
                }
#pragma unroll
                for (int b = 0; b < B; b++) {
                    const int kl = kb + b * pg, q = (K.j + z0 + kl + c) & 1;
                    const int g = K.g0 + q + gp * (kl + 1);
                    const bool ok = exists(kl, q);
                    if (ok) u[g] = v[b];
                    if (ok && kl == 0 && lo != CL_NOWHERE) cl_st(lo + (unsigned)sizeof(T) * (unsigned)g, v[b]);
                    if (ok && kl == nl - 1 && hi != CL_NOWHERE) cl_st(hi + (unsigned)sizeof(T) * (unsigned)g, v[b]);
                }
            }
        }
        if (push && split) cl_arrive();
    }
}

// the children of coarse position p along one axis: first fine index and count
// (geometric: the last coarse cell takes the odd cell too)
__device__ __forceinline__ void cl_children(int geom, int nf, int nc, int p, int& lo, int& n)
{
    lo = nf == nc ? p : 2 * p;
    n = nf == nc ? 1 : ((geom && p == nc - 1) ? nf - 2 * (nc - 1) : 2);
}

// sum over the children of coarse column (I,J) in the fine planes lk ..
// lk+nk-1 (rows part, part + nparts, ... of them) of volume times residual
template <class T, bool RF>
__device__ __forceinline__ T cl_children_resid(const ClPlan<T>& P, const ClMem<T>& M, int s, int z0, int I, int J,
                                               int lk, int nk, int part, int nparts)
{
    const ClLev<T>& F = P.lev[s];
    const ClLev<T>& C = P.lev[s + 1];
    const T* u = M.S + F.uo;
    const ClAx<T>* ax = M.ax + F.ax0;
    const bool red_only = P.nu1 >= 1;  // after a black pass the black residuals vanish up to rounding
    int li, ni, lj, nj;
    cl_children(P.geom, F.nx, C.nx, I, li, ni);
    cl_children(P.geom, F.ny, C.ny, J, lj, nj);
    T sum = T(0);
    for (int q = part; q < nj * nk; q += nparts) {
        const int dk = nj == 2 ? q >> 1 : q / nj, j = lj + (q - dk * nj), k = lk + dk;
        const T vyz = (j == F.ny - 1 ? F.wl[1] : F.w[1]) * (k == F.nz - 1 ? F.wl[2] : F.w[2]);
        const int row = j + F.ny * (k - z0);
        const ClAx<T> Y = ax[F.nx + j];
        for (int i = li + (red_only ? ((li + j + k) & 1) : 0); i < li + ni; i += red_only ? 2 : 1) {
            const int g = (i + 1) + F.gx * (j + 1) + F.gp * (k - z0 + 1);
            ClCell<T, RF> W;
            cl_load<T, RF>(F.rows + ((i + j + k) & 1 ? 8 * F.half : 0), (i >> 1) + F.P * (j + F.ny * k), W);
            const T fv = M.S[F.fo + i + F.nx * row];
            const ClAx<T> X = ax[i];
            T r;
            if constexpr (RF) {
                const T off = ((W.a[2] * u[g + X.om] + W.a[3] * u[g + X.op]) +
                               (W.a[4] * u[g + Y.om] + W.a[5] * u[g + Y.op])) +
                              (W.a[6] * u[g - F.gp] + W.a[7] * u[g + F.gp]);
                r = fv - (W.a[0] * u[g] + off);
            } else {
                const ClAx<T> Z = ax[F.nx + F.ny + k];
                const T d = P.dexc + (((X.cm + X.cp) + (Y.cm + Y.cp)) + (Z.cm + Z.cp));
                const T sum6 = ((X.cm * u[g + X.om] + X.cp * u[g + X.op]) + (Y.cm * u[g + Y.om] + Y.cp * u[g + Y.op])) +
                               (Z.cm * u[g - F.gp] + Z.cp * u[g + F.gp]);
                r = fv - (d * u[g] - sum6);
            }
            sum += ((i == F.nx - 1 ? F.wl[0] : F.w[0]) * vyz) * r;
        }
    }
    return sum;
}
// the volume of the children of coarse cell (I,J,K)
template <class T>
__device__ __forceinline__ T cl_volume(const ClPlan<T>& P, const ClLev<T>& F, const ClLev<T>& C, int I, int J, int K)
{
    auto width = [&](int a, int nf, int nc, int p) {
        int lo, n;
        cl_children(P.geom, nf, nc, p, lo, n);
        return lo + n == nf ? (T)(n - 1) * F.w[a] + F.wl[a] : (T)n * F.w[a];
    };
    return width(0, F.nx, C.nx, I) * width(1, F.ny, C.ny, J) * width(2, F.nz, C.nz, K);
}

// f_{s+1} = R(f_s - A_s u_s) between levels of one split (or of the first
// block): 2^rlog lanes per coarse cell, each a share of the children's rows
template <class T, bool RF>
__device__ __forceinline__ void cl_restrict(const ClPlan<T>& P, const ClMem<T>& M, int s)
{
    const ClLev<T>& F = P.lev[s];
    const ClLev<T>& C = P.lev[s + 1];
    int zf, nlf, zc, nlc;
    cl_span(P, M.rank, s, zf, nlf);
    cl_span(P, M.rank, s + 1, zc, nlc);
    const int lg = F.rlog, NL = 1 << lg, part = (int)threadIdx.x & (NL - 1);
    const int n = C.nx * C.ny * nlc, per = CL_TPB >> lg;
    const int trips = (n + per - 1) / per;
    T* fc = M.S + C.fo;
    cl_begin(P, s);
    for (int t = 0; t < trips; t++) {  // the same trips for every lane (shuffles below)
        const int idx = t * per + ((int)threadIdx.x >> lg);
        T sum = T(0), vol = T(1);
        if (idx < n) {
            const int r = (int)C.dnx.div((unsigned)idx), I = idx - r * C.nx;
            const int kc = (int)C.dny.div((unsigned)r), J = r - kc * C.ny, K = zc + kc;
            int lk, nk;
            cl_children(P.geom, F.nz, C.nz, K, lk, nk);
            sum = cl_children_resid<T, RF>(P, M, s, zf, I, J, lk, nk, part, NL);
            vol = cl_volume(P, F, C, I, J, K);
        }
        for (int o = NL >> 1; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        if (idx < n && part == 0) fc[idx] = sum / vol;
    }
    __syncthreads();  // the coarse right-hand side is read by this block alone
}

// the same from the last split level into the first block's level: each block
// sums its own fine planes into the first block's staging planes ...
template <class T, bool RF>
__device__ __forceinline__ void cl_restrict_push(const ClPlan<T>& P, const ClMem<T>& M, int s)
{
    const ClLev<T>& C = P.lev[s + 1];
    int zf, nlf;
    cl_span(P, M.rank, s, zf, nlf);
    const int n = C.nx * C.ny * nlf;
    cl_begin(P, s);
    for (int idx = threadIdx.x; idx < n; idx += CL_TPB) {
        const int r = (int)C.dnx.div((unsigned)idx), I = idx - r * C.nx;
        const int kl = (int)C.dny.div((unsigned)r), J = r - kl * C.ny;
        const T v = cl_children_resid<T, RF>(P, M, s, zf, I, J, zf + kl, 1, 0, 1);
        cl_st(M.zero + (unsigned)P.stage_off + (unsigned)sizeof(T) * (unsigned)(C.nx * C.ny * zf + idx), v);
    }
    cl_end(P, s);
}
// ... which the first block adds up plane by plane
template <class T>
__device__ __forceinline__ void cl_restrict_sum(const ClPlan<T>& P, const ClMem<T>& M, int s)
{
    const ClLev<T>& F = P.lev[s];
    const ClLev<T>& C = P.lev[s + 1];
    const T* stage = reinterpret_cast<const T*>(reinterpret_cast<const unsigned char*>(M.S) + P.stage_off);
    const int np = C.nx * C.ny, n = np * C.nz;
    T* fc = M.S + C.fo;
    for (int idx = threadIdx.x; idx < n; idx += CL_TPB) {
        const int r = (int)C.dnx.div((unsigned)idx), I = idx - r * C.nx;
        const int K = (int)C.dny.div((unsigned)r), J = r - K * C.ny;
        int lk, nk;
        cl_children(P.geom, F.nz, C.nz, K, lk, nk);
        T sum = T(0);
        for (int q = 0; q < nk; q++) sum += stage[np * (lk + q) + (idx - np * K)];
        fc[idx] = sum / cl_volume(P, F, C, I, J, K);
    }
    __syncthreads();
}

// u_s += P u_{s+1}: the black cells (the first post-smoothing pass rewrites the
// red ones), or both colours without post-smoothing; a thread keeps one fine
// column as in cl_smooth.  A split level below the first block's level copies
// the coarse planes it reads first.
template <class T>
__device__ __forceinline__ void cl_prolong(const ClPlan<T>& P, const ClMem<T>& M, int s)
{
    const ClLev<T>& F = P.lev[s];
    const ClLev<T>& C = P.lev[s + 1];
    int z0, nl, cz, cnl;
    cl_span(P, M.rank, s, z0, nl);
    cl_span(P, M.rank, s + 1, cz, cnl);
    T* u = M.S + F.uo;
    T* ec = M.S + C.uo;
    if (s < P.m && s + 1 >= P.m) {
        cl_wait();
        if (M.rank != 0) {
            // ghosted planes K0 .. K1 (indices one above the cell's): parents of the own planes and one more each side
            const int K0 = F.nz == C.nz ? z0 : min(z0 >> 1, C.nz - 1);
            const int K1 = (F.nz == C.nz ? z0 + nl - 1 : min((z0 + nl - 1) >> 1, C.nz - 1)) + 2;
            for (int q = C.gp * K0 + (int)threadIdx.x; q < C.gp * (K1 + 1); q += CL_TPB)
                cl_ld(M.zero + (unsigned)sizeof(T) * (unsigned)(C.uo + q), ec[q]);
        }
        __syncthreads();
    } else {
        cl_begin(P, s);
    }
    const ClPush pd = cl_pushes(P, M, s, z0, nl);
    const T* e = ec - C.gp * cz;
    const ClLin<T>* lz = M.lin + F.lin0[2] + z0;
    const int p0 = F.pg > 1 ? (int)F.dcol.div(threadIdx.x) : 0;
    const int c0 = (int)threadIdx.x - p0 * F.ncol;
    if (p0 < F.pg)
        for (int cc = c0; cc < F.ncol; cc += CL_TPB) {
            const int j = (int)F.dnh.div((unsigned)cc), h = cc - j * F.nh;
            const bool has1 = 2 * h + 1 < F.nx;
            const int g0 = 2 * h + 1 + F.gx * (j + 1);
            const ClLin<T> lx0 = M.lin[F.lin0[0] + 2 * h], lx1 = M.lin[F.lin0[0] + 2 * h + (has1 ? 1 : 0)];
            const ClLin<T> ly = M.lin[F.lin0[1] + j];
            // the reference's form corrects from the parent and leaves an odd last cell alone
            const int I = h, J = j >> 1;
            const int par = (I + 1) + C.gx * (J + 1);
            if (!P.geom && (I >= C.nx || J >= C.ny)) continue;
            for (int kl = p0; kl < nl; kl += F.pg)
                for (int c = P.only_black ? 1 : 0; c < 2; c++) {
                    const int q = (j + z0 + kl + c) & 1;
                    if (q && !has1) continue;
                    const ClLin<T> z = lz[kl];
                    const int x0 = q ? lx1.o0 : lx0.o0, x1 = q ? lx1.o1 : lx0.o1;
                    const T wx0 = q ? lx1.w0 : lx0.w0, wx1 = q ? lx1.w1 : lx0.w1;
                    T v;
                    if (P.geom) {
                        const T* a = e + z.o0;
                        const T* b = e + z.o1;
                        const T pa = ly.w0 * (wx0 * a[ly.o0 + x0] + wx1 * a[ly.o0 + x1]) +
                                     ly.w1 * (wx0 * a[ly.o1 + x0] + wx1 * a[ly.o1 + x1]);
                        const T pb = ly.w0 * (wx0 * b[ly.o0 + x0] + wx1 * b[ly.o0 + x1]) +
                                     ly.w1 * (wx0 * b[ly.o1 + x0] + wx1 * b[ly.o1 + x1]);
                        v = z.w0 * pa + z.w1 * pb;
                    } else {
                        const int Kc = (z0 + kl) >> 1;
                        if (Kc >= C.nz) continue;
                        const int pz = C.gp * (Kc + 1), oy = C.gx * (J + 1);
                        v = e[par + pz] + (((wx0 * e[x0 + oy + pz] + wx1 * e[x1 + oy + pz]) +
                                            (ly.w0 * e[I + 1 + ly.o0 + pz] + ly.w1 * e[I + 1 + ly.o1 + pz])) +
                                           (z.w0 * e[par + z.o0] + z.w1 * e[par + z.o1]));
                    }
                    const int g = g0 + q + F.gp * (kl + 1);
                    v += u[g];
                    u[g] = v;
                    cl_push<T>(pd, g, kl, nl, v);
                }
        }
    cl_end(P, s);
}

// u = A^{-1} f on the coarsest level (FP64 sums): thread (row r, part) sums
// every parts-th column, the rows' parts are added through shared memory
template <class T>
__device__ __forceinline__ void cl_coarse_solve(const ClPlan<T>& P, const ClMem<T>& M, const double* __restrict__ ainv)
{
    const int s = P.nl - 1;
    const ClLev<T>& C = P.lev[s];
    const int n = C.nx * C.ny * C.nz;
    const T* f = M.S + C.fo;
    T* u = M.S + C.uo;
    double* sh = reinterpret_cast<double*>(reinterpret_cast<unsigned char*>(M.S) + P.part_off);
    const int parts = min(max(CL_TPB / n, 1), n);
    const int part = (int)threadIdx.x / n, r = (int)threadIdx.x - part * n;
    __syncthreads();
    if (part < parts) {
        double acc = 0.0;
#pragma unroll 4
        for (int q = part; q < n; q += parts) acc += __ldg(&ainv[q * n + r]) * (double)f[q];
        sh[part * n + r] = acc;
    }
    __syncthreads();
    if (part == 0) {
        double acc = 0.0;
        for (int q = 0; q < parts; q++) acc += sh[q * n + r];
        const int row = (int)C.dnx.div((unsigned)r), i = r - row * C.nx;
        const int k = (int)C.dny.div((unsigned)row), j = row - k * C.ny;
        const int g = (i + 1) + C.gx * (j + 1) + C.gp * (k + 1);
        u[g] = (T)acc;
        cl_push<T>(cl_pushes(P, M, s, 0, C.nz), g, k, C.nz, (T)acc);
    }
}

// the V-cycle from lev[0] (right-hand side fin; from zero, or from the state in
// uout) down to the coarsest and back; the result is written to uout
template <class T, bool RF>
__global__ void __launch_bounds__(CL_TPB, 1) k_cluster(const __grid_constant__ ClPlan<T> P, CSplit<T> fin,
                                                             Split<T> uout, const unsigned char* __restrict__ tab,
                                                             const double* __restrict__ ainv)
{
    extern __shared__ __align__(16) unsigned char cl_smem[];
    ClMem<T> M;
    M.S = reinterpret_cast<T*>(cl_smem);
    ClAx<T>* axt = reinterpret_cast<ClAx<T>*>(cl_smem + P.ax_off);
    ClLin<T>* lint = reinterpret_cast<ClLin<T>*>(cl_smem + P.lin_off);
    M.ax = axt;
    M.lin = lint;
    M.rank = P.nc > 1 ? (int)cl_rank() : 0;
    const unsigned base = (unsigned)__cvta_generic_to_shared(cl_smem);
    M.rlo = M.rank > 0 ? M.rank - 1 : P.nc - 1;
    M.rhi = M.rank < P.nc - 1 ? M.rank + 1 : 0;
    M.lo = cl_map(base, (unsigned)M.rlo);
    M.hi = cl_map(base, (unsigned)M.rhi);
    M.zero = cl_map(base, 0);
    M.self = cl_map(base, (unsigned)M.rank);
    // constant tables and cleared fields before the predecessor's results are needed
    {
        uint4* z = reinterpret_cast<uint4*>(cl_smem);
        for (int e = threadIdx.x; e < P.zero_vecs; e += CL_TPB) z[e] = make_uint4(0u, 0u, 0u, 0u);
        const ClAx<T>* ga = reinterpret_cast<const ClAx<T>*>(tab);
        const ClLin<T>* gl = reinterpret_cast<const ClLin<T>*>(tab + (P.lin_off - P.ax_off));
        for (int e = threadIdx.x; e < P.nax; e += CL_TPB) {
            ClAx<T> x = ga[e];
            x.cm *= P.kc;
            x.cp *= P.kc;
            axt[e] = x;
        }
        for (int e = threadIdx.x; e < P.nlin; e += CL_TPB) lint[e] = gl[e];
    }
    pdl_wait();
    const ClLev<T>& T0 = P.lev[0];
    int z0, nl;
    cl_span(P, M.rank, 0, z0, nl);
    __syncthreads();
    // the top level's columns: both colours of local planes k0 .. k1-1 (ghost planes -1 and nl)
    auto columns = [&](int k0, int k1, auto&& cell) {
        const int p0 = T0.pg > 1 ? (int)T0.dcol.div(threadIdx.x) : 0;
        if (p0 >= T0.pg) return;
        for (int cc = (int)threadIdx.x - p0 * T0.ncol; cc < T0.ncol; cc += CL_TPB) {
            const int j = (int)T0.dnh.div((unsigned)cc), h = cc - j * T0.nh;
            const bool has1 = 2 * h + 1 < T0.nx;
#pragma unroll 4
            for (int kl = k0 + p0; kl < k1; kl += T0.pg) {
                int k = z0 + kl;
                if (k < 0 || k >= T0.nz) {
                    if (!(T0.per & 4)) continue;
                    k = k < 0 ? T0.nz - 1 : 0;
                }
                // split offset, ghosted and natural index of the even cell; its colour
                const int q = (j + k) & 1, o = h + T0.P * (j + T0.ny * k);
                cell(q, has1, o, 2 * h + 1 + T0.gx * (j + 1) + T0.gp * (kl + 1), 2 * h + T0.nx * (j + T0.ny * kl));
            }
        }
    };
    T* ut = M.S + T0.uo;
    T* ft = M.S + T0.fo;
    columns(0, nl, [&](int q, bool has1, int o, int, int n) {
        ft[n] = __ldg(fin.half(q) + o);
        if (has1) ft[n + 1] = __ldg(fin.half(q ^ 1) + o);
    });
    if (P.load_u)
        columns(-1, nl + 1, [&](int q, bool has1, int o, int g, int) {
            ut[g] = uout.half(q)[o];
            if (has1) ut[g + 1] = uout.half(q ^ 1)[o];
        });
    __syncthreads();
    if (P.m > 0) cl_arrive();  // every block's fields are cleared before a neighbour stores into them
    // down (s = 0 .. nl-2), coarsest solve, up (s = nl-2 .. 0), as one loop: one
    // copy of each phase's code (the instruction cache starts cold)
    for (int t = 0; t < 2 * (P.nl - 1); t++) {
        const bool down = t < P.nl - 1;
        const int s = down ? t : 2 * (P.nl - 1) - 1 - t;
        if (t == P.nl - 1 && M.rank == 0) cl_coarse_solve(P, M, ainv);
        if (!down && s == P.m - 1) {  // back on the split levels: the first block is done
            __syncthreads();
            cl_arrive();
        }
        if (s >= P.m && M.rank != 0) continue;
        if (!down) cl_prolong(P, M, s);
        cl_smooth<T, RF>(P, M, s, down);
        if (!down) continue;
        if (s != P.m - 1) {
            cl_restrict<T, RF>(P, M, s);
            if (s < P.m) cl_arrive();  // (the next level's first phase waits)
        } else {
            cl_restrict_push<T, RF>(P, M, s);
            cl_wait();
            if (M.rank == 0) cl_restrict_sum(P, M, s);
        }
    }
    if (P.m > 0 && P.nu2 == 0) cl_wait();
    __syncthreads();
    columns(0, nl, [&](int q, bool has1, int o, int g, int) {
        uout.half(q)[o] = ut[g];
        if (has1) uout.half(q ^ 1)[o] = ut[g + 1];
    });
}

// explicit rows of the levels of k_cluster, all levels in one launch: eight
// words per cell (diagonal, its reciprocal, the six off-diagonal weights), of a
// cell coefficient (row_eval's: arithmetic face mean times the face coefficient,
// Dirichlet faces on the diagonal) or copied from row arrays
template <class T, class Op>
struct CRowsPlan {
    int n;
    unsigned blk0[CL_MAXL + 1];
    Lev L[CL_MAXL];
    Op op[CL_MAXL];
    T* rows[CL_MAXL];
};
template <class T, class Op>
__global__ void __launch_bounds__(TPB) k_crows(const __grid_constant__ CRowsPlan<T, Op> P)
{
    pdl_wait();
    int l = 0;
    while (l + 1 < P.n && blockIdx.x >= P.blk0[l + 1]) l++;
    const Lev& L = P.L[l];
    const Op& op = P.op[l];
    // both colours' halves one after the other
    const unsigned t = (blockIdx.x - P.blk0[l]) * TPB + threadIdx.x;
    const int cc = t >= (unsigned)L.half;
    const unsigned o = t - (cc ? (unsigned)L.half : 0u);
    int i, j, k;
    if (o >= (unsigned)L.half || !decode(L, o, cc, i, j, k)) return;
    T a[8];
    if constexpr (std::is_same<Op, ROp<T>>::value) {
        a[0] = __ldg(&sel(op.r[0], cc)[o]);
#pragma unroll
        for (int f = 0; f < 6; f++) a[2 + f] = __ldg(&sel(op.r[1 + f], cc)[o]);
    } else {
        const T kc = kval(op, L, i, j, k);
        T d = op.dex[0] ? __ldg(&sel(op.dex, cc)[o]) : op.dexc;
#pragma unroll
        for (int f = 0; f < 6; f++) {
            const int ax = f >> 1, s = (f & 1) ? 1 : -1;
            const int p = ax == 0 ? i : (ax == 1 ? j : k);
            int x = i, y = j, z = k;
            T w = T(0);
            if (nbr(L, ax, s, x, y, z)) {
                const int q = ax == 0 ? x : (ax == 1 ? y : z);
                w = T(0.5) * (kc + kval(op, L, x, y, z)) * (T)fcoef(L, ax, p, q);
                d += w;
            } else if (L.bc[f] == BC_DIRC) {
                d += kc * (T)dcoef(L, ax, p);
            }
            a[2 + f] = -w;
        }
        a[0] = d;
    }
    a[1] = T(1) / a[0];
    T* r = P.rows[l] + 8 * ((size_t)cc * L.half + o);
    constexpr int W = 32 / (int)sizeof(T);
#pragma unroll
    for (int q = 0; q < 8; q += W) {
        VecW<T, W> v;
#pragma unroll
        for (int e = 0; e < W; e++) v.v[e] = a[q + e];
        stv<T, W>(r + q, v);
    }
}

}  // namespace mps
