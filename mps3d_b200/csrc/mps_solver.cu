// mps_solver.cu -- host driver and C ABI of the B200 multigrid / Krylov
// solver.  One handle = one CUDA stream + a device workspace reused across
// calls with the same grid signature.
//
// Solve structure (correction scheme; equivalent to the reference's FAS
// V-cycle, mgridlib/mgridsteps.f90:384-579, because the operator is linear):
//   V(l): nu1 red-black GS sweeps; f_{l+1} = R(f_l - A_l u_l) (fused);
//         u_{l+1} = 0; V(l+1); u_l += P u_{l+1}; nu2 sweeps.
//   coarsest: u = A^{-1} f with a precomputed dense inverse.
// Outer loops: FP64 stationary V-cycle iteration; MIXED = FP64 residual +
// FP32 V-cycles + FP64 update (defect correction); FGMRES(m) right
// preconditioned by the V-cycle with FP64 Gram-Schmidt and Givens.
#include <algorithm>
#include <array>
#include <cmath>
#include <cstdint>
#include <memory>
#include <mutex>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <string>
#include <thread>
#include <type_traits>
#include <vector>

#include "../../include/mps_linsolve.h"

#include <cstddef>

// The Fortran module include/mps_linsolve_c.f90 declares bind(C) twins of
// these structs with the same components in the same order; a Fortran
// compiler lays them out by the C rules.  These offsets are what that module
// (and the ctypes mirror in mps3d_b200/capi.py) assume: a change of a struct
// that moves one fails here instead of corrupting a caller's arguments.
static_assert(offsetof(mps_grid, llenx) == 16 && sizeof(mps_grid) == 40, "mps_grid layout");
static_assert(offsetof(mps_solver_opts, tol_kind) == 8 && offsetof(mps_solver_opts, ranks) == 28 &&
                  offsetof(mps_solver_opts, max_coarse) == 40 && offsetof(mps_solver_opts, flux) == 72 &&
                  sizeof(mps_solver_opts) == 80,
              "mps_solver_opts layout");
static_assert(offsetof(mps_solve_info, rel_res) == 16 && offsetof(mps_solve_info, launches) == 48 &&
                  sizeof(mps_solve_info) == 56,
              "mps_solve_info layout");
static_assert(offsetof(mps_profile, ms) == 32 && offsetof(mps_profile, precision_bytes) == 96 &&
                  offsetof(mps_profile, cells) == 104 && sizeof(mps_profile) == 112,
              "mps_profile layout");
static_assert(offsetof(mps_problem, timederiv) == 40 && offsetof(mps_problem, dt) == 48 &&
                  offsetof(mps_problem, vel) == 56 && offsetof(mps_problem, bc_code) == 88 &&
                  offsetof(mps_problem, bcval) == 112 && offsetof(mps_problem, mgridsterm) == 160 &&
                  offsetof(mps_problem, soln) == 168 && sizeof(mps_problem) == 176,
              "mps_problem layout");
#include "mps_kernels.cuh"
#include "mps_tma.cuh"
#include "mps_cluster.cuh"

#include <cudaTypedefs.h>

namespace mps {

constexpr int MAXL = 24;
constexpr int MAX_DENSE = 1024;

static inline unsigned nblk(long long n, int tpb = TPB) { return (unsigned)((n + tpb - 1) / tpb); }

// launch with the programmatic stream-serialization attribute: the kernel may
// be scheduled before its predecessor on the stream finishes, and waits for it
// in its first statement (pdl_wait); inside a captured graph this becomes a
// programmatic edge, which shortens the gap between dependent launches
template <class... KArgs, class... Args>
static cudaError_t pdl_launch(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t s,
                              Args&&... args)
{
    cudaLaunchConfig_t cfg;
    std::memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kern, std::forward<Args>(args)...);
}


// a kernel attribute (the shared-memory limit) set once per device: the call
// costs host time, and attributes belong to each device's context
template <class F>
static bool once_per_device(int dev, signed char* state, F&& set)
{
    static std::mutex m;
    std::lock_guard<std::mutex> lock(m);
    if (dev < 0 || dev >= 64) return set();
    if (state[dev] == 0) state[dev] = set() ? 1 : -1;
    return state[dev] == 1;
}

struct Err {
    int code = 0;
    std::string msg;
};

#define CK(call)                                                                                   \
    do {                                                                                           \
        cudaError_t e_ = (call);                                                                   \
        if (e_ != cudaSuccess) {                                                                   \
            ctx.err.code = MPS_ERR_CUDA;                                                           \
            ctx.err.msg = std::string(#call) + ": " + cudaGetErrorString(e_);                     \
            return MPS_ERR_CUDA;                                                                   \
        }                                                                                          \
    } while (0)
#define CKL()                                                                                      \
    do {                                                                                           \
        ctx.launches++;                                                                            \
        cudaError_t e_ = cudaGetLastError();                                                       \
        if (e_ != cudaSuccess) {                                                                   \
            ctx.err.code = MPS_ERR_CUDA;                                                           \
            ctx.err.msg = std::string("launch at ") + __FILE__ + ":" + std::to_string(__LINE__) +   \
                          ": " + cudaGetErrorString(e_);                                           \
            return MPS_ERR_CUDA;                                                                   \
        }                                                                                          \
    } while (0)

struct Arena {
    std::vector<void*> blocks;
    size_t bytes = 0;
    size_t limit = 0;  // 0: no cap; else get() fails once the arena would exceed it
    void* get(size_t n)
    {
        void* p = nullptr;
        if (n == 0) n = 16;
        if (limit && bytes + n > limit) return nullptr;
        if (cudaMalloc(&p, n) != cudaSuccess) return nullptr;
        if (cudaMemset(p, 0, n) != cudaSuccess) { cudaFree(p); return nullptr; }
        blocks.push_back(p);
        bytes += n;
        return p;
    }
    void clear()
    {
        for (void* p : blocks) cudaFree(p);
        blocks.clear();
        bytes = 0;
    }
};

template <class T>
struct Hier {
    T* U[MAXL][2] = {};  // two full split buffers (2*half) per level
    T* F[MAXL] = {};     // right-hand side (split)
    T* R[MAXL] = {};     // residual scratch (split)
    T* D[MAXL] = {};     // diagonal of the red rows (levels 1 .. nlev-2; the red pass written by the restriction)
    int ri[MAXL] = {}, bi[MAXL] = {};
    KOp<T> kop[MAXL];
    ROp<T> rop[MAXL];
    double* AinvT = nullptr;
    int cl_l0 = -1;                   // first level of the cluster's V-cycle (k_cluster), -1: none
    unsigned char* cltab = nullptr;   // its axis and interpolation tables
    std::vector<unsigned char> climg; // the host copy of the tables on the device (cl_tables)
    double cl_len[3] = {0, 0, 0};     // the box that they hold
    T* crow[MAXL] = {};               // explicit rows on its levels, eight words a cell (k_crows)
    double* Dprev = nullptr;  // the coarsest matrix whose inverse AinvT holds
    int* gj = nullptr;        // its inversion state (k_gauss_jordan)
};

struct Signature {
    int dims[3] = {0, 0, 0};
    int bc[6] = {0, 0, 0, 0, 0, 0};
    int hier = -1, ranks[3] = {0, 0, 0}, max_coarse = 0, opclass = -1, prec = -1, krylov = -1, restart = 0;
    int has_reac = -1, kuni = -1, transpose = -1;
    bool operator==(const Signature& o) const { return std::memcmp(this, &o, sizeof(Signature)) == 0; }
};

struct Prof {
    bool on = false;
    int level = 0;  // the level whose smoothing/transfer launches are timed
    std::vector<cudaEvent_t> ev;
    std::vector<int> cls;
    int used = 0;
    int count[MPS_PROF_NCLASS] = {};
    double ms[MPS_PROF_NCLASS] = {};
    int precision_bytes = 8, coeff_field = 0;
    long long cells = 0;
};

// a captured iteration, replayed with cudaGraphLaunch; keyed by everything
// that is baked into its kernel parameters
struct GraphKey {
    Signature sig;
    int kind = -1, prec = -1, inner = 0, nu1 = 0, nu2 = 0, nlev = 0, flux = 0, transpose = 0, prof = 0, relaxed = 0, extra_q = 0, kseg = 0;
    double kc = 0, dexc = 0;
    double len[3] = {0, 0, 0};  // the box: the levels' face coefficients
    const void* ws = nullptr;  // workspace identity (first arena block)
    bool operator==(const GraphKey& o) const
    {
        return sig == o.sig && std::equal(len, len + 3, o.len) && relaxed == o.relaxed && extra_q == o.extra_q && kseg == o.kseg && kind == o.kind && prec == o.prec && inner == o.inner && nu1 == o.nu1 &&
               nu2 == o.nu2 && nlev == o.nlev && flux == o.flux && transpose == o.transpose && prof == o.prof &&
               kc == o.kc &&
               dexc == o.dexc && ws == o.ws;
    }
};
struct GraphEntry {
    GraphKey key;
    cudaGraphExec_t exec = nullptr;
    int kernels = 0;
    std::vector<cudaEvent_t> ev;  // profiling event-record nodes (pairs)
    std::vector<int> cls;
};

struct BatchState;

struct Ctx {
    int dev = 0;
    int nsm = 148;  // streaming multiprocessors of the device
    BatchState* batch = nullptr;  // batched solves (mps_linsolve_batched_dev)
    long long launches = 0;
    Prof prof;
    std::vector<GraphEntry> graphs;
    GraphEntry* capturing = nullptr;
    cudaStream_t s = nullptr;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    Err err;
    Arena ar;       // grid-dependent workspace (both precisions)
    Arena kar;      // Krylov basis (FGMRES), keyed by (length, restart)
    long long kar_n = 0;
    int kar_m = 0;
    int kar_dims[3] = {0, 0, 0};  // the cells whose pads its vectors hold zero
    Arena inbuf;    // host-API staging of the inputs
    struct Lane {   // one host thread of the pageable copies: a stream, two pinned buffers
        cudaStream_t s = nullptr;
        double* pin[2] = {nullptr, nullptr};
        cudaEvent_t ev[2] = {nullptr, nullptr};
    };
    std::vector<Lane> lanes;  // created at the first host call with pageable arrays
    bool tma_ok = false;      // the shared-memory colour pass can run (set at workspace set-up)
    bool tma_allowed = true;  // MPS_TMA=0 at handle creation: the register-fed kernels only (for comparisons)
    bool red0_ready = false;  // the finest level's first red pass from zero was written by the outer residual
    bool redz[MAXL] = {};     // level l's first red pass from zero was written by the restriction into it
    bool sub_allowed = true;  // MPS_SUBCYCLE=0 at handle creation: one launch per pass on every level (for comparisons)
    bool relaxed = false;     // over-relaxed passes and averaged-face coarse coefficients (solve_impl)
    int extra_q = 0;          // the diagonal extra's weight (extra_step), and with it
    double relax[MAXL] = {};  // the part of the over-relaxation that each level takes
    size_t inbuf_bytes = 0;
    Signature sig;
    int nlev = 0;
    double len[3] = {0, 0, 0};  // edge lengths of the box that lev describes
    Lev lev[MAXL];
    Xfer xf[MAXL];
    Lin* dtab = nullptr;      // device prolongation tables of the current plan
    size_t dtab_n = 0;
    std::vector<Lin> htab;
    // FP64 coefficient pyramid (split cell fields)
    double* pk[MAXL] = {};
    double* pka[MAXL] = {};   // arithmetic means of the finest coefficient (levels >= 1; k_restrict_coef)
    double* seg64[MAXL] = {};  // rows of one coefficient on the large levels (k_kseg)
    float* seg32[MAXL] = {};
    double* preac[MAXL] = {};
    double* pv[3][MAXL] = {};
    double* dex64[MAXL] = {};
    float* k32[MAXL] = {};
    float* dex32[MAXL] = {};
    double* rows64[MAXL] = {};
    float* rows32[MAXL] = {};
    double* trows = nullptr;  // forward rows of one level, while a transposed operator's are built
    Hier<double> h64;
    Hier<float> h32;
    double* x64 = nullptr;  // outer iterate (mixed / fgmres)
    double* b64 = nullptr;
    int kseg = 0;             // this solve's operators carry the rows of one coefficient: 2 most rows are, 1 fewer
    KOp<double> kop64;      // fine-level FP64 operator for outer residuals
    ROp<double> rop64;
    double* dense = nullptr;
    double* gjM = nullptr;
    int* dstatus = nullptr;
    RedBuf rb;
    unsigned long long* dmax = nullptr;
    double* hpin = nullptr;  // pinned host scratch
    // FGMRES
    double* V = nullptr;
    void* Z = nullptr;
    double* w = nullptr;
    double* hcol = nullptr;
    double** Vptr = nullptr;
    double* dpart = nullptr;
    int mdot_blocks = 0;
    double* zero_face = nullptr;
    size_t zero_face_n = 0;
};

}  // namespace mps

struct mps_handle_s {
    mps::Ctx ctx;
};

namespace mps {

// ----------------------------------------------------------------------
static Lev make_lev(int nx, int ny, int nz, const double w[3], const double wl[3], const int bc[6])
{
    Lev L;
    std::memset(&L, 0, sizeof(L));
    L.nx = nx; L.ny = ny; L.nz = nz;
    L.nh = (nx + 1) / 2;
    L.P = ((L.nh + 7) / 8) * 8;
    L.half = (long long)L.P * ny * nz;
    for (int f = 0; f < 6; f++) L.bc[f] = bc[f];
    for (int a = 0; a < 3; a++) L.per[a] = bc[2 * a] == BC_PERI;
    const int n[3] = {nx, ny, nz};
    for (int a = 0; a < 3; a++) {
        const double ww = w[a], wwl = wl[a];
        L.w[a] = ww;
        L.wl[a] = wwl;
        const double dl = 0.5 * (ww + wwl);
        L.cr[a] = 1.0 / (ww * ww);
        L.cl[a] = n[a] == 1 ? 1.0 / (wwl * wwl) : 1.0 / (dl * wwl);
        L.cp[a] = 1.0 / (dl * ww);
        L.dr[a] = 2.0 / (ww * ww);
        L.dlast[a] = 2.0 / (wwl * wwl);
    }
    L.uniform = (w[0] == wl[0] && w[1] == wl[1] && w[2] == wl[2]) ? 1 : 0;
    L.divP.init((unsigned)L.P);
    L.divNy.init((unsigned)ny);
    L.divG.init((unsigned)(L.P / 4));
    L.rows = (unsigned)ny * (unsigned)nz;
    return L;
}

static Lev make_lev_uniform(int nx, int ny, int nz, const double llen[3], const int bc[6])
{
    const double w[3] = {llen[0] / nx, llen[1] / ny, llen[2] / nz};
    return make_lev(nx, ny, nz, w, w, bc);
}

// level sizes and cell widths.  CELL = the reference (l/2 by integer division,
// mgridsteps.f90:21-23; dx = llen/l on every level, find_AX :724-726; coarsest
// when a per-rank size reaches LMIN=1, :512).  GEOM = l/2 with the odd cell of
// an odd size merged into the last coarse cell and exact widths; coarsest when
// a level has at most max_coarse cells.
static int plan_levels(const mps_grid* g, const mps_solver_opts* o, const int bc[6], Lev* lev, Xfer* xf,
                       std::string& why)
{
    int d[3] = {g->lx, g->ly, g->lz};
    const double llen[3] = {g->llenx, g->lleny, g->llenz};
    double w[3], wl[3];
    for (int a = 0; a < 3; a++) w[a] = wl[a] = llen[a] / d[a];
    int n = 0;
    const int* P = o->ranks;
    const bool cell = o->hierarchy == MPS_HIER_CELL;
    if (cell) {
        for (int a = 0; a < 3; a++)
            if (P[a] < 1 || d[a] % P[a] != 0) { why = "CELL hierarchy: size not divisible by ranks"; return -1; }
    }
    for (;;) {
        lev[n] = make_lev(d[0], d[1], d[2], w, wl, bc);
        long long cells = (long long)d[0] * d[1] * d[2];
        bool coarsest;
        if (cell)
            coarsest = d[0] / P[0] <= 1 || d[1] / P[1] <= 1 || d[2] / P[2] <= 1;
        else
            coarsest = cells <= o->max_coarse || (d[0] == 1 && d[1] == 1 && d[2] == 1);
        if (coarsest || n == MAXL - 1) {
            if (!coarsest) { why = "too many levels"; return -1; }
            if (cells > MAX_DENSE) { why = "coarsest level too large for the dense solve"; return -1; }
            return n + 1;
        }
        int c[3];
        double cw[3], cwl[3];
        Xfer X;
        std::memset(&X, 0, sizeof(X));
        X.geom = !cell;
        for (int a = 0; a < 3; a++) {
            if (cell) {
                int l = d[a] / P[a];
                if ((l & 1) && P[a] > 1) { why = "CELL hierarchy: odd per-rank size with several ranks"; return -1; }
                c[a] = P[a] * (l / 2);
                cw[a] = cwl[a] = llen[a] / c[a];
            } else if (d[a] == 1) {
                c[a] = 1;
                cw[a] = cwl[a] = wl[a];
            } else {
                c[a] = d[a] / 2;
                cw[a] = 2.0 * w[a];
                cwl[a] = (d[a] & 1) ? 2.0 * w[a] + wl[a] : w[a] + wl[a];
                if (c[a] == 1) cw[a] = cwl[a];
            }
            X.nf[a] = d[a];
            X.nc[a] = c[a];
            X.rf[a] = wl[a] / w[a];
            X.Rc[a] = cwl[a] / w[a];
            X.per[a] = bc[2 * a] == BC_PERI;
        }
        xf[n] = X;
        for (int a = 0; a < 3; a++) { d[a] = c[a]; w[a] = cw[a]; wl[a] = cwl[a]; }
        n++;
    }
}

template <class T>
static Split<T> cur(Hier<T>& H, const Lev& L, int l)
{
    Split<T> s;
    s.c[0] = H.U[l][H.ri[l]];
    s.c[1] = H.U[l][H.bi[l]] + L.half;
    return s;
}
template <class T>
static CSplit<T> ccur(Hier<T>& H, const Lev& L, int l)
{
    CSplit<T> s;
    s.c[0] = H.U[l][H.ri[l]];
    s.c[1] = H.U[l][H.bi[l]] + L.half;
    return s;
}
template <class T>
static CSplit<T> csplit(const T* base, const Lev& L)
{
    CSplit<T> s;
    s.c[0] = base;
    s.c[1] = base + L.half;
    return s;
}
template <class T>
static Split<T> split(T* base, const Lev& L)
{
    Split<T> s;
    s.c[0] = base;
    s.c[1] = base + L.half;
    return s;
}

// ---- finest-level profiling (events around launches on the handle's stream) ----
static void prof_begin(Ctx& ctx, int cls)
{
    Prof& P = ctx.prof;
    if (!P.on) return;
    if (ctx.capturing) {  // event-record node inside the graph being captured
        GraphEntry& G = *ctx.capturing;
        cudaEvent_t a;
        if (cudaEventCreate(&a) != cudaSuccess) return;
        G.ev.push_back(a);
        G.cls.push_back(cls);
        cudaEventRecordWithFlags(a, ctx.s, cudaEventRecordExternal);
        return;
    }
    if (P.used + 2 > (int)P.ev.size()) {
        for (int q = 0; q < 256; q++) {
            cudaEvent_t e;
            if (cudaEventCreate(&e) != cudaSuccess) return;
            P.ev.push_back(e);
        }
    }
    cudaEventRecord(P.ev[P.used], ctx.s);
    P.cls.push_back(cls);
}
static void prof_end(Ctx& ctx)
{
    Prof& P = ctx.prof;
    if (!P.on) return;
    if (ctx.capturing) {
        GraphEntry& G = *ctx.capturing;
        if (G.ev.size() != 2 * G.cls.size() - 1) return;
        cudaEvent_t b;
        if (cudaEventCreate(&b) != cudaSuccess) return;
        G.ev.push_back(b);
        cudaEventRecordWithFlags(b, ctx.s, cudaEventRecordExternal);
        return;
    }
    if (P.cls.size() * 2 != (size_t)P.used + 2) return;
    cudaEventRecord(P.ev[P.used + 1], ctx.s);
    P.used += 2;
}
// after a synchronize that followed a replay of G: add its event pairs
static void prof_collect_graph(Ctx& ctx, const GraphEntry& G)
{
    Prof& P = ctx.prof;
    if (!P.on) return;
    for (size_t q = 0; q < G.cls.size() && 2 * q + 1 < G.ev.size(); q++) {
        float ms = 0.f;
        if (cudaEventElapsedTime(&ms, G.ev[2 * q], G.ev[2 * q + 1]) == cudaSuccess) {
            P.ms[G.cls[q]] += ms;
            P.count[G.cls[q]]++;
        }
    }
}
static void destroy_graphs(Ctx& ctx)
{
    for (GraphEntry& G : ctx.graphs) {
        if (G.exec) cudaGraphExecDestroy(G.exec);
        for (cudaEvent_t e : G.ev) cudaEventDestroy(e);
    }
    ctx.graphs.clear();
}

static void prof_collect(Ctx& ctx)  // after a stream synchronize
{
    Prof& P = ctx.prof;
    for (size_t q = 0; q < P.cls.size() && (int)(2 * q + 1) < P.used; q++) {
        float ms = 0.f;
        if (cudaEventElapsedTime(&ms, P.ev[2 * q], P.ev[2 * q + 1]) == cudaSuccess) {
            P.ms[P.cls[q]] += ms;
            P.count[P.cls[q]]++;
        }
    }
    P.cls.clear();
    P.used = 0;
}

// Replay the captured graph for `key`, capturing `body` first when needed.
// Graphs hold kernel parameters (buffer pointers, operator constants) by
// value; the red/black buffer parities return to their start after an even
// number of sweeps per level, which the callers guarantee.  Returns the entry.
template <class F>
static int run_graph(Ctx& ctx, const GraphKey& key, GraphEntry** out, F&& body)
{
    GraphEntry* G = nullptr;
    for (GraphEntry& e : ctx.graphs)
        if (e.key == key) { G = &e; break; }
    if (!G) {
        if (ctx.graphs.size() >= 16) destroy_graphs(ctx);
        ctx.graphs.emplace_back();
        G = &ctx.graphs.back();
        G->key = key;
        cudaGraph_t graph = nullptr;
        const long long l0 = ctx.launches;
        if (cudaStreamBeginCapture(ctx.s, cudaStreamCaptureModeThreadLocal) != cudaSuccess) {
            ctx.graphs.pop_back();
            ctx.err.msg = "stream capture failed to start";
            return MPS_ERR_CUDA;
        }
        ctx.capturing = G;
        int st = body();
        ctx.capturing = nullptr;
        cudaError_t ce = cudaStreamEndCapture(ctx.s, &graph);
        if (st || ce != cudaSuccess) {
            if (graph) cudaGraphDestroy(graph);
            for (cudaEvent_t e : G->ev) cudaEventDestroy(e);
            ctx.graphs.pop_back();
            cudaGetLastError();
            if (!st) { ctx.err.msg = std::string("stream capture: ") + cudaGetErrorString(ce); st = MPS_ERR_CUDA; }
            return st;
        }
        G->kernels = (int)(ctx.launches - l0);
        ctx.launches = l0;
        ce = cudaGraphInstantiate(&G->exec, graph, 0);
        cudaGraphDestroy(graph);
        if (ce != cudaSuccess) {
            for (cudaEvent_t e : G->ev) cudaEventDestroy(e);
            ctx.graphs.pop_back();
            ctx.err.msg = std::string("graph instantiate: ") + cudaGetErrorString(ce);
            return MPS_ERR_CUDA;
        }
    }
    if (cudaGraphLaunch(G->exec, ctx.s) != cudaSuccess) {
        ctx.err.msg = "graph launch failed";
        return MPS_ERR_CUDA;
    }
    ctx.launches += G->kernels;
    *out = G;
    return 0;
}

static bool odd_periodic(const Lev& L)
{
    return (L.per[0] && (L.nx & 1)) || (L.per[1] && (L.ny & 1)) || (L.per[2] && (L.nz & 1));
}

// ---- transfer boxes ----
// coarse cells whose 2x2x2 children are regular cells of uniform coefficients
// away from odd periodic seams (false when an axis does not halve)
static bool restrict_box(const Lev& F, const Lev& C, Box& b)
{
    const int nf[3] = {F.nx, F.ny, F.nz}, nc[3] = {C.nx, C.ny, C.nz};
    for (int a = 0; a < 3; a++) {
        if (nf[a] != 2 * nc[a] && nf[a] != 2 * nc[a] + 1) return false;
        const bool seam = F.per[a] && (nf[a] & 1);
        const bool irregular_end = nf[a] != 2 * nc[a] || !F.uniform;  // unequal children
        b.lo[a] = seam ? 1 : 0;
        b.hi[a] = nc[a] - 1 - ((irregular_end || seam) ? 1 : 0);
        if (b.hi[a] < b.lo[a]) return false;
    }
    return true;
}
// fine cells whose bracketing coarse centres are regular cells (geometric hierarchy)
static bool prolong_box(const Lev& F, const Lev& C, const Xfer& X, Box& b)
{
    if (!X.geom) return false;
    const int nf[3] = {F.nx, F.ny, F.nz}, nc[3] = {C.nx, C.ny, C.nz};
    for (int a = 0; a < 3; a++) {
        if (nf[a] != 2 * nc[a] && nf[a] != 2 * nc[a] + 1) return false;
        const int creg = nc[a] - ((nf[a] != 2 * nc[a] || !F.uniform) ? 1 : 0);
        b.lo[a] = 1;
        b.hi[a] = 2 * creg - 3;
        // along y and z the regular rows go in pairs (2J+1, 2J+2) between
        // coarse rows J and J+1: an odd count leaves its last row to the shell
        if (a > 0 && ((b.hi[a] - b.lo[a] + 1) & 1)) b.hi[a]--;
        if (b.hi[a] < b.lo[a]) return false;
    }
    return true;
}
static long long box_cells(const Box& b)
{
    return (long long)(b.hi[0] - b.lo[0] + 1) * (b.hi[1] - b.lo[1] + 1) * (b.hi[2] - b.lo[2] + 1);
}

// the launch description of the prolongation bulk (k_prolong_v) of fine
// level L with box pb and W cells per thread: the regular rows in 2 x 2
// blocks, their x ends, the rows outside the box, and the red cells of odd
// periodic seams; pp.blk0[4] blocks in all
static void prolong_form(const Lev& L, const Box& pb, int W, ProlongDiv& dv, Box& sb, ProlongDiv& sv,
                         ProlongParts& pp)
{
    const long long G = (L.nh + W - 1) / W;  // groups holding a cell (the rest of the P / W are pads)
    const long long rall = (long long)L.ny * L.nz;
    const long long rin = (long long)(pb.hi[1] - pb.lo[1] + 1) * (pb.hi[2] - pb.lo[2] + 1);
    dv.g.init((unsigned)G);
    dv.yin.init((unsigned)(pb.hi[1] - pb.lo[1] + 1));
    dv.yin2.init((unsigned)(pb.hi[1] - pb.lo[1] + 1) / 2);
    dv.nh.init((unsigned)((L.nx + 1) / 2));
    // groups with every cell in the box for both row parities: 2Wg >= lo,
    // 2W(g+1) - 1 <= hi
    dv.g_lo = (pb.lo[0] + 2 * W - 1) / (2 * W);
    dv.g_hi = (pb.hi[0] + 1) / (2 * W) - 1;
    const long long gin = dv.g_hi >= dv.g_lo ? dv.g_hi - dv.g_lo + 1 : 0;
    if (gin == 0) { dv.g_lo = 0; dv.g_hi = -1; }
    dv.gin.init((unsigned)std::max<long long>(gin, 1));
    dv.gout.init((unsigned)std::max<long long>(G - gin, 1));
    // red cells on odd periodic seams (read by the next red pass)
    const int sy = L.per[1] && (L.ny & 1), sz = L.per[2] && (L.nz & 1), sx = L.per[0] && (L.nx & 1);
    sb.lo[0] = 0;
    sb.hi[0] = L.nx - 1;
    sb.lo[1] = sy;
    sb.hi[1] = L.ny - 1 - sy;
    sb.lo[2] = sz;
    sb.hi[2] = L.nz - 1 - sz;
    const long long rin2 = (long long)(sb.hi[1] - sb.lo[1] + 1) * (sb.hi[2] - sb.lo[2] + 1);
    sv = dv;
    sv.yin.init((unsigned)(sb.hi[1] - sb.lo[1] + 1));
    pp.cnt[0] = (unsigned)(rin / 4 * gin);  // 2 x 2 row blocks
    pp.cnt[1] = (unsigned)(rin * (G - gin));
    pp.cnt[2] = (unsigned)((rall - rin) * G);
    pp.cnt[3] = odd_periodic(L) ? (unsigned)((rall - rin2) * ((L.nx + 1) / 2) + (sx ? 2 * rin2 : 0)) : 0u;
    pp.blk0[0] = 0;
    for (int q = 0; q < 4; q++) pp.blk0[q + 1] = pp.blk0[q] + nblk(pp.cnt[q]);
}

// colour passes and the outer residual: interior groups (no boundary code)
// and the shell as two parts of a launch (measured at 257^3: FP32 colour
// pass 54.6 against 58.3 us, FP64 91 against 126 us, outer residual 156
// against 201 us)
#ifndef MPS_COLOUR_SPLIT
#define MPS_COLOUR_SPLIT 1
#endif
#ifndef MPS_RESID_SPLIT
#define MPS_RESID_SPLIT 1
#endif

// the interior / shell decomposition of a level's groups of W cells
// (k_colourv_split, k_residv_split); false when the level has no interior
static bool make_split(const Lev& L, int W, ColourSplit& cs)
{
    // the interior: cells 1 .. n-2 along each axis; on a level with merged
    // last cells 1 .. n-3, whose faces all have the regular coefficients
    const int m = L.uniform ? 2 : 3;
    if (L.ny < m + 1 || L.nz < m + 1) return false;
    cs.g_lo = 1;
    cs.g_hi = (L.nx - m + 1) / (2 * W) - 1;
    if (cs.g_hi < cs.g_lo) return false;
    const unsigned G = (unsigned)((L.nh + W - 1) / W);
    const unsigned gin = (unsigned)(cs.g_hi - cs.g_lo + 1);
    const unsigned rin = (unsigned)(L.ny - m) * (unsigned)(L.nz - m);
    cs.gin.init(gin);
    cs.yin.init((unsigned)(L.ny - m));
    cs.gx.init(std::max(G - gin, 1u));
    cs.g.init(G);
    cs.n_in = rin * gin;
    cs.n_xe = rin * (G - gin);
    cs.n_face = ((unsigned)L.ny * (unsigned)L.nz - rin) * G;
    cs.nb_in = nblk(cs.n_in);
    cs.nb_xe = nblk(cs.n_xe);
    cs.nb_face = nblk(cs.n_face);
    cs.b.lo[0] = 0;
    cs.b.hi[0] = L.nx - 1;
    cs.b.lo[1] = 1;
    cs.b.hi[1] = L.ny - m;
    cs.b.lo[2] = 1;
    cs.b.hi[2] = L.nz - m;
    return true;
}

// the restriction bulk's interior coarse rows and groups (every fine cell
// evaluated has its neighbours inside the grid and regular faces: fine cells
// 1 .. n-2, or 1 .. n-3 on a level with merged last cells) and the rest; an
// empty interior leaves everything to the rest part
static RestrictSplit make_restrict_split(const Lev& F, const Lev& C, const Box& bx, int W)
{
    RestrictSplit rs;
    std::memset(&rs, 0, sizeof(rs));
    const int m = F.uniform ? 2 : 3;
    const int G = F.P / W;
    rs.J0 = std::max(bx.lo[1], 1);
    rs.K0 = std::max(bx.lo[2], 1);
    const int J1 = std::min(bx.hi[1], (F.ny - m - 1) / 2), K1 = std::min(bx.hi[2], (F.nz - m - 1) / 2);
    rs.ga = 1;
    rs.gb = ((F.nx - m - 1) / 2 - W + 1) / W;
    int nJ = J1 - rs.J0 + 1, nK = K1 - rs.K0 + 1, ng = rs.gb - rs.ga + 1;
    if (nJ < 1 || nK < 1 || ng < 1) {  // no interior: the rectangle is empty
        nJ = nK = 0;
        ng = 0;
        rs.ga = 0;
        rs.gb = -1;
    }
    rs.gin.init((unsigned)std::max(ng, 1));
    rs.yin.init((unsigned)std::max(nJ, 1));
    rs.gx.init((unsigned)std::max(G - ng, 1));
    rs.g.init((unsigned)G);
    rs.n_in = (unsigned)nJ * (unsigned)nK * (unsigned)ng;
    rs.n_xe = (unsigned)nJ * (unsigned)nK * (unsigned)(G - ng);
    rs.n_out = ((unsigned)C.ny * (unsigned)C.nz - (unsigned)nJ * (unsigned)nK) * (unsigned)G;
    rs.nb_in = nblk(rs.n_in);
    rs.nb_xe = nblk(rs.n_xe);
    rs.nb_out = nblk(rs.n_out);
    rs.rect.lo[0] = 0;
    rs.rect.hi[0] = C.nx - 1;
    rs.rect.lo[1] = rs.J0;
    rs.rect.hi[1] = rs.J0 + nJ - 1;
    rs.rect.lo[2] = rs.K0;
    rs.rect.hi[2] = rs.K0 + nK - 1;
    return rs;
}

// ---- the finest colour pass through shared memory (k_colour_tma) ----
#ifndef MPS_TMA_COLOUR
#define MPS_TMA_COLOUR 1
#endif
#ifndef MPS_TMA_LEVELS
#define MPS_TMA_LEVELS 1  // the finest level only
#endif
// tile rows and blocks per SM of the FP32 pass.  With a staged coefficient
// (257^3 mixed plasma solve, ms): 6 rows at 3 blocks per SM 12.72-12.75, 8 rows
// at 2 blocks 12.79-12.81, 5 rows at 4 blocks 13.40, 7 rows at 3 blocks 13.78.
// Without one (uniform, or uniform in most rows; 257^3 Poisson / plasma,
// ms): 6 rows at 3, 4, 5 blocks - / 10.73, 5.39 / 10.37, - / 10.56; 7 rows at 4
// blocks 5.48 / 10.86, 8 rows at 4 blocks 5.13 / 10.40
template <bool KF>
struct TmaShape {  // rows per block, one warp each; blocks per SM the tiling aims at; cells per thread
    static constexpr int TJ = KF ? 6 : 8;
    static constexpr int BPS = KF ? 3 : 4;
    static constexpr int W = 4;
};
// planes of a tile's chunk at least: one of fewer spends its time filling the
// slots, and the register-fed pass is faster (129^3 mixed plasma / Poisson
// solve, 5 planes: 3.27 / 1.69 ms against 3.47 / 1.78; 193^3 Poisson, 8 planes:
// 3.24 against 3.10)
constexpr int TMA_PLANES = 8;

static PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder()
{
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    static bool tried = false;
    if (!tried) {
        tried = true;
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess && p)
            fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
        else
            cudaGetLastError();
    }
    return fn;
}

// 3-D map of one colour half (P x ny x nz elements) with boxes of `rows`
// full rows of one plane
static bool encode_half(CUtensorMap* m, const float* base, const Lev& L, int rows)
{
    auto fn = tensor_map_encoder();
    if (!fn) return false;
    const cuuint64_t dims[3] = {(cuuint64_t)L.P, (cuuint64_t)L.ny, (cuuint64_t)L.nz};
    const cuuint64_t strides[2] = {(cuuint64_t)L.P * sizeof(float), (cuuint64_t)L.P * L.ny * sizeof(float)};
    const cuuint32_t box[3] = {(cuuint32_t)L.P, (cuuint32_t)rows, 1};
    const cuuint32_t es[3] = {1, 1, 1};
    return fn(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<float*>(base), dims, strides, box, es,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// the finest level's FP32 colour pass from a valid state with k_colour_tma (the
// FP64 pass measured slower through shared memory, 104-117 against 87 us at 257^3,
// the FP32 pass faster, 49.6 against 51.2 us, both with a staged coefficient);
// returns 1 when the pass was launched, 0 when this level or operator does
// not qualify (the caller runs the register-fed pass), < 0 on an error
template <bool KF>
static int colour_pass_tma_kf(Ctx& ctx, Hier<float>& H, const KOp<float>& op, int l, int c, float* out,
                              const float* fh, float om)
{
    constexpr int TJ = TmaShape<KF>::TJ, W = TmaShape<KF>::W;
    const Lev& L = ctx.lev[l];
    if (!ctx.tma_ok || L.P > 256 || op.dex[0] || L.ny < 3 || L.nz < 3) return 0;
    ColourSplit cs;
    if (!make_split(L, W, cs)) return 0;
    const int oc = c ^ 1;
    const float* uo = oc == 0 ? H.U[l][H.ri[l]] : H.U[l][H.bi[l]] + L.half;
    CUtensorMap mU, mKo, mKc, mF;
    std::memset(&mKo, 0, sizeof(mKo));
    std::memset(&mKc, 0, sizeof(mKc));
    if (!encode_half(&mU, uo, L, TJ + 2) || !encode_half(&mF, fh, L, TJ)) return 0;
    if (KF && (!encode_half(&mKo, op.k[oc], L, TJ + 2) || !encode_half(&mKc, op.k[c], L, TJ))) return 0;
    TmaColour tc;
    std::memset(&tc, 0, sizeof(tc));
    auto pad128 = [](unsigned elems) { return (unsigned)((elems * sizeof(float) + 127) / 128 * 128 / sizeof(float)); };
    tc.tile_elems = pad128((unsigned)L.P * (TJ + 2));
    tc.own_elems = pad128((unsigned)L.P * TJ);
    tc.slot_bytes = (unsigned)(L.P * sizeof(float)) * ((TJ + 2) + TJ) * (KF ? 2 : 1);
    const size_t smem = tma_smem_bytes<float, KF>(tc);
    if (smem > 220 * 1024) return 0;
    // tiles for the blocks that fit on an SM (shared memory, threads, at most
    // TmaShape::BPS): each tile streams its planes plus two halo planes, so
    // more tiles re-read more
    const int bps = std::max(1, std::min({(int)(227 * 1024 / (smem + 1024)), 2048 / (TJ * 32), TmaShape<KF>::BPS}));
    // the interior box of the split: rows 1 .. jhi, planes 1 .. khi (one cell
    // short of merged last cells); the shell blocks take every other row
    tc.jhi = cs.b.hi[1];
    tc.khi = cs.b.hi[2];
    if (cs.b.lo[1] != 1 || cs.b.lo[2] != 1 || tc.jhi < 1 || tc.khi < 1) return 0;
    tc.njb = (tc.jhi + TJ - 1) / TJ;
    const int want = std::max(1, ctx.nsm * bps / tc.njb);
    tc.tk = std::max(1, (tc.khi + want - 1) / want);
    if (tc.tk < TMA_PLANES) return 0;
    tc.nkb = (tc.khi + tc.tk - 1) / tc.tk;
    tc.ntile = tc.njb * tc.nkb;
    tc.g_lo = cs.g_lo;
    tc.g_hi = cs.g_hi;
    tc.n_xe = cs.n_xe;
    tc.n_face = cs.n_face;
    const unsigned nsh = tc.n_xe + tc.n_face;
    tc.nb_shell = std::min<unsigned>((nsh + TJ * 32 - 1) / (TJ * 32), (unsigned)ctx.nsm * 4);
    tc.flag = ctx.rb.out + 3;
    auto launch = [&](auto kern) -> int {
        const cudaError_t e = pdl_launch(kern, tc.ntile + tc.nb_shell, TJ * 32, smem, ctx.s, L, op, c, ccur(H, L, l),
                                         out, fh, cs, tc, om, mU, mKo, mKc, mF);
        if (e != cudaSuccess) {
            ctx.err.code = MPS_ERR_CUDA;
            ctx.err.msg = std::string("k_colour_tma launch: ") + cudaGetErrorString(e);
            return -1;
        }
        return 1;
    };
    if (L.uniform) return launch(k_colour_tma<float, W, TJ, KF, true>);
    return launch(k_colour_tma<float, W, TJ, KF, false>);
}
static int colour_pass_tma(Ctx& ctx, Hier<float>& H, const KOp<float>& op, int l, int c, float* out, const float* fh,
                           float om)
{
    // (a coefficient that is one along most rows is not staged)
    if (op.k[0] && ctx.kseg != 2) return colour_pass_tma_kf<true>(ctx, H, op, l, c, out, fh, om);
    return colour_pass_tma_kf<false>(ctx, H, op, l, c, out, fh, om);
}

// the attributes the shared-memory colour pass needs, set outside any stream
// capture (at workspace set-up); false when the device or driver cannot run it
static bool tma_prepare(int dev)
{
    static signed char state[64] = {};
    if (!MPS_TMA_COLOUR || !tensor_map_encoder()) return false;
    return once_per_device(dev, state, [] {
        const int bytes = 220 * 1024;
        auto set = [&](auto kern) {
            return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) == cudaSuccess;
        };
        constexpr int W = TmaShape<true>::W, JK = TmaShape<true>::TJ, JU = TmaShape<false>::TJ;
        bool ok = set(k_colour_tma<float, W, JK, true, true>) && set(k_colour_tma<float, W, JU, false, true>) &&
                  set(k_colour_tma<float, W, JK, true, false>) && set(k_colour_tma<float, W, JU, false, false>);
        if (!ok) cudaGetLastError();
        return ok;
    });
}

// the explicit-row colour pass in two parts (k_colourv_split_rop); cells
// per thread measured on the 129^3 SG step (finest pass FP32 / FP64, live
// events): one cell 17.7 / 24.7 us, 2 / 1 cells 17.3 / 24.9, 2 / 2 cells
// 17.2 / 25.4, 4 / 2 cells 21.3 / 25.5, against 20.9 / 28.8 us for k_colour
// (one cell per thread, boundary code everywhere); the solve times move
// by less than their noise (2.13-2.19 / 1.46-1.51 ms)
#ifndef MPS_ROP_SPLIT
#define MPS_ROP_SPLIT 1
#endif
#ifndef MPS_ROP_W32
#define MPS_ROP_W32 1
#endif
#ifndef MPS_ROP_W64
#define MPS_ROP_W64 1
#endif

// ---- the relaxation of a V-cycle's colour passes ----
// Over-relaxed red-black passes smooth better than plain ones in three
// dimensions, and reading a cell's own old value costs nothing where the state
// is zero (the first sweep of a coarse level, of the finest level in the first
// inner V-cycle of a mixed solve) or stays in cache (coarse levels).  So: 1.6
// in the first pre-smoothing sweep of every level, 1.4 in the other passes of
// the coarse levels, plain where the transfers count on it.  V-cycles to 1e-11
// in an FP64 CPU model, plain -> this schedule with k_restrict_coef: 65^3 Dirichlet
// 10.4 -> 8.0, 100x83x61 15.4 -> 10.5, 129^3 plasma slab 15.4 -> 12.6, odd
// periodic along all axes 15.2 -> 11.5; also 1.4 in the finest level's other
// passes saves another 5% of the cycles on large grids and costs a read of
// the colour's half in each.
constexpr double OMEGA_FIRST = 1.6;   // the first pre-smoothing sweep
constexpr double OMEGA_LATER = 1.4;   // the other passes of the levels below the finest
// Where the diagonal extra (1/dt, a sink) outweighs the faces, a plain pass is nearly
// exact and an over-relaxed one overshoots.  So a level relaxes by 1 + (w - 1) / (1 + r)^2,
// r its smallest diagonal extra over its face sum (which falls by four from level to
// level), and plainly where less than RELAX_LEAST is left.  V-cycles to 1e-11 in an FP64
// CPU model, 32^3, extra over the finest face sum 0.1 / 0.3 / 1 / 3 / 10 / 100, plain ->
// relaxed alike on every level -> this: V(2,2) 7 / 5 / 4 / 3 / 2 / 1 -> 7 / 6 / 5 / 3 / 2 / 2 ->
// 6 / 5 / 3 / 2 / 2 / 1, V(1,1) 12 / 9 / 7 / 5 / 4 / 2 -> 9 / 9 / 8 / 8 / 6 / 4 ->
// 8 / 7 / 6 / 4 / 3 / 2.  Of the powers of 1 / (1 + r), 2 is the lowest that took no more cycles
// than plain passes anywhere (1.5 to 4, V(1,1) to V(3,3), three boxes, r to 1000)
constexpr double RELAX_LEAST = 0.02;
// the smallest diagonal extra of a cell, from the detection's words
static double diag_extra_min(double dtinv, double maxreac, unsigned long long top)
{
    if (!(maxreac > 0.0) || !top) return dtinv;
    const long long b = ordered_bits(top);
    double r;
    std::memcpy(&r, &b, sizeof(r));
    return dtinv - r;
}
// the diagonal extra over the finest face sum in half powers of two: what the
// relaxation depends on, and a captured launch sequence with it, must not change with
// every digit of a reaction field.  EXTRA_NONE: none that a level would feel
constexpr int EXTRA_NONE = -1000;
static double face_sum(const Lev& L)
{
    double s = 0.0;
    for (int a = 0; a < 3; a++) s += lev_n(L, a) > 1 ? 2.0 * L.cr[a] : 0.0;
    return s;
}
static int extra_step(const Lev& L0, double extra, double maxk)
{
    if (!(extra > 1e-6 * maxk * face_sum(L0))) return EXTRA_NONE;
    return (int)std::lround(2.0 * std::log2(std::min(extra / std::max(maxk * face_sum(L0), 1e-300), 1e6)));
}
// Ctx::relax of every level; without a level that relaxes, Ctx::relaxed goes
static void set_relaxation(Ctx& ctx)
{
    const double r0 = ctx.extra_q == EXTRA_NONE ? 0.0 : std::exp2(0.5 * ctx.extra_q), f0 = face_sum(ctx.lev[0]);
    for (int l = 0; l < ctx.nlev; l++) {
        const double f = face_sum(ctx.lev[l]), r = f > 0.0 ? r0 * f0 / f : r0;
        ctx.relax[l] = 1.0 / ((1.0 + r) * (1.0 + r));
    }
    ctx.relaxed = ctx.relaxed && (OMEGA_FIRST - 1.0) * ctx.relax[0] >= RELAX_LEAST;
}
// pre: pre-smoothing, sw: sweep, c: colour
static double pass_omega(const Ctx& ctx, int l, const mps_solver_opts* o, bool pre, int sw, int c)
{
    if (!ctx.relaxed) return 1.0;
    if (pre && c == 1 && sw == o->nu1 - 1) return 1.0;  // the restriction counts on a vanishing black residual
    double w = OMEGA_LATER;
    if (pre && sw == 0) w = OMEGA_FIRST;
    else if (l == 0 || (!pre && sw == 0 && c == 0)) return 1.0;  // the prolongation corrects the black cells only
    const double excess = (w - 1.0) * ctx.relax[l];
    return excess < RELAX_LEAST ? 1.0 : 1.0 + excess;
}

// ---- one colour pass ----
// zero_state 2: the whole state is zero, 1: colour c is, 0: neither; om: the
// pass's relaxation
template <class T, class Op>
static int colour_pass(Ctx& ctx, Hier<T>& H, const Op& op, int l, int c, int zero_state, double omega)
{
    const T om = (T)omega;
    const Lev& L = ctx.lev[l];
    const unsigned nb = nblk((long long)L.P * L.rows);
    T* out;
    const T* fh = H.F[l] + (c ? L.half : 0);
    if (c == 0) out = H.U[l][H.ri[l] ^ 1];
    else out = H.U[l][H.bi[l] ^ 1] + L.half;
    if (l == ctx.prof.level) prof_begin(ctx, MPS_PROF_SMOOTH);
    if constexpr (std::is_same<Op, KOp<T>>::value) {
        if (zero_state == 2 && c == 0 && H.D[l]) {  // from zero: f / diag, elementwise
            pdl_launch(k_red_from_zero<T>, nb, TPB, 0, ctx.s, L, (const T*)fh, (const T*)H.D[l], out);
            if (l == ctx.prof.level) prof_end(ctx);
            CKL();
            H.ri[l] ^= 1;
            return 0;
        }
    }
    if constexpr (std::is_same<Op, KOp<float>>::value) {
        if (l <= MPS_TMA_LEVELS - 1 && zero_state == 0) {
            const int r = colour_pass_tma(ctx, H, op, l, c, out, fh, om);
            if (r < 0) return MPS_ERR_CUDA;
            if (r == 1) {
                if (l == ctx.prof.level) prof_end(ctx);
                CKL();
                if (c == 0) H.ri[l] ^= 1;
                else H.bi[l] ^= 1;
                return 0;
            }
        }
    }
    if constexpr (std::is_same<Op, KOp<T>>::value) {
        if (L.uniform || L.nx >= 16) {
            // vector kernel, W cells per thread (faces at a merged last cell
            // take their own coefficients inside the row evaluation); the
            // levels below the finest have their own shape
            auto launch = [&](auto wc, auto mbc) {
                constexpr int W = decltype(wc)::value, MB = decltype(mbc)::value;
                ColourSplit cs;
                if (MPS_COLOUR_SPLIT && make_split(L, W, cs)) {
                    // interior groups without boundary code, the shell apart
                    const unsigned nbt = cs.nb_in + cs.nb_xe + cs.nb_face;
                    auto go = [&](auto uc) {
                        constexpr bool UNI = decltype(uc)::value;
                        if (zero_state == 2) {
                            pdl_launch(k_colourv_split<T, W, ZeroU<T>, MB, UNI>, nbt, TPB, 0, ctx.s, L, op, c, ZeroU<T>(),
                                       out, fh, cs, om);
                        } else if (zero_state == 1) {
                            OtherOnlyU<T> u;
                            u.c = c;
                            u.other = c == 0 ? H.U[l][H.bi[l]] + L.half : H.U[l][H.ri[l]];
                            pdl_launch(k_colourv_split<T, W, OtherOnlyU<T>, MB, UNI>, nbt, TPB, 0, ctx.s, L, op, c, u, out,
                                       fh, cs, om);
                        } else {
                            pdl_launch(k_colourv_split<T, W, CSplit<T>, MB, UNI>, nbt, TPB, 0, ctx.s, L, op, c,
                                       ccur(H, L, l), out, fh, cs, om);
                        }
                    };
                    if (L.uniform) go(std::true_type());
                    else go(std::false_type());
                    return;
                }
                FastDiv dg;
                dg.init((unsigned)(L.P / W));
                const unsigned nbv = nblk((long long)(L.P / W) * L.rows);
                if (zero_state == 2) {
                    pdl_launch(k_colourv<T, W, ZeroU<T>, MB>, nbv, TPB, 0, ctx.s, L, op, c, ZeroU<T>(), out, fh, dg, om);
                } else if (zero_state == 1) {
                    OtherOnlyU<T> u;
                    u.c = c;
                    u.other = c == 0 ? H.U[l][H.bi[l]] + L.half : H.U[l][H.ri[l]];
                    pdl_launch(k_colourv<T, W, OtherOnlyU<T>, MB>, nbv, TPB, 0, ctx.s, L, op, c, u, out, fh, dg, om);
                } else {
                    pdl_launch(k_colourv<T, W, CSplit<T>, MB>, nbv, TPB, 0, ctx.s, L, op, c, ccur(H, L, l), out, fh,
                               dg, om);
                }
            };
            if (l == 0)
                launch(std::integral_constant<int, ColourShape<T>::W>(), std::integral_constant<int, ColourShape<T>::MINB>());
            else if (l == 1)
                launch(std::integral_constant<int, CoarseShape<T>::W>(), std::integral_constant<int, CoarseShape<T>::MINB>());
            else
                launch(std::integral_constant<int, SmallShape<T>::W>(), std::integral_constant<int, SmallShape<T>::MINB>());
            if (l == ctx.prof.level) prof_end(ctx);
            CKL();
            if (c == 0) H.ri[l] ^= 1;
            else H.bi[l] ^= 1;
            return 0;
        }
    }
    if constexpr (std::is_same<Op, ROp<T>>::value) {
        // explicit rows: interior groups W cells per thread, the shell cell by cell
        constexpr int W = sizeof(T) == 4 ? MPS_ROP_W32 : MPS_ROP_W64;
        ColourSplit cs;
        if (MPS_ROP_SPLIT && L.nx >= 16 && make_split(L, W, cs)) {
            const unsigned nbt = cs.nb_in + cs.nb_xe + cs.nb_face;
            if (zero_state == 2) {
                pdl_launch(k_colourv_split_rop<T, W, ZeroU<T>>, nbt, TPB, 0, ctx.s, L, op, c, ZeroU<T>(), out, fh, cs);
            } else if (zero_state == 1) {
                OtherOnlyU<T> u;
                u.c = c;
                u.other = c == 0 ? H.U[l][H.bi[l]] + L.half : H.U[l][H.ri[l]];
                pdl_launch(k_colourv_split_rop<T, W, OtherOnlyU<T>>, nbt, TPB, 0, ctx.s, L, op, c, u, out, fh, cs);
            } else {
                pdl_launch(k_colourv_split_rop<T, W, CSplit<T>>, nbt, TPB, 0, ctx.s, L, op, c, ccur(H, L, l), out, fh,
                           cs);
            }
            if (l == ctx.prof.level) prof_end(ctx);
            CKL();
            if (c == 0) H.ri[l] ^= 1;
            else H.bi[l] ^= 1;
            return 0;
        }
    }
    if (zero_state == 2) {  // whole state zero
        pdl_launch(k_colour<T, Op, ZeroU<T>>, nb, TPB, 0, ctx.s, L, op, c, ZeroU<T>(), out, fh, om);
    } else if (zero_state == 1) {  // colour c zero, other colour valid
        OtherOnlyU<T> u;
        u.c = c;
        u.other = c == 0 ? H.U[l][H.bi[l]] + L.half : H.U[l][H.ri[l]];
        pdl_launch(k_colour<T, Op, OtherOnlyU<T>>, nb, TPB, 0, ctx.s, L, op, c, u, out, fh, om);
    } else {
        pdl_launch(k_colour<T, Op, CSplit<T>>, nb, TPB, 0, ctx.s, L, op, c, ccur(H, L, l), out, fh, om);
    }
    if (l == ctx.prof.level) prof_end(ctx);
    CKL();
    if (c == 0) H.ri[l] ^= 1;
    else H.bi[l] ^= 1;
    return 0;
}

template <class T>
static int coarse_solve(Ctx& ctx, Hier<T>& H, int l)
{
    const Lev& L = ctx.lev[l];
    const int n = L.nx * L.ny * L.nz;
    pdl_launch(k_coarse_solve<T>, 1, 512, n * sizeof(double), ctx.s, L, H.AinvT, csplit<T>(H.F[l], L), cur(H, L, l));
    CKL();
    return 0;
}

// ---- the small levels in one cluster (k_cluster) ----
// the kernel's attributes, set outside any stream capture (at workspace
// set-up); false when the device cannot hold a cluster of 16 blocks
static bool cl_prepare(int dev)
{
    static signed char state[64] = {};
    return once_per_device(dev, state, [] {
        auto set = [](const void* kern) {
            if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, CL_SMEM_MAX) != cudaSuccess ||
                cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess)
                return false;
            cudaLaunchConfig_t cfg;
            std::memset(&cfg, 0, sizeof(cfg));
            cfg.gridDim = dim3(CL_MAXC);
            cfg.blockDim = dim3(CL_TPB);
            cfg.dynamicSmemBytes = CL_SMEM_MAX;
            cudaLaunchAttribute at[1];
            at[0].id = cudaLaunchAttributeClusterDimension;
            at[0].val.clusterDim.x = CL_MAXC;
            at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
            cfg.attrs = at;
            cfg.numAttrs = 1;
            int n = 0;
            return cudaOccupancyMaxActiveClusters(&n, kern, &cfg) == cudaSuccess && n >= 1;
        };
        const bool ok = set((const void*)k_cluster<float, false>) &&
                        set((const void*)k_cluster<float, true>) &&
                        set((const void*)k_cluster<double, false>) &&
                        set((const void*)k_cluster<double, true>);
        if (!ok) cudaGetLastError();
        return ok;
    });
}

// the axis entries of one level in the ghosted layout of row pitch gx: the
// face coefficients of fcoef / dcoef by position
template <class T>
static void cl_axes(const Lev& L, int gx, std::vector<ClAx<T>>& out)
{
    const int n3[3] = {L.nx, L.ny, L.nz};
    const int st3[3] = {1, gx, gx * (L.ny + 2)};
    for (int a = 0; a < 3; a++) {
        const int n = n3[a], st = st3[a];
        const bool per = L.per[a] != 0, wrap = per && a < 2;  // along z the ghost planes hold the wrapped cells
        const bool dm = !per && L.bc[2 * a] == BC_DIRC, dp = !per && L.bc[2 * a + 1] == BC_DIRC;
        for (int p = 0; p < n; p++) {
            ClAx<T> x;
            x.om = -st;
            x.op = st;
            if (p > 0) x.cm = (T)(p == n - 1 ? L.cl[a] : L.cr[a]);
            else if (per) x.cm = (T)(n == 1 ? L.cl[a] : L.cp[a]);
            else x.cm = dm ? (T)(n == 1 ? L.dlast[a] : L.dr[a]) : T(0);
            if (p < n - 1) x.cp = (T)(p + 1 == n - 1 ? L.cp[a] : L.cr[a]);
            else if (per) x.cp = (T)L.cl[a];
            else x.cp = dp ? (T)L.dlast[a] : T(0);
            if (wrap && p == 0) x.om = (n - 1) * st;
            if (wrap && p == n - 1) x.op = -(n - 1) * st;
            out.push_back(x);
        }
    }
}

// the launch plan from level l0: split levels and their planes, shared-memory
// layout, tables (ax, lin); false when it does not fit
template <class T>
static bool cl_layout(const Ctx& ctx, int l0, ClPlan<T>& P, size_t& smem, std::vector<ClAx<T>>& ax,
                      std::vector<ClLin<T>>& lin)
{
    std::memset(&P, 0, sizeof(P));
    ax.clear();
    lin.clear();
    const int nl = ctx.nlev - l0;
    if (nl < 2 || nl > CL_MAXL) return false;
    P.nl = nl;
    P.geom = ctx.xf[l0].geom;
    auto cells = [&](int s) { const Lev& L = ctx.lev[l0 + s]; return (long long)L.nx * L.ny * L.nz; };
    P.m = 0;
    while (P.m < nl - 1 && cells(P.m) > CL_GATHER) P.m++;
    P.nc = 1;
    if (P.m > 0) {
        // the planes of the coarsest split level over the blocks; a finer plane
        // belongs to the block of its parent
        const int nzb = ctx.lev[l0 + P.m - 1].nz;
        P.nc = std::min(CL_MAXC, nzb);
        for (int s = P.m - 1; s >= 0; s--) {
            ClLev<T>& G = P.lev[s];
            const int nz = ctx.lev[l0 + s].nz;
            for (int r = 0; r < P.nc; r++) {
                if (s == P.m - 1) G.z[r] = (int)((long long)r * nz / P.nc);
                else G.z[r] = (nz == ctx.lev[l0 + s + 1].nz ? 1 : 2) * P.lev[s + 1].z[r];
            }
            G.z[P.nc] = nz;
        }
    }
    long long off = 0;
    for (int s = 0; s < nl; s++) {
        const Lev& L = ctx.lev[l0 + s];
        ClLev<T>& G = P.lev[s];
        G.nx = L.nx; G.ny = L.ny; G.nz = L.nz; G.nh = L.nh;
        G.P = L.P;
        G.gx = L.nx + 2;
        G.gp = G.gx * (L.ny + 2);
        int held = L.nz;  // planes of the largest share
        if (s < P.m) {
            held = 0;
            for (int r = 0; r < P.nc; r++) held = std::max(held, G.z[r + 1] - G.z[r]);
        }
        if (s == 0) P.share = L.nh * L.ny * held;
        G.uo = (int)off;
        off += (long long)G.gp * (held + 2);
        G.fo = (int)off;
        off += (long long)L.nx * L.ny * held;
        if (off * (long long)sizeof(T) > CL_SMEM_MAX) return false;
        G.ax0 = (int)ax.size();
        cl_axes<T>(L, G.gx, ax);
        for (int a = 0; a < 3; a++) {
            G.per |= L.per[a] ? 1 << a : 0;
            G.w[a] = (T)L.w[a];
            G.wl[a] = (T)L.wl[a];
        }
        G.ncol = L.nh * L.ny;
        G.pg = std::max(1, std::min(held, CL_TPB / G.ncol));
        G.dcol.init((unsigned)G.ncol);
        G.dnh.init((unsigned)L.nh);
        G.dny.init((unsigned)L.ny);
        G.dnx.init((unsigned)L.nx);
        if (s < nl - 1) {
            const Xfer& X = ctx.xf[l0 + s];
            const int nf[3] = {L.nx, L.ny, L.nz};
            for (int a = 0; a < 3; a++) {
                G.lin0[a] = (int)lin.size();
                const Lev& C = ctx.lev[l0 + s + 1];
                const int nc = lev_n(C, a), st = a == 0 ? 1 : (a == 1 ? C.nx + 2 : (C.nx + 2) * (C.ny + 2));
                // coarse index x (possibly -1 or nc) -> offset and the sign of its weight
                auto at = [&](int x, int& o) {
                    T sgn = T(1);
                    if (x < 0 || x >= nc) {
                        if (C.per[a]) {
                            if (a < 2) x = x < 0 ? nc - 1 : 0;  // along z: the ghost plane
                        } else {
                            if (C.bc[2 * a + (x < 0 ? 0 : 1)] == BC_DIRC) sgn = T(-1);
                            x = x < 0 ? 0 : nc - 1;
                        }
                    }
                    o = st * (x + 1);
                    return sgn;
                };
                for (int i = 0; i < nf[a]; i++) {
                    ClLin<T> e;
                    if (P.geom) {
                        Lin b;
                        geom_lin(X, a, i, b.j0, b.j1, b.t);
                        e.w0 = at(b.j0, e.o0) * (T)(1.0 - b.t);
                        e.w1 = at(b.j1, e.o1) * (T)b.t;
                    } else if (i / 2 < nc) {
                        const T w = (i & 1) ? T(0.125) : T(-0.125);
                        e.w0 = at(i / 2 + 1, e.o0) * w;
                        e.w1 = -at(i / 2 - 1, e.o1) * w;
                    } else {  // odd last cell: not read
                        e.o0 = e.o1 = st;
                        e.w0 = e.w1 = T(0);
                    }
                    lin.push_back(e);
                }
            }
            // lanes per coarse cell: up to 4 (the rows of a cell's children) while the cells leave threads idle
            const Lev& C = ctx.lev[l0 + s + 1];
            const long long nc = (long long)C.nx * C.ny * ((held + 1) / 2);
            G.rlog = nc * 4 <= CL_TPB ? 2 : (nc * 2 <= CL_TPB ? 1 : 0);
        }
    }
    size_t bytes = ((size_t)off * sizeof(T) + 15) & ~(size_t)15;
    P.zero_vecs = (int)(bytes / 16);
    P.stage_off = (int)bytes;
    if (P.m > 0) {
        const Lev& F = ctx.lev[l0 + P.m - 1];
        const Lev& C = ctx.lev[l0 + P.m];
        bytes += ((size_t)C.nx * C.ny * F.nz * sizeof(T) + 15) & ~(size_t)15;
    }
    const long long n = cells(nl - 1);
    P.part_off = (int)bytes;
    bytes += sizeof(double) * (size_t)std::max<long long>(CL_TPB, n);
    P.ax_off = (int)bytes;
    P.nax = (int)ax.size();
    bytes += (ax.size() * sizeof(ClAx<T>) + 15) & ~(size_t)15;
    P.lin_off = (int)bytes;
    P.nlin = (int)lin.size();
    bytes += (lin.size() * sizeof(ClLin<T>) + 15) & ~(size_t)15;
    smem = bytes;
    return n <= CL_TPB && bytes <= (size_t)CL_SMEM_MAX;
}

// the cluster's part of a hierarchy: the first level whose V-cycle fits, room
// for its tables, and the row arrays of its explicit rows;
// cl_l0 -1: none (odd periodic sizes: cells of one colour touch, and in-place
// passes would read new values)
template <class T>
static bool cl_setup(Ctx& ctx, Hier<T>& H, const Signature& sig, bool lean)
{
    H.cl_l0 = -1;
    H.cltab = nullptr;
    H.cl_len[0] = H.cl_len[1] = H.cl_len[2] = 0.0;
    for (int l = 0; l < MAXL; l++) H.crow[l] = nullptr;
    if (lean || !ctx.sub_allowed || !cl_prepare(ctx.dev)) return true;
    std::unique_ptr<ClPlan<T>> P(new ClPlan<T>);
    std::vector<ClAx<T>> ax;
    std::vector<ClLin<T>> lin;
    size_t smem = 0;
    const bool rows = sig.opclass == 1 || !sig.kuni || sig.has_reac;  // explicit rows
    int odd = -1;  // the deepest level with an odd periodic size
    for (int l = 0; l < ctx.nlev; l++)
        if (odd_periodic(ctx.lev[l])) odd = l;
    for (int l = odd + 1; l < ctx.nlev - 1; l++) {
        if (!cl_layout<T>(ctx, l, *P, smem, ax, lin) ||
            P->share > cl_max_share<T>(rows, sig.opclass == 1, l > 0, P->nc))
            continue;
        H.cl_l0 = l;
        break;
    }
    if (H.cl_l0 < 0) return true;
    H.cltab = (unsigned char*)ctx.ar.get(smem - (size_t)P->ax_off);
    if (!H.cltab) return false;
    if (rows)
        for (int l = H.cl_l0; l < ctx.nlev - 1; l++) {
            H.crow[l] = (T*)ctx.ar.get(sizeof(T) * 8 * 2 * ctx.lev[l].half);
            if (!H.crow[l]) return false;
        }
    return true;
}

// the cluster's tables for the present box, in stream order.  They hold the face
// coefficients, which scale with the box, and the workspace outlives it: the
// tables on the device are kept while the box stays the same
template <class T>
static int cl_tables(Ctx& ctx, Hier<T>& H)
{
    if (H.cl_l0 < 0 || std::equal(ctx.len, ctx.len + 3, H.cl_len)) return 0;
    std::unique_ptr<ClPlan<T>> P(new ClPlan<T>);
    std::vector<ClAx<T>> ax;
    std::vector<ClLin<T>> lin;
    size_t smem = 0;
    if (!cl_layout<T>(ctx, H.cl_l0, *P, smem, ax, lin)) {
        ctx.err.msg = "cluster plan";
        return MPS_ERR_CUDA;
    }
    H.climg.assign(smem - (size_t)P->ax_off, 0);
    std::memcpy(H.climg.data(), ax.data(), ax.size() * sizeof(ClAx<T>));
    if (!lin.empty())
        std::memcpy(H.climg.data() + (P->lin_off - P->ax_off), lin.data(), lin.size() * sizeof(ClLin<T>));
    CK(cudaMemcpyAsync(H.cltab, H.climg.data(), H.climg.size(), cudaMemcpyHostToDevice, ctx.s));
    std::copy(ctx.len, ctx.len + 3, H.cl_len);
    return 0;
}

// the explicit rows of the cluster's levels (once per solve)
template <class T, class Op>
static int cl_rows(Ctx& ctx, Hier<T>& H, const Op* ops)
{
    if (H.cl_l0 < 0 || !H.crow[H.cl_l0]) return 0;
    std::unique_ptr<CRowsPlan<T, Op>> pp(new CRowsPlan<T, Op>);
    CRowsPlan<T, Op>& P = *pp;
    std::memset((void*)&P, 0, sizeof(P));
    for (int l = H.cl_l0; l < ctx.nlev - 1; l++) {
        const Lev& L = ctx.lev[l];
        P.L[P.n] = L;
        P.op[P.n] = ops[l];
        P.rows[P.n] = H.crow[l];
        P.blk0[P.n + 1] = P.blk0[P.n] + nblk(2 * L.half);
        P.n++;
    }
    pdl_launch(k_crows<T, Op>, P.blk0[P.n], TPB, 0, ctx.s, P);
    CKL();
    return 0;
}

static double pass_omega(const Ctx& ctx, int l, const mps_solver_opts* o, bool pre, int sw, int c);

// the V-cycle from level H.cl_l0 to the coarsest and back in one launch
template <class T, class Op>
static int cluster_cycle(Ctx& ctx, Hier<T>& H, const Op* ops, const mps_solver_opts* o, bool zero_guess)
{
    const int l0 = H.cl_l0;
    std::unique_ptr<ClPlan<T>> pp(new ClPlan<T>);  // the kernel parameter (copied at launch)
    ClPlan<T>& P = *pp;
    std::vector<ClAx<T>> ax;
    std::vector<ClLin<T>> lin;
    size_t smem = 0;
    const bool rows = H.crow[l0] != nullptr;
    if (!cl_layout<T>(ctx, l0, P, smem, ax, lin)) {
        ctx.err.msg = "cluster plan";
        return MPS_ERR_CUDA;
    }
    P.nu1 = o->nu1;
    P.nu2 = o->nu2;
    P.only_black = o->nu2 >= 1;
    P.load_u = !zero_guess;
    for (int s = 0; s < P.nl; s++) {
        const int l = l0 + s;
        P.lev[s].om0 = (T)pass_omega(ctx, l, o, true, 0, 0);
        P.lev[s].om1 = (T)pass_omega(ctx, l, o, false, 0, 1);
        P.lev[s].half = ctx.lev[l].half;
        P.lev[s].rows = H.crow[l];
    }
    if constexpr (std::is_same<Op, KOp<T>>::value) {
        P.kc = ops[l0].kc;
        P.dexc = ops[l0].dexc;
    }
    CSplit<T> fin = csplit<T>(H.F[l0], ctx.lev[l0]);
    Split<T> uout = cur(H, ctx.lev[l0], l0);
    const unsigned char* tab = H.cltab;
    const double* ainv = H.AinvT;
    void* args[] = {(void*)&P, (void*)&fin, (void*)&uout, (void*)&tab, (void*)&ainv};
    const void* kern = rows ? (const void*)k_cluster<T, true> : (const void*)k_cluster<T, false>;
    cudaLaunchConfig_t cfg;
    std::memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3((unsigned)P.nc);
    cfg.blockDim = dim3(CL_TPB);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = ctx.s;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim.x = (unsigned)P.nc;
    at[1].val.clusterDim.y = at[1].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 2;
    cudaLaunchKernelExC(&cfg, kern, args);
    CKL();
    return 0;
}

template <class T, class Op>
static int vcycle_rec(Ctx& ctx, Hier<T>& H, const Op* ops, int l, const mps_solver_opts* o, bool zero_guess)
{
    if (l == ctx.nlev - 1) return coarse_solve(ctx, H, l);
    if (l == H.cl_l0) return cluster_cycle(ctx, H, ops, o, zero_guess);
    const Lev& L = ctx.lev[l];
    const Lev& C = ctx.lev[l + 1];
    int st;
    auto om = [&](bool pre, int sw, int c) { return pass_omega(ctx, l, o, pre, sw, c); };
    for (int s = 0; s < o->nu1; s++) {
        bool z = zero_guess && s == 0;
        if (z && ((l == 0 && ctx.red0_ready) || ctx.redz[l])) {
            // the red pass from zero (red = om f / diag) came with the outer
            // residual (finest level) or with the restriction (coarse levels)
            H.ri[l] ^= 1;
            ctx.redz[l] = false;
        } else if ((st = colour_pass(ctx, H, ops[l], l, 0, z ? 2 : 0, om(true, s, 0)))) {
            return st;
        }
        if ((st = colour_pass(ctx, H, ops[l], l, 1, z ? 1 : 0, om(true, s, 1)))) return st;
    }
    if (o->nu1 == 0 && zero_guess) {
        // no pre-smoothing from a zero guess: materialise the zero state
        CK(cudaMemsetAsync(H.U[l][H.ri[l]], 0, sizeof(T) * L.half, ctx.s));
        CK(cudaMemsetAsync(H.U[l][H.bi[l]] + L.half, 0, sizeof(T) * L.half, ctx.s));
    }
    if (l == ctx.prof.level) prof_begin(ctx, MPS_PROF_RESTRICT);
    // the coarse level's first red pass from zero comes with its right-hand
    // side (cell-coefficient operators; not for the coarsest level, a level
    // the cluster takes, or from the finest level, whose
    // restriction has no registers to spare: the launches below pass rz only
    // to the forms that write it and then set the level's flag)
    RedZ<T> rz{nullptr, nullptr};
    if constexpr (std::is_same<Op, KOp<T>>::value) {
        if (l >= 1 && o->nu1 >= 1 && l + 1 < ctx.nlev - 1 && H.D[l + 1] && l + 1 != H.cl_l0) {
            rz.u = H.U[l + 1][H.ri[l + 1] ^ 1];
            rz.d = H.D[l + 1];
        }
    }
    bool done = false;
    {
        Box bx;
        if (o->nu1 >= 1 && L.nx >= 16 && restrict_box(L, C, bx)) {
            // red residual of the bulk's children restricted in registers, the
            // shell with the general body
            auto launch = [&](auto wc, auto mbc) {
                constexpr int W = decltype(wc)::value, MB = decltype(mbc)::value;
                const RestrictSplit rs = make_restrict_split(L, C, bx, W);
                const long long shell = (long long)C.nx * C.ny * C.nz - box_cells(bx);
                const unsigned nbb = rs.nb_in + rs.nb_xe + rs.nb_out;
                const unsigned nbs = shell > 0 ? nblk(8 * shell) : 0;
                const RedZ<T> rzw = W <= 2 ? rz : RedZ<T>{nullptr, nullptr};
                if (rzw.u) ctx.redz[l + 1] = true;
                if (L.uniform)
                    pdl_launch(k_resid_restrict_v<T, W, MB, true, Op>, nbb + nbs, TPB, 0, ctx.s, L, ops[l],
                               ccur(H, L, l), H.F[l], C, split<T>(H.F[l + 1], C), rs, bx, nbb, ctx.xf[l].geom,
                               (unsigned)shell, rzw);
                else
                    pdl_launch(k_resid_restrict_v<T, W, MB, false, Op>, nbb + nbs, TPB, 0, ctx.s, L, ops[l],
                               ccur(H, L, l), H.F[l], C, split<T>(H.F[l + 1], C), rs, bx, nbb, ctx.xf[l].geom,
                               (unsigned)shell, rzw);
            };
            if constexpr (!std::is_same<Op, KOp<T>>::value)  // explicit rows: one coarse cell per thread
                launch(std::integral_constant<int, 1>(), std::integral_constant<int, RestrictShape<T>::MINB>());
            else if (l == 0)
                launch(std::integral_constant<int, RestrictShape<T>::W>(), std::integral_constant<int, RestrictShape<T>::MINB>());
            else if (l == 1)
                launch(std::integral_constant<int, CoarseXferShape<T>::W>(), std::integral_constant<int, CoarseXferShape<T>::MINB>());
            else
                launch(std::integral_constant<int, SmallXferShape<T>::W>(), std::integral_constant<int, SmallXferShape<T>::MINB>());
            CKL();
            done = true;
        }
    }
    if (!done) {
        if (rz.u) ctx.redz[l + 1] = true;
        pdl_launch(k_resid_restrict<T, Op>, nblk((long long)C.nx * C.ny * C.nz), TPB, 0, ctx.s, 
            L, ops[l], ccur(H, L, l), csplit<T>(H.F[l], L), C, split<T>(H.F[l + 1], C), ctx.xf[l].geom, rz);
        CKL();
    }
    if (l == ctx.prof.level) prof_end(ctx);
    if ((st = vcycle_rec(ctx, H, ops, l + 1, o, true))) return st;
    if (l == ctx.prof.level) prof_begin(ctx, MPS_PROF_PROLONG);
    // the first post-smoothing pass overwrites the red cells from the black
    // ones, so only black cells need the correction (unless an odd periodic
    // seam makes red cells read red neighbours)
    Box pb{};
    auto prolong_bulk = [&](auto wc) {
        constexpr int W = decltype(wc)::value;
        ProlongDiv dv, sv;
        Box sb;
        ProlongParts pp;
        prolong_form(L, pb, W, dv, sb, sv, pp);
        pdl_launch(k_prolong_v<T, W>, pp.blk0[4], TPB, 0, ctx.s, L, cur(H, L, l), C, ccur(H, C, l + 1), ctx.xf[l],
                   pb, dv, sb, sv, pp);
    };
    if (o->nu2 >= 1 && L.nx >= 16 && prolong_box(L, C, ctx.xf[l], pb)) {
        if (l == 0) prolong_bulk(std::integral_constant<int, ProlongShape<T>::W>());
        else if (l == 1) prolong_bulk(std::integral_constant<int, CoarseXferShape<T>::W>());
        else prolong_bulk(std::integral_constant<int, SmallXferShape<T>::W>());
        CKL();
    } else if (o->nu2 >= 1) {
        pdl_launch(k_prolong_correct<T>, nblk((long long)L.P * L.rows), TPB, 0, ctx.s, L, cur(H, L, l), C,
                                                                               ccur(H, C, l + 1), ctx.xf[l], 1);
        CKL();
        if (odd_periodic(L)) {
            pdl_launch(k_prolong_correct<T>, nblk((long long)L.P * L.rows), TPB, 0, ctx.s, L, cur(H, L, l), C,
                                                                                   ccur(H, C, l + 1), ctx.xf[l], 2);
            CKL();
        }
    } else {
        pdl_launch(k_prolong_correct<T>, nblk((long long)L.nx * L.ny * L.nz), TPB, 0, ctx.s, 
            L, cur(H, L, l), C, ccur(H, C, l + 1), ctx.xf[l], -1);
        CKL();
    }
    if (l == ctx.prof.level) prof_end(ctx);
    for (int s = 0; s < o->nu2; s++) {
        if ((st = colour_pass(ctx, H, ops[l], l, 0, 0, om(false, s, 0)))) return st;
        if ((st = colour_pass(ctx, H, ops[l], l, 1, 0, om(false, s, 1)))) return st;
    }
    return 0;
}

template <class T>
static int vcycle(Ctx& ctx, Hier<T>& H, int opclass, const mps_solver_opts* o, bool zero_guess)
{
    for (int l = 0; l < MAXL; l++) ctx.redz[l] = false;  // set and consumed within one V-cycle
    if (opclass == 0) return vcycle_rec(ctx, H, H.kop, 0, o, zero_guess);
    return vcycle_rec(ctx, H, H.rop, 0, o, zero_guess);
}

// r = f - A u, sums (r.r, f.f) -> ctx.rb.out; optional r written to rout (type R);
// ured (optional): the red half that a V-cycle's first red pass from a zero
// state on rout would write (om r / diag); *ured_done tells whether it was
// written (the split kernel only)
template <class T, class Op, class R>
static int resid_norm(Ctx& ctx, const Op& op, CSplit<T> u, CSplit<T> f, Split<R> rout, R* ured = nullptr,
                      bool* ured_done = nullptr, double om = 1.0)
{
    if (ured_done) *ured_done = false;
    const Lev& L = ctx.lev[0];
    prof_begin(ctx, MPS_PROF_RESID);
    if constexpr (std::is_same<Op, KOp<T>>::value) {
        if (L.uniform) {  // vector kernel, one launch per colour, norms accumulated
            constexpr int W = ResidShape<T>::W;
            FastDiv dg;
            dg.init((unsigned)(L.P / W));
            // grid-stride over one wave of resident blocks: no partial last
            // wave, and few partials for the norm reduction (measured at 257^3:
            // 193 us against 220 us for 8 blocks per SM and 233 us for one
            // thread per group)
            const unsigned nall = nblk((long long)(L.P / W) * L.rows);
            const unsigned nbv = std::min<unsigned>(nall, (unsigned)(ctx.nsm * ResidShape<T>::MINB));
            ColourSplit cs;
            if (MPS_RESID_SPLIT && make_split(L, W, cs)) {  // interior without boundary code, the shell apart
                R* ur = rout.c[0] ? ured : nullptr;
                pdl_launch(k_residv_split<T, W, R>, nbv, TPB, 0, ctx.s, L, op, u, f.half(0),
                           rout.c[0] ? rout.half(0) : nullptr, ctx.rb, cs, ur, (R)om);
                CKL();
                prof_end(ctx);
                if (ured_done) *ured_done = ur != nullptr;
                return 0;
            }
            // both colours in one pass (f and rout as split bases, halves L.half apart)
            pdl_launch(k_residv<T, W, R>, nbv, TPB, 0, ctx.s, L, op, -1, u, f.half(0), rout.c[0] ? rout.half(0) : nullptr,
                                                       ctx.rb, 0, dg);
            CKL();
            prof_end(ctx);
            return 0;
        }
    } else {
        // explicit rows: interior cells without boundary code, the shell cell by cell
        ColourSplit cs;
        if (MPS_RESID_SPLIT && L.uniform && L.nx >= 16 && make_split(L, 1, cs)) {
            const unsigned nbv = std::min<unsigned>(cs.nb_in + cs.nb_xe + cs.nb_face,
                                                    (unsigned)(ctx.nsm * ResidShape<T>::MINB));
            pdl_launch(k_residv_split<T, 1, R, Op>, nbv, TPB, 0, ctx.s, L, op, u, f.half(0),
                       rout.c[0] ? rout.half(0) : nullptr, ctx.rb, cs, (R*)nullptr, R(1));
            CKL();
            prof_end(ctx);
            return 0;
        }
    }
    pdl_launch(k_resid_norm<T, Op, R>, nblk((long long)L.P * L.rows), TPB, 0, ctx.s, L, op, u, f, rout, ctx.rb);
    prof_end(ctx);
    CKL();
    return 0;
}

static int fetch(Ctx& ctx, const double* dsrc, int n)
{
    CK(cudaMemcpyAsync(ctx.hpin, dsrc, sizeof(double) * n, cudaMemcpyDeviceToHost, ctx.s));
    CK(cudaStreamSynchronize(ctx.s));
    return 0;
}

// the residual norms (rb.out[0..1]) and the device failure word rb.out[3],
// which a kernel whose bounded wait gave up sets (k_colour_tma)
static int fetch_norms(Ctx& ctx)
{
    if (int st = fetch(ctx, ctx.rb.out, 4)) return st;
    if (ctx.hpin[3] != 0.0) {
        CK(cudaMemsetAsync(ctx.rb.out + 3, 0, sizeof(double), ctx.s));
        ctx.err.code = MPS_ERR_TIMEOUT;
        ctx.err.msg = "a bounded device-side wait expired (colour pass copies)";
        return MPS_ERR_TIMEOUT;
    }
    return 0;
}

// ----------------------------------------------------------------------
struct Inputs {  // device pointers (ghosted Fortran-order fields)
    const double* vel;
    const double* dcoeff;
    const double* reac;
    const double* source;
    const double* bcval[6];
    const double* sterm;
    double* soln;
};

template <class T>
static void alloc_hier(Ctx& ctx, Hier<T>& H, bool& ok)
{
    for (int l = 0; l < ctx.nlev; l++) {
        const Lev& L = ctx.lev[l];
        size_t b = sizeof(T) * 2 * L.half;
        H.U[l][0] = (T*)ctx.ar.get(b);
        H.U[l][1] = (T*)ctx.ar.get(b);
        H.F[l] = (T*)ctx.ar.get(b);
        H.R[l] = (T*)ctx.ar.get(b);
        H.D[l] = (l >= 1 && l < ctx.nlev - 1) ? (T*)ctx.ar.get(sizeof(T) * L.half) : nullptr;
        H.ri[l] = H.bi[l] = 0;
        ok = ok && H.U[l][0] && H.U[l][1] && H.F[l] && H.R[l] && (H.D[l] || l < 1 || l >= ctx.nlev - 1);
    }
    const Lev& C = ctx.lev[ctx.nlev - 1];
    const long long n = (long long)C.nx * C.ny * C.nz;
    H.AinvT = (double*)ctx.ar.get(sizeof(double) * n * n);
    H.Dprev = (double*)ctx.ar.get(sizeof(double) * n * n);
    H.gj = (int*)ctx.ar.get(sizeof(int) * 4);
    ok = ok && H.AinvT && H.Dprev && H.gj;
}

// levels whose rows of one coefficient are marked where most are (figures of 32-cell
// segments, which the rows replaced):
// those bound by bytes (a smaller level's passes are bound by latency, which the
// row's own load would lengthen).  257^3 plasma solve without / on the finest
// level / on the finest two: 11.80 / 10.79 / 10.73 ms mixed, 18.0 / 15.52 / 15.44 ms
// FP64; the 129^3 step 5.58 / 5.51 / 5.51 ms
constexpr long long SEG_MIN_CELLS = 1 << 19;
static bool seg_level(const Lev& L) { return (long long)L.nx * L.ny * L.nz >= SEG_MIN_CELLS && L.nx >= 32; }

// the arrays of one signature; lean: only what a solve cannot do without -- no averaged-
// face coarse coefficients and their means, no rows of one coefficient, no cluster (its rows
// are eight words a cell), the transposed rows' scratch per solve
static bool alloc_workspace(Ctx& ctx, const Signature& sig, int need64, int need32, bool lean)
{
    bool ok = true;
    const int nl = ctx.nlev;
    for (int l = 0; l < nl; l++) {
        const Lev& L = ctx.lev[l];
        const size_t b64 = sizeof(double) * 2 * L.half, b32 = sizeof(float) * 2 * L.half;
        ctx.pk[l] = (double*)ctx.ar.get(b64);
        const bool means = !lean && sig.opclass == 0 && !sig.kuni && l >= 1;
        ctx.pka[l] = means ? (double*)ctx.ar.get(b64) : nullptr;
        ctx.preac[l] = sig.has_reac ? (double*)ctx.ar.get(b64) : nullptr;
        ctx.dex64[l] = sig.has_reac ? (double*)ctx.ar.get(b64) : nullptr;
        for (int a = 0; a < 3; a++) ctx.pv[a][l] = sig.opclass == 1 ? (double*)ctx.ar.get(b64) : nullptr;
        ok = ok && ctx.pk[l] && (ctx.pka[l] || !means);
        if (sig.opclass == 1) {
            ctx.rows64[l] = (need64 || l == 0) ? (double*)ctx.ar.get(7 * b64) : nullptr;  // l>0: FP64 solves
            ctx.rows32[l] = need32 ? (float*)ctx.ar.get(7 * b32) : nullptr;
        } else {
            ctx.k32[l] = (need32 && !sig.kuni) ? (float*)ctx.ar.get(b32) : nullptr;
            const bool segs = !lean && !sig.kuni && seg_level(L);
            const size_t ns = L.rows;
            ctx.seg64[l] = segs ? (double*)ctx.ar.get(sizeof(double) * ns) : nullptr;
            ctx.seg32[l] = segs ? (float*)ctx.ar.get(sizeof(float) * ns) : nullptr;
            ok = ok && (!segs || (ctx.seg64[l] && ctx.seg32[l]));
            ctx.dex32[l] = (need32 && sig.has_reac) ? (float*)ctx.ar.get(b32) : nullptr;
        }
    }
    // (kept with the signature instead of allocated for every level of every solve; the
    // 65^3 gradient, 14 to 24 ms from run to run, does not resolve the gain)
    const bool trows = !lean && sig.transpose;
    ctx.trows = trows ? (double*)ctx.ar.get(sizeof(double) * 7 * 2 * ctx.lev[0].half) : nullptr;
    ok = ok && (ctx.trows || !trows);
    if (need64) alloc_hier(ctx, ctx.h64, ok);
    if (need32) alloc_hier(ctx, ctx.h32, ok);
    const Lev& L0 = ctx.lev[0];
    ctx.x64 = (double*)ctx.ar.get(sizeof(double) * 2 * L0.half);
    ctx.b64 = (double*)ctx.ar.get(sizeof(double) * 2 * L0.half);
    const Lev& C = ctx.lev[nl - 1];
    const long long nc = (long long)C.nx * C.ny * C.nz;
    ctx.dense = (double*)ctx.ar.get(sizeof(double) * nc * nc);
    ctx.gjM = (double*)ctx.ar.get(sizeof(double) * nc * nc * 2);
    ctx.dstatus = (int*)ctx.ar.get(sizeof(int) * 4);
    const unsigned maxb = nblk((long long)L0.P * L0.rows);
    ctx.rb.partial = (double*)ctx.ar.get(sizeof(double) * 2 * (maxb + 1));
    ctx.rb.counter = (unsigned*)ctx.ar.get(sizeof(unsigned) * 4);
    ctx.rb.out = (double*)ctx.ar.get(sizeof(double) * 4);
    ok = ok && ctx.x64 && ctx.b64 && ctx.dense && ctx.gjM && ctx.dstatus && ctx.rb.partial && ctx.rb.counter &&
         ctx.rb.out;
    // the small levels in one cluster
    if (need64) ok = ok && cl_setup<double>(ctx, ctx.h64, sig, lean);
    if (need32) ok = ok && cl_setup<float>(ctx, ctx.h32, sig, lean);
    return ok;
}

static int setup_workspace(Ctx& ctx, const Signature& sig, int need64, int need32)
{
    if (sig == ctx.sig) return 0;
    destroy_graphs(ctx);
    ctx.ar.clear();
    ctx.sig = Signature();
    bool ok = alloc_workspace(ctx, sig, need64, need32, false);
    if (!ok) {  // past the cap, or the device is full: without the arrays that only buy time
        cudaGetLastError();
        ctx.ar.clear();
        ok = alloc_workspace(ctx, sig, need64, need32, true);
    }
    if (!ok) {
        cudaGetLastError();
        ctx.ar.clear();
        ctx.err.code = MPS_ERR_NOMEM;
        ctx.err.msg = "device allocation failed";
        return MPS_ERR_NOMEM;
    }
    // the arena zeroes new blocks with cudaMemset on the legacy stream; the
    // solver's stream does not synchronise with it, so wait here
    if (cudaDeviceSynchronize() != cudaSuccess) return MPS_ERR_CUDA;
    ctx.tma_ok = ctx.tma_allowed && tma_prepare(ctx.dev);
    ctx.sig = sig;
    return 0;
}

// FGMRES basis: V (m+1 FP64 vectors), Z (m preconditioned vectors, FP32 in
// mixed precision), w, the Hessenberg column and the dot-product partials
static int setup_krylov(Ctx& ctx, long long n, int m)
{
    const Lev& L0 = ctx.lev[0];
    const int dims[3] = {L0.nx, L0.ny, L0.nz};
    if (ctx.kar_n == n && ctx.kar_m == m) {
        if (std::equal(dims, dims + 3, ctx.kar_dims)) return 0;
        // another grid of the same padded length: its pads held the other's cells, and
        // the dot products run over the pads
        CK(cudaMemsetAsync(ctx.V, 0, sizeof(double) * n * (m + 1), ctx.s));
        CK(cudaMemsetAsync(ctx.Z, 0, sizeof(double) * n * m, ctx.s));
        CK(cudaMemsetAsync(ctx.w, 0, sizeof(double) * n, ctx.s));
        std::copy(dims, dims + 3, ctx.kar_dims);
        return 0;
    }
    destroy_graphs(ctx);
    ctx.kar.clear();
    ctx.kar_n = 0;
    ctx.kar_m = 0;
    bool ok = true;
    ctx.V = (double*)ctx.kar.get(sizeof(double) * n * (m + 1));
    ctx.Z = ctx.kar.get(sizeof(double) * n * m);
    ctx.w = (double*)ctx.kar.get(sizeof(double) * n);
    ctx.hcol = (double*)ctx.kar.get(sizeof(double) * 2 * (m + 2));
    ctx.Vptr = (double**)ctx.kar.get(sizeof(double*) * (m + 2));
    ctx.mdot_blocks = 592;
    ctx.dpart = (double*)ctx.kar.get(sizeof(double) * (m + 2) * ctx.mdot_blocks);
    ok = ctx.V && ctx.Z && ctx.w && ctx.hcol && ctx.Vptr && ctx.dpart;
    if (ok) {
        std::vector<double*> hp(m + 2);
        for (int j = 0; j <= m; j++) hp[j] = ctx.V + (size_t)j * n;
        hp[m + 1] = ctx.w;
        if (cudaMemcpy(ctx.Vptr, hp.data(), sizeof(double*) * (m + 2), cudaMemcpyHostToDevice) != cudaSuccess)
            ok = false;
    }
    if (!ok || cudaDeviceSynchronize() != cudaSuccess) {
        ctx.kar.clear();
        ctx.err.code = MPS_ERR_NOMEM;
        ctx.err.msg = "device allocation failed (Krylov basis)";
        return MPS_ERR_NOMEM;
    }
    ctx.kar_n = n;
    ctx.kar_m = m;
    std::copy(dims, dims + 3, ctx.kar_dims);
    return 0;
}

template <class T>
static void set_kop(Ctx& ctx, KOp<T>* ops, T* const* kT, T* const* dexT, double kc, double dtinv, bool kuni,
                    bool has_reac)
{
    for (int l = 0; l < ctx.nlev; l++) {
        const Lev& L = ctx.lev[l];
        KOp<T> op;
        op.seg = nullptr;
        if (kuni) { op.k[0] = op.k[1] = nullptr; op.kc = (T)kc; }
        else { op.k[0] = kT[l]; op.k[1] = kT[l] + L.half; op.kc = T(0); }
        if (has_reac) { op.dex[0] = dexT[l]; op.dex[1] = dexT[l] + L.half; op.dexc = T(0); }
        else { op.dex[0] = op.dex[1] = nullptr; op.dexc = (T)dtinv; }
        ops[l] = op;
    }
}
template <class T>
static ROp<T> make_rop(T* rows, const Lev& L)
{
    ROp<T> r;
    for (int q = 0; q < 7; q++) {
        r.r[q][0] = rows + (size_t)q * 2 * L.half;
        r.r[q][1] = rows + (size_t)q * 2 * L.half + L.half;
    }
    return r;
}

template <class T>
static int build_rows_level(Ctx& ctx, int l, T* rows, double dtinv, int flux, int transpose, T* tmp)
{
    const Lev& L = ctx.lev[l];
    const double* z = ctx.pk[l];  // any valid pointer for unused fields
    auto cs = [&](const double* p) { return csplit<double>(p ? p : z, L); };
    T* dst = transpose ? tmp : rows;
    pdl_launch(k_build_rows<T>, nblk((long long)L.nx * L.ny * L.nz), TPB, 0, ctx.s, 
        L, cs(ctx.pv[0][l]), cs(ctx.pv[1][l]), cs(ctx.pv[2][l]), cs(ctx.pk[l]), cs(ctx.preac[l]),
        ctx.preac[l] != nullptr, dtinv, flux, make_rop<T>(dst, L));
    CKL();
    if (transpose) {
        pdl_launch(k_transpose_rows<T>, nblk((long long)L.nx * L.ny * L.nz), TPB, 0, ctx.s, L, make_rop<T>(tmp, L),
                                                                                   make_rop<T>(rows, L));
        CKL();
    }
    return 0;
}

template <class T, class Op>
static int coarse_inverse(Ctx& ctx, Hier<T>& H, const Op& op)
{
    const int l = ctx.nlev - 1;
    const Lev& L = ctx.lev[l];
    const int n = L.nx * L.ny * L.nz;
    CK(cudaMemsetAsync(ctx.dense, 0, sizeof(double) * n * n, ctx.s));
    pdl_launch(k_dense_assemble<T, Op>, nblk(n), TPB, 0, ctx.s, L, op, ctx.dense);
    CKL();
    // an unchanged matrix (repeated solves with one operator) keeps its inverse
    pdl_launch(k_dense_same, 1, 1024, 0, ctx.s, n, (const double*)ctx.dense, H.Dprev, H.gj);
    CKL();
    pdl_launch(k_gj_prepare, nblk(2LL * n * n), TPB, 0, ctx.s, n, ctx.dense, ctx.gjM, (const int*)H.gj);
    CKL();
    const size_t smem = sizeof(double) * 2 * (size_t)n * n;
    static signed char gj_state[64] = {};
    const bool gj_smem = once_per_device(ctx.dev, gj_state, [] {
        return cudaFuncSetAttribute(k_gauss_jordan, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024) ==
               cudaSuccess;
    });
    if (smem <= 200 * 1024 && gj_smem) {
        pdl_launch(k_gauss_jordan, 1, 1024, smem, ctx.s, n, ctx.gjM, H.AinvT, ctx.dstatus, 1, H.gj);
    } else {
        pdl_launch(k_gauss_jordan, 1, 1024, 0, ctx.s, n, ctx.gjM, H.AinvT, ctx.dstatus, 0, H.gj);
    }
    CKL();
    return 0;
}

// ----------------------------------------------------------------------
// prepare_only: stop after the set-up (hierarchy, operators, right-hand side,
// initial guess, coarsest inverse), for the batched driver
// det (optional): the operator detection of these inputs already read back
// (DET_WORDS words); the batched solve detects every problem with one
// device->host read
static int solve_impl(Ctx& ctx, const mps_grid* g, int timederiv, double dt, const Inputs& in, const int bc[6],
                      const mps_solver_opts* o, mps_solve_info* info, int ref_norm_only, int prepare_only = 0,
                      const unsigned long long* det = nullptr)
{
    mps_solve_info inf;
    std::memset(&inf, 0, sizeof(inf));
    inf.status = MPS_OK;
    // ---- argument checks ----
    if (!g || g->lx < 1 || g->ly < 1 || g->lz < 1 || !(g->llenx > 0) || !(g->lleny > 0) || !(g->llenz > 0) ||
        !in.dcoeff || !in.source || !in.soln) {
        ctx.err.msg = "bad grid or null field";
        return MPS_ERR_BAD_ARG;
    }
    if ((long long)g->lx * g->ly * g->lz >= (1LL << 31) / 2) { ctx.err.msg = "grid too large"; return MPS_ERR_BAD_ARG; }
    for (int f = 0; f < 6; f++)
        if (bc[f] < 1 || bc[f] > 5) { ctx.err.msg = "bad BC code"; return MPS_ERR_BAD_ARG; }
    for (int a = 0; a < 3; a++)
        if ((bc[2 * a] == BC_PERI) != (bc[2 * a + 1] == BC_PERI)) {
            ctx.err.msg = "PERI must be set on both faces of a direction";
            return MPS_ERR_BAD_ARG;
        }
    if (timederiv && !(dt > 0)) { ctx.err.msg = "dt must be positive"; return MPS_ERR_BAD_ARG; }
    if (o->nu1 < 0 || o->nu2 < 0 || o->maxit < 0 || o->restart < 1 || o->restart > 250 || o->max_coarse < 1 ||
        o->max_coarse > MAX_DENSE) {
        ctx.err.msg = "bad solver option";
        return MPS_ERR_BAD_ARG;
    }
    for (int f = 0; f < 6; f++)
        if (!in.bcval[f] && (bc[f] == BC_DIRC || bc[f] == BC_FLUX)) {
            ctx.err.msg = "missing boundary values for a DIRC/FLUX face";
            return MPS_ERR_BAD_ARG;
        }
    std::string why;
    int nl = plan_levels(g, o, bc, ctx.lev, ctx.xf, why);
    if (nl < 1) { ctx.err.msg = why; return MPS_ERR_BAD_ARG; }
    ctx.nlev = nl;
    ctx.len[0] = g->llenx;
    ctx.len[1] = g->lleny;
    ctx.len[2] = g->llenz;
    const Lev& L0 = ctx.lev[0];
    {  // 1-D prolongation tables of the geometric transfers
        size_t total = 0;
        for (int l = 0; l + 1 < nl; l++)
            for (int a = 0; a < 3; a++) total += ctx.xf[l].nf[a];
        std::vector<Lin> tab(total > 0 ? total : 1);
        size_t pos = 0;
        for (int l = 0; l + 1 < nl; l++)
            for (int a = 0; a < 3; a++) {
                for (int i = 0; i < ctx.xf[l].nf[a]; i++) {
                    Lin e;
                    geom_lin(ctx.xf[l], a, i, e.j0, e.j1, e.t);
                    tab[pos + i] = e;
                }
                pos += ctx.xf[l].nf[a];
            }
        // the device copy is kept while the tables do not change (a copy from
        // pageable host memory would hold the host until the stream drains)
        const bool same = ctx.dtab && tab.size() == ctx.htab.size() &&
                          std::memcmp(tab.data(), ctx.htab.data(), sizeof(Lin) * tab.size()) == 0;
        if (!same) {
            if (tab.size() > ctx.dtab_n) {
                if (ctx.dtab) cudaFree(ctx.dtab);
                ctx.dtab = nullptr;
                ctx.dtab_n = 0;
                CK(cudaMalloc((void**)&ctx.dtab, sizeof(Lin) * tab.size()));
                ctx.dtab_n = tab.size();
            }
            ctx.htab.swap(tab);
            CK(cudaMemcpyAsync(ctx.dtab, ctx.htab.data(), sizeof(Lin) * ctx.htab.size(), cudaMemcpyHostToDevice,
                               ctx.s));
        }
        pos = 0;
        for (int l = 0; l + 1 < nl; l++)
            for (int a = 0; a < 3; a++) {
                ctx.xf[l].tab[a] = ctx.dtab + pos;
                pos += ctx.xf[l].nf[a];
            }
    }
    const double dtinv = timederiv ? 1.0 / dt : 0.0;

    const long long launches0 = ctx.launches;
    CK(cudaEventRecord(ctx.e0, ctx.s));
    // ---- operator detection (one small device->host read) ----
    unsigned long long* dm = ctx.dmax;
    const long long ncell = (long long)L0.nx * L0.ny * L0.nz;
    const long long ng = (long long)(L0.nx + 2) * (L0.ny + 2) * (L0.nz + 2);
    unsigned long long hm[DET_WORDS];
    double k0 = 0.0;
    if (det) {
        std::memcpy(hm, det, sizeof(hm));
        std::memcpy(&k0, det + DET_REF, sizeof(double));
    } else {
        CK(cudaMemsetAsync(dm, 0, sizeof(hm), ctx.s));
        const unsigned mb = std::min<unsigned>(nblk(ncell), 1184);
        pdl_launch(k_maxabs_all, mb, TPB, 0, ctx.s, L0, in.vel, in.reac, in.dcoeff, in.source, in.soln, dm);
        CKL();
        if (in.reac) {
            pdl_launch(k_max_reac, mb, TPB, 0, ctx.s, L0, in.reac, dm + DET_REAC);
            CKL();
        }
        CK(cudaMemcpyAsync(hm, dm, sizeof(hm), cudaMemcpyDeviceToHost, ctx.s));
        CK(cudaMemcpyAsync(&k0, in.dcoeff + 1 + (L0.nx + 2) * (1 + (long long)(L0.ny + 2)), sizeof(double),
                           cudaMemcpyDeviceToHost, ctx.s));
        CK(cudaStreamSynchronize(ctx.s));
    }
    auto asd = [](unsigned long long b) { double d; std::memcpy(&d, &b, 8); return d; };
    const double maxvel = asd(hm[0]), maxreac = asd(hm[1]), dkvar = asd(hm[2]), maxsrc = asd(hm[3]),
                 maxsol = asd(hm[4]), maxk = asd(hm[5]);
    if (!(maxvel <= 1e308) || !(maxreac <= 1e308) || !(dkvar <= 1e308) || !(maxsrc <= 1e308) ||
        !(maxsol <= 1e308) || !(maxk <= 1e308)) {
        ctx.err.msg = "NaN or Inf in the inputs";
        inf.status = MPS_ERR_NAN;
        if (info) *info = inf;
        return MPS_ERR_NAN;
    }
    Signature sig;
    sig.dims[0] = g->lx; sig.dims[1] = g->ly; sig.dims[2] = g->lz;
    for (int f = 0; f < 6; f++) sig.bc[f] = bc[f];
    sig.hier = o->hierarchy;
    for (int a = 0; a < 3; a++) sig.ranks[a] = o->hierarchy == MPS_HIER_CELL ? o->ranks[a] : 0;
    sig.max_coarse = o->hierarchy == MPS_HIER_GEOM ? o->max_coarse : 0;
    sig.opclass = (o->transpose == 0 && o->flux == MPS_FLUX_UPWIND && maxvel == 0.0) ? 0 : 1;
    if (o->flux == MPS_FLUX_UPWIND && maxvel == 0.0) sig.opclass = 0;  // symmetric: A^T = A
    sig.prec = 0;
    sig.krylov = 0;
    sig.restart = 0;
    sig.has_reac = maxreac > 0.0;
    sig.kuni = dkvar == 0.0;
    sig.transpose = o->transpose && sig.opclass == 1;
    const bool mixed = o->precision == MPS_PREC_MIXED;
    // both hierarchies stay allocated (switching precision costs no allocation);
    // only the one this solve uses is filled
    int st = setup_workspace(ctx, sig, 1, 1);
    const int need64 = !mixed, need32 = mixed;
    if (st) return st;
    // The solves on the geometric hierarchy with a cell coefficient over-relax
    // their passes (pass_omega) and take the coarse coefficients of
    // k_restrict_coef; mps_vcycle_once, which is one perform_vcycle, the
    // reference's hierarchy, explicit rows (not symmetric) and V-cycles
    // without a relaxed first sweep or post-smoothing keep plain Gauss-Seidel
    // and arithmetic means, and so does a workspace without room for both means.
    ctx.relaxed = sig.opclass == 0 && o->hierarchy == MPS_HIER_GEOM && !ref_norm_only && o->nu1 >= 1 && o->nu2 >= 1 &&
                  (sig.kuni || nl < 2 || ctx.pka[1]);
    ctx.extra_q = extra_step(L0, diag_extra_min(dtinv, maxreac, hm[DET_REAC]), maxk);
    set_relaxation(ctx);
    if (o->krylov == MPS_KRYLOV_FGMRES && (st = setup_krylov(ctx, 2 * ctx.lev[0].half, o->restart))) return st;

    // ---- coefficient pyramid (FP64) ----
    // (no level of a cell-coefficient operator reads a uniform coefficient's field)
    const bool kpyr = sig.opclass == 1 || !sig.kuni;
    if (kpyr) {
        pdl_launch(k_pack<double>, nblk(ncell), TPB, 0, ctx.s, L0, in.dcoeff, split<double>(ctx.pk[0], L0), 1.0, 0.0);
        CKL();
    }
    if (sig.has_reac) {
        pdl_launch(k_pack<double>, nblk(ncell), TPB, 0, ctx.s, L0, in.reac, split<double>(ctx.preac[0], L0), 1.0, 0.0);
        CKL();
    }
    if (sig.opclass == 1)
        for (int a = 0; a < 3; a++) {
            pdl_launch(k_pack<double>, nblk(ncell), TPB, 0, ctx.s, L0, in.vel ? in.vel + a * ng : nullptr,
                                                           split<double>(ctx.pv[a][0], L0), 1.0, 0.0);
            CKL();
        }
    for (int l = 0; l + 1 < nl; l++) {
        const Lev& F = ctx.lev[l];
        const Lev& C = ctx.lev[l + 1];
        const unsigned nb = nblk((long long)C.nx * C.ny * C.nz);
        const int geom = ctx.xf[l].geom;
        if (kpyr) {
            if (ctx.relaxed)
                pdl_launch(k_restrict_coef, nb, TPB, 0, ctx.s, F, csplit<double>(ctx.pk[l], F),
                           csplit<double>(l ? ctx.pka[l] : ctx.pk[0], F), C, split<double>(ctx.pk[l + 1], C),
                           split<double>(ctx.pka[l + 1], C));
            else
                pdl_launch(k_restrict_field, nb, TPB, 0, ctx.s, F, csplit<double>(ctx.pk[l], F), C,
                           split<double>(ctx.pk[l + 1], C), geom);
            CKL();
        }
        if (sig.has_reac) {
            pdl_launch(k_restrict_field, nb, TPB, 0, ctx.s, F, csplit<double>(ctx.preac[l], F), C,
                                                    split<double>(ctx.preac[l + 1], C), geom);
            CKL();
        }
        if (sig.opclass == 1)
            for (int a = 0; a < 3; a++) {
                pdl_launch(k_restrict_field, nb, TPB, 0, ctx.s, F, csplit<double>(ctx.pv[a][l], F), C,
                                                        split<double>(ctx.pv[a][l + 1], C), geom);
                CKL();
            }
    }
    // ---- operators ----
    if (sig.opclass == 0) {
        for (int l = 0; l < nl; l++) {
            const long long n2 = 2 * ctx.lev[l].half;
            if (sig.has_reac) {
                pdl_launch(k_cast_field<double>, std::min<unsigned>(nblk(n2), 2368), TPB, 0, ctx.s, n2, ctx.preac[l], ctx.dex64[l], -1.0, dtinv);
                CKL();
            }
            if (need32) {
                if (!sig.kuni) {
                    pdl_launch(k_cast_field<float>, std::min<unsigned>(nblk(n2), 2368), TPB, 0, ctx.s, n2, ctx.pk[l], ctx.k32[l], 1.0, 0.0);
                    CKL();
                }
                if (sig.has_reac) {
                    pdl_launch(k_cast_field<float>, std::min<unsigned>(nblk(n2), 2368), TPB, 0, ctx.s, n2, ctx.preac[l], ctx.dex32[l], -1.0, dtinv);
                    CKL();
                }
            }
        }
        KOp<double> k64[MAXL];
        set_kop<double>(ctx, k64, ctx.pk, ctx.dex64, k0, dtinv, sig.kuni, sig.has_reac);
        if (need32) set_kop<float>(ctx, ctx.h32.kop, ctx.k32, ctx.dex32, k0, dtinv, sig.kuni, sig.has_reac);
        // a coefficient that changes seldom: along x at most once in four 32-cell chunks of
        // the rows, from row to row in a quarter of the sampled columns (four a row).
        // A row with a change along x has no single coefficient: with more than one such
        // change in two rows the colour pass stages the field as without the marks
        const unsigned long long nchunk = (unsigned long long)L0.rows * (unsigned)((L0.nx + 31) / 32);
        ctx.kseg = 0;
        if (!prepare_only && !sig.kuni && ctx.seg64[0] && !in.vel && hm[6] <= nchunk / 4 &&
            hm[7] <= (unsigned long long)L0.rows)
            ctx.kseg = hm[6] <= L0.rows / 2 ? 2 : 1;
        if (ctx.kseg) {
            auto segments = [&](auto* k, auto* seg, auto& op, int l) -> int {
                using TT = typename std::remove_pointer<decltype(seg)>::type;
                const Lev& L = ctx.lev[l];
                op.seg = seg;
                pdl_launch(k_kseg<TT>, nblk(32LL * L.rows), TPB, 0, ctx.s, L, csplit<TT>(k, L), seg);
                CKL();
                return 0;
            };
            for (int l = 0; l < nl && ctx.seg64[l]; l++) {
                if ((need64 || l == 0) && (st = segments(ctx.pk[l], ctx.seg64[l], k64[l], l))) return st;
                if (need32 && (st = segments(ctx.k32[l], ctx.seg32[l], ctx.h32.kop[l], l))) return st;
            }
        }
        ctx.kop64 = k64[0];
        if (need64) std::copy(k64, k64 + nl, ctx.h64.kop);
    } else {
        double* trows = ctx.trows;
        if (sig.transpose && !trows) CK(cudaMallocAsync((void**)&trows, sizeof(double) * 7 * 2 * L0.half, ctx.s));
        auto release = [&]() { if (trows != ctx.trows) cudaFreeAsync(trows, ctx.s); };
        for (int l = 0; l < nl; l++) {
            if (ctx.rows64[l] && (need64 || l == 0)) {
                if ((st = build_rows_level<double>(ctx, l, ctx.rows64[l], dtinv, o->flux, sig.transpose, trows))) {
                    release();
                    return st;
                }
                if (need64) ctx.h64.rop[l] = make_rop<double>(ctx.rows64[l], ctx.lev[l]);
            }
            if (ctx.rows32[l] && need32) {
                if (ctx.rows64[l] && (need64 || l == 0)) {
                    // the FP64 rows of this level rounded: a pass over 21 words a cell against
                    // the face fluxes' exponentials again (185 us at 129^3 SG; the electron step
                    // 1830 -> 1674 us, the plasma step 5.22 -> 5.03 ms)
                    const long long n7 = 7 * 2 * ctx.lev[l].half;
                    pdl_launch(k_cast_field<float>, std::min<unsigned>(nblk(n7), 2368), TPB, 0, ctx.s, n7,
                               ctx.rows64[l], ctx.rows32[l], 1.0, 0.0);
                    CKL();
                } else if ((st = build_rows_level<float>(ctx, l, ctx.rows32[l], dtinv, o->flux, sig.transpose,
                                                         (float*)trows))) {
                    release();
                    return st;
                }
                ctx.h32.rop[l] = make_rop<float>(ctx.rows32[l], ctx.lev[l]);
            }
        }
        release();
        ctx.rop64 = make_rop<double>(ctx.rows64[0], L0);
    }
    // ---- right-hand side and initial guess ----
    {
        const double* bv[6];
        for (int f = 0; f < 6; f++) bv[f] = in.bcval[f];
        pdl_launch(k_find_bvec, nblk(ncell), TPB, 0, ctx.s, L0, in.vel, in.dcoeff, in.source, bv[0], bv[1], bv[2], bv[3],
                                                    bv[4], bv[5], in.sterm, o->flux, split<double>(ctx.b64, L0));
        CKL();
        if (maxsol == 0.0) {  // a zero initial guess (every interior cell): clear instead of packing
            CK(cudaMemsetAsync(ctx.x64, 0, sizeof(double) * 2 * L0.half, ctx.s));
        } else {
            pdl_launch(k_pack<double>, nblk(ncell), TPB, 0, ctx.s, L0, in.soln, split<double>(ctx.x64, L0), 1.0, 0.0);
            CKL();
        }
    }
    // ---- coarsest inverse ----
    CK(cudaMemsetAsync(ctx.dstatus, 0, sizeof(int) * 4, ctx.s));
    if (need64) {
        if (sig.opclass == 0) st = coarse_inverse(ctx, ctx.h64, ctx.h64.kop[nl - 1]);
        else st = coarse_inverse(ctx, ctx.h64, ctx.h64.rop[nl - 1]);
    } else {
        if (sig.opclass == 0) st = coarse_inverse(ctx, ctx.h32, ctx.h32.kop[nl - 1]);
        else st = coarse_inverse(ctx, ctx.h32, ctx.h32.rop[nl - 1]);
    }
    if (st) return st;
    if (!prepare_only) {  // the tables and rows of the cluster's levels
        if ((st = need64 ? cl_tables(ctx, ctx.h64) : cl_tables(ctx, ctx.h32))) return st;
        if (sig.opclass == 0) st = need64 ? cl_rows(ctx, ctx.h64, ctx.h64.kop) : cl_rows(ctx, ctx.h32, ctx.h32.kop);
        else st = need64 ? cl_rows(ctx, ctx.h64, ctx.h64.rop) : cl_rows(ctx, ctx.h32, ctx.h32.rop);
        if (st) return st;
    }
    if (sig.opclass == 0 && !prepare_only) {
        // the red rows' diagonals of the levels with their own launches (the
        // restriction into such a level also writes its first red pass)
        auto diag_red = [&](auto& H) -> int {
            using TT = typename std::remove_reference<decltype(*H.D[0])>::type;
            const int lend = H.cl_l0 >= 0 ? H.cl_l0 : nl - 1;
            for (int l = 1; l < lend && l < nl - 1; l++) {
                if (!H.D[l]) continue;
                const Lev& Ll = ctx.lev[l];
                pdl_launch(k_diag_red<TT, KOp<TT>>, nblk((long long)Ll.P * Ll.rows), TPB, 0, ctx.s, Ll, H.kop[l],
                           H.D[l], (TT)pass_omega(ctx, l, o, true, 0, 0));
                CKL();
            }
            return 0;
        };
        if (need64) st = diag_red(ctx.h64);
        else st = diag_red(ctx.h32);
        if (st) return st;
    }
    if (prepare_only) {
        inf.levels = nl;
        if (info) *info = inf;
        return 0;
    }

    // ---- iterations ----
    const Lev& L = L0;
    const long long n2 = 2 * L.half;
    double bnorm = 0.0, rel = 0.0, rms = 0.0;
    int it = 0, vcycles = 0;
    auto norms = [&](double rr, double ff) {
        rel = ff > 0.0 ? std::sqrt(rr) / std::sqrt(ff) : std::sqrt(rr);
        rms = std::sqrt(rr / (double)ncell);
    };
    auto conv = [&]() { return o->tol_kind == MPS_TOL_RMS_ABS ? rms <= o->tol : rel <= o->tol; };
    Split<double> no64;
    no64.c[0] = no64.c[1] = nullptr;

    GraphKey gk;
    gk.sig = sig;
    gk.prec = mixed;
    gk.nu1 = o->nu1;
    gk.nu2 = o->nu2;
    gk.nlev = nl;
    gk.flux = o->flux;
    gk.transpose = sig.transpose;  // a symmetric operator's transposed solve replays the forward graphs
    gk.kc = sig.kuni ? k0 : 0.0;
    gk.dexc = sig.has_reac ? 0.0 : dtinv;
    std::copy(ctx.len, ctx.len + 3, gk.len);
    gk.ws = ctx.ar.blocks.empty() ? nullptr : ctx.ar.blocks[0];
    gk.relaxed = ctx.relaxed;
    gk.extra_q = ctx.relaxed ? ctx.extra_q : 0;
    gk.kseg = sig.opclass == 0 ? ctx.kseg : 0;
    gk.prof = ctx.prof.on ? 1 + ctx.prof.level : 0;  // profiled graphs carry event-record nodes
    // graphs need the buffer parities to return after one iteration
    const bool graphs = o->use_graph && ((o->nu1 + o->nu2) % 2 == 0);

    if (o->krylov == MPS_KRYLOV_NONE && !mixed) {
        // FP64 stationary V-cycle iteration on h64 (x lives in level-0 U)
        Hier<double>& H = ctx.h64;
        CK(cudaMemcpyAsync(H.U[0][0], ctx.x64, sizeof(double) * n2, cudaMemcpyDeviceToDevice, ctx.s));
        CK(cudaMemcpyAsync(H.F[0], ctx.b64, sizeof(double) * n2, cudaMemcpyDeviceToDevice, ctx.s));
        for (int l = 0; l < nl; l++) H.ri[l] = H.bi[l] = 0;
        auto residual = [&]() -> int {
            if (sig.opclass == 0) return resid_norm(ctx, H.kop[0], ccur(H, L, 0), csplit<double>(H.F[0], L), no64);
            return resid_norm(ctx, H.rop[0], ccur(H, L, 0), csplit<double>(H.F[0], L), no64);
        };
        auto iteration = [&]() -> int {
            int s2 = vcycle(ctx, H, sig.opclass, o, false);
            if (s2) return s2;
            return residual();
        };
        if ((st = residual())) return st;
        for (;;) {
            if ((st = fetch_norms(ctx))) return st;
            if (!(ctx.hpin[0] <= 1e308)) { inf.status = MPS_ERR_NAN; break; }
            norms(ctx.hpin[0], ctx.hpin[1]);
            if (it == 0) inf.rel_res0 = rel;
            if (ref_norm_only ? it >= o->maxit : (conv() || it >= o->maxit)) break;
            if (graphs) {
                gk.kind = 1;
                GraphEntry* G = nullptr;
                for (;;) {  // each replay ends with the residual norms of the new iterate
                    if ((st = run_graph(ctx, gk, &G, iteration))) return st;
                    if ((st = fetch_norms(ctx))) return st;
                    prof_collect_graph(ctx, *G);
                    vcycles++;
                    it++;
                    if (!(ctx.hpin[0] <= 1e308)) { inf.status = MPS_ERR_NAN; break; }
                    norms(ctx.hpin[0], ctx.hpin[1]);
                    if (ref_norm_only ? it >= o->maxit : (conv() || it >= o->maxit)) break;
                }
                break;
            }
            if ((st = iteration())) return st;
            vcycles++;
            it++;
        }
        // copy the iterate back to x64 (split, both colours)
        CK(cudaMemcpyAsync(ctx.x64, H.U[0][H.ri[0]], sizeof(double) * L.half, cudaMemcpyDeviceToDevice, ctx.s));
        CK(cudaMemcpyAsync(ctx.x64 + L.half, H.U[0][H.bi[0]] + L.half, sizeof(double) * L.half,
                           cudaMemcpyDeviceToDevice, ctx.s));
    } else if (o->krylov == MPS_KRYLOV_NONE && mixed) {
        // FP64 defect correction with FP32 V-cycles
        Hier<float>& H = ctx.h32;
        const int inner = o->inner_cycles > 0 ? o->inner_cycles : 2;
        for (int l = 0; l < nl; l++) H.ri[l] = H.bi[l] = 0;
        gk.inner = inner;
        // the residual also writes the first V-cycle's red pass from zero on the
        // finest level (r / diag) where its split kernel runs; the V-cycle then
        // skips that pass
        bool red_ready = false;
        auto residual = [&]() -> int {
            Split<float> r32 = split<float>(H.F[0], L);
            float* ured = o->nu1 >= 1 && H.cl_l0 != 0 ? H.U[0][H.ri[0] ^ 1] : nullptr;
            if (sig.opclass == 0)
                return resid_norm(ctx, ctx.kop64, csplit<double>(ctx.x64, L), csplit<double>(ctx.b64, L), r32, ured,
                                  &red_ready, pass_omega(ctx, 0, o, true, 0, 0));
            return resid_norm(ctx, ctx.rop64, csplit<double>(ctx.x64, L), csplit<double>(ctx.b64, L), r32, ured,
                              &red_ready);
        };
        auto iteration = [&]() -> int {
            int s2;
            for (int c = 0; c < inner; c++) {
                ctx.red0_ready = c == 0 && red_ready;
                s2 = vcycle(ctx, H, sig.opclass, o, c == 0);
                ctx.red0_ready = false;
                if (s2) return s2;
            }
            const unsigned ab = std::min<unsigned>(nblk(2 * L.half), 4736);
            pdl_launch(k_axpy2<float, double>, ab, TPB, 0, ctx.s, L.half, 1.0, (const float*)H.U[0][H.ri[0]], ctx.x64,
                       (const float*)(H.U[0][H.bi[0]] + L.half), ctx.x64 + L.half);
            CKL();
            return residual();
        };
        if ((st = residual())) return st;
        for (;;) {
            if ((st = fetch_norms(ctx))) return st;
            if (!(ctx.hpin[0] <= 1e308)) { inf.status = MPS_ERR_NAN; break; }
            norms(ctx.hpin[0], ctx.hpin[1]);
            if (it == 0) inf.rel_res0 = rel;
            if (conv() || it >= o->maxit) break;
            if (graphs) {
                gk.kind = 2;
                GraphEntry* G = nullptr;
                for (;;) {  // each replay ends with the residual norms of the new iterate
                    if ((st = run_graph(ctx, gk, &G, iteration))) return st;
                    if ((st = fetch_norms(ctx))) return st;
                    prof_collect_graph(ctx, *G);
                    vcycles += inner;
                    it++;
                    if (!(ctx.hpin[0] <= 1e308)) { inf.status = MPS_ERR_NAN; break; }
                    norms(ctx.hpin[0], ctx.hpin[1]);
                    if (conv() || it >= o->maxit) break;
                }
                break;
            }
            if ((st = iteration())) return st;
            vcycles += inner;
            it++;
        }
    } else {
        // FGMRES(m), right preconditioned by one V-cycle (FP32 when MIXED)
        for (int l = 0; l < nl; l++) ctx.h32.ri[l] = ctx.h32.bi[l] = ctx.h64.ri[l] = ctx.h64.bi[l] = 0;
        const int m = o->restart;
        const long long n = n2;
        const unsigned db = ctx.mdot_blocks;
        std::vector<double> H((size_t)(m + 1) * m), cs(m), sn(m), gq(m + 1), y(m);
        auto HH = [&](int i, int j) -> double& { return H[(size_t)i + (size_t)(m + 1) * j]; };
        for (;;) {
            // w = b - A x, beta = ||w||
            if (sig.opclass == 0)
                st = resid_norm(ctx, ctx.kop64, csplit<double>(ctx.x64, L), csplit<double>(ctx.b64, L),
                                split<double>(ctx.w, L));
            else
                st = resid_norm(ctx, ctx.rop64, csplit<double>(ctx.x64, L), csplit<double>(ctx.b64, L),
                                split<double>(ctx.w, L));
            if (st) return st;
            if ((st = fetch_norms(ctx))) return st;
            if (!(ctx.hpin[0] <= 1e308)) { inf.status = MPS_ERR_NAN; break; }
            norms(ctx.hpin[0], ctx.hpin[1]);
            if (it == 0) { inf.rel_res0 = rel; bnorm = std::sqrt(ctx.hpin[1]); }
            if (conv() || it >= o->maxit) break;
            const double beta = std::sqrt(ctx.hpin[0]);
            // v0 = w / beta
            ctx.hpin[0] = beta;
            CK(cudaMemcpyAsync(ctx.hcol, ctx.hpin, sizeof(double), cudaMemcpyHostToDevice, ctx.s));
            pdl_launch(k_scale_to, std::min<unsigned>(nblk(n), 2368), TPB, 0, ctx.s, n, ctx.w, ctx.hcol, 0, ctx.V, nullptr);
            CKL();
            std::fill(H.begin(), H.end(), 0.0);
            std::fill(gq.begin(), gq.end(), 0.0);
            gq[0] = beta;
            int j = 0;
            bool done = false;
            for (j = 0; j < m && it < o->maxit; j++) {
                double* vj = ctx.V + (size_t)j * n;
                GraphEntry* pg = nullptr;  // the preconditioner's graph replayed this iteration
                // z_j = M^{-1} v_j (one V-cycle from zero), then w = A z_j in FP64
                if (mixed) {
                    Hier<float>& P = ctx.h32;
                    pdl_launch(k_cast_field<float>, std::min<unsigned>(nblk(n), 2368), TPB, 0, ctx.s, n, vj, P.F[0], 1.0, 0.0);
                    CKL();
                    if (graphs) {
                        gk.kind = 3;
                        if ((st = run_graph(ctx, gk, &pg, [&]() { return vcycle(ctx, P, sig.opclass, o, true); })))
                            return st;
                    } else if ((st = vcycle(ctx, P, sig.opclass, o, true))) {
                        return st;
                    }
                    float* zj = (float*)ctx.Z + (size_t)j * n;
                    CK(cudaMemcpyAsync(zj, P.U[0][P.ri[0]], sizeof(float) * L.half, cudaMemcpyDeviceToDevice, ctx.s));
                    CK(cudaMemcpyAsync(zj + L.half, P.U[0][P.bi[0]] + L.half, sizeof(float) * L.half,
                                       cudaMemcpyDeviceToDevice, ctx.s));
                    if (sig.opclass == 0)
                        pdl_launch(k_apply<double, KOp<double>, float>, nblk((long long)L.P * L.rows), TPB, 0, ctx.s, 
                            L, ctx.kop64, csplit<float>(zj, L), split<double>(ctx.w, L));
                    else
                        pdl_launch(k_apply<double, ROp<double>, float>, nblk((long long)L.P * L.rows), TPB, 0, ctx.s, 
                            L, ctx.rop64, csplit<float>(zj, L), split<double>(ctx.w, L));
                    CKL();
                } else {
                    Hier<double>& P = ctx.h64;
                    CK(cudaMemcpyAsync(P.F[0], vj, sizeof(double) * n, cudaMemcpyDeviceToDevice, ctx.s));
                    if (graphs) {
                        gk.kind = 4;
                        if ((st = run_graph(ctx, gk, &pg, [&]() { return vcycle(ctx, P, sig.opclass, o, true); })))
                            return st;
                    } else if ((st = vcycle(ctx, P, sig.opclass, o, true))) {
                        return st;
                    }
                    double* zj = (double*)ctx.Z + (size_t)j * n;
                    CK(cudaMemcpyAsync(zj, P.U[0][P.ri[0]], sizeof(double) * L.half, cudaMemcpyDeviceToDevice, ctx.s));
                    CK(cudaMemcpyAsync(zj + L.half, P.U[0][P.bi[0]] + L.half, sizeof(double) * L.half,
                                       cudaMemcpyDeviceToDevice, ctx.s));
                    if (sig.opclass == 0)
                        pdl_launch(k_apply<double, KOp<double>, double>, nblk((long long)L.P * L.rows), TPB, 0, ctx.s, 
                            L, ctx.kop64, csplit<double>(zj, L), split<double>(ctx.w, L));
                    else
                        pdl_launch(k_apply<double, ROp<double>, double>, nblk((long long)L.P * L.rows), TPB, 0, ctx.s, 
                            L, ctx.rop64, csplit<double>(zj, L), split<double>(ctx.w, L));
                    CKL();
                }
                vcycles++;
                // CGS2 against v_0..v_j: pass 1 coefficients in hcol[0..j], pass 2 in
                // hcol[m+2 ..]; the Hessenberg column is their sum
                for (int pass = 0; pass < 2; pass++) {
                    double* hp = ctx.hcol + (pass ? m + 2 : 0);
                    pdl_launch(k_multidot, db, TPB, 0, ctx.s, n, j + 1, ctx.Vptr, ctx.w, ctx.dpart);
                    CKL();
                    pdl_launch(k_multidot_finish, j + 1, TPB, 0, ctx.s, j + 1, db, ctx.dpart, hp, 0);
                    CKL();
                    pdl_launch(k_multiaxpy, std::min<unsigned>(nblk(n), 2368), TPB, 0, ctx.s, n, j + 1, ctx.Vptr, hp, ctx.w);
                    CKL();
                }
                // ||w||^2 (Vptr[m+1] points at w) into hcol[j+1]
                pdl_launch(k_multidot, db, TPB, 0, ctx.s, n, 1, ctx.Vptr + m + 1, ctx.w, ctx.dpart);
                CKL();
                pdl_launch(k_multidot_finish, 1, TPB, 0, ctx.s, 1, db, ctx.dpart, ctx.hcol + j + 1, 0);
                CKL();
                CK(cudaMemcpyAsync(ctx.hpin, ctx.hcol, sizeof(double) * (j + 2), cudaMemcpyDeviceToHost, ctx.s));
                CK(cudaMemcpyAsync(ctx.hpin + 256, ctx.hcol + m + 2, sizeof(double) * (j + 1), cudaMemcpyDeviceToHost,
                                   ctx.s));
                CK(cudaStreamSynchronize(ctx.s));
                if (pg) prof_collect_graph(ctx, *pg);
                for (int i = 0; i <= j; i++) HH(i, j) = ctx.hpin[i] + ctx.hpin[256 + i];
                double hn = std::sqrt(std::max(ctx.hpin[j + 1], 0.0));
                if (!(hn <= 1e308)) { inf.status = MPS_ERR_NAN; done = true; break; }
                HH(j + 1, j) = hn;
                ctx.hpin[0] = hn;
                CK(cudaMemcpyAsync(ctx.hcol + j + 1, ctx.hpin, sizeof(double), cudaMemcpyHostToDevice, ctx.s));
                if (hn > 0.0) {
                    pdl_launch(k_scale_to, std::min<unsigned>(nblk(n), 2368), TPB, 0, ctx.s, n, ctx.w, ctx.hcol, j + 1,
                                                                                    ctx.V + (size_t)(j + 1) * n, nullptr);
                    CKL();
                }
                for (int i = 0; i < j; i++) {
                    double t = cs[i] * HH(i, j) + sn[i] * HH(i + 1, j);
                    HH(i + 1, j) = -sn[i] * HH(i, j) + cs[i] * HH(i + 1, j);
                    HH(i, j) = t;
                }
                double a = HH(j, j), b = HH(j + 1, j), rr = std::sqrt(a * a + b * b);
                cs[j] = rr == 0.0 ? 1.0 : a / rr;
                sn[j] = rr == 0.0 ? 0.0 : b / rr;
                HH(j, j) = cs[j] * a + sn[j] * b;
                HH(j + 1, j) = 0.0;
                gq[j + 1] = -sn[j] * gq[j];
                gq[j] = cs[j] * gq[j];
                it++;
                const double est = std::fabs(gq[j + 1]) / (bnorm > 0 ? bnorm : 1.0);
                if ((o->tol_kind == MPS_TOL_REL_L2 && est <= o->tol) || hn == 0.0) { j++; break; }
            }
            if (done) break;
            // y = H^{-1} g ; x += Z y
            for (int i = j - 1; i >= 0; i--) {
                double s = gq[i];
                for (int q = i + 1; q < j; q++) s -= HH(i, q) * y[q];
                y[i] = (HH(i, i) != 0.0) ? s / HH(i, i) : 0.0;
            }
            for (int i = 0; i < j; i++) {
                if (mixed)
                    pdl_launch(k_axpy<float, double>, std::min<unsigned>(nblk(n), 2368), TPB, 0, ctx.s, n, y[i], (float*)ctx.Z + (size_t)i * n, ctx.x64);
                else
                    pdl_launch(k_axpy<double, double>, std::min<unsigned>(nblk(n), 2368), TPB, 0, ctx.s, n, y[i], (double*)ctx.Z + (size_t)i * n, ctx.x64);
                CKL();
            }
        }
    }
    // ---- output ----
    int gst = 0;
    CK(cudaMemcpyAsync(&gst, ctx.dstatus, sizeof(int), cudaMemcpyDeviceToHost, ctx.s));
    pdl_launch(k_unpack<double>, nblk(ncell), TPB, 0, ctx.s, L0, csplit<double>(ctx.x64, L0), in.soln);
    CKL();
    if (o->fill_ghosts) {
        const int mx = std::max(std::max(L0.ny * L0.nz, L0.nx * L0.nz), L0.nx * L0.ny);
        const double* zf[6];
        for (int f = 0; f < 6; f++) zf[f] = in.bcval[f];
        pdl_launch(k_fill_ghosts, nblk(mx), TPB, 0, ctx.s, L0, in.soln, zf[0], zf[1], zf[2], zf[3], zf[4], zf[5]);
        CKL();
    }
    CK(cudaEventRecord(ctx.e1, ctx.s));
    CK(cudaStreamSynchronize(ctx.s));
    float ms = 0.f;
    CK(cudaEventElapsedTime(&ms, ctx.e0, ctx.e1));
    if (ctx.prof.on) {
        prof_collect(ctx);
        ctx.prof.precision_bytes = mixed ? 4 : 8;
        ctx.prof.coeff_field = sig.opclass == 0 ? !sig.kuni && ctx.kseg != 2 : 7;
        ctx.prof.cells = ncell;
    }
    inf.launches = (int)(ctx.launches - launches0);
    inf.iters = it;
    inf.vcycles = vcycles;
    inf.levels = nl;
    inf.rel_res = rel;
    inf.rms_res = rms;
    inf.time_ms = ms;
    if (inf.status == MPS_OK && !ref_norm_only && !conv()) inf.status = MPS_ERR_NOT_CONVERGED;
    (void)gst;
    if (info) *info = inf;
    return inf.status == MPS_ERR_NAN ? MPS_ERR_NAN : 0;
}

}  // namespace mps

#include "mps_batch.cuh"

// ======================================================================
// C ABI
// ======================================================================
using namespace mps;

extern "C" {

void mps_default_opts(mps_solver_opts* o)
{
    if (!o) return;
    std::memset(o, 0, sizeof(*o));
    o->tol = 1e-10;
    o->tol_kind = MPS_TOL_REL_L2;
    o->maxit = 50;
    o->nu1 = 2;
    o->nu2 = 2;
    o->hierarchy = MPS_HIER_GEOM;
    o->ranks[0] = o->ranks[1] = o->ranks[2] = 1;
    o->max_coarse = 125;
    o->precision = MPS_PREC_FP64;
    o->inner_cycles = 0;
    o->krylov = MPS_KRYLOV_NONE;
    o->restart = 30;
    o->fill_ghosts = 0;
    o->use_graph = 1;
    o->transpose = 0;
    o->flux = MPS_FLUX_UPWIND;
}

const char* mps_version(void) { return "mps3d_b200 0.1 (sm_100a)"; }

int mps_create(mps_handle* h, int device)
{
    if (!h) return MPS_ERR_BAD_ARG;
    *h = nullptr;
    mps_handle_s* H = new (std::nothrow) mps_handle_s();
    if (!H) return MPS_ERR_NOMEM;
    Ctx& ctx = H->ctx;
    int dev = device;
    if (dev < 0 && cudaGetDevice(&dev) != cudaSuccess) { delete H; return MPS_ERR_CUDA; }
    if (cudaSetDevice(dev) != cudaSuccess) { delete H; return MPS_ERR_CUDA; }
    ctx.dev = dev;
    // optional cap on the grid-dependent workspace (bytes, per arena), for
    // callers that share the device with other large allocations
    if (const char* cap = std::getenv("MPS_WORKSPACE_LIMIT_BYTES")) {
        const long long v = std::atoll(cap);
        if (v > 0) ctx.ar.limit = ctx.kar.limit = (size_t)v;
    }
    // the shared-memory (TMA) kernels and the register-fed ones give the same
    // results; the variable selects the register-fed ones (for comparisons)
    if (const char* tv = std::getenv("MPS_TMA")) ctx.tma_allowed = std::atoi(tv) != 0;
    // the cluster form of the small levels and the per-level launches
    // solve the same systems; the variable selects the per-level launches
    if (const char* sv = std::getenv("MPS_SUBCYCLE")) ctx.sub_allowed = std::atoi(sv) != 0;
    if (cudaDeviceGetAttribute(&ctx.nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || ctx.nsm < 1) {
        delete H;
        return MPS_ERR_CUDA;
    }
    if (cudaStreamCreateWithFlags(&ctx.s, cudaStreamNonBlocking) != cudaSuccess ||
        cudaEventCreate(&ctx.e0) != cudaSuccess || cudaEventCreate(&ctx.e1) != cudaSuccess ||
        cudaMallocHost((void**)&ctx.hpin, sizeof(double) * 512) != cudaSuccess ||
        cudaMalloc((void**)&ctx.dmax, sizeof(unsigned long long) * DET_WORDS) != cudaSuccess) {
        delete H;
        return MPS_ERR_CUDA;
    }
    *h = H;
    return MPS_OK;
}

int mps_destroy(mps_handle h)
{
    if (!h) return MPS_ERR_BAD_ARG;
    Ctx& ctx = h->ctx;
    cudaSetDevice(ctx.dev);
    cudaStreamSynchronize(ctx.s);
    destroy_batch(ctx);
    destroy_graphs(ctx);
    ctx.ar.clear();
    ctx.kar.clear();
    ctx.inbuf.clear();
    for (auto& ln : ctx.lanes) {
        if (ln.s) cudaStreamSynchronize(ln.s);
        for (int b = 0; b < 2; b++) {
            if (ln.pin[b]) cudaFreeHost(ln.pin[b]);
            if (ln.ev[b]) cudaEventDestroy(ln.ev[b]);
        }
        if (ln.s) cudaStreamDestroy(ln.s);
    }
    ctx.lanes.clear();
    for (cudaEvent_t e : ctx.prof.ev) cudaEventDestroy(e);
    if (ctx.dtab) cudaFree(ctx.dtab);
    if (ctx.dmax) cudaFree(ctx.dmax);
    if (ctx.hpin) cudaFreeHost(ctx.hpin);
    if (ctx.e0) cudaEventDestroy(ctx.e0);
    if (ctx.e1) cudaEventDestroy(ctx.e1);
    if (ctx.s) cudaStreamDestroy(ctx.s);
    delete h;
    return MPS_OK;
}

void* mps_stream(mps_handle h) { return h ? (void*)h->ctx.s : nullptr; }

const char* mps_last_error(mps_handle h) { return h ? h->ctx.err.msg.c_str() : "null handle"; }

static int run_dev(mps_handle h, const mps_grid* g, int timederiv, double dt, const double* vel, const double* dcoeff,
                   const double* reac, const double* source, const int bc_code[6], const double* const bcval[6],
                   const double* sterm, double* soln, const mps_solver_opts* opts, mps_solve_info* info,
                   void* stream, int ref_norm_only)
{
    if (!h || !bc_code) return MPS_ERR_BAD_ARG;
    Ctx& ctx = h->ctx;
    ctx.err = Err();
    if (cudaSetDevice(ctx.dev) != cudaSuccess) return MPS_ERR_CUDA;
    mps_solver_opts o;
    if (opts) o = *opts;
    else mps_default_opts(&o);
    cudaStream_t user = (cudaStream_t)stream;
    cudaEvent_t ev = nullptr;
    if (user && user != ctx.s) {  // order the handle's stream after the caller's
        if (cudaEventCreateWithFlags(&ev, cudaEventDisableTiming) != cudaSuccess) return MPS_ERR_CUDA;
        cudaEventRecord(ev, user);
        cudaStreamWaitEvent(ctx.s, ev, 0);
    }
    Inputs in;
    in.vel = vel; in.dcoeff = dcoeff; in.reac = reac; in.source = source; in.sterm = sterm; in.soln = soln;
    for (int f = 0; f < 6; f++) in.bcval[f] = bcval ? bcval[f] : nullptr;
    int st = solve_impl(ctx, g, timederiv, dt, in, bc_code, &o, info, ref_norm_only);
    if (ev) {
        cudaEventRecord(ev, ctx.s);
        cudaStreamWaitEvent(user, ev, 0);
        cudaEventDestroy(ev);
    }
    if (st && info) info->status = st;
    return st;
}

int mps_linsolve_batched_dev(mps_handle h, int nprob, const mps_problem* probs, const mps_solver_opts* opts,
                             mps_solve_info* infos, void* stream)
{
    if (!h) return MPS_ERR_BAD_ARG;
    Ctx& ctx = h->ctx;
    ctx.err = Err();
    if (nprob < 1 || nprob > MPS_BATCH_MAX || !probs) { ctx.err.msg = "batched: bad problem count"; return MPS_ERR_BAD_ARG; }
    if (cudaSetDevice(ctx.dev) != cudaSuccess) return MPS_ERR_CUDA;
    mps_solver_opts o;
    if (opts) o = *opts;
    else mps_default_opts(&o);
    if (o.krylov != MPS_KRYLOV_NONE || o.transpose || o.flux != MPS_FLUX_UPWIND || o.nu1 < 1 ||
        (o.nu1 + o.nu2) % 2 != 0 || (o.precision != MPS_PREC_MIXED && o.precision != MPS_PREC_FP64)) {
        ctx.err.msg = "batched: stationary iteration only (krylov NONE, upwind, no transpose), nu1 >= 1, nu1+nu2 even";
        return MPS_ERR_BAD_ARG;
    }
    cudaStream_t user = (cudaStream_t)stream;
    cudaEvent_t ev = nullptr;
    if (user && user != ctx.s) {
        if (cudaEventCreateWithFlags(&ev, cudaEventDisableTiming) != cudaSuccess) return MPS_ERR_CUDA;
        cudaEventRecord(ev, user);
        cudaStreamWaitEvent(ctx.s, ev, 0);
    }
    int st = o.precision == MPS_PREC_MIXED ? batched_solve<float>(ctx, nprob, probs, &o, infos)
                                           : batched_solve<double>(ctx, nprob, probs, &o, infos);
    if (ev) {
        cudaEventRecord(ev, ctx.s);
        cudaStreamWaitEvent(user, ev, 0);
        cudaEventDestroy(ev);
    }
    if (st && st != MPS_ERR_NAN) cudaStreamSynchronize(ctx.s);
    return st;
}

int mps_set_profile(mps_handle h, int on)
{
    if (!h) return MPS_ERR_BAD_ARG;
    h->ctx.prof.on = on != 0;
    h->ctx.prof.level = on > 1 ? on - 1 : 0;
    return MPS_OK;
}

int mps_get_profile(mps_handle h, mps_profile* p, int reset)
{
    if (!h || !p) return MPS_ERR_BAD_ARG;
    Prof& P = h->ctx.prof;
    std::memset(p, 0, sizeof(*p));
    for (int c = 0; c < MPS_PROF_NCLASS; c++) { p->count[c] = P.count[c]; p->ms[c] = P.ms[c]; }
    p->precision_bytes = P.precision_bytes;
    p->coeff_field = P.coeff_field;
    p->cells = P.cells;
    if (reset)
        for (int c = 0; c < MPS_PROF_NCLASS; c++) { P.count[c] = 0; P.ms[c] = 0.0; }
    return MPS_OK;
}

int mps_linsolve_dev(mps_handle h, const mps_grid* g, int timederiv, double dt, const double* vel,
                     const double* dcoeff, const double* reac, const double* source, const int bc_code[6],
                     const double* const bcval[6], const double* mgridsterm, double* soln,
                     const mps_solver_opts* opts, mps_solve_info* info, void* stream)
{
    int st = run_dev(h, g, timederiv, dt, vel, dcoeff, reac, source, bc_code, bcval, mgridsterm, soln, opts, info,
                     stream, 0);
    if (st) return st;
    return info ? info->status : MPS_OK;
}

// host-pointer front end: stage the ghosted inputs on the device
// ---- copies between pageable host arrays and the device ----
// A pageable array cannot be read by the DMA engines directly; the driver
// would stage it through its own small pinned buffers one piece at a time.
// Here each of several host threads owns a contiguous part of the array, a
// stream and two pinned chunk buffers: it copies chunk i+1 into one buffer
// (a plain memcpy, in parallel with the other threads) while the DMA engine
// moves chunk i from the other.  Pinned (page-locked or device) arrays go
// straight to cudaMemcpyAsync on the handle's stream.
constexpr size_t kLaneChunk = 1u << 20;  // doubles per chunk buffer (8 MiB)
constexpr int kMaxLanes = 8;

static bool is_pageable(const void* p)
{
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return true;
    }
    return a.type == cudaMemoryTypeUnregistered;
}

static int ensure_lanes(Ctx& ctx)
{
    if (!ctx.lanes.empty()) return 0;
    const unsigned hc = std::thread::hardware_concurrency();
    const int n = std::max(1, std::min<int>(kMaxLanes, hc ? (int)hc / 2 : 4));
    ctx.lanes.resize(n);
    for (auto& ln : ctx.lanes) {
        if (cudaStreamCreateWithFlags(&ln.s, cudaStreamNonBlocking) != cudaSuccess) return MPS_ERR_CUDA;
        for (int b = 0; b < 2; b++) {
            if (cudaMallocHost((void**)&ln.pin[b], sizeof(double) * kLaneChunk) != cudaSuccess) return MPS_ERR_NOMEM;
            if (cudaEventCreateWithFlags(&ln.ev[b], cudaEventDisableTiming) != cudaSuccess) return MPS_ERR_CUDA;
        }
    }
    return 0;
}

struct HostCopy {
    double* dev;        // device array
    double* host;       // pageable host array (const for H2D)
    size_t n;           // doubles
};

// all copies of one direction, each array split across the lanes; the
// handle's stream is ordered after (H2D) or the host waits for (D2H) them
static int staged_copies(Ctx& ctx, const std::vector<HostCopy>& cps, bool h2d)
{
    if (cps.empty()) return 0;
    if (int st = ensure_lanes(ctx)) return st;
    const int nl = (int)ctx.lanes.size();
    if (!h2d) {  // the results must be complete before the lanes read them
        cudaEvent_t e = ctx.e1;
        if (cudaEventRecord(e, ctx.s) != cudaSuccess) return MPS_ERR_CUDA;
        for (auto& ln : ctx.lanes)
            if (cudaStreamWaitEvent(ln.s, e, 0) != cudaSuccess) return MPS_ERR_CUDA;
    }
    std::vector<int> status(nl, 0);
    auto work = [&](int li) {
        Ctx::Lane& ln = ctx.lanes[li];
        int b = 0;
        bool used[2] = {false, false};
        for (const HostCopy& cp : cps) {
            // lane shares start on 4 KiB boundaries of the device array
            const size_t part = ((cp.n + nl - 1) / nl + 511) / 512 * 512;
            const size_t lo = std::min(cp.n, part * li), hi = std::min(cp.n, lo + part);
            for (size_t o = lo; o < hi; o += kLaneChunk) {
                const size_t m = std::min(kLaneChunk, hi - o);
                if (used[b] && cudaEventSynchronize(ln.ev[b]) != cudaSuccess) { status[li] = MPS_ERR_CUDA; return; }
                if (h2d) {
                    std::memcpy(ln.pin[b], cp.host + o, sizeof(double) * m);
                    if (cudaMemcpyAsync(cp.dev + o, ln.pin[b], sizeof(double) * m, cudaMemcpyHostToDevice, ln.s) !=
                        cudaSuccess) { status[li] = MPS_ERR_CUDA; return; }
                    if (cudaEventRecord(ln.ev[b], ln.s) != cudaSuccess) { status[li] = MPS_ERR_CUDA; return; }
                } else {
                    if (cudaMemcpyAsync(ln.pin[b], cp.dev + o, sizeof(double) * m, cudaMemcpyDeviceToHost, ln.s) !=
                            cudaSuccess ||
                        cudaStreamSynchronize(ln.s) != cudaSuccess) { status[li] = MPS_ERR_CUDA; return; }
                    std::memcpy(cp.host + o, ln.pin[b], sizeof(double) * m);
                }
                used[b] = true;
                b ^= 1;
            }
        }
        if (cudaStreamSynchronize(ln.s) != cudaSuccess) status[li] = MPS_ERR_CUDA;
    };
    std::vector<std::thread> th;
    for (int li = 1; li < nl; li++) th.emplace_back(work, li);
    work(0);
    for (auto& t : th) t.join();
    for (int st : status)
        if (st) return st;
    return 0;
}

static int run_host(mps_handle h, const mps_grid* g, int timederiv, double dt, const double* vel,
                    const double* dcoeff, const double* reac, const double* source, const int bc_code[6],
                    const double* const bcval[6], const double* mgridsterm, double* soln,
                    const mps_solver_opts* opts, mps_solve_info* info, int ref_norm_only)
{
    if (!h || !g || !dcoeff || !source || !soln || !bc_code) return MPS_ERR_BAD_ARG;
    if (g->lx < 1 || g->ly < 1 || g->lz < 1) return MPS_ERR_BAD_ARG;
    Ctx& ctx = h->ctx;
    if (cudaSetDevice(ctx.dev) != cudaSuccess) return MPS_ERR_CUDA;
    const size_t ng = (size_t)(g->lx + 2) * (g->ly + 2) * (g->lz + 2);
    const size_t ni = (size_t)g->lx * g->ly * g->lz;
    const size_t fs[6] = {(size_t)g->ly * g->lz, (size_t)g->ly * g->lz, (size_t)g->lx * g->lz,
                          (size_t)g->lx * g->lz, (size_t)g->lx * g->ly, (size_t)g->lx * g->ly};
    // one device block for the staged inputs, every field starting on a
    // 4 KiB boundary (copies into 8-byte aligned destinations ran at 37-40
    // GB/s over the host link, aligned ones at 55 GB/s)
    auto al = [](size_t n) { return (n * sizeof(double) + 4095) / 4096 * 4096 / sizeof(double); };
    size_t need = al(3 * ng) + 4 * al(ng) + al(ni) + al(fs[0] * 2 + fs[2] * 2 + fs[4] * 2);
    need *= sizeof(double);
    if (ctx.inbuf_bytes < need) {
        ctx.inbuf.clear();
        ctx.inbuf_bytes = 0;
        if (!ctx.inbuf.get(need)) return MPS_ERR_NOMEM;
        if (cudaDeviceSynchronize() != cudaSuccess) return MPS_ERR_CUDA;
        ctx.inbuf_bytes = need;
    }
    double* base = (double*)ctx.inbuf.blocks[0];
    double* d_vel = base;
    double* d_dc = d_vel + al(3 * ng);
    double* d_re = d_dc + al(ng);
    double* d_src = d_re + al(ng);
    double* d_sol = d_src + al(ng);
    double* d_st = d_sol + al(ng);
    double* d_bc = d_st + al(ni);
    const double* dbv[6];
    cudaStream_t s = ctx.s;
    // pinned (or device) arrays: one cudaMemcpyAsync each on the handle's
    // stream; pageable arrays: the staged, multi-threaded copies above
    std::vector<HostCopy> staged;
    auto h2d = [&](double* dst, const double* src, size_t n) -> int {
        if (is_pageable(src)) {
            staged.push_back({dst, const_cast<double*>(src), n});
            return 0;
        }
        return cudaMemcpyAsync(dst, src, sizeof(double) * n, cudaMemcpyHostToDevice, s) == cudaSuccess ? 0
                                                                                                       : MPS_ERR_CUDA;
    };
    int st = 0;
    if (vel && (st = h2d(d_vel, vel, 3 * ng))) return st;
    if ((st = h2d(d_dc, dcoeff, ng))) return st;
    if (reac && (st = h2d(d_re, reac, ng))) return st;
    if ((st = h2d(d_src, source, ng))) return st;
    if ((st = h2d(d_sol, soln, ng))) return st;
    if (mgridsterm && (st = h2d(d_st, mgridsterm, ni))) return st;
    double* p = d_bc;
    for (int f = 0; f < 6; f++) {
        dbv[f] = nullptr;
        if (bcval && bcval[f]) {
            if ((st = h2d(p, bcval[f], fs[f]))) return st;
            dbv[f] = p;
        }
        p += fs[f];
    }
    if ((st = staged_copies(ctx, staged, true))) return st;  // complete when it returns
    st = run_dev(h, g, timederiv, dt, vel ? d_vel : nullptr, d_dc, reac ? d_re : nullptr, d_src, bc_code, dbv,
                 mgridsterm ? d_st : nullptr, d_sol, opts, info, nullptr, ref_norm_only);
    if (st) return st;
    if (is_pageable(soln)) {
        if ((st = staged_copies(ctx, {HostCopy{d_sol, soln, ng}}, false))) return st;
    } else {
        if (cudaMemcpyAsync(soln, d_sol, sizeof(double) * ng, cudaMemcpyDeviceToHost, s) != cudaSuccess)
            return MPS_ERR_CUDA;
        if (cudaStreamSynchronize(s) != cudaSuccess) return MPS_ERR_CUDA;
    }
    return info ? info->status : MPS_OK;
}

int mps_linsolve(mps_handle h, const mps_grid* g, int timederiv, double dt, const double* vel, const double* dcoeff,
                 const double* reac, const double* source, const int bc_code[6], const double* const bcval[6],
                 const double* mgridsterm, double* soln, const mps_solver_opts* opts, mps_solve_info* info)
{
    return run_host(h, g, timederiv, dt, vel, dcoeff, reac, source, bc_code, bcval, mgridsterm, soln, opts, info, 0);
}

int mps_vcycle_once(mps_handle h, const mps_grid* g, int timederiv, double dt, const double* vel,
                    const double* dcoeff, const double* reac, const double* source, const int bc_code[6],
                    const double* const bcval[6], const double* mgridsterm, double* soln, double* resnorm,
                    const mps_solver_opts* opts)
{
    mps_solver_opts o;
    if (opts) o = *opts;
    else {
        mps_default_opts(&o);
        o.hierarchy = MPS_HIER_CELL;
    }
    o.maxit = 1;
    o.krylov = MPS_KRYLOV_NONE;
    o.precision = MPS_PREC_FP64;
    mps_solve_info info;
    int st = run_host(h, g, timederiv, dt, vel, dcoeff, reac, source, bc_code, bcval, mgridsterm, soln, &o, &info, 1);
    if (resnorm) *resnorm = info.rms_res;
    return st;
}

int mps_apply_A_dev(mps_handle h, const mps_grid* g, int timederiv, double dt, const double* vel,
                    const double* dcoeff, const double* reac, const int bc_code[6], const double* soln, double* AX,
                    const mps_solver_opts* opts, void* stream)
{
    if (!h || !g || !dcoeff || !soln || !AX || !bc_code) return MPS_ERR_BAD_ARG;
    Ctx& ctx = h->ctx;
    ctx.err = Err();
    if (cudaSetDevice(ctx.dev) != cudaSuccess) return MPS_ERR_CUDA;
    mps_solver_opts o;
    if (opts) o = *opts;
    else mps_default_opts(&o);
    // A u through the same operator setup as a solve: run a zero-iteration
    // solve to build the fine operator, then apply it
    o.maxit = 0;
    o.krylov = MPS_KRYLOV_NONE;
    o.precision = MPS_PREC_FP64;
    o.hierarchy = MPS_HIER_GEOM;
    const size_t ng = (size_t)(g->lx + 2) * (g->ly + 2) * (g->lz + 2);
    double* tmp = nullptr;
    double* zsrc = nullptr;
    cudaStream_t s = ctx.s;
    cudaStream_t user = (cudaStream_t)stream;
    if (user && user != s) {  // soln is read below, before the solve orders the streams
        cudaEvent_t ev = nullptr;
        if (cudaEventCreateWithFlags(&ev, cudaEventDisableTiming) != cudaSuccess) return MPS_ERR_CUDA;
        cudaEventRecord(ev, user);
        cudaStreamWaitEvent(s, ev, 0);
        cudaEventDestroy(ev);
    }
    if (cudaMallocAsync((void**)&tmp, sizeof(double) * ng * 2, s) != cudaSuccess) return MPS_ERR_CUDA;
    zsrc = tmp + ng;
    cudaMemcpyAsync(tmp, soln, sizeof(double) * ng, cudaMemcpyDeviceToDevice, s);
    cudaMemsetAsync(zsrc, 0, sizeof(double) * ng, s);
    int bcfix[6];
    for (int f = 0; f < 6; f++) bcfix[f] = bc_code[f];
    mps_solve_info info;
    // DIRC/FLUX faces need value arrays for find_bvec; they do not enter A
    int st = MPS_OK;
    std::vector<double*> fb;
    const double* bv[6] = {nullptr, nullptr, nullptr, nullptr, nullptr, nullptr};
    for (int f = 0; f < 6 && st == MPS_OK; f++) {
        if (bc_code[f] == BC_DIRC || bc_code[f] == BC_FLUX) {
            size_t n = (f < 2) ? (size_t)g->ly * g->lz : (f < 4 ? (size_t)g->lx * g->lz : (size_t)g->lx * g->ly);
            double* d = nullptr;
            if (cudaMallocAsync((void**)&d, sizeof(double) * n, s) != cudaSuccess) {
                st = MPS_ERR_CUDA;
                break;
            }
            cudaMemsetAsync(d, 0, sizeof(double) * n, s);
            fb.push_back(d);
            bv[f] = d;
        }
    }
    if (st == MPS_OK)
        st = run_dev(h, g, timederiv, dt, vel, dcoeff, reac, zsrc, bcfix, bv, nullptr, tmp, &o, &info, stream, 1);
    if (st == MPS_OK) {
        const Lev& L = ctx.lev[0];
        double* out = nullptr;
        if (cudaMallocAsync((void**)&out, sizeof(double) * 2 * L.half, s) != cudaSuccess) {
            st = MPS_ERR_CUDA;
        } else {
            if (ctx.sig.opclass == 0)
                k_apply<double, KOp<double>, double><<<nblk((long long)L.P * L.rows), TPB, 0, s>>>(
                    L, ctx.kop64, csplit<double>(ctx.x64, L), split<double>(out, L));
            else
                k_apply<double, ROp<double>, double><<<nblk((long long)L.P * L.rows), TPB, 0, s>>>(
                    L, ctx.rop64, csplit<double>(ctx.x64, L), split<double>(out, L));
            k_unpack_nat<double><<<nblk((long long)L.nx * L.ny * L.nz), TPB, 0, s>>>(L, csplit<double>(out, L), AX);
            cudaFreeAsync(out, s);
            if (cudaGetLastError() != cudaSuccess) st = MPS_ERR_CUDA;
        }
    }
    // every exit path frees what this call allocated and waits for the stream
    for (double* d : fb) cudaFreeAsync(d, s);
    cudaFreeAsync(tmp, s);
    if (cudaStreamSynchronize(s) != cudaSuccess && st == MPS_OK) st = MPS_ERR_CUDA;
    return st;
}

int mps_find_bvec_dev(mps_handle h, const mps_grid* g, const double* vel, const double* dcoeff,
                      const double* source, const int bc_code[6], const double* const bcval[6],
                      const double* mgridsterm, double* b, const mps_solver_opts* opts, void* stream)
{
    if (!h || !g || !dcoeff || !source || !b || !bc_code) return MPS_ERR_BAD_ARG;
    Ctx& ctx = h->ctx;
    if (cudaSetDevice(ctx.dev) != cudaSuccess) return MPS_ERR_CUDA;
    for (int f = 0; f < 6; f++)
        if (bc_code[f] < 1 || bc_code[f] > 5 || (!(bcval && bcval[f]) && (bc_code[f] == BC_DIRC || bc_code[f] == BC_FLUX)))
            return MPS_ERR_BAD_ARG;
    const double llen[3] = {g->llenx, g->lleny, g->llenz};
    Lev L = make_lev_uniform(g->lx, g->ly, g->lz, llen, bc_code);
    cudaStream_t s = stream ? (cudaStream_t)stream : ctx.s;
    double* buf = nullptr;
    if (cudaMallocAsync((void**)&buf, sizeof(double) * 2 * L.half, s) != cudaSuccess) return MPS_ERR_CUDA;
    cudaMemsetAsync(buf, 0, sizeof(double) * 2 * L.half, s);
    const long long n = (long long)L.nx * L.ny * L.nz;
    k_find_bvec<<<nblk(n), TPB, 0, s>>>(L, vel, dcoeff, source, bcval[0], bcval[1], bcval[2], bcval[3], bcval[4],
                                        bcval[5], mgridsterm, opts ? opts->flux : 0, split<double>(buf, L));
    k_unpack_nat<double><<<nblk(n), TPB, 0, s>>>(L, csplit<double>(buf, L), b);
    cudaFreeAsync(buf, s);
    if (cudaGetLastError() != cudaSuccess) return MPS_ERR_CUDA;
    if (cudaStreamSynchronize(s) != cudaSuccess) return MPS_ERR_CUDA;
    return MPS_OK;
}

int mps_fill_ghosts_dev(mps_handle h, const mps_grid* g, const int bc_code[6], const double* const bcval[6],
                        double* soln, void* stream)
{
    if (!h || !g || !soln || !bc_code) return MPS_ERR_BAD_ARG;
    Ctx& ctx = h->ctx;
    if (cudaSetDevice(ctx.dev) != cudaSuccess) return MPS_ERR_CUDA;
    for (int f = 0; f < 6; f++)
        if (bc_code[f] < 1 || bc_code[f] > 5 || (!(bcval && bcval[f]) && bc_code[f] == BC_DIRC)) return MPS_ERR_BAD_ARG;
    const double llen[3] = {g->llenx, g->lleny, g->llenz};
    Lev L = make_lev_uniform(g->lx, g->ly, g->lz, llen, bc_code);
    cudaStream_t s = stream ? (cudaStream_t)stream : ctx.s;
    const int mx = std::max(std::max(L.ny * L.nz, L.nx * L.nz), L.nx * L.ny);
    k_fill_ghosts<<<nblk(mx), TPB, 0, s>>>(L, soln, bcval ? bcval[0] : nullptr, bcval ? bcval[1] : nullptr,
                                           bcval ? bcval[2] : nullptr, bcval ? bcval[3] : nullptr,
                                           bcval ? bcval[4] : nullptr, bcval ? bcval[5] : nullptr);
    if (cudaGetLastError() != cudaSuccess) return MPS_ERR_CUDA;
    if (cudaStreamSynchronize(s) != cudaSuccess) return MPS_ERR_CUDA;
    return MPS_OK;
}

}  // extern "C"
