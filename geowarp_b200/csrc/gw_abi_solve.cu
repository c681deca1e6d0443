// C ABI, Krylov solvers: BiCGSTAB / CG, restarted GMRES, multigrid-
// preconditioned flexible GMRES, the workspace-free Krylov entry point and
// SpMV (declarations and reference citations in include/geowarp_b200.h).
#include <limits.h>

#include <algorithm>
#include <memory>
#include <mutex>
#include <type_traits>
#include <vector>

#include "gw_host.cuh"
#include "gw_mg.cuh"
#include "gw_mg_tail.cuh"

using namespace gw;
using namespace gwh;

namespace {
struct KWs {
    double *r, *rh, *p, *v, *y, *s, *z, *t, *Minv, *partials;
    KScalars *sc;
};

int64_t krylov_ws_bytes(int64_t n_rows, int nf) {
    const int64_t n = n_rows * nf;
    return 8 * align256(8 * n) + align256(8 * n_rows * nf * nf) + align256(8 * (int64_t)kRedBlocks * 4) +
           align256(sizeof(KScalars));
}

KWs carve(void *ws, int64_t n_rows, int nf) {
    const int64_t n = n_rows * nf;
    char *w = (char *)ws;
    KWs k;
    double **vecs[8] = {&k.r, &k.rh, &k.p, &k.v, &k.y, &k.s, &k.z, &k.t};
    for (int i = 0; i < 8; ++i) { *vecs[i] = (double *)w; w += align256(8 * n); }
    k.Minv = (double *)w; w += align256(8 * n_rows * nf * nf);
    k.partials = (double *)w; w += align256(8 * (int64_t)kRedBlocks * 4);
    k.sc = (KScalars *)w;
    return k;
}

template <int NF, typename VT>
int krylov(const gw_bsr_t *A, int method, int precond, const double *b, double *x, double rtol, int max_iter, void *ws,
           int *iters, double *relres, cudaStream_t s) {
    PtrsA a = make_ptrs(*A);
    KWs k = carve(ws, A->n_rows, NF);
    const int D = (A->mask_words == 1) ? 2 : 3;
    const int nr = A->n_rows;
    if (nr == 0) { *iters = 0; *relres = 0.0; return GW_OK; }
    BicgVecs V;
    V.x = x; V.b = b; V.r = k.r; V.rh = k.rh; V.p = k.p; V.v = k.v; V.y = k.y; V.s = k.s; V.z = k.z; V.t = k.t;
    V.Minv = k.Minv; V.partials = k.partials; V.sc = k.sc;
    GW_CUDA(cudaMemsetAsync(k.sc, 0, sizeof(KScalars), s));
    KScalars h;
    memset(&h, 0, sizeof(h));
    h.max_iter = max_iter;
    GW_CUDA(cudaMemcpyAsync(&k.sc->max_iter, &h.max_iter, sizeof(int), cudaMemcpyHostToDevice, s));
    k_precond_setup<NF, VT><<<gw_count_launch(nblk(nr, kThreads)), kThreads, 0, s>>>(a, D, precond, k.Minv);
    GW_LAUNCHED();
    const int gw_rows = red_grid_rows(nr), ge_rows = red_grid_elems(nr);
    if (method == GW_KRYLOV_CG) k_cg_init<NF, VT><<<gw_count_launch(gw_rows), kThreads, 0, s>>>(a, V, rtol);
    else k_bicg_init<NF, VT><<<gw_count_launch(gw_rows), kThreads, 0, s>>>(a, V, rtol);
    GW_LAUNCHED();
    int chunk = 2;
    for (;;) {
        GW_CUDA(cudaMemcpyAsync(&h, k.sc, sizeof(KScalars), cudaMemcpyDeviceToHost, s));
        GW_CUDA(cudaStreamSynchronize(s));
        if (h.done) break;
        for (int it = 0; it < chunk; ++it) {
            if (method == GW_KRYLOV_CG) {
                k_cg_p<NF><<<gw_count_launch(red_grid_elems((int64_t)nr * NF)), kThreads, 0, s>>>(nr, V);
                k_cg_q<NF, VT><<<gw_count_launch(gw_rows), kThreads, 0, s>>>(a, V);
                k_cg_xr<NF><<<gw_count_launch(ge_rows), kThreads, 0, s>>>(nr, V);
            } else {
                k_bicg_p<NF><<<gw_count_launch(ge_rows), kThreads, 0, s>>>(nr, V);
                k_bicg_v<NF, VT><<<gw_count_launch(gw_rows), kThreads, 0, s>>>(a, V);
                k_bicg_s<NF><<<gw_count_launch(ge_rows), kThreads, 0, s>>>(nr, V);
                k_bicg_t<NF, VT><<<gw_count_launch(gw_rows), kThreads, 0, s>>>(a, V);
                k_bicg_xr<NF><<<gw_count_launch(ge_rows), kThreads, 0, s>>>(nr, V);
            }
        }
        GW_LAUNCHED();
        chunk = chunk < 64 ? chunk * 2 : 64;
    }
    *iters = h.iters;
    *relres = (h.bb > 0.0) ? ::sqrt(h.rr / h.bb) : 0.0;
    const int gc = guard_check(s, "Krylov");
    if (gc) return gc;
    if (h.status == ST_BREAKDOWN) return GW_EBREAKDOWN;
    if (h.status == ST_NAN) return GW_ENAN;
    if (h.rr > h.tol2) return GW_ENOCONV;
    return GW_OK;
}

template <typename VT>
int krylov_nf(const gw_bsr_t *A, int method, int precond, const double *b, double *x, double rtol, int max_iter,
              void *ws, int *iters, double *relres, cudaStream_t s) {
    switch (A->nf) {
        case 1: return krylov<1, VT>(A, method, precond, b, x, rtol, max_iter, ws, iters, relres, s);
        case 2: return krylov<2, VT>(A, method, precond, b, x, rtol, max_iter, ws, iters, relres, s);
        case 3: return krylov<3, VT>(A, method, precond, b, x, rtol, max_iter, ws, iters, relres, s);
        case 4: return krylov<4, VT>(A, method, precond, b, x, rtol, max_iter, ws, iters, relres, s);
        default: return GW_EINVAL;
    }
}
}  // namespace

namespace {
// block partials of a GMRES solve: the Gram-Schmidt items, or two values per block of k_gm_residual
constexpr int kGmresPartials = kGsPartials > 2 * kRedBlocks ? kGsPartials : 2 * kRedBlocks;
// second Gram-Schmidt passes of the last GMRES solve on this host thread
thread_local int g_last_reorths = 0;
// whether the last GMRES solve on this host thread stopped on stagnation
thread_local int g_last_stalled = 0;

// Restarted GMRES can stagnate for good: the true residual at each cycle start
// stops falling (a preconditioned operator whose field of values contains
// zero, or a preconditioner too weak for the accuracy asked).  A solve whose
// residual fell by less than 10% over the last GW_TUNE_GMRES_STALL restart
// cycles stops there, and returns GW_ENOCONV, instead of running on to
// max_iter: at that rate 650 more cycles would gain less than a factor 4.
// 0 turns the check off.
class StallWatch {
  public:
    StallWatch() : window_(g_tune[GW_TUNE_GMRES_STALL]) {}
    // beta: the true residual norm at the start of a restart cycle
    bool stalled(double beta) {
        if (window_ <= 0) return false;
        hist_.push_back(beta);
        const size_t n = hist_.size();
        return n > (size_t)window_ && beta > 0.9 * hist_[n - 1 - window_];
    }

  private:
    int window_;
    std::vector<double> hist_;
};

// Launches one kernel of the Arnoldi step with programmatic dependent launch.
template <typename... KA, typename... A>
void launch_pdl(void (*k)(KA...), int grid, int block, size_t smem, cudaStream_t s, A... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(gw_count_launch(grid));
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    (void)cudaLaunchKernelEx(&cfg, k, KA(args)...);  // checked by the caller's GW_LAUNCHED / end of capture
}

// The Gram-Schmidt kernels of one column: both passes, or the first one alone.
void gs_dots(const GmresVecs &G, int restart, int pass, cudaStream_t s) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(gw_count_launch(gs_dots_blocks(G.n)), (restart + 1 + kGsGroup - 1) / kGsGroup);
    cfg.blockDim = dim3(kGsThreads);
    cfg.stream = s;
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    (void)cudaLaunchKernelEx(&cfg, k_gm_dots, G, pass);
}
void gs_update(const GmresVecs &G, int pass, cudaStream_t s) {
    launch_pdl(k_gm_update, gs_update_blocks(G.n), kGsThreads, 0, s, G, pass);
}
template <int NF>
void gs_next(int n_rows, const GmresVecs &G, int start, const double *Minv, double *zout, double scale, cudaStream_t s) {
    // block 0 closes the column, the others take one row per thread
    launch_pdl(k_gm_next<NF>, 1 + nblk(n_rows, kGsThreads), kGsThreads, 0, s, n_rows, G, start, Minv, zout, scale);
}

// Profiling only: whether column k takes the second Gram-Schmidt pass (read
// after pass 0), so that the timed launches queue it where it is needed.  Runs
// without profiling never read it.
int prof_reorth(GScalars *sc, cudaStream_t s) {
    int re = 1;
    if (cudaMemcpyAsync(&re, &sc->reorth, sizeof(int), cudaMemcpyDeviceToHost, s) != cudaSuccess) return 1;
    if (cudaStreamSynchronize(s) != cudaSuccess) return 1;
    return re;
}

// The Gram-Schmidt kernels of a column; profiled runs queue the second pass only
// where the column takes it.
void gs_column(const GmresVecs &G, int restart, double vb, cudaStream_t s) {
    const double n8 = 8.0 * G.n;
    { ProfScope ps(PC_DOTS, s, vb + n8); gs_dots(G, restart, 0, s); }
    { ProfScope ps(PC_UPDATE, s, vb + n8); gs_update(G, 0, s); }
    if (g_prof_on && !prof_reorth(G.sc, s)) return;
    { ProfScope ps(PC_DOTS, s, vb); gs_dots(G, restart, 1, s); }
    { ProfScope ps(PC_UPDATE, s, vb + n8); gs_update(G, 1, s); }
}
// An instantiated graph and the launches it replays.
struct StepGraph {
    cudaGraphExec_t exec = nullptr;
    int64_t launches = 0;
    StepGraph() = default;
    StepGraph(const StepGraph &) = delete;
    ~StepGraph() { if (exec) cudaGraphExecDestroy(exec); }
    int replay(cudaStream_t s) const {
        GW_CUDA(cudaGraphLaunch(exec, s));
        g_launches += launches;
        return GW_OK;
    }
};

// Graph of the launches that record(stream) makes.  The solvers' captures share one
// stream per device, so one host thread records at a time.
std::mutex g_capture_mu;
cudaStream_t g_capture_stream[64] = {};

template <typename F>
int capture_graph(F record, StepGraph *g) {
    int dev = 0;
    GW_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return GW_EINVAL;
    cudaGraph_t graph;
    {
        std::lock_guard<std::mutex> lk(g_capture_mu);
        cudaStream_t &cs = g_capture_stream[dev];
        if (!cs) GW_CUDA(cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking));
        GW_CUDA(cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal));
        t_captured = &g->launches;
        record(cs);
        t_captured = nullptr;
        GW_CUDA(cudaStreamEndCapture(cs, &graph));
    }
    const cudaError_t ie = cudaGraphInstantiate(&g->exec, graph, 0);
    cudaGraphDestroy(graph);
    GW_CUDA(ie);
    return GW_OK;
}

int64_t gmres_ws_bytes(int64_t n_rows, int nf, int restart) {
    const int64_t n = n_rows * nf;
    return align256(8 * n * (restart + 1)) + 2 * align256(8 * n) + align256(8 * n_rows * nf * nf) +
           align256(8 * (int64_t)kGmresPartials) + align256(sizeof(GScalars));
}

template <int NF, typename VT>
int gmres(const gw_bsr_t *A, int precond, const double *b, double *x, double rtol, int max_iter, int restart,
          void *ws, int *iters, double *relres, cudaStream_t s) {
    PtrsA a = make_ptrs(*A);
    const int nr = A->n_rows;
    if (nr == 0) { *iters = 0; *relres = 0.0; return GW_OK; }
    const int64_t n = (int64_t)nr * NF;
    char *w = (char *)ws;
    GmresVecs G;
    G.V = (double *)w; w += align256(8 * n * (restart + 1));
    G.w = (double *)w; w += align256(8 * n);
    G.z = (double *)w; w += align256(8 * n);
    G.Minv = (double *)w; w += align256(8 * (int64_t)nr * NF * NF);
    G.partials = (double *)w; w += align256(8 * (int64_t)kGmresPartials);
    G.sc = (GScalars *)w;
    G.x = x; G.b = b; G.n = (size_t)n;
    const size_t head = offsetof(GScalars, H);
    k_gm_begin<<<gw_count_launch(1), 32, 0, s>>>(G.sc, max_iter, restart, ::pow(10.0, -0.1 * g_tune[GW_TUNE_GS_CANCEL]));
    const int D = (A->mask_words == 1) ? 2 : 3;
    k_precond_setup<NF, VT><<<gw_count_launch(nblk(nr, kThreads)), kThreads, 0, s>>>(a, D, precond, G.Minv);
    GW_LAUNCHED();
    const int gr = red_grid_rows(nr), ge = red_grid_elems(nr);
    // A warp per row where the rows alone do not fill the device and are long enough
    // for it (below 16 blocks most of its lanes would idle).  A solve of 24 columns with
    // eight lanes per row -> a warp: 1,000 rows of 125 blocks 4 x 4 FP64 987 -> 622 us, 4,096
    // rows of 27 649 -> 617, 3,600 of 25 2 x 2 522 -> 477, of 9 499 -> 482; FP32 4 x 4 rows of
    // 27: 4,096 602 -> 591, 8,000 646 -> 690, 13,824 742 -> 861 (FP64 there 982 -> 910).
    const bool wide = nr <= 8192 && (int64_t)A->nnzb >= 16 * (int64_t)nr;
    GScalars h;
    memset(&h, 0, head);
    int first = 1;
    StallWatch stall;
    g_last_stalled = 0;
    StepGraph step;  // kStepCols columns, for this solve only
    constexpr int kStepCols = 8, kStepFrom = 24;
    int queued = 0;  // columns of this solve so far
    for (int cycle = 0; cycle < 1000000; ++cycle) {
        k_gm_residual<NF, VT><<<gw_count_launch(gr), kThreads, 0, s>>>(a, G, first, rtol);
        gs_next<NF>(nr, G, 1, G.Minv, G.z, 1.0, s);
        GW_LAUNCHED();
        first = 0;
        GW_CUDA(cudaMemcpyAsync(&h, G.sc, head, cudaMemcpyDeviceToHost, s));
        GW_CUDA(cudaStreamSynchronize(s));
        if (h.done) break;
        if (stall.stalled(h.beta)) { g_last_stalled = 1; break; }
        int chunk = 8;
        int kk = 0;  // columns queued in this cycle: at most `restart` of them can count
        const double spmv_bytes = (double)A->nnzb * (NF * NF * sizeof(VT) + 4) + 4.0 * (nr + 1) + 16.0 * n;
        auto column = [&](cudaStream_t st) {
            {
                ProfScope ps(PC_SPMV, st, spmv_bytes);
                if (wide) launch_pdl(k_gm_spmv_wide<NF, VT>, nblk(nr, 4), 128, 0, st, a, G);
                else launch_pdl(k_gm_spmv<NF, VT>, gr, kThreads, 0, st, a, G);
            }
            gs_column(G, restart, 8.0 * n * (kk + 2), st);
            ProfScope ps(PC_NEXT, st, 8.0 * n * 3 + 8.0 * nr * NF * NF);
            gs_next<NF>(nr, G, 0, G.Minv, G.z, 1.0, st);
        };
        for (;;) {
            chunk = std::min(chunk, restart - kk);
            int it = 0;
            if (!g_prof_on && (step.exec || queued >= kStepFrom)) {
                // A long solve replays eight columns at a time: six launches of 2-3 us of
                // work each cost the host 20 us.  Recording them costs 140-250 us a solve, so
                // a solve of up to 24 columns launches its kernels.  4,096 rows of 4 x 4 FP64
                // blocks, recorded after 8 columns -> after 24: 9 columns 727 -> 501 us, 24
                // columns 840 -> 606, 25 columns 1,166 -> 1,187, 100 columns 3,260 -> 3,270
                // (the former kernels, no column recorded: 547, 1,267, 1,301, 5,820).
                if (!step.exec && chunk >= kStepCols) {
                    auto columns = [&](cudaStream_t cs) {
                        for (int q = 0; q < kStepCols; ++q) column(cs);
                    };
                    const int rc = capture_graph(columns, &step);
                    if (rc) return rc;
                }
                for (; step.exec && it + kStepCols <= chunk; it += kStepCols, kk += kStepCols, queued += kStepCols) {
                    const int rc = step.replay(s);
                    if (rc) return rc;
                }
            }
            for (; it < chunk; ++it, ++kk, ++queued) column(s);
            GW_LAUNCHED();
            GW_CUDA(cudaMemcpyAsync(&h, G.sc, head, cudaMemcpyDeviceToHost, s));
            GW_CUDA(cudaStreamSynchronize(s));
            if (h.cycle_done || kk >= restart) break;
            chunk = chunk < 32 ? chunk * 2 : 32;
        }
        if (h.status) break;
        k_gm_solve_y<<<gw_count_launch(1), 32, 0, s>>>(G.sc);
        k_gm_update_x<NF><<<gw_count_launch(ge), kThreads, 0, s>>>(nr, G);
        GW_LAUNCHED();
    }
    *iters = h.iters;
    g_last_reorths = h.reorths;
    *relres = (h.bnorm > 0.0) ? h.resid / h.bnorm : 0.0;
    // the header carries the guard of every kernel up to the last residual
    const int gc = (h.guard || h.status) ? guard_check(s, "GMRES") : GW_OK;
    if (gc) return gc;
    if (h.status == ST_NAN) return GW_ENAN;
    if (h.resid > h.tol) return GW_ENOCONV;
    return GW_OK;
}

template <typename VT>
int gmres_nf(const gw_bsr_t *A, int precond, const double *b, double *x, double rtol, int max_iter, int restart,
             void *ws, int *iters, double *relres, cudaStream_t s) {
    switch (A->nf) {
        case 1: return gmres<1, VT>(A, precond, b, x, rtol, max_iter, restart, ws, iters, relres, s);
        case 2: return gmres<2, VT>(A, precond, b, x, rtol, max_iter, restart, ws, iters, relres, s);
        case 3: return gmres<3, VT>(A, precond, b, x, rtol, max_iter, restart, ws, iters, relres, s);
        case 4: return gmres<4, VT>(A, precond, b, x, rtol, max_iter, restart, ws, iters, relres, s);
        default: return GW_EINVAL;
    }
}
}  // namespace

extern "C" int64_t gw_gmres_workspace_bytes(int32_t n_rows, int32_t nf, int32_t restart) {
    if (restart < 1 || restart > kGmresMaxRestart) return -1;
    return gmres_ws_bytes(n_rows, nf, restart);
}

extern "C" int gw_bsr_gmres_solve(const gw_bsr_t *A, int32_t prec, int32_t precond, const double *b, double *x,
                                  double rtol, int32_t max_iter, int32_t restart, void *workspace, int32_t *iters_host,
                                  double *relres_host, void *stream) {
    GW_REQUIRE(A && b && x && workspace && iters_host && relres_host && max_iter > 0);
    GW_REQUIRE(vec_ok(A, b, x));
    GW_REQUIRE(restart >= 1 && restart <= kGmresMaxRestart);
    int it = 0;
    double rr = 0.0;
    int rc = (prec == GW_PREC_F64)
                 ? gmres_nf<double>(A, precond, b, x, rtol, max_iter, restart, workspace, &it, &rr, S(stream))
                 : gmres_nf<float>(A, precond, b, x, rtol, max_iter, restart, workspace, &it, &rr, S(stream));
    *iters_host = it;
    *relres_host = rr;
    return rc;
}

// ==================================================================== multigrid-preconditioned flexible GMRES
namespace {
// damping of the block-Jacobi smoother (GW_TUNE_MG_OMEGA, in percent)
inline double mg_omega() { return 0.01 * g_tune[GW_TUNE_MG_OMEGA]; }
// smoothing sweeps before / after the coarse correction: two, or one from
// level GW_TUNE_MG_ONE_SWEEP down (fewer launches on the latency-bound coarse
// levels against more Krylov iterations; the autotuner weighs the two)
inline int mg_sweeps(int l) {
    if (l == 0) return g_tune[GW_TUNE_MG_FINE_SWEEPS];
    return l >= g_tune[GW_TUNE_MG_ONE_SWEEP] ? 1 : g_tune[GW_TUNE_MG_SWEEPS];
}

// Bump allocator over the caller's workspace; with p == nullptr it only counts,
// so sizing and carving run the same code.
struct Bump {
    char *p;
    int64_t used;
    void *take(int64_t b) {
        b = align256(b);
        void *r = p ? (void *)(p + used) : nullptr;
        used += b;
        return r;
    }
};

struct MgLevel {
    gw_grid_t g;
    Lat L;
    gw_bsr_t A;             // level 0: the caller's matrix; coarse levels: FP64 in the workspace
    double *Minv, *b, *x, *x2, *r;
    uint8_t *fixed;
    int *tmp, *sws, *blockrow;
    int *child;             // coarse levels: fine rows of the 3^D children of each row (pattern phase)
    int *parent;            // levels with a coarser one: coarse rows of the 2^D parents of each row
    void *pvals;            // level 0: BF16 copy of the fine Jacobian read by the V-cycle (mixed);
                            // in 2D past the FP32 values in svals, which has room for FP64
    uint8_t *flags;
    // 2D: the sliced layout (gw_sell.cuh) of this level's matrix
    int *scols, *strips;
    void *svals;
};
struct MgHier {
    int nl = 0;             // levels holding a matrix; the last one is solved with a dense inverse
    MgLevel lv[kMgMaxLevels];
    double *dM = nullptr, *dInv = nullptr;
    int dn = 0;
    int *counts = nullptr;  // pattern phase: row and block counts of the levels, the index guard
    unsigned char *timg = nullptr;  // 2D: shared-memory images of the fused tail
};

gw_grid_t coarse_grid(const gw_grid_t &g) {
    gw_grid_t c = g;
    int nn = 1;
    for (int k = 0; k < 3; ++k) {
        if (k < g.dim) {
            c.n_grid[k] = (g.n_grid[k] + 1) / 2;  // fine nodes N -> coarse nodes N/2 + 1
            nn *= c.n_grid[k] + 1;
        } else {
            c.n_grid[k] = 0;
        }
        c.h[k] = 2.0 * g.h[k];
        c.inv_h[k] = 0.5 * g.inv_h[k];
        c.h_nodes[k] = 2.0 * g.h_nodes[k];
    }
    c.n_nodes = nn;
    return c;
}

// Carves (or, with a counting Bump, sizes) every level of the hierarchy at its
// upper bound -- a coarse level holds at most its lattice's node count of rows
// and 5^D blocks per row -- and then the flexible-GMRES vectors.  The hierarchy
// comes first, so its addresses depend only on (grid, n_rows, nf): a plan built
// in a workspace stays valid for any restart length.
struct FlexVecs {
    double *V, *Z, *w, *partials;
    GScalars *sc;
};
constexpr int kTailSmem = 224 * 1024;  // dynamic shared memory of one CTA of the fused tail at most
void mg_carve_sell(Bump &bp, MgLevel &v, int64_t n_rows, int nf) {
    const int64_t e = sell_elems(n_rows);
    v.scols = (int *)bp.take(4 * e);
    v.strips = (int *)bp.take(4 * (n_rows / 8 + 1));  // chunks of at least 8 rows
    v.svals = bp.take(8 * e * nf * nf);
}
void mg_carve_hier(Bump &bp, MgHier &h, const gw_grid_t &g0, int64_t n_rows0, int nf) {
    const int64_t n0 = n_rows0 * nf;
    const int D = g0.dim, mw = D == 2 ? 1 : 4, S = D == 2 ? 25 : 125;
    MgLevel &l0 = h.lv[0];
    l0.g = g0;
    l0.Minv = (double *)bp.take(8 * n_rows0 * nf * nf);
    l0.b = (double *)bp.take(8 * n0);
    l0.x = (double *)bp.take(8 * n0);
    l0.x2 = (double *)bp.take(8 * n0);
    l0.r = (double *)bp.take(8 * n0);
    l0.fixed = (uint8_t *)bp.take(n_rows0);
    const int CN = D == 2 ? 9 : 27, PN = D == 2 ? 4 : 8;
    l0.parent = (int *)bp.take(4 * n_rows0 * PN);
    if (D == 2) {
        mg_carve_sell(bp, l0, n_rows0, nf);
        if (l0.svals) l0.pvals = (float *)l0.svals + sell_elems(n_rows0) * nf * nf;
    } else {
        l0.pvals = bp.take(2 * n_rows0 * S * nf * nf);
    }
    gw_grid_t g = g0;
    int64_t nodes = g0.n_nodes;
    int l = 0;
    // levels carved for the smallest coarsest-level bound a caller may set
    for (; l + 1 < kMgMaxLevels && nodes * nf > kMgCoarseMin; ++l) {
        g = coarse_grid(g);
        nodes = g.n_nodes;
        MgLevel &c = h.lv[l + 1];
        c.g = g;
        c.A.node2row = (int *)bp.take(4 * nodes);
        c.A.row2node = (int *)bp.take(4 * nodes);
        c.A.row_ptr = (int *)bp.take(4 * (nodes + 1));
        c.A.stencil = (uint32_t *)bp.take(4 * nodes * mw);
        c.A.cols = (int *)bp.take(4 * nodes * S);
        c.A.vals = bp.take(8 * nodes * S * nf * nf);
        c.blockrow = (int *)bp.take(4 * nodes * S);
        c.tmp = (int *)bp.take(4 * (nodes + 1));
        c.sws = (int *)bp.take(4 * (scan_ws_ints(nodes + 1) + 64));
        c.flags = (uint8_t *)bp.take(nodes);
        c.Minv = (double *)bp.take(8 * nodes * nf * nf);
        c.b = (double *)bp.take(8 * nodes * nf);
        c.x = (double *)bp.take(8 * nodes * nf);
        c.x2 = (double *)bp.take(8 * nodes * nf);
        c.r = (double *)bp.take(8 * nodes * nf);
        c.fixed = (uint8_t *)bp.take(nodes);
        c.child = (int *)bp.take(4 * nodes * CN);
        c.parent = (int *)bp.take(4 * nodes * PN);
        if (D == 2) mg_carve_sell(bp, c, nodes, nf);
    }
    h.nl = l + 1;  // upper bound; the plan may stop earlier
    h.dM = (double *)bp.take(8 * (int64_t)kMgCoarseMax * kMgCoarseMax);
    h.dInv = (double *)bp.take(8 * (int64_t)kMgCoarseMax * kMgCoarseMax);
    h.counts = (int *)bp.take(4 * (kMgMaxLevels + 1));
    if (D == 2) h.timg = (unsigned char *)bp.take((int64_t)kTailSmem * kTailMaxCluster);
}
void mg_carve_flex(Bump &bp, FlexVecs &fv, int64_t n0, int restart) {
    fv.V = (double *)bp.take(8 * n0 * (restart + 1));
    fv.Z = (double *)bp.take(8 * n0 * restart);
    fv.w = (double *)bp.take(8 * n0);
    fv.partials = (double *)bp.take(8 * (int64_t)kGmresPartials);
    fv.sc = (GScalars *)bp.take(sizeof(GScalars));
}

int64_t mg_ws_bytes(const gw_grid_t &g0, int64_t n_rows, int nf, int restart) {
    Bump bp{nullptr, 0};
    MgHier h;
    FlexVecs fv;
    mg_carve_hier(bp, h, g0, n_rows, nf);
    mg_carve_flex(bp, fv, n_rows * nf, restart);
    return bp.used;
}

// Pattern phase: the coarse active sets, row maps, stencils, row pointers and
// columns of every level below A0 (two host reads: the levels' row counts, then
// their block counts with the index guard).  Depends on A0's pattern only.
template <int NF>
int mg_pattern(MgHier &h, const gw_bsr_t *A0, gw_mg_plan_t *plan, cudaStream_t s) {
    const int D = h.lv[0].g.dim, mw = D == 2 ? 1 : 4;
    const int nl_bound = h.nl;
    h.lv[0].L = lat_of(h.lv[0].g);
    h.lv[0].A = *A0;
    // active nodes and row counts of the levels that may be needed (none below one whose
    // whole lattice is small enough for the dense level), read once
    const int64_t coarse = g_tune[GW_TUNE_MG_COARSE];
    int counts[kMgMaxLevels + 1] = {0};
    if ((int64_t)A0->n_rows * NF > coarse) {
        GW_CUDA(cudaMemsetAsync(h.counts, 0, 4 * kMgMaxLevels, s));
        int q = 0;
        for (; q + 1 < nl_bound && (int64_t)h.lv[q].g.n_nodes * NF > coarse; ++q) {
            MgLevel &f = h.lv[q], &c = h.lv[q + 1];
            c.L = lat_of(c.g);
            k_mg_coarse_flags<<<gw_count_launch(nblk(c.g.n_nodes, kThreads)), kThreads, 0, s>>>(
                f.L, q == 0 ? (const int *)f.A.node2row : nullptr, q == 0 ? nullptr : f.flags, c.L, c.flags, h.counts + q + 1);
        }
        GW_LAUNCHED();
        GW_CUDA(cudaMemcpyAsync(counts, h.counts, 4 * (q + 1), cudaMemcpyDeviceToHost, s));
        GW_CUDA(cudaStreamSynchronize(s));
    }
    int l = 0;
    while (h.lv[l].A.n_rows * NF > g_tune[GW_TUNE_MG_COARSE]) {
        if (l + 1 >= nl_bound) {
            snprintf(g_msg, sizeof(g_msg), "multigrid: coarsest level still has %d unknowns", h.lv[l].A.n_rows * NF);
            return GW_EINVAL;
        }
        MgLevel &f = h.lv[l], &c = h.lv[l + 1];
        const int N = c.g.n_nodes, nrc = counts[l + 1];
        PtrsA fa = make_ptrs(f.A);
        if (nrc <= 0 || nrc > N) {
            snprintf(g_msg, sizeof(g_msg), "multigrid: empty coarse level");
            return GW_EINVAL;
        }
        k_flags_to_int<<<gw_count_launch(nblk(N, kThreads)), kThreads, 0, s>>>(c.flags, N, c.tmp);
        GW_LAUNCHED();
        int rc = scan_exclusive(c.tmp, c.tmp, N, c.sws + 64, s);
        if (rc) return rc;
        k_compact<<<gw_count_launch(nblk(N, kThreads)), kThreads, 0, s>>>(c.flags, c.tmp, N, NF, nullptr,
                                                                          (int *)c.A.node2row, (int *)c.A.row2node, nullptr);
        GW_LAUNCHED();
        GW_CUDA(cudaMemsetAsync((void *)c.A.stencil, 0, 4 * (size_t)N * mw, s));
        GW_CUDA(cudaMemsetAsync(c.tmp, 0, 4 * ((size_t)nrc + 1), s));
        if (D == 2)
            k_mg_coarse_stencil2<<<gw_count_launch(nblk((int64_t)nrc * 32, kThreads)), kThreads, 0, s>>>(
                f.L, fa, c.L, nrc, c.A.row2node, (uint32_t *)c.A.stencil, c.tmp);
        else
            k_mg_coarse_stencil<<<gw_count_launch(nblk(nrc, kThreads)), kThreads, 0, s>>>(
                f.L, fa, c.L, nrc, c.A.row2node, (uint32_t *)c.A.stencil, mw, c.tmp);
        GW_LAUNCHED();
        rc = scan_exclusive(c.tmp, (int *)c.A.row_ptr, nrc + 1, c.sws, s);
        if (rc) return rc;
        c.A.n_rows = nrc;
        c.A.nf = NF;
        // its capacity, until the block counts are read below (which are ints: rows of a
        // lattice of more than 2^31 / 125 nodes need not be)
        c.A.nnzb = (int)std::min<int64_t>((int64_t)N * (D == 2 ? 25 : 125), INT_MAX);
        c.A.mask_words = mw;
        PtrsA ca = make_ptrs(c.A);
        if (D == 2) k_pattern_fill<2><<<gw_count_launch(nblk(nrc, kThreads)), kThreads, 0, s>>>(c.g, ca, (int *)c.A.cols);
        else k_pattern_fill<3><<<gw_count_launch(nblk(nrc, kThreads)), kThreads, 0, s>>>(c.g, ca, (int *)c.A.cols);
        k_mg_blockrow<<<gw_count_launch(nblk(nrc, kThreads)), kThreads, 0, s>>>(c.A.row_ptr, nrc, c.A.nnzb, c.blockrow);
        if (D == 2) {
            k_mg_children<2><<<gw_count_launch(nblk(nrc, kThreads)), kThreads, 0, s>>>(f.L, fa, c.L, ca, c.child);
            k_mg_parents<2><<<gw_count_launch(nblk(f.A.n_rows, kThreads)), kThreads, 0, s>>>(f.L, fa, c.L, ca, f.parent);
        } else {
            k_mg_children<3><<<gw_count_launch(nblk(nrc, kThreads)), kThreads, 0, s>>>(f.L, fa, c.L, ca, c.child);
            k_mg_parents<3><<<gw_count_launch(nblk(f.A.n_rows, kThreads)), kThreads, 0, s>>>(f.L, fa, c.L, ca, f.parent);
        }
        GW_LAUNCHED();
        ++l;
    }
    h.nl = l + 1;
    h.dn = h.lv[l].A.n_rows * NF;
    if (D == 2)
        for (int q = 0; q < (h.nl > 1 ? h.nl - 1 : 1); ++q) {
            MgLevel &v = h.lv[q];
            const int lpr = sell_lpr(v.A.n_rows);
            k_sell_pattern<<<gw_count_launch(nblk((int64_t)sell_chunks(v.A.n_rows, lpr) * 32, kThreads)), kThreads, 0, s>>>(
                make_ptrs(v.A), lpr, v.strips, v.scols);
            GW_LAUNCHED();
        }
    if (h.nl > 1) {
        MgTotals tot;
        memset(&tot, 0, sizeof(tot));
        tot.n = h.nl;
        for (int q = 0; q < h.nl; ++q) {
            tot.row_ptr[q] = h.lv[q].A.row_ptr;
            tot.n_rows[q] = h.lv[q].A.n_rows;
        }
        k_mg_totals<<<gw_count_launch(1), 32, 0, s>>>(tot, h.counts);
        GW_LAUNCHED();
        GW_CUDA(cudaMemcpyAsync(counts, h.counts, 4 * (kMgMaxLevels + 1), cudaMemcpyDeviceToHost, s));
        GW_CUDA(cudaStreamSynchronize(s));
        for (int q = 1; q < h.nl; ++q) h.lv[q].A.nnzb = counts[q];
        if (counts[kMgMaxLevels]) {  // an index guard failed
            const int gc = guard_check(s, "multigrid plan");
            if (gc) return gc;
        }
    }
    memset(plan, 0, sizeof(*plan));
    plan->levels = h.nl;
    plan->dense_n = h.dn;
    for (int q = 0; q < h.nl; ++q) {
        plan->n_rows[q] = h.lv[q].A.n_rows;
        plan->nnzb[q] = h.lv[q].A.nnzb;
    }
    plan->nf = NF;
    plan->fine_n_rows = A0->n_rows;
    plan->fine_nnzb = A0->nnzb;
    plan->row_ptr = A0->row_ptr;
    plan->cols = A0->cols;
    return GW_OK;
}

// Restores the level sizes a plan recorded into a freshly carved hierarchy.
void mg_apply_plan(MgHier &h, const gw_bsr_t *A0, const gw_mg_plan_t *plan, int nf) {
    const int mw = h.lv[0].g.dim == 2 ? 1 : 4;
    h.nl = plan->levels;
    h.dn = plan->dense_n;
    h.lv[0].L = lat_of(h.lv[0].g);
    h.lv[0].A = *A0;
    for (int q = 1; q < h.nl; ++q) {
        MgLevel &c = h.lv[q];
        c.L = lat_of(c.g);
        c.A.n_rows = plan->n_rows[q];
        c.A.nnzb = plan->nnzb[q];
        c.A.nf = nf;
        c.A.mask_words = mw;
    }
}

// Numeric phase: smoother blocks and fixed-DOF masks of every level, Galerkin
// values of the coarse levels, dense inverse of the coarsest.  No host reads.
template <typename VT>
inline bool mg_bf16_fine() { return std::is_same<VT, float>::value && g_tune[GW_TUNE_MG_BF16] != 0; }

template <int NF, typename VT>
int mg_numeric(MgHier &h, cudaStream_t s) {
    const int D = h.lv[0].g.dim;
    {
        const MgLevel &l0 = h.lv[0];
        PtrsA a0 = make_ptrs(l0.A);
        k_mg_smoother_setup<NF, VT><<<gw_count_launch(nblk(l0.A.n_rows, kThreads)), kThreads, 0, s>>>(a0, D, l0.Minv);
        k_mg_fixed_mask<NF, VT><<<gw_count_launch(nblk(l0.A.n_rows, kThreads)), kThreads, 0, s>>>(a0, l0.fixed);
        GW_LAUNCHED();
    }
    for (int l = 0; l + 1 < h.nl; ++l) {
        MgLevel &f = h.lv[l], &c = h.lv[l + 1];
        PtrsA fa = make_ptrs(f.A), ca = make_ptrs(c.A);
        const int nb = c.A.nnzb;
        if (D == 2) k_mg_rap2<NF, VT><<<gw_count_launch(nblk((int64_t)nb * 16, kThreads)), kThreads, 0, s>>>(fa, f.fixed, c.child, c.L, ca, c.blockrow);
        else k_mg_rap<NF, VT><<<gw_count_launch(nblk(nb, kThreads)), kThreads, 0, s>>>(f.L, fa, f.fixed, c.L, ca, c.blockrow);
        GW_LAUNCHED();
        const int nrc = c.A.n_rows;
        k_mg_fix_empty_rows<NF, VT><<<gw_count_launch(nblk(nrc, kThreads)), kThreads, 0, s>>>(ca);
        k_mg_smoother_setup<NF, VT><<<gw_count_launch(nblk(nrc, kThreads)), kThreads, 0, s>>>(ca, D, c.Minv);
        k_mg_fixed_mask<NF, VT><<<gw_count_launch(nblk(nrc, kThreads)), kThreads, 0, s>>>(ca, c.fixed);
        GW_LAUNCHED();
    }
    const int l = h.nl - 1;
    const MgLevel &lc = h.lv[l];
    const int n = h.dn;
    GW_CUDA(cudaMemsetAsync(h.dM, 0, 8 * (size_t)n * n, s));
    PtrsA ac = make_ptrs(lc.A);
    k_mg_dense_build<NF, VT><<<gw_count_launch(nblk(lc.A.n_rows, kThreads)), kThreads, 0, s>>>(ac, h.dM, n);
    auto inv = k_mg_dense_invert<1>;
    switch ((n + 31) / 32) {  // columns per lane: n <= kMgCoarseMax = 160
        case 2: inv = k_mg_dense_invert<2>; break;
        case 3: inv = k_mg_dense_invert<3>; break;
        case 4: inv = k_mg_dense_invert<4>; break;
        case 5: inv = k_mg_dense_invert<5>; break;
        default: break;
    }
    inv<<<gw_count_launch(1), 512, 0, s>>>(h.dM, h.dInv, n);
    GW_LAUNCHED();
    return GW_OK;
}

// -------------------------------------------------------------- 2D: sliced rows
SellA sell_of(const MgLevel &v, bool bf16) {
    SellA a;
    a.n_rows = v.A.n_rows;
    a.n_chunks = sell_chunks(v.A.n_rows, sell_lpr(v.A.n_rows));
    a.cols = v.scols;
    a.trips = v.strips;
    a.vals = bf16 ? v.pvals : v.svals;
    return a;
}

// warps per CTA of the sliced row kernels: at most 8 (their register bound)
int sell_block() { return 32 * std::min(g_tune[GW_TUNE_ROW_WARPS], 8); }
int sell_grid(const SellA &a) {
    const int b = nblk(a.n_chunks, sell_block() / 32);
    return b < 1 ? 1 : b;
}

// Values of the sliced layout: the finest level on every solve (fresh = false),
// and after a numeric phase the smoothed coarse levels too, in one launch.
template <int NF, typename VT>
int sell_values(const MgHier &h, bool fresh, cudaStream_t s) {
    SellJobs js;
    js.n = 0;
    js.warps = 0;
    const int last = fresh ? std::max(h.nl - 1, 1) : 1;
    auto add = [&](const MgLevel &v, void *out) {
        SellJob &j = js.j[js.n++];
        j.A = make_ptrs(v.A);
        j.lpr = sell_lpr(v.A.n_rows);
        j.first_warp = js.warps;
        j.trips = v.strips;
        j.cols = v.scols;
        j.vals = out;
        js.warps += sell_chunks(v.A.n_rows, j.lpr);
    };
    for (int l = 0; l < last; ++l) add(h.lv[l], h.lv[l].svals);
    k_sell_values<NF, VT, VT><<<gw_count_launch(nblk((int64_t)js.warps * 32, kThreads)), kThreads, 0, s>>>(js);
    if constexpr (std::is_same<VT, float>::value) {
        if (mg_bf16_fine<VT>()) {
            js.n = js.warps = 0;
            add(h.lv[0], h.lv[0].pvals);
            k_sell_values<NF, float, __nv_bfloat16><<<gw_count_launch(nblk((int64_t)js.warps * 32, kThreads)), kThreads, 0, s>>>(js);
        }
    }
    GW_LAUNCHED();
    return GW_OK;
}

template <int NF, typename VT>
void sell_jacobi(const MgHier &h, int l, VecRef b, const double *xin, VecRef xout, const GScalars *sc, cudaStream_t s) {
    const MgLevel &v = h.lv[l];
    const bool bf = l == 0 && mg_bf16_fine<VT>();
    const SellA a = sell_of(v, bf);
    const double vs = 8.0 * v.A.n_rows * NF, mat = (double)v.A.nnzb * (NF * NF * (bf ? 2 : sizeof(VT)) + 4);
    ProfScope ps(l == 0 ? PC_MG_JACOBI : PC_MG_JACOBI_COARSE, s, 3 * vs + 8.0 * v.A.n_rows * NF * NF + mat);
    const bool one = sell_lpr(v.A.n_rows) == 1;
    void (*k)(SellA, const double *, VecRef, const double *, VecRef, double, const GScalars *);
    if (bf) k = one ? k_sell_jacobi<NF, __nv_bfloat16, 1> : k_sell_jacobi<NF, __nv_bfloat16, 4>;
    else k = one ? k_sell_jacobi<NF, VT, 1> : k_sell_jacobi<NF, VT, 4>;
    launch_pdl(k, sell_grid(a), sell_block(), 0, s, a, (const double *)v.Minv, b, xin, xout, mg_omega(), sc);
}

template <int NF, typename VT>
void sell_residual(const MgHier &h, int l, VecRef b, const double *x, const GScalars *sc, cudaStream_t s) {
    const MgLevel &v = h.lv[l];
    const bool bf = l == 0 && mg_bf16_fine<VT>();
    const SellA a = sell_of(v, bf);
    ProfScope ps(PC_MG_RESID, s, 3 * 8.0 * v.A.n_rows * NF + (double)v.A.nnzb * (NF * NF * (bf ? 2 : sizeof(VT)) + 4));
    const bool one = sell_lpr(v.A.n_rows) == 1;
    void (*k)(SellA, VecRef, const double *, double *, const GScalars *);
    if (bf) k = one ? k_sell_residual<NF, __nv_bfloat16, 1> : k_sell_residual<NF, __nv_bfloat16, 4>;
    else k = one ? k_sell_residual<NF, VT, 1> : k_sell_residual<NF, VT, 4>;
    launch_pdl(k, sell_grid(a), sell_block(), 0, s, a, b, x, v.r, sc);
}

template <int NF, typename VT>
void sell_spmv(const MgHier &h, VecRef z, const GmresVecs &G, cudaStream_t s) {
    const SellA a = sell_of(h.lv[0], false);
    void (*k)(SellA, VecRef, double *, const GScalars *) =
        sell_lpr(a.n_rows) == 1 ? k_sell_spmv<NF, VT, 1> : k_sell_spmv<NF, VT, 4>;
    launch_pdl(k, sell_grid(a), sell_block(), 0, s, a, z, G.w, (const GScalars *)G.sc);
}

// Next basis vector and what the V-cycle starts from: in 2D the finest level's
// zero-start sweep (nothing when the finest level is the dense one), in 3D its
// right-hand side.
template <int NF>
void mg_next(const MgHier &h, const GmresVecs &G, int start, cudaStream_t s) {
    const MgLevel &v = h.lv[0];
    const bool flat = v.g.dim == 2, smooth = flat && h.nl > 1;
    gs_next<NF>(v.A.n_rows, G, start, smooth ? v.Minv : nullptr, flat ? (smooth ? v.x : nullptr) : v.b,
                smooth ? mg_omega() : 1.0, s);
}

// -------------------------------------------------------------- fused coarse tail
// Largest cluster of the tail that the current device keeps resident: 16 CTAs
// where it can (a size above 8 is not portable), else 8, 0 when neither fits
// (then every level keeps its own launches).  Queried once per device, before
// any stream capture (gmres_mg calls it first).
template <int NF, typename VT>
int tail_cluster_max() {
    static int cached[64] = {0};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
    const int got = __atomic_load_n(&cached[dev], __ATOMIC_ACQUIRE);
    if (got) return got > 0 ? got : 0;
    int size = -1;
    auto k = k_sell_tail<NF, VT>;
    if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kTailSmem) == cudaSuccess)
        for (int cand : {kTailMaxCluster, 8}) {
            if (cand > 8 && cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess)
                continue;
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3(cand);
            cfg.blockDim = dim3(kTailThreads);
            cfg.dynamicSmemBytes = kTailSmem;
            cudaLaunchAttribute at;
            at.id = cudaLaunchAttributeClusterDimension;
            at.val.clusterDim.x = cand;
            at.val.clusterDim.y = 1;
            at.val.clusterDim.z = 1;
            cfg.attrs = &at;
            cfg.numAttrs = 1;
            int n = 0;
            if (cudaOccupancyMaxActiveClusters(&n, (void *)k, &cfg) == cudaSuccess && n >= 1) {
                size = cand;
                break;
            }
        }
    (void)cudaGetLastError();  // a refused query leaves no error behind
    __atomic_store_n(&cached[dev], size, __ATOMIC_RELEASE);
    return size > 0 ? size : 0;
}

struct TailShape {
    int l0;       // first level of the tail; h.nl - 1: none
    int cluster;
    int smem;     // bytes
};
// log2 of a level's rows per CTA: a power of two, at least one chunk of 8
int tail_sh(int n_rows, int cluster) {
    int sh = 3;
    while (((int64_t)cluster << sh) < n_rows) ++sh;
    return sh;
}
// shared memory of one CTA; off (may be null): every level's vectors, the dense one's
// at h.nl - 1, the image's start at h.nl
template <int NF, typename VT>
int64_t tail_bytes(const MgHier &h, int l0, int cluster, int *off) {
    const int last = h.nl - 1;
    int64_t d = 0, img = sizeof(TailHead);
    for (int l = l0; l < last; ++l) {
        const int sh = tail_sh(h.lv[l].A.n_rows, cluster);
        if (off) off[l] = (int)d;
        d += 4 * tail_vec<NF>(sh);
        img += TailPart<NF, VT>(sh, kTailT).bytes();
    }
    if (off) off[last] = (int)d;
    d += (16 * (int64_t)h.dn + 15) / 16 * 16;
    if (off) off[last + 1] = (int)d;
    return d + img + tail_dense_bytes(h.dn, h.lv[last].A.n_rows, cluster);
}
// First level of at most GW_TUNE_MG_TAIL rows (0: kTailRows) whose rows, with
// those of the levels below, fit the cluster's shared memory; at least as many
// CTAs as give each warp one chunk of that level and one row of the dense inverse.
// 30 Arnoldi steps with the bound at 512 / 1024 / 2048 / 4096 rows: 26k rows FP64 2.15 /
// 2.16 / 2.00 / 2.00 ms, 5k rows FP32 1.52 / 1.53 / 1.38 / 1.38 ms, 2.6k u-p rows FP32 1.71 /
// 1.50 / 1.49 / 1.49 ms.
constexpr int kTailRows = 2048;
template <int NF, typename VT>
TailShape tail_shape(const MgHier &h) {
    const int last = h.nl - 1, cmax = tail_cluster_max<NF, VT>();
    const int bound = g_tune[GW_TUNE_MG_TAIL] > 0 ? std::min(g_tune[GW_TUNE_MG_TAIL], 16384) : kTailRows;
    TailShape t{last, 0, 0};
    if (cmax == 0) return t;
    for (int l = mg_bf16_fine<VT>() ? 1 : 0; l < last; ++l) {  // the tail reads the solve's own values
        const int n = h.lv[l].A.n_rows;
        if (n > bound || sell_lpr(n) != 4) continue;
        int c = 1;
        while (c < cmax && (c * kTailWarps * 8 < n || c * kTailWarps < h.dn || tail_bytes<NF, VT>(h, l, c, nullptr) > kTailSmem)) c *= 2;
        const int64_t b = tail_bytes<NF, VT>(h, l, c, nullptr);
        if (b > kTailSmem) continue;
        return TailShape{l, c, (int)b};
    }
    return t;
}

template <int NF, typename VT>
TailArgs tail_args(const MgHier &h, const TailShape &t) {
    const int last = h.nl - 1;
    TailArgs a;
    memset(&a, 0, sizeof(a));
    a.l0 = t.l0;
    a.last = last;
    a.cluster = t.cluster;
    int off[kMgMaxLevels + 1];
    (void)tail_bytes<NF, VT>(h, t.l0, t.cluster, off);
    for (int l = t.l0; l < last; ++l) {
        const MgLevel &v = h.lv[l];
        TailLevel &w = a.lv[l];
        w.A = sell_of(v, false);
        w.Minv = v.Minv;
        w.fixed = v.fixed;
        w.child = v.child;
        w.parent = v.parent;
        w.sh = tail_sh(v.A.n_rows, t.cluster);
        w.off = off[l];
        w.sweeps = mg_sweeps(l);
    }
    a.dInv = h.dInv;
    a.dn = h.dn;
    a.n_last = h.lv[last].A.n_rows;
    a.child_last = h.lv[last].child;
    a.off_last = off[last];
    a.off_img = off[last + 1];
    a.img = h.timg;
    a.img_stride = kTailSmem;
    a.omega = mg_omega();
    return a;
}

// The images of the tail's shared memory, after the values they copy (on every
// solve: the tail may hold the finest level, and its knobs may have changed).
template <int NF, typename VT>
int tail_image(const MgHier &h, cudaStream_t s) {
    const TailShape t = tail_shape<NF, VT>(h);
    if (t.l0 == h.nl - 1) return GW_OK;
    k_tail_image<NF, VT><<<dim3(gw_count_launch(t.cluster), h.nl - t.l0), 256, 0, s>>>(tail_args<NF, VT>(h, t));
    GW_LAUNCHED();
    return GW_OK;
}

template <int NF, typename VT>
void sell_tail(const MgHier &h, const TailShape &t, VecRef b, VecRef out, const GScalars *sc, cudaStream_t s) {
    TailArgs a = tail_args<NF, VT>(h, t);
    a.b = b;
    a.out = out;
    a.x1 = h.lv[t.l0].x;
    a.sc = sc;
    double bytes = 8.0 * h.dn * h.dn;
    for (int l = t.l0; l + 1 < h.nl; ++l)
        bytes += (double)h.lv[l].A.nnzb * (NF * NF * sizeof(VT) + 4) + 8.0 * h.lv[l].A.n_rows * NF * (NF + 2);
    ProfScope ps(PC_MG_TAIL, s, bytes);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(gw_count_launch(t.cluster));
    cfg.blockDim = dim3(kTailThreads);
    cfg.dynamicSmemBytes = t.smem;
    cfg.stream = s;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = t.cluster;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 2;
    (void)cudaLaunchKernelEx(&cfg, k_sell_tail<NF, VT>, a);
}

// One V-cycle on v_k, result in Z[k].  The zero-start sweep of every level comes
// with its right-hand side (mg_next, k_sell_restrict).
template <int NF, typename VT>
void sell_vcycle(const MgHier &h, const GmresVecs &G, VecRef z, cudaStream_t s) {
    const int last = h.nl - 1;
    const GScalars *sc = G.sc;
    const VecRef v0{G.V, G.n};
    const TailShape tail = tail_shape<NF, VT>(h);
    const int l0 = tail.l0;
    double *cur[kMgMaxLevels], *oth[kMgMaxLevels];
    for (int l = 0; l < l0; ++l) {
        const MgLevel &v = h.lv[l], &c = h.lv[l + 1];
        const VecRef b = l == 0 ? v0 : VecRef{v.b, 0};
        double *x = v.x, *y = v.x2;
        for (int it = 1; it < mg_sweeps(l); ++it) {
            sell_jacobi<NF, VT>(h, l, b, x, VecRef{y, 0}, sc, s);
            std::swap(x, y);
        }
        sell_residual<NF, VT>(h, l, b, x, sc, s);
        {
            ProfScope ps(PC_MG_TRANSFER, s, 8.0 * NF * (v.A.n_rows + c.A.n_rows));
            launch_pdl(k_sell_restrict<NF>, nblk(c.A.n_rows, 128), 128, 0, s, c.A.n_rows, v.A.n_rows,
                       (const int *)c.child, (const uint8_t *)v.fixed, (const double *)v.r, c.b,
                       (const double *)(l + 1 < last ? c.Minv : nullptr), c.x, mg_omega(), sc);
        }
        cur[l] = x;
        oth[l] = y;
    }
    const VecRef bl = l0 == 0 ? v0 : VecRef{h.lv[l0].b, 0};
    if (l0 < last) {
        sell_tail<NF, VT>(h, tail, bl, l0 == 0 ? z : VecRef{h.lv[l0].x2, 0}, sc, s);
        cur[l0] = h.lv[l0].x2;
    } else {
        launch_pdl(k_sell_dense_apply, nblk((int64_t)h.dn * 32, kThreads), kThreads, 0, s, (const double *)h.dInv, bl,
                   last == 0 ? z : VecRef{h.lv[last].x, 0}, h.dn, sc);
        cur[last] = h.lv[last].x;
    }
    for (int l = l0 - 1; l >= 0; --l) {
        const MgLevel &v = h.lv[l], &c = h.lv[l + 1];
        const VecRef b = l == 0 ? v0 : VecRef{v.b, 0};
        double *x = cur[l], *y = oth[l];
        {
            ProfScope ps(PC_MG_TRANSFER, s, 8.0 * NF * (2.0 * v.A.n_rows + c.A.n_rows));
            launch_pdl(k_sell_prolong<NF>, nblk(v.A.n_rows, 128), 128, 0, s, v.A.n_rows, c.A.n_rows,
                       (const int *)v.parent, (const uint8_t *)v.fixed, (const double *)cur[l + 1], x, sc);
        }
        for (int it = 0; it < mg_sweeps(l); ++it) {
            const bool out = l == 0 && it + 1 == mg_sweeps(0);
            sell_jacobi<NF, VT>(h, l, b, x, out ? z : VecRef{y, 0}, sc, s);
            std::swap(x, y);
        }
        cur[l] = x;
    }
}

template <int NF, typename VT>
void mg_jacobi(const MgHier &h, int l, const double *b, const double *xin, double *xout, int zero, const int *skip,
               cudaStream_t s) {
    const MgLevel &v = h.lv[l];
    PtrsA a = make_ptrs(v.A);
    const int tb = zero ? kThreads : tune_rows_block();
    const bool bf = l == 0 && mg_bf16_fine<VT>();
    if (bf) a.vals = v.pvals;
    const int g = zero ? red_grid_elems(v.A.n_rows)
                       : (bf ? resident_rows_grid((const void *)k_mg_jacobi<NF, __nv_bfloat16>, tb, v.A.n_rows)
                             : resident_rows_grid((const void *)k_mg_jacobi<NF, VT>, tb, v.A.n_rows));
    // algorithmic bytes: b, x_out, Minv; with a previous iterate also x_in and the matrix
    const double vs = 8.0 * v.A.n_rows * NF, mat = (double)v.A.nnzb * (NF * NF * (bf ? 2 : sizeof(VT)) + 4);
    ProfScope ps(l == 0 ? PC_MG_JACOBI : PC_MG_JACOBI_COARSE, s,
                 2 * vs + 8.0 * v.A.n_rows * NF * NF + (zero ? 0.0 : vs + mat));
    if (bf) k_mg_jacobi<NF, __nv_bfloat16><<<gw_count_launch(g), tb, 0, s>>>(a, v.Minv, b, xin, xout, mg_omega(), zero, skip);
    else k_mg_jacobi<NF, VT><<<gw_count_launch(g), tb, 0, s>>>(a, v.Minv, b, xin, xout, mg_omega(), zero, skip);
}

// 3D (block-CSR rows of up to 125 blocks): one V-cycle on h.lv[0].b; returns the buffer that holds the result (the same
// buffer on every call).
template <int NF, typename VT>
double *mg_vcycle(const MgHier &h, const int *skip, cudaStream_t s) {
    const int last = h.nl - 1;
    double *cur[kMgMaxLevels], *oth[kMgMaxLevels];
    for (int l = 0; l < last; ++l) {
        const MgLevel &v = h.lv[l], &c = h.lv[l + 1];
        double *x = v.x, *y = v.x2;
        if (mg_sweeps(l) >= 2) {
            // both zero-start sweeps in one launch, into the buffer the
            // second separate sweep would have written
            PtrsA a = make_ptrs(v.A);
            const bool bf = l == 0 && mg_bf16_fine<VT>();
            if (bf) a.vals = v.pvals;
            const double vs = 8.0 * v.A.n_rows * NF;
            const double mat = (double)v.A.nnzb * (NF * NF * (bf ? 2 : sizeof(VT)) + 4);
            ProfScope ps(l == 0 ? PC_MG_JACOBI : PC_MG_JACOBI_COARSE, s, 2 * vs + 8.0 * v.A.n_rows * NF * NF + mat);
            if (bf)
                k_mg_presmooth2<NF, __nv_bfloat16><<<gw_count_launch(resident_rows_grid(
                                                         (const void *)k_mg_presmooth2<NF, __nv_bfloat16>,
                                                         tune_rows_block(), v.A.n_rows)),
                                                     tune_rows_block(), 0, s>>>(a, v.Minv, v.b, y, mg_omega(), skip);
            else
                k_mg_presmooth2<NF, VT><<<gw_count_launch(resident_rows_grid(
                                              (const void *)k_mg_presmooth2<NF, VT>, tune_rows_block(), v.A.n_rows)),
                                          tune_rows_block(), 0, s>>>(a, v.Minv, v.b, y, mg_omega(), skip);
            double *t = x; x = y; y = t;
            for (int it = 2; it < mg_sweeps(l); ++it) {
                mg_jacobi<NF, VT>(h, l, v.b, x, y, 0, skip, s);
                t = x; x = y; y = t;
            }
        } else {
            mg_jacobi<NF, VT>(h, l, v.b, nullptr, x, 1, skip, s);
            for (int it = 1; it < mg_sweeps(l); ++it) {
                mg_jacobi<NF, VT>(h, l, v.b, x, y, 0, skip, s);
                double *t = x; x = y; y = t;
            }
        }
        PtrsA a = make_ptrs(v.A), ca = make_ptrs(c.A);
        const double vs = 8.0 * v.A.n_rows * NF;
        {
        const bool bf = l == 0 && mg_bf16_fine<VT>();
        PtrsA ar = a;
        if (bf) ar.vals = v.pvals;
        ProfScope ps(PC_MG_RESID, s, 3 * vs + (double)v.A.nnzb * (NF * NF * (bf ? 2 : sizeof(VT)) + 4));
        if (bf)
            k_mg_residual<NF, __nv_bfloat16><<<gw_count_launch(resident_rows_grid(
                                                   (const void *)k_mg_residual<NF, __nv_bfloat16>, tune_rows_block(),
                                                   v.A.n_rows)),
                                               tune_rows_block(), 0, s>>>(ar, v.b, x, v.r, skip);
        else
            k_mg_residual<NF, VT><<<gw_count_launch(resident_rows_grid((const void *)k_mg_residual<NF, VT>,
                                                                       tune_rows_block(), v.A.n_rows)),
                                    tune_rows_block(), 0, s>>>(a, v.b, x, v.r, skip);
        }
        ProfScope ps(PC_MG_TRANSFER, s, vs + 8.0 * c.A.n_rows * NF);
        k_mg_restrict_list<NF><<<gw_count_launch(nblk(c.A.n_rows, kThreads)), kThreads, 0, s>>>(
                c.A.n_rows, v.A.n_rows, c.child, v.fixed, v.r, c.b, skip);
        cur[l] = x;
        oth[l] = y;
    }
    const MgLevel &lc = h.lv[last];
    k_mg_dense_apply<<<gw_count_launch(nblk((int64_t)h.dn * 32, kThreads)), kThreads, 0, s>>>(h.dInv, lc.b, lc.x, h.dn, skip);
    cur[last] = lc.x;
    for (int l = last - 1; l >= 0; --l) {
        const MgLevel &v = h.lv[l], &c = h.lv[l + 1];
        PtrsA a = make_ptrs(v.A), ca = make_ptrs(c.A);
        double *x = cur[l], *y = oth[l];
        {
        ProfScope ps(PC_MG_TRANSFER, s, 16.0 * v.A.n_rows * NF + 8.0 * c.A.n_rows * NF);
        k_mg_prolong_list<NF><<<gw_count_launch(nblk(v.A.n_rows, kThreads)), kThreads, 0, s>>>(
                v.A.n_rows, c.A.n_rows, v.parent, v.fixed, cur[l + 1], x, skip);
        }
        for (int it = 0; it < mg_sweeps(l); ++it) {
            mg_jacobi<NF, VT>(h, l, v.b, x, y, 0, skip, s);
            double *t = x; x = y; y = t;
        }
        cur[l] = x;
    }
    return cur[0];
}

// One Arnoldi step with its V-cycle is ~40 small kernels.  Issuing them one by
// one costs more host time than the GPU spends running them, so the step is
// captured once as a CUDA graph and replayed.  Every kernel argument of the
// step is fixed by the key below (matrix, vectors, workspace, plan), so one
// instantiated graph serves all Newton iterations of a load step.  The graphs
// are held in a small cache (least recently used entry replaced).
struct MgGraphKey {
    int device, nf, vt_bytes, restart, nl, dn, dim, row_warps, one_sweep, sweeps, omega, tail, bf16, fine_sweeps;
    int n_grid[3];
    int n_rows[kMgMaxLevels], nnzb[kMgMaxLevels];
    gw_bsr_t A;
    const void *ws;
    const double *b;
    double *x, *z;
};
struct MgGraphEntry {
    MgGraphKey key;
    std::shared_ptr<const StepGraph> graph;  // null: an empty slot
    uint64_t stamp;
};
constexpr int kMgGraphCache = 8;
// Shared by the host threads: entries change under the lock, and a solve keeps its
// graph alive, so an entry replaced by another thread goes when that solve is done.
struct MgGraphs {
    std::mutex mu;
    MgGraphEntry e[kMgGraphCache];
    uint64_t clock = 0;
};
MgGraphs &mg_graphs() {
    static MgGraphs *const g = new MgGraphs();  // not destroyed at exit, when CUDA may be gone
    return *g;
}
// The next basis vector (start: the first of a cycle) and its V-cycle.
template <int NF, typename VT>
void mg_step_tail(const MgHier &h, GmresVecs &G, VecRef z, int start, const int *skip, cudaStream_t s) {
    { ProfScope ps(PC_NEXT, s, 8.0 * G.n * 3); mg_next<NF>(h, G, start, s); }
    if (h.lv[0].g.dim == 2) sell_vcycle<NF, VT>(h, G, z, s);
    else G.z = mg_vcycle<NF, VT>(h, skip, s);
}

// One Arnoldi step and the V-cycle of the new basis vector.
template <int NF, typename VT>
void mg_arnoldi_step(const MgHier &h, const PtrsA &a, GmresVecs &G, double *Z, int restart,
                     const int *skip, cudaStream_t s) {
    const VecRef z{Z, G.n};
    const bool flat = h.lv[0].g.dim == 2;
    {
        ProfScope ps(PC_SPMV, s, (double)h.lv[0].A.nnzb * (NF * NF * sizeof(VT) + 4) + 4.0 * (a.n_rows + 1) + 24.0 * G.n);
        if (flat) sell_spmv<NF, VT>(h, z, G, s);
        else k_gm_spmv_keep<NF, VT><<<gw_count_launch(resident_rows_grid((const void *)k_gm_spmv_keep<NF, VT>, kThreads, a.n_rows)),
                                      kThreads, 0, s>>>(a, G, Z);
    }
    gs_column(G, restart, 8.0 * G.n * (restart / 2), s);
    mg_step_tail<NF, VT>(h, G, z, 0, skip, s);
}

// Returns the cached (or newly captured) graph of one Arnoldi step.
template <int NF, typename VT>
int mg_step_graph(const MgHier &h, const gw_grid_t &grid, const gw_bsr_t *A, GmresVecs &G, double *Z, void *ws,
                  int restart, const int *skip, std::shared_ptr<const StepGraph> *out) {
    MgGraphKey k;
    memset(&k, 0, sizeof(k));
    GW_CUDA(cudaGetDevice(&k.device));
    k.nf = NF; k.vt_bytes = sizeof(VT); k.restart = restart; k.nl = h.nl; k.dn = h.dn; k.dim = grid.dim;
    k.row_warps = g_tune[GW_TUNE_ROW_WARPS];
    k.one_sweep = g_tune[GW_TUNE_MG_ONE_SWEEP];
    k.sweeps = g_tune[GW_TUNE_MG_SWEEPS];
    k.omega = g_tune[GW_TUNE_MG_OMEGA];
    k.tail = g_tune[GW_TUNE_MG_TAIL];
    k.bf16 = g_tune[GW_TUNE_MG_BF16];
    k.fine_sweeps = g_tune[GW_TUNE_MG_FINE_SWEEPS];
    for (int q = 0; q < 3; ++q) k.n_grid[q] = grid.n_grid[q];
    for (int q = 0; q < h.nl; ++q) { k.n_rows[q] = h.lv[q].A.n_rows; k.nnzb[q] = h.lv[q].A.nnzb; }
    k.A = *A; k.ws = ws; k.b = G.b; k.x = G.x; k.z = G.z;
    MgGraphs &cache = mg_graphs();
    {
        std::lock_guard<std::mutex> lk(cache.mu);
        for (MgGraphEntry &ent : cache.e)
            if (ent.graph && memcmp(&ent.key, &k, sizeof(k)) == 0) {
                ent.stamp = ++cache.clock;
                *out = ent.graph;
                return GW_OK;
            }
    }
    PtrsA a = make_ptrs(*A);
    auto made = std::make_shared<StepGraph>();
    auto step = [&](cudaStream_t cs) { mg_arnoldi_step<NF, VT>(h, a, G, Z, restart, skip, cs); };
    const int rc = capture_graph(step, made.get());
    if (rc) return rc;
    *out = made;
    std::shared_ptr<const StepGraph> replaced;  // released outside the lock
    std::lock_guard<std::mutex> lk(cache.mu);
    MgGraphEntry *slot = &cache.e[0];  // an empty slot first, else the least recently used one
    for (MgGraphEntry &ent : cache.e)
        if (slot->graph && (!ent.graph || ent.stamp < slot->stamp)) slot = &ent;
    replaced = std::move(slot->graph);
    slot->key = k;
    slot->graph = std::move(made);
    slot->stamp = ++cache.clock;
    return GW_OK;
}

template <int NF, typename VT>
int gmres_mg(const gw_grid_t *grid, const gw_bsr_t *A, gw_mg_plan_t *plan_in, const double *b, double *x,
             double rtol, int max_iter, int restart, void *ws, int64_t ws_bytes, int *iters, double *relres,
             cudaStream_t s) {
    const int nr = A->n_rows;
    if (nr == 0) { *iters = 0; *relres = 0.0; return GW_OK; }
    const int64_t n = (int64_t)nr * NF;
    (void)tail_cluster_max<NF, VT>();  // device queries before any stream capture
    {
        const int tb = tune_rows_block();
        (void)resident_rows_grid((const void *)k_mg_jacobi<NF, VT>, tb, 1);
        (void)resident_rows_grid((const void *)k_mg_presmooth2<NF, VT>, tb, 1);
        (void)resident_rows_grid((const void *)k_mg_residual<NF, VT>, tb, 1);
        (void)resident_rows_grid((const void *)k_mg_jacobi<NF, __nv_bfloat16>, tb, 1);
        (void)resident_rows_grid((const void *)k_mg_presmooth2<NF, __nv_bfloat16>, tb, 1);
        (void)resident_rows_grid((const void *)k_mg_residual<NF, __nv_bfloat16>, tb, 1);
        (void)resident_rows_grid((const void *)k_gm_spmv_keep<NF, VT>, kThreads, 1);
    }
    Bump bp{(char *)ws, 0};
    MgHier h;
    FlexVecs fv;
    mg_carve_hier(bp, h, *grid, nr, NF);
    mg_carve_flex(bp, fv, n, restart);
    if (bp.used > ws_bytes) {
        snprintf(g_msg, sizeof(g_msg), "multigrid GMRES: workspace of %lld bytes, %lld needed", (long long)ws_bytes,
                 (long long)bp.used);
        return GW_EINVAL;
    }
    int rc;
    {
        ProfScope ps(PC_MG_SETUP, s, (double)A->nnzb * (NF * NF * sizeof(VT) + 4));
        gw_mg_plan_t local;
        if (plan_in) {
            if (plan_in->workspace != ws || plan_in->nf != NF || plan_in->fine_n_rows != nr ||
                plan_in->fine_nnzb != A->nnzb || plan_in->row_ptr != A->row_ptr || plan_in->cols != A->cols ||
                plan_in->levels < 1 || plan_in->levels > h.nl ||
                plan_in->dense_n != plan_in->n_rows[plan_in->levels - 1] * NF || plan_in->dense_n > kMgCoarseMax) {
                snprintf(g_msg, sizeof(g_msg), "multigrid GMRES: the plan was built for another workspace or pattern");
                return GW_EINVAL;
            }
            mg_apply_plan(h, A, plan_in, NF);
        } else {
            rc = mg_pattern<NF>(h, A, &local, s);
            if (rc) return rc;
        }
        // lag: the previous solve's coarse operators, smoothers and dense
        // inverse are still in the workspace; GMRES itself applies A
        rc = (plan_in && plan_in->lag) ? GW_OK : mg_numeric<NF, VT>(h, s);
        // the V-cycle's BF16 copy of the fine level follows the current A on
        // every solve, lagged or not (the fine level's own rows are never lagged)
        if (!rc && grid->dim == 2) {
            const bool fresh = !(plan_in && plan_in->lag);
            rc = sell_values<NF, VT>(h, fresh, s);
            if (!rc) rc = tail_image<NF, VT>(h, s);
        } else if (!rc && mg_bf16_fine<VT>()) {
            const size_t nv = (size_t)A->nnzb * NF * NF;
            k_to_bf16<<<gw_count_launch(red_grid_elems((int64_t)nv)), kThreads, 0, s>>>(
                (const float *)A->vals, (__nv_bfloat16 *)h.lv[0].pvals, nv);
            GW_LAUNCHED();
        }
    }
    if (rc) return rc;
    PtrsA a = make_ptrs(*A);
    GmresVecs G;
    G.V = fv.V; G.w = fv.w; G.partials = fv.partials; G.sc = fv.sc; G.Minv = nullptr;
    G.x = x; G.b = b; G.n = (size_t)n;
    G.z = nullptr;
    const size_t head = offsetof(GScalars, H);
    k_gm_begin<<<gw_count_launch(1), 32, 0, s>>>(G.sc, max_iter, restart, ::pow(10.0, -0.1 * g_tune[GW_TUNE_GS_CANCEL]));
    const int gr = red_grid_rows(nr), gv = red_grid_elems(n);
    const VecRef z{fv.Z, (size_t)n};
    const int *skip = &G.sc->cycle_done;
    std::shared_ptr<const StepGraph> step_graph;
    GScalars hs;
    memset(&hs, 0, head);
    int first = 1;
    StallWatch stall;
    g_last_stalled = 0;
    for (int cycle = 0; cycle < 1000000; ++cycle) {
        k_gm_residual<NF, VT><<<gw_count_launch(gr), kThreads, 0, s>>>(a, G, first, rtol);
        GW_LAUNCHED();
        mg_step_tail<NF, VT>(h, G, z, 1, skip, s);
        GW_LAUNCHED();
        // the first cycle of a plan that has solved before queues its steps at once:
        // from a zero start |r| / tol is 1 / rtol, and a wrong guess costs steps that
        // return at once
        const bool ahead = first && plan_in && plan_in->last_rate > 0 && rtol > 0.0 && rtol < 1.0;
        first = 0;
        if (!ahead) {
            GW_CUDA(cudaMemcpyAsync(&hs, G.sc, head, cudaMemcpyDeviceToHost, s));
            GW_CUDA(cudaStreamSynchronize(s));
            if (hs.done) break;
        }
        if (!ahead && stall.stalled(hs.beta)) { g_last_stalled = 1; break; }
        // Arnoldi steps queued before the next host check.  A step queued past
        // convergence costs as much as one that counts, a check 10-15 us of idle
        // device: nine tenths of the steps that the previous solve's convergence
        // rate predicts (solves of one load step contract alike), then what the
        // observed rate leaves.
        int chunk = 4;
        if (ahead)
            chunk = (int)std::min(-0.9 * ::log(rtol) / (1e-3 * plan_in->last_rate), 1e6);
        else if (plan_in && plan_in->last_rate > 0 && hs.tol > 0.0 && hs.beta > hs.tol)
            chunk = (int)std::min(0.9 * ::log(hs.beta / hs.tol) / (1e-3 * plan_in->last_rate), 1e6);
        else if (plan_in && plan_in->last_iters > 0)
            chunk = std::min(plan_in->last_iters, 16);
        chunk = std::min(std::max(chunk, 1), std::min(restart, std::max(max_iter - hs.iters, 1)));
        bool counted = false;
        for (;;) {
            if (!g_prof_on && !step_graph) {  // timed runs launch kernel by kernel, bracketed by events
                rc = mg_step_graph<NF, VT>(h, *grid, A, G, fv.Z, ws, restart, skip, &step_graph);
                if (rc) return rc;
            }
            for (int it = 0; it < chunk; ++it) {
                if (step_graph) {
                    rc = step_graph->replay(s);
                    if (rc) return rc;
                } else {
                    mg_arnoldi_step<NF, VT>(h, a, G, fv.Z, restart, skip, s);
                }
            }
            GW_LAUNCHED();
            GW_CUDA(cudaMemcpyAsync(&hs, G.sc, head, cudaMemcpyDeviceToHost, s));
            GW_CUDA(cudaStreamSynchronize(s));
            if (ahead && !counted) {
                counted = true;
                (void)stall.stalled(hs.beta);  // the first cycle's entry of the window
            }
            if (hs.cycle_done) break;
            int next = std::min(chunk < 16 ? chunk * 2 : 16, restart - hs.k);
            if (hs.k > 0 && hs.beta > 0.0 && hs.resid > 0.0 && hs.resid < hs.beta && hs.tol > 0.0) {
                const double rate = ::pow(hs.resid / hs.beta, 1.0 / hs.k);
                if (rate < 1.0) {
                    const double left = ::ceil(::log(hs.tol / hs.resid) / ::log(rate));
                    next = (int)std::min(std::max(left, 1.0), (double)(restart - hs.k));
                }
            }
            chunk = next;
        }
        if (hs.status) break;
        k_gm_solve_y<<<gw_count_launch(1), 32, 0, s>>>(G.sc);
        k_gm_update_x_flex<<<gw_count_launch(gv), kThreads, 0, s>>>((size_t)n, G, fv.Z);
        GW_LAUNCHED();
    }
    *iters = hs.iters;
    g_last_reorths = hs.reorths;
    *relres = (hs.bnorm > 0.0) ? hs.resid / hs.bnorm : 0.0;
    if (plan_in) {
        plan_in->last_iters = hs.iters;
        plan_in->last_rate = 0;
        if (hs.iters > 0 && hs.resid > 0.0 && hs.resid < hs.bnorm)
            plan_in->last_rate = (int)(1e3 * ::log(hs.bnorm / hs.resid) / hs.iters);
    }
    // the header carries the guard of every kernel up to the last residual
    rc = (hs.guard || hs.status) ? guard_check(s, "multigrid GMRES") : GW_OK;
    if (rc) return rc;
    if (hs.status == ST_NAN) return GW_ENAN;
    if (hs.resid > hs.tol) return GW_ENOCONV;
    return GW_OK;
}

template <typename VT>
int gmres_mg_nf(const gw_grid_t *grid, const gw_bsr_t *A, gw_mg_plan_t *plan, const double *b, double *x,
                double rtol, int max_iter, int restart, void *ws, int64_t ws_bytes, int *iters, double *relres,
                cudaStream_t s) {
    switch (A->nf) {
        case 1: return gmres_mg<1, VT>(grid, A, plan, b, x, rtol, max_iter, restart, ws, ws_bytes, iters, relres, s);
        case 2: return gmres_mg<2, VT>(grid, A, plan, b, x, rtol, max_iter, restart, ws, ws_bytes, iters, relres, s);
        case 3: return gmres_mg<3, VT>(grid, A, plan, b, x, rtol, max_iter, restart, ws, ws_bytes, iters, relres, s);
        case 4: return gmres_mg<4, VT>(grid, A, plan, b, x, rtol, max_iter, restart, ws, ws_bytes, iters, relres, s);
        default: return GW_EINVAL;
    }
}

int mg_check_args(const gw_grid_t *grid, const gw_bsr_t *A) {
    GW_REQUIRE(grid->dim == 2 || grid->dim == 3);
    GW_REQUIRE(A->mask_words == (grid->dim == 2 ? 1 : 4));
    GW_REQUIRE(A->n_rows <= grid->n_nodes);
    GW_REQUIRE(A->nf >= 1 && A->nf <= 4);
    return GW_OK;
}
}  // namespace

extern "C" int64_t gw_gmres_mg_workspace_bytes(const gw_grid_t *grid, int32_t n_rows, int32_t nf, int32_t restart) {
    if (!grid || restart < 1 || restart > kGmresMaxRestart || nf < 1 || nf > 4 || n_rows < 0) return -1;
    return mg_ws_bytes(*grid, n_rows, nf, restart);
}

extern "C" int gw_mg_plan_build(const gw_grid_t *grid, const gw_bsr_t *A, void *workspace, int64_t workspace_bytes,
                                gw_mg_plan_t *plan_host, void *stream) {
    GW_REQUIRE(grid && A && workspace && plan_host);
    int rc = mg_check_args(grid, A);
    if (rc) return rc;
    Bump bp{(char *)workspace, 0};
    MgHier h;
    mg_carve_hier(bp, h, *grid, A->n_rows, A->nf);
    if (bp.used > workspace_bytes) {
        snprintf(g_msg, sizeof(g_msg), "multigrid plan: workspace of %lld bytes, %lld needed",
                 (long long)workspace_bytes, (long long)bp.used);
        return GW_EINVAL;
    }
    cudaStream_t s = S(stream);
    switch (A->nf) {
        case 1: rc = mg_pattern<1>(h, A, plan_host, s); break;
        case 2: rc = mg_pattern<2>(h, A, plan_host, s); break;
        case 3: rc = mg_pattern<3>(h, A, plan_host, s); break;
        default: rc = mg_pattern<4>(h, A, plan_host, s); break;
    }
    if (rc) return rc;
    plan_host->workspace = workspace;
    return GW_OK;
}

extern "C" int32_t gw_gmres_last_reorths(void) { return g_last_reorths; }
extern "C" int32_t gw_gmres_last_stalled(void) { return g_last_stalled; }

extern "C" int gw_bsr_gmres_mg_solve(const gw_grid_t *grid, const gw_bsr_t *A, int32_t prec,
                                     gw_mg_plan_t *plan_host, const double *b, double *x, double rtol,
                                     int32_t max_iter, int32_t restart, void *workspace, int64_t workspace_bytes,
                                     int32_t *iters_host, double *relres_host, void *stream) {
    GW_REQUIRE(grid && A && b && x && workspace && iters_host && relres_host && max_iter > 0);
    GW_REQUIRE(vec_ok(A, b, x));
    GW_REQUIRE(restart >= 1 && restart <= kGmresMaxRestart);
    int rc = mg_check_args(grid, A);
    if (rc) return rc;
    int it = 0;
    double rr = 0.0;
    rc = (prec == GW_PREC_F64)
             ? gmres_mg_nf<double>(grid, A, plan_host, b, x, rtol, max_iter, restart, workspace, workspace_bytes, &it,
                                   &rr, S(stream))
             : gmres_mg_nf<float>(grid, A, plan_host, b, x, rtol, max_iter, restart, workspace, workspace_bytes, &it,
                                  &rr, S(stream));
    *iters_host = it;
    *relres_host = rr;
    return rc;
}

extern "C" int64_t gw_krylov_workspace_bytes(int32_t n_rows, int32_t nf, int32_t prec) {
    (void)prec;
    return krylov_ws_bytes(n_rows, nf);
}

extern "C" int gw_bsr_krylov_solve(const gw_bsr_t *A, int32_t prec, int32_t method, int32_t precond, const double *b,
                                   double *x, double rtol, int32_t max_iter, void *workspace, int32_t *iters_host,
                                   double *relres_host, void *stream) {
    GW_REQUIRE(A && b && x && workspace && iters_host && relres_host && max_iter > 0);
    GW_REQUIRE(vec_ok(A, b, x));
    int it = 0;
    double rr = 0.0;
    int rc = (prec == GW_PREC_F64)
                 ? krylov_nf<double>(A, method, precond, b, x, rtol, max_iter, workspace, &it, &rr, S(stream))
                 : krylov_nf<float>(A, method, precond, b, x, rtol, max_iter, workspace, &it, &rr, S(stream));
    *iters_host = it;
    *relres_host = rr;
    return rc;
}

// ==================================================================== Krylov without a caller workspace
// For callers that cannot allocate device memory themselves: a host whose own
// memory manager owns the device heap, or a code path where calling cudaMalloc
// is not allowed.  The scratch the BiCGSTAB / CG driver needs lives in one
// file-scope device array, sized for at most kStaticKrylovMaxUnknowns unknowns
// (n_rows * nf); every GPU that loads the library holds it (about 12.6 MB)
// until the process exits.
namespace {
constexpr int64_t kStaticKrylovMaxUnknowns = 131072;
constexpr int64_t align256c(int64_t b) { return (b + 255) & ~(int64_t)255; }
// krylov_ws_bytes at the limit, for the largest block size (nf = 4)
constexpr int64_t kStaticKrylovBytes = 8 * align256c(8 * kStaticKrylovMaxUnknowns) +
                                       align256c(8 * kStaticKrylovMaxUnknowns * 4) +
                                       align256c(8 * (int64_t)kRedBlocks * 4) + align256c(sizeof(KScalars));
static __device__ __align__(256) unsigned char g_krylov_scratch[kStaticKrylovBytes];

constexpr int kMaxStaticDevices = 64;
void *g_krylov_scratch_addr[kMaxStaticDevices] = {};

// Device address of g_krylov_scratch on the current device.  The name is only a
// host-side stand-in, so the address is looked up once per device, with that
// device current, and cached.
int static_krylov_scratch(void **out) {
    int dev = 0;
    GW_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kMaxStaticDevices) {
        snprintf(g_msg, sizeof(g_msg), "gw_bsr_krylov_solve_static: device ordinal %d above %d", dev,
                 kMaxStaticDevices - 1);
        return GW_EINVAL;
    }
    void *p = __atomic_load_n(&g_krylov_scratch_addr[dev], __ATOMIC_ACQUIRE);
    if (!p) {
        GW_CUDA(cudaGetSymbolAddress(&p, g_krylov_scratch));
        __atomic_store_n(&g_krylov_scratch_addr[dev], p, __ATOMIC_RELEASE);
    }
    *out = p;
    return GW_OK;
}
}  // namespace

extern "C" int64_t gw_krylov_static_max_unknowns(void) { return kStaticKrylovMaxUnknowns; }

extern "C" int gw_bsr_krylov_solve_static(const gw_bsr_t *A, int32_t prec, int32_t method, int32_t precond,
                                          const double *b, double *x, double rtol, int32_t max_iter,
                                          int32_t *iters_host, double *relres_host, void *stream) {
    GW_REQUIRE(A && b && x && iters_host && relres_host && max_iter > 0);
    GW_REQUIRE(vec_ok(A, b, x));
    const int64_t unknowns = (int64_t)A->n_rows * A->nf;
    if (A->n_rows < 0 || A->nf < 1 || A->nf > 4 || unknowns > kStaticKrylovMaxUnknowns ||
        krylov_ws_bytes(A->n_rows, A->nf) > kStaticKrylovBytes) {
        snprintf(g_msg, sizeof(g_msg),
                 "gw_bsr_krylov_solve_static: %lld unknowns (n_rows %d x nf %d) exceed the static scratch limit of "
                 "%lld unknowns; use gw_bsr_krylov_solve with a caller workspace",
                 (long long)unknowns, A->n_rows, A->nf, (long long)kStaticKrylovMaxUnknowns);
        return GW_EINVAL;
    }
    void *ws = nullptr;
    const int rs = static_krylov_scratch(&ws);
    if (rs != GW_OK) return rs;
    // the driver clears the scalar block (reduction ticket, flags) on every call
    // and writes every vector before reading it, so the contents a previous call
    // left in the scratch are never used
    int it = 0;
    double rr = 0.0;
    int rc = (prec == GW_PREC_F64)
                 ? krylov_nf<double>(A, method, precond, b, x, rtol, max_iter, ws, &it, &rr, S(stream))
                 : krylov_nf<float>(A, method, precond, b, x, rtol, max_iter, ws, &it, &rr, S(stream));
    *iters_host = it;
    *relres_host = rr;
    return rc;
}

namespace {
template <typename VT>
int spmv_any(const gw_bsr_t *A, const double *x, double *y, bool trans, cudaStream_t s) {
    PtrsA a = make_ptrs(*A);
    const int g = red_grid_rows(A->n_rows);
    if (A->n_rows == 0) return GW_OK;
    if (trans) GW_CUDA(cudaMemsetAsync(y, 0, sizeof(double) * (size_t)A->n_rows * A->nf, s));
#define GW_SPMV_CASE(NF_)                                                  \
    case NF_:                                                              \
        if (trans) k_spmv_t<NF_, VT><<<gw_count_launch(g), kThreads, 0, s>>>(a, x, y);      \
        else k_spmv<NF_, VT><<<gw_count_launch(g), kThreads, 0, s>>>(a, x, y);              \
        break;
    switch (A->nf) {
        GW_SPMV_CASE(1) GW_SPMV_CASE(2) GW_SPMV_CASE(3) GW_SPMV_CASE(4)
        default: return GW_EINVAL;
    }
#undef GW_SPMV_CASE
    GW_LAUNCHED();
    return GW_OK;
}
}  // namespace

extern "C" int gw_bsr_spmv(const gw_bsr_t *A, int32_t prec, const double *x, double *y, void *stream) {
    GW_REQUIRE(A && x && y);
    GW_REQUIRE(vec_ok(A, x, y));
    return prec == GW_PREC_F64 ? spmv_any<double>(A, x, y, false, S(stream)) : spmv_any<float>(A, x, y, false, S(stream));
}

extern "C" int gw_bsr_spmv_t(const gw_bsr_t *A, int32_t prec, const double *x, double *y, void *stream) {
    GW_REQUIRE(A && x && y);
    return prec == GW_PREC_F64 ? spmv_any<double>(A, x, y, true, S(stream)) : spmv_any<float>(A, x, y, true, S(stream));
}