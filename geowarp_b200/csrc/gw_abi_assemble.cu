// C ABI, residual and element-tangent assembly (declarations and reference
// citations in include/geowarp_b200.h): the deterministic cell-sum
// assembly of the 2D kinds (gw_assemble_sorted) and the atomic one
// (gw_assemble, used for the 3D kind).
#include <algorithm>

#include "gw_host.cuh"
#include "gw_assemble.cuh"

using namespace gw;
using namespace gwh;

namespace {
template <int KIND, typename VT>
void assemble_per_model(const LaunchConst &c, const PtrsP &p, const int *perm, const uint8_t *fm, const double *un,
                        const double *uo, const PtrsA &a, double *R, double *force, int b, cudaStream_t s) {
    const int pb = g_tune[GW_TUNE_PARTICLE_BLOCK];
    switch (c.mc.model) {
        case GW_MODEL_HENCKY: k_assemble<KIND, true, VT, GW_MODEL_HENCKY><<<gw_count_launch(b), pb, 0, s>>>(c, p, perm, fm, un, uo, a, R, force); break;
        case GW_MODEL_J2: k_assemble<KIND, true, VT, GW_MODEL_J2><<<gw_count_launch(b), pb, 0, s>>>(c, p, perm, fm, un, uo, a, R, force); break;
        case GW_MODEL_NEOHOOKEAN: k_assemble<KIND, true, VT, GW_MODEL_NEOHOOKEAN><<<gw_count_launch(b), pb, 0, s>>>(c, p, perm, fm, un, uo, a, R, force); break;
        case GW_MODEL_LINEAR: k_assemble<KIND, true, VT, GW_MODEL_LINEAR><<<gw_count_launch(b), pb, 0, s>>>(c, p, perm, fm, un, uo, a, R, force); break;
        case GW_MODEL_DP: k_assemble<KIND, true, VT, GW_MODEL_DP><<<gw_count_launch(b), pb, 0, s>>>(c, p, perm, fm, un, uo, a, R, force); break;
        default: k_assemble<KIND, true, VT><<<gw_count_launch(b), pb, 0, s>>>(c, p, perm, fm, un, uo, a, R, force); break;
    }
}

// 3D: whether one thread per particle (k_assemble) is the faster assembly of n.
// Residual only: its 27 nodes are too little work to spread (10,648 particles 84 us
// against 87, 32,768: 91 against 175, 262,144: 546 against 1,290; 8,000: 82 against 65).
// With an FP64 tangent it takes one wave of 148 x 256 threads (255 registers) after the
// other, 2.1 ms each, and k_assemble3 59 ns a particle: worth it where the waves are
// full (110,592 particles 6.29 ms against 6.61, 262,144: 14.7 against 15.5; 175,616,
// 93% full: 10.35 against 10.40; 64,000: 4.07 against 3.86).  With an FP32 tangent
// never (110,592: 5.95 against 6.01, 262,144: 13.9 against 13.8).
bool thread_per_particle3(int n, bool want_K, int prec) {
    if (!want_K) return n > 10240;
    constexpr int64_t wave = 148 * 256;
    return prec == GW_PREC_F64 && 15 * ((n + wave - 1) / wave * wave) < 16 * (int64_t)n;
}

// k_assemble3: eight particles per CTA (27 threads each) up to two CTAs per SM, then
// 32, a whole warp's worth of evaluations.  FP64 with tangent, 8 / 32 a CTA: 1,000 particles
// 146 / 302 us, 1,728: 233 / 305, 2,744: 322 / 304, 4,096: 435 / 304; residual only 47 / 47,
// 58 / 48, 73 / 41, 91 / 41.
template <bool WANT_K, typename VT>
int launch_assemble3(const LaunchConst &c, const PtrsP &p, const int *perm, const uint8_t *fm, const double *un,
                     const double *uo, const PtrsA &a, double *R, double *force, cudaStream_t s) {
    const int P = p.n <= 8 * 2 * 148 ? 8 : 32;
    auto k = k_assemble3<WANT_K, VT>;
    const int smem = P * (int)sizeof(Scatter3<WANT_K>);
    GW_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, 32 * (int)sizeof(Scatter3<WANT_K>)));
    k<<<gw_count_launch(nblk(p.n, P)), 256, smem, s>>>(c, p, P, perm, fm, un, uo, a, R, force);
    GW_LAUNCHED();
    return GW_OK;
}

template <int KIND>
int launch_assemble(const LaunchConst &c, const PtrsP &p, const int *perm, const uint8_t *fm, const double *un,
                    const double *uo, const gw_bsr_t *A, int prec, double *R, double *force, const PtrsA &a,
                    cudaStream_t s) {
    const int pb = g_tune[GW_TUNE_PARTICLE_BLOCK];
    const int b = nblk(p.n, pb);
    if (p.n > 0) {
        const int D = KindTraits<KIND>::D, NF = KindTraits<KIND>::NF, NS = KindTraits<KIND>::NS;
        // algorithmic bytes, each array once: particle state in (x, lp, F_old,
        // b_old, E) and out (F_new, b_new, sigma), the grid vectors (u_new, u_old,
        // R) and the matrix values
        (void)NS;
        const double per_p = 8.0 * (2 * D + 9 + 9 + 1) + 8.0 * 27;
        const double grid = 8.0 * 3 * (double)A->n_rows * NF;
        const bool want_K = A->vals != nullptr;
        const double mat = want_K ? (double)A->nnzb * NF * NF * (prec == GW_PREC_F64 ? 8 : 4) : 0.0;
        ProfScope ps(PC_ASSEMBLE, s, per_p * p.n + grid + mat);
        if constexpr (KIND == GW_KIND_COUPLED3D) {
            int rc;
            if (thread_per_particle3(p.n, want_K, prec)) {
                if (want_K) k_assemble<KIND, true, double><<<gw_count_launch(b), pb, 0, s>>>(c, p, perm, fm, un, uo, a, R, force);
                else k_assemble<KIND, false, double><<<gw_count_launch(b), pb, 0, s>>>(c, p, perm, fm, un, uo, a, R, force);
                rc = GW_OK;
            } else if (!want_K) rc = launch_assemble3<false, double>(c, p, perm, fm, un, uo, a, R, force, s);
            else if (prec == GW_PREC_F64) rc = launch_assemble3<true, double>(c, p, perm, fm, un, uo, a, R, force, s);
            else rc = launch_assemble3<true, float>(c, p, perm, fm, un, uo, a, R, force, s);
            if (rc) return rc;
        } else if (!want_K) {
            k_assemble<KIND, false, double><<<gw_count_launch(b), pb, 0, s>>>(c, p, perm, fm, un, uo, a, R, force);
        } else if constexpr (KIND == GW_KIND_SOLID2D) {
            // the 2D solid tangent kernel is instantiated per material, so each
            // carries only its own constitutive code (fewer registers and spills)
            if (prec == GW_PREC_F64) assemble_per_model<KIND, double>(c, p, perm, fm, un, uo, a, R, force, b, s);
            else assemble_per_model<KIND, float>(c, p, perm, fm, un, uo, a, R, force, b, s);
        } else {
            if (prec == GW_PREC_F64) k_assemble<KIND, true, double><<<gw_count_launch(b), pb, 0, s>>>(c, p, perm, fm, un, uo, a, R, force);
            else k_assemble<KIND, true, float><<<gw_count_launch(b), pb, 0, s>>>(c, p, perm, fm, un, uo, a, R, force);
        }
        GW_LAUNCHED();
    }
    if (A->vals && A->n_rows > 0) {
        const int D = KindTraits<KIND>::D;
        if (prec == GW_PREC_F64) k_identity_dirichlet<D, double><<<gw_count_launch(nblk(A->n_rows, kThreads)), kThreads, 0, s>>>(a, fm);
        else k_identity_dirichlet<D, float><<<gw_count_launch(nblk(A->n_rows, kThreads)), kThreads, 0, s>>>(a, fm);
        GW_LAUNCHED();
    }
    return GW_OK;
}
}  // namespace

extern "C" int gw_assemble(const gw_grid_t *grid, const gw_material_t *mat, const gw_step_t *st,
                           const gw_particles_t *pt, const int32_t *perm, const uint8_t *free_mask,
                           const double *u_new, const double *u_old, const gw_bsr_t *A, int32_t prec, double *R_rows,
                           double *force, void *stream) {
    GW_REQUIRE(grid && mat && st && pt && perm && free_mask && u_new && u_old && R_rows);
    // the row map is needed for the residual even without a matrix
    GW_REQUIRE(A && A->node2row && (A->n_rows == 0 || A->row2node));
    GW_REQUIRE(mat->model >= 0 && mat->model <= GW_MODEL_NORSAND);
    cudaStream_t s = S(stream);
    LaunchConst c = make_lc(grid, mat, st);
    PtrsP p = make_ptrs(*pt);
    PtrsA a = make_ptrs(*A);
    if (A->vals) {
        GW_REQUIRE(A->row_ptr && A->cols && A->stencil);
        const size_t vb = (prec == GW_PREC_F64 ? 8 : 4) * (size_t)A->nnzb * A->nf * A->nf;
        GW_CUDA(cudaMemsetAsync(A->vals, 0, vb, s));
    }
    GW_CUDA(cudaMemsetAsync(R_rows, 0, sizeof(double) * (size_t)A->n_rows * A->nf, s));
    switch (grid->kind) {
        case GW_KIND_SOLID2D: return launch_assemble<GW_KIND_SOLID2D>(c, p, perm, free_mask, u_new, u_old, A, prec, R_rows, force, a, s);
        case GW_KIND_COUPLED2D: return launch_assemble<GW_KIND_COUPLED2D>(c, p, perm, free_mask, u_new, u_old, A, prec, R_rows, force, a, s);
        case GW_KIND_COUPLED3D: return launch_assemble<GW_KIND_COUPLED3D>(c, p, perm, free_mask, u_new, u_old, A, prec, R_rows, force, a, s);
        default: return GW_EINVAL;
    }
}

// ==================================================================== deterministic assembly
namespace {
// The workspace: cell starts and ends, boxes, particle records, cell sums.
struct AsmParts {
    int64_t cend, box, rec, sums, bytes;
};
// Cells whose sums are held at once: all of them in batches of up to half a million
// (1.4 GB in the solid kind, 3.2 GB in u-p); a larger grid goes in bands of rows of
// cells, at least 16 rows high, whose last two rows the next band computes again.
// Where particles are fewer than cells, the sums lie at a cell's first particle, unless
// they are more than a band and at least a quarter of the cells (each band looks at every
// row, which a grid of mostly empty cells would not repay).
constexpr int64_t kSumCells = 1 << 19;
int64_t sum_cells(const gw_grid_t &g) {
    const int64_t nc = (int64_t)g.n_grid[0] * g.n_grid[1], most = std::max<int64_t>(kSumCells, 16 * g.n_grid[0]);
    return nc < most ? nc : most / g.n_grid[0] * g.n_grid[0];
}
bool sums_by_cell(const gw_grid_t &g, int64_t n) {
    const int64_t nc = (int64_t)g.n_grid[0] * g.n_grid[1];
    return nc <= n || (sum_cells(g) < n && nc <= 4 * n);
}
AsmParts asm_parts(const gw_grid_t &g, int64_t n, int64_t rec_bytes, int64_t sum_bytes) {
    AsmParts w;
    const int64_t n_cells = (int64_t)g.n_grid[0] * g.n_grid[1], c = align256(4 * n_cells);
    w.cend = c;
    w.box = 2 * c;
    w.rec = 3 * c;
    w.sums = w.rec + align256(rec_bytes * n);
    w.bytes = w.sums + sum_bytes * (sums_by_cell(g, n) ? sum_cells(g) : n);
    return w;
}

template <int KIND, typename VT>
int64_t q_record_bytes() { return QRecord<KIND, VT>::BYTES; }

int64_t record_bytes(int kind, int prec) {
    switch (kind) {
        case GW_KIND_SOLID2D: return prec == GW_PREC_F64 ? q_record_bytes<GW_KIND_SOLID2D, double>() : q_record_bytes<GW_KIND_SOLID2D, float>();
        case GW_KIND_COUPLED2D: return prec == GW_PREC_F64 ? q_record_bytes<GW_KIND_COUPLED2D, double>() : q_record_bytes<GW_KIND_COUPLED2D, float>();
        default: return 0;
    }
}

template <int KIND, bool WANT_K, typename VT>
void launch_particle_q(const LaunchConst &c, const PtrsP &p, const int *perm, const double *un, const double *uo,
                       unsigned char *scratch, double *force, cudaStream_t s) {
    const int pb = g_tune[GW_TUNE_PARTICLE_BLOCK];
    const int b = nblk(p.n, pb);
    if constexpr (KIND == GW_KIND_SOLID2D && WANT_K) {
        // one instantiation per material: each carries only its own constitutive code
        switch (c.mc.model) {
            case GW_MODEL_HENCKY: k_particle_q<KIND, WANT_K, VT, GW_MODEL_HENCKY><<<gw_count_launch(b), pb, 0, s>>>(c, p, perm, un, uo, scratch, force); return;
            case GW_MODEL_J2: k_particle_q<KIND, WANT_K, VT, GW_MODEL_J2><<<gw_count_launch(b), pb, 0, s>>>(c, p, perm, un, uo, scratch, force); return;
            case GW_MODEL_NEOHOOKEAN: k_particle_q<KIND, WANT_K, VT, GW_MODEL_NEOHOOKEAN><<<gw_count_launch(b), pb, 0, s>>>(c, p, perm, un, uo, scratch, force); return;
            case GW_MODEL_LINEAR: k_particle_q<KIND, WANT_K, VT, GW_MODEL_LINEAR><<<gw_count_launch(b), pb, 0, s>>>(c, p, perm, un, uo, scratch, force); return;
            case GW_MODEL_DP: k_particle_q<KIND, WANT_K, VT, GW_MODEL_DP><<<gw_count_launch(b), pb, 0, s>>>(c, p, perm, un, uo, scratch, force); return;
            default: break;
        }
    }
    k_particle_q<KIND, WANT_K, VT><<<gw_count_launch(b), pb, 0, s>>>(c, p, perm, un, uo, scratch, force);
}

template <int KIND, bool WANT_K, typename VT>
int assemble_sorted(const LaunchConst &c, const PtrsP &p, const int *perm, const int *keys, const uint8_t *fm,
                    const double *un, const double *uo, const gw_bsr_t *A, double *R, double *force, const PtrsA &a,
                    char *ws, int64_t ws_bytes, cudaStream_t s) {
    const int ncx = c.g.n_grid[0], ncy = c.g.n_grid[1];
    // the records written below must fit the caller's workspace (record size
    // of this instantiation, not of another precision)
    const AsmParts w = asm_parts(c.g, p.n, QRecord<KIND, VT>::BYTES, 8 * CellSums<KIND>::ND);
    if (w.bytes > ws_bytes) {
        snprintf(g_msg, sizeof(g_msg), "gw_assemble_sorted: workspace of %lld bytes, %lld needed",
                 (long long)ws_bytes, (long long)w.bytes);
        return GW_EINVAL;
    }
    int *cstart = (int *)ws, *cend = (int *)(ws + w.cend), *box = (int *)(ws + w.box);
    unsigned char *scratch = (unsigned char *)(ws + w.rec);
    double *sums = (double *)(ws + w.sums);
    const int by_cell = sums_by_cell(c.g, p.n);
    const int D = KindTraits<KIND>::D, NF = KindTraits<KIND>::NF;
    // algorithmic bytes, each array once: particle state in (x, lp, F_old, b_old,
    // E) and out (F_new, b_new, sigma), the scratch records written and read
    // back, the grid vectors (u_new, u_old, R) and the matrix values
    const double per_p = 8.0 * (2 * D + 9 + 9 + 1) + 8.0 * 27 + 2.0 * QRecord<KIND, VT>::BYTES;
    const double grid = 8.0 * 3 * (double)A->n_rows * NF;
    const double mat = WANT_K ? (double)A->nnzb * NF * NF * sizeof(VT) : 0.0;
    ProfScope ps(PC_ASSEMBLE, s, per_p * p.n + grid + mat);
    GW_CUDA(cudaMemsetAsync(ws, 0, w.box, s));  // cells without particles: start = end = 0
    k_cell_ranges<<<gw_count_launch(nblk(p.n, kThreads)), kThreads, 0, s>>>(c.g, keys, p.n, fm, a.node2row, a.n_rows, cstart,
                                                                         cend);
    GW_LAUNCHED();
    launch_particle_q<KIND, WANT_K, VT>(c, p, perm, un, uo, scratch, force, s);
    GW_LAUNCHED();
    const int rows = by_cell ? (int)(sum_cells(c.g) / ncx) : ncy;  // rows of cells at once
    for (int y0 = 0;; y0 += rows - 2) {
        const int y1 = std::min(y0 + rows, ncy);
        k_cell_blocks<KIND, WANT_K, VT><<<gw_count_launch(nblk((int64_t)ncx * (y1 - y0), kCellGroups)), 16 * kCellGroups, 0, s>>>(
            c, y0 * ncx, y1 * ncx, by_cell, cstart, cend, scratch, sums, box);
        if (A->n_rows > 0)  // a node's cells start up to two rows below it
            k_row_gather<KIND, WANT_K, VT><<<gw_count_launch(nblk(A->n_rows, kGatherRows)), 32 * kGatherRows, 0, s>>>(
                c.g, by_cell, y0 * ncx, y0 ? y0 + 2 : 0, y1 < ncy ? y1 : ncy + 1, cstart, box, sums, fm, a, R);
        if (y1 == ncy) break;
    }
    GW_LAUNCHED();
    return GW_OK;
}

template <int KIND>
int assemble_sorted_kind(const LaunchConst &c, const PtrsP &p, const int *perm, const int *keys, const uint8_t *fm,
                         const double *un, const double *uo, const gw_bsr_t *A, int prec, double *R, double *force,
                         const PtrsA &a, char *ws, int64_t ws_bytes, cudaStream_t s) {
    int rc;
    if (p.n > 0) {
        // residual only (A->vals NULL) keeps the record layout of prec: the
        // workspace was sized for it (gw_assemble_workspace_bytes)
        const bool f64 = prec == GW_PREC_F64;
        if (!A->vals)
            rc = f64 ? assemble_sorted<KIND, false, double>(c, p, perm, keys, fm, un, uo, A, R, force, a, ws, ws_bytes, s)
                     : assemble_sorted<KIND, false, float>(c, p, perm, keys, fm, un, uo, A, R, force, a, ws, ws_bytes, s);
        else
            rc = f64 ? assemble_sorted<KIND, true, double>(c, p, perm, keys, fm, un, uo, A, R, force, a, ws, ws_bytes, s)
                     : assemble_sorted<KIND, true, float>(c, p, perm, keys, fm, un, uo, A, R, force, a, ws, ws_bytes, s);
        return rc;
    }
    // no particles: the rows the gather would write are zero, with their identity entries
    if (A->vals) GW_CUDA(cudaMemsetAsync(A->vals, 0, (prec == GW_PREC_F64 ? 8 : 4) * (size_t)A->nnzb * A->nf * A->nf, s));
    GW_CUDA(cudaMemsetAsync(R, 0, sizeof(double) * (size_t)A->n_rows * A->nf, s));
    if (A->vals && A->n_rows > 0) {
        if (prec == GW_PREC_F64) k_identity_dirichlet<2, double><<<gw_count_launch(nblk(A->n_rows, kThreads)), kThreads, 0, s>>>(a, fm);
        else k_identity_dirichlet<2, float><<<gw_count_launch(nblk(A->n_rows, kThreads)), kThreads, 0, s>>>(a, fm);
        GW_LAUNCHED();
    }
    return GW_OK;
}
}  // namespace

extern "C" int64_t gw_assemble_workspace_bytes(const gw_grid_t *grid, int32_t n_particles, int32_t prec) {
    if (!grid || n_particles < 0) return -1;
    if (grid->dim != 2) return 0;  // the 3D kind assembles with atomics and needs no workspace
    const int64_t sum = 8 * (grid->kind == GW_KIND_SOLID2D ? CellSums<GW_KIND_SOLID2D>::ND : CellSums<GW_KIND_COUPLED2D>::ND);
    return asm_parts(*grid, n_particles, record_bytes(grid->kind, prec), sum).bytes;
}

extern "C" int gw_assemble_sorted(const gw_grid_t *grid, const gw_material_t *mat, const gw_step_t *st,
                                  const gw_particles_t *pt, const int32_t *perm, const int32_t *keys,
                                  const uint8_t *free_mask, const double *u_new, const double *u_old, const gw_bsr_t *A,
                                  int32_t prec, double *R_rows, double *force, void *workspace, int64_t workspace_bytes,
                                  void *stream) {
    if (grid && grid->dim == 3)  // 3D: the atomic assembly
        return gw_assemble(grid, mat, st, pt, perm, free_mask, u_new, u_old, A, prec, R_rows, force, stream);
    GW_REQUIRE(grid && mat && st && pt && perm && keys && free_mask && u_new && u_old && R_rows && workspace);
    GW_REQUIRE(grid->kind == GW_KIND_SOLID2D || grid->kind == GW_KIND_COUPLED2D);
    GW_REQUIRE(A && A->node2row && (A->n_rows == 0 || A->row2node));
    GW_REQUIRE(mat->model >= 0 && mat->model <= GW_MODEL_NORSAND);
    GW_REQUIRE(((uintptr_t)workspace & 255u) == 0);
    const int64_t need = gw_assemble_workspace_bytes(grid, pt->n, prec);
    if (workspace_bytes < need) {
        snprintf(g_msg, sizeof(g_msg), "gw_assemble_sorted: workspace of %lld bytes, %lld needed",
                 (long long)workspace_bytes, (long long)need);
        return GW_EINVAL;
    }
    cudaStream_t s = S(stream);
    LaunchConst c = make_lc(grid, mat, st);
    PtrsP p = make_ptrs(*pt);
    PtrsA a = make_ptrs(*A);
    if (A->vals) GW_REQUIRE(A->row_ptr && A->cols && A->stencil);
    char *ws = (char *)workspace;
    if (grid->kind == GW_KIND_SOLID2D)
        return assemble_sorted_kind<GW_KIND_SOLID2D>(c, p, perm, keys, free_mask, u_new, u_old, A, prec, R_rows, force, a, ws, workspace_bytes, s);
    return assemble_sorted_kind<GW_KIND_COUPLED2D>(c, p, perm, keys, free_mask, u_new, u_old, A, prec, R_rows, force, a, ws, workspace_bytes, s);
}
