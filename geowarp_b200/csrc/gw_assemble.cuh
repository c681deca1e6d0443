// Deterministic residual and element-tangent assembly for the 2D kinds
// (solid and u-p).  Replaces the per-particle atomic scatter of the
// reference's residual kernels (mpm/mpm_utils.py:586-596, 990-1017: one
// wp.atomic_add per node and field) and of its coloured-AD Jacobian
// (solvers/sparse_differentiation.py:213-401).
//
// Three passes:
//
//  1. k_particle_q (one thread per particle, cell-sorted order): kinematics,
//     return map and stress, written back as F_new / b_new / sigma like the
//     reference, and the particle's stress resultants Q (FP64) and their
//     derivatives Dm = dQ/dtheta (FP64, or FP32 in mixed precision) with respect to
//     the gathered nodal quantities theta (displacement gradient H, ubar, and for
//     u-p pbar, grad p, dp~).  These go to a scratch record per sorted particle;
//     there is no scatter in this pass.
//
//  2. k_cell_blocks (16 lanes per occupied cell): the particles of one cell share
//     their lower corner, so they touch the same 3 x 3 nodes.  A lane sums whole
//     element blocks (slot a, slot b) and residual entries over the cell's
//     particles in sorted order and leaves them, in FP64, in the cell's buffer.
//
//  3. k_row_gather (a warp per block row): a row's entries and blocks are the sums
//     over the up to nine cells that reach its node; it is written once, with its
//     Dirichlet identity entries.
//
// The summation order of a row is fixed (its cells by (cy mod 3, cx mod 3), a cell's
// particles in sorted order, FP32 blocks rounded after each cell), so R and K are
// bitwise reproducible.  The former cell scatter kept the order by nine colour
// phases of cells three apart: nine dependent launches of 8-10 us each however small
// the problem (640 particles FP64: 79 us), 994 us on 1.03 M particles; the two passes
// take 9 us and 786 us.  (Rows gathering straight from the records, each read four to
// nine times: 27 us and 2,135 us.)
//
// The residual rows follow residual_rows(): for field j < D
//   r_a[j] = -sum_k G_a[k] Q_U[k][j] + W_a (Q_S g_j + fx_j) + [j = D-1] W_a Q_PEN,
// and for the pressure row (u-p)
//   r_a[D] = W_a Q_M1 + sum_k G_a[k] Q_M2[k] + (W_a - Wavg_a) Q_M3,
// and the element blocks are K_ab = -d r_a / d u_b with
//   d Q_q / d u_b[g] = C_b[q][g] = sum_k Dm[q][TH + k D + g] G_b[k] + [g = D-1] Dm[q][TU] W_b
// (pressure column: Dm[q][TP] W_b + Dm[q][TD] (W_b - Wavg_b) + sum_k Dm[q][TG+k] G_b[k]).
#pragma once
#include "gw_step_kernels.cuh"

namespace gw {
namespace {  // internal linkage: each translation unit compiles the kernels it launches

// Scratch record of one sorted particle: doubles x[D], lp[D], Q[NQ], fx[D] (point
// load and traction per unit weight), then VT Dm from a 16-byte boundary; padded to
// 32 bytes.  The solid kind's only nonzero derivatives are those of Qu with respect
// to H (4 x 4) and of the footing penalty with respect to ubar (1).
template <int KIND, typename VT>
struct QRecord {
    typedef Layout<KIND> L;
    static const int D = KindTraits<KIND>::D;
    static const bool UP = KindTraits<KIND>::UP;
    static const int Q0 = 2 * D, FX = Q0 + L::NQ;
    static const int ND = (FX + D + 1) / 2 * 2;          // doubles
    static const int NDM = UP ? L::NQ * L::NT : 17;      // tangent entries
    static const int BYTES = ((ND * 8 + NDM * (int)sizeof(VT)) + 31) / 32 * 32;
};
// Sums of one cell, FP64: the blocks (a, b) of its box of ns slots, row a after row a
// (a row's reader takes ns blocks in a piece), then the slots' residual entries.
template <int KIND>
struct CellSums {
    static const int NF = KindTraits<KIND>::NF;
    static const int ND = (81 * NF * NF + 9 * NF + 1) / 2 * 2;  // doubles, for the largest box
};

// sorted keys -> [start, end) of every occupied cell (cells without particles keep start = end = 0).
// The cell's first thread also looks up the rows of its nodes that have free DOFs: a
// contribution to a node that no row gathers (a stale row map) fails the guard.  (Here
// it costs at most 1% of the assembly; in pass 2, 1-5%.)
__global__ void k_cell_ranges(gw_grid_t grid, const int *__restrict__ keys, int n, const uint8_t *__restrict__ free_mask,
                              const int *__restrict__ node2row, int n_rows, int *__restrict__ cstart,
                              int *__restrict__ cend) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    const int k = keys[t], ncx = grid.n_grid[0], ncy = grid.n_grid[1];
    if (!in_range(k, ncx * ncy, GS_ASSEMBLE)) return;
    if (t == n - 1 || keys[t + 1] != k) cend[k] = t + 1;
    if (t > 0 && keys[t - 1] == k) return;
    cstart[k] = t;
    const int cx = k % ncx, cy = k / ncx;
    unsigned m[9];
    int row[9];
#pragma unroll
    for (int a = 0; a < 9; ++a) {
        const int nx = cx + a % 3, ny = cy + a / 3, node = nx + ny * (ncx + 1);
        const bool in = nx <= ncx && ny <= ncy;
        m[a] = in ? free_mask[node] : 0u;
        row[a] = in ? node2row[node] : 0;
    }
#pragma unroll
    for (int a = 0; a < 9; ++a)
        if (m[a]) in_range(row[a], n_rows, GS_ASSEMBLE);
}

// Pass 1: one thread per particle in sorted order.
template <int KIND, bool WANT_K, typename VT, int MODEL = -1>
__global__ void __launch_bounds__(kThreads) k_particle_q(LaunchConst c, PtrsP p, const int *__restrict__ perm,
                                                         const double *__restrict__ u_new,
                                                         const double *__restrict__ u_old,
                                                         unsigned char *__restrict__ scratch,
                                                         double *__restrict__ force) {
    typedef KindTraits<KIND> KT;
    typedef Layout<KIND> L;
    typedef QRecord<KIND, VT> RC;
    const int D = KT::D;
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= p.n) return;
    const int pid = perm[t];
    double x[D], lp[D], Fo[9], bo[9];
    for (int k = 0; k < D; ++k) { x[k] = p.x[pid * D + k]; lp[k] = p.lp[pid * D + k]; }
    for (int k = 0; k < 9; ++k) { Fo[k] = p.F_old[(size_t)pid * 9 + k]; bo[k] = p.b_old[(size_t)pid * 9 + k]; }
    const double E = p.E ? p.E[pid] : c.E0;
    const double pi_old = p.pi_old ? p.pi_old[pid] : 0.0;
    const double pi_new = p.pi_new ? p.pi_new[pid] : 0.0;
    PState<KIND> s;
    if (!particle_shape<KIND>(c.g, x, lp, s)) atomicOr(&g_status, ST_RANGE);
    particle_gather<KIND>(u_new, u_old, s);
    PEval<KIND> ev;
    particle_eval<KIND, WANT_K, MODEL>(c, s, x, Fo, bo, E, pi_old, pi_new, c.st.p_vol, ev);
    for (int i = 0; i < 3; ++i)
        for (int j = 0; j < 3; ++j) {
            p.F_new[(size_t)pid * 9 + i * 3 + j] = ev.F_new[i][j];
            p.b_new[(size_t)pid * 9 + i * 3 + j] = ev.b_new[i][j];
            p.sigma[(size_t)pid * 9 + i * 3 + j] = ev.sigma[i][j];
        }
    if (p.pi_new) p.pi_new[pid] = ev.pi_new;
    if (ev.pen_on && force) atomicAdd(force, -ev.pen);
    const double ramp = (c.st.current_step + 1.0) / c.st.total_steps;
    double *rd = (double *)(scratch + (size_t)t * RC::BYTES);
    bool bad = false;
    for (int k = 0; k < D; ++k) {
        double f = (p.ext_flag && p.ext_flag[pid]) ? c.st.point_load[k] * ramp : 0.0;
        if (KIND == GW_KIND_COUPLED2D && p.trac_flag && p.trac_flag[pid]) f += c.st.traction[k] * c.g.h[k] / c.st.PPD;
        rd[k] = x[k];
        rd[D + k] = lp[k];
        rd[RC::FX + k] = f;
    }
    for (int q = 0; q < L::NQ; ++q) {
        rd[RC::Q0 + q] = ev.Q[q];
        if (!isfinite(ev.Q[q])) bad = true;
    }
    if (bad) atomicOr(&g_status, ST_NAN);
    if (!WANT_K) return;
    VT *rm = (VT *)(rd + RC::ND);
    if (RC::UP) {
        for (int q = 0; q < L::NQ; ++q)
            for (int tt = 0; tt < L::NT; ++tt) rm[q * L::NT + tt] = (VT)ev.Dm[q][tt];
    } else {
        for (int q = 0; q < 4; ++q)
            for (int tt = 0; tt < 4; ++tt) rm[q * 4 + tt] = (VT)ev.Dm[L::QU + q][L::TH + tt];
        rm[16] = (VT)ev.Dm[L::QPEN][L::TU];
    }
}

__device__ __forceinline__ void record_row(const float *p, double d[4]) {
    const float4 v = *reinterpret_cast<const float4 *>(p);
    d[0] = v.x; d[1] = v.y; d[2] = v.z; d[3] = v.w;
}
__device__ __forceinline__ void record_row(const double *p, double d[4]) {
    const double2 a = reinterpret_cast<const double2 *>(p)[0], b = reinterpret_cast<const double2 *>(p)[1];
    d[0] = a.x; d[1] = a.y; d[2] = b.x; d[3] = b.y;
}

// Pass 2: 16 lanes per cell.  The axes of eight particles are evaluated one per
// lane; then lane l takes block l, l + 16, ... of the cell's box (the union of its
// particles' spans: 16 blocks where they lie inside one cell, up to 81) and residual
// entries l, l + 16, one at a time over all the cell's particles, so it holds one
// block in registers and the SM many cells.  (A cell of more than eight particles
// evaluates its axes again for each round.)  box[cell]: the box's extents, 0 without
// particles.  Cells cell0 .. cell1 - 1, their sums from the buffer's start (by_cell) or
// at their first particle.
constexpr int kCellGroups = 8;   // cells per CTA
constexpr int kCellBatch = 8;
struct CellAxis {
    double w[3], g[3], a[3];
    int off, span;  // corner offset from the cell (a particle clamped at the grid edge), nodes
};
template <int KIND, bool WANT_K, typename VT>
__global__ void __launch_bounds__(16 * kCellGroups) k_cell_blocks(LaunchConst c, int cell0, int cell1, int by_cell,
                                                                  const int *__restrict__ cstart,
                                                                  const int *__restrict__ cend,
                                                                  const unsigned char *__restrict__ scratch,
                                                                  double *__restrict__ sums, int *__restrict__ box) {
    typedef KindTraits<KIND> KT;
    typedef Layout<KIND> L;
    typedef QRecord<KIND, VT> RC;
    typedef CellSums<KIND> CS;
    static_assert(KT::D == 2, "the cell pass covers the 2D kinds");
    constexpr int D = 2, NF = KT::NF;
    __shared__ CellAxis axs[kCellGroups][kCellBatch][2];
    const int lane = threadIdx.x & 15, grp = threadIdx.x >> 4;
    const int cell = cell0 + blockIdx.x * kCellGroups + grp;
    const unsigned gmask = 0xffffu << (threadIdx.x & 16);  // this cell's half of the warp
    if (cell >= cell1) return;  // whole groups; group-wide syncs below
    const int p0 = cstart[cell], p1 = cend[cell];
    if (p1 <= p0) {
        if (lane == 0) box[cell] = 0;
        return;
    }
    const int ncx = c.g.n_grid[0], cx = cell % ncx, cy = cell / ncx;
    const double ramp = (c.st.current_step + 1.0) / c.st.total_steps;
    const double gv = -c.st.gravity_mag * (c.st.gravity_full ? 1.0 : ramp);
    auto axes = [&](int t0) {  // axes of the batch from t0 into shared memory; the extent of this lane's
        const int pp = lane >> 1, k = lane & 1;
        if (t0 + pp >= p1) return 0;
        const double *rd = (const double *)(scratch + (size_t)(t0 + pp) * RC::BYTES);
        Axis ax;
        gimp_axis(rd[k], rd[D + k], c.g.h[k], c.g.inv_h[k], ax);
        CellAxis &o = axs[grp][pp][k];
        for (int i = 0; i < 3; ++i) { o.w[i] = ax.w[i]; o.g[i] = ax.gw[i]; o.a[i] = ax.wavg[i]; }
        o.off = ax.lower - (k == 0 ? cx : cy);
        o.span = ax.span;
        return min(3, max(0, o.off + o.span));
    };
    int e0 = 0, e1 = 0;
    for (int t0 = p0; t0 < p1; t0 += kCellBatch) {
        const int e = axes(t0);
        if (lane & 1) e1 = max(e1, e);
        else e0 = max(e0, e);
    }
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) {
        e0 = max(e0, __shfl_xor_sync(gmask, e0, o, 16));
        e1 = max(e1, __shfl_xor_sync(gmask, e1, o, 16));
    }
    const int ns = e0 * e1, nb = ns * ns;
    const bool one = p1 - p0 <= kCellBatch;  // the axes of the only batch are in place
    const float ins = 1.0f / (float)max(ns, 1), ie0 = 1.0f / (float)max(e0, 1);  // exact quotients of small integers below
    double *const out = sums + (size_t)(by_cell ? cell - cell0 : p0) * CS::ND;
    __syncwarp(gmask);

    for (int q0 = 0; q0 < ns * NF; q0 += 16) {  // residual entries (slot a, field f)
        const int q = q0 + lane, a = q / NF, f = q % NF;
        const int ay = (int)(((float)a + 0.5f) * ie0), ax = a - ay * e0;
        double racc = 0.0;
        for (int t0 = p0; t0 < p1; t0 += kCellBatch) {
            if (!one) {
                __syncwarp(gmask);
                axes(t0);
                __syncwarp(gmask);
            }
            const int np = q < ns * NF ? min(kCellBatch, p1 - t0) : 0;
            for (int pp = 0; pp < np; ++pp) {
                const CellAxis &X = axs[grp][pp][0], &Y = axs[grp][pp][1];
                const int a0 = ax - X.off, a1 = ay - Y.off;
                if ((unsigned)a0 >= (unsigned)X.span || (unsigned)a1 >= (unsigned)Y.span) continue;
                const double *rd = (const double *)(scratch + (size_t)(t0 + pp) * RC::BYTES);
                const double *Q = rd + RC::Q0;
                const double Wa = X.w[a0] * Y.w[a1], Ga0 = X.g[a0] * Y.w[a1], Ga1 = X.w[a0] * Y.g[a1];
                double v;
                if (f < D) {
                    v = -(Ga0 * Q[L::QU + f] + Ga1 * Q[L::QU + D + f]);
                    v += Wa * (Q[L::QS] * (f == D - 1 ? gv : 0.0) + rd[RC::FX + f]);
                    if (f == D - 1) v += Wa * Q[L::QPEN];
                } else {
                    const double Waa = X.a[a0] * Y.a[a1];
                    v = Wa * Q[L::QM1] + (Wa - Waa) * Q[L::QM3] + Ga0 * Q[L::QM2] + Ga1 * Q[L::QM2 + 1];
                }
                racc += v;
            }
        }
        if (q < ns * NF) out[nb * NF * NF + q] = racc;
    }
    if (WANT_K)
        for (int q0 = 0; q0 < nb; q0 += 16) {
            const int q = q0 + lane;
            const int a = (int)(((float)q + 0.5f) * ins), b = q - a * ns;
            const int ay = (int)(((float)a + 0.5f) * ie0), ax = a - ay * e0;
            const int by = (int)(((float)b + 0.5f) * ie0), bx = b - by * e0;
            double kacc[NF][NF];
#pragma unroll
            for (int f = 0; f < NF; ++f)
#pragma unroll
                for (int g = 0; g < NF; ++g) kacc[f][g] = 0.0;
            for (int t0 = p0; t0 < p1; t0 += kCellBatch) {
                if (!one) {
                    __syncwarp(gmask);
                    axes(t0);
                    __syncwarp(gmask);
                }
                const int np = q < nb ? min(kCellBatch, p1 - t0) : 0;
                for (int pp = 0; pp < np; ++pp) {
                    const CellAxis &X = axs[grp][pp][0], &Y = axs[grp][pp][1];
                    const int xo = X.off, xs = X.span, yo = Y.off, ys = Y.span;
                    const int a0 = ax - xo, a1 = ay - yo, b0 = bx - xo, b1 = by - yo;
                    if ((unsigned)a0 >= (unsigned)xs || (unsigned)a1 >= (unsigned)ys || (unsigned)b0 >= (unsigned)xs ||
                        (unsigned)b1 >= (unsigned)ys)
                        continue;
                    const VT *Dm = (const VT *)((const double *)(scratch + (size_t)(t0 + pp) * RC::BYTES) + RC::ND);
                    const double Wa = X.w[a0] * Y.w[a1], Ga0 = X.g[a0] * Y.w[a1], Ga1 = X.w[a0] * Y.g[a1];
                    const double Wb = X.w[b0] * Y.w[b1], Gb0 = X.g[b0] * Y.w[b1], Gb1 = X.w[b0] * Y.g[b1];
                    if (!RC::UP) {
                        double C[4][2];  // dQu / du_b
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            double d[4];
                            record_row(Dm + u * 4, d);
                            C[u][0] = d[0] * Gb0 + d[D] * Gb1;
                            C[u][1] = d[1] * Gb0 + d[D + 1] * Gb1;
                        }
#pragma unroll
                        for (int g = 0; g < 2; ++g)
#pragma unroll
                            for (int f = 0; f < 2; ++f) {
                                double v = -(Ga0 * C[f][g] + Ga1 * C[D + f][g]);
                                if (f == 1 && g == 1) v += Wa * ((double)Dm[16] * Wb);
                                kacc[f][g] -= v;
                            }
                    } else {
                        const double Waa = X.a[a0] * Y.a[a1], Wbb = X.a[b0] * Y.a[b1];
                        double C[L::NQ][NF];
#pragma unroll
                        for (int u = 0; u < L::NQ; ++u) {
                            const VT *dq = Dm + u * L::NT;
                            C[u][0] = (double)dq[L::TH + 0] * Gb0 + (double)dq[L::TH + D] * Gb1;
                            C[u][1] = (double)dq[L::TH + 1] * Gb0 + (double)dq[L::TH + D + 1] * Gb1 + (double)dq[L::TU] * Wb;
                            C[u][NF - 1] = (double)dq[L::TP] * Wb + (double)dq[L::TD] * (Wb - Wbb) + (double)dq[L::TG] * Gb0 +
                                           (double)dq[L::TG + 1] * Gb1;
                        }
#pragma unroll
                        for (int g = 0; g < NF; ++g) {
#pragma unroll
                            for (int f = 0; f < D; ++f) {
                                double v = -(Ga0 * C[L::QU + f][g] + Ga1 * C[L::QU + D + f][g]);
                                if (f == D - 1) v += Wa * gv * C[L::QS][g] + Wa * C[L::QPEN][g];
                                kacc[f][g] -= v;
                            }
                            const double v = Wa * C[L::QM1][g] + (Wa - Waa) * C[L::QM3][g] + Ga0 * C[L::QM2][g] + Ga1 * C[L::QM2 + 1][g];
                            kacc[NF - 1][g] -= v;
                        }
                    }
                }
            }
            if (q < nb) {
                double *d = out + q * NF * NF;
#pragma unroll
                for (int f = 0; f < NF; ++f)
#pragma unroll
                    for (int g = 0; g < NF; ++g) d[f * NF + g] = kacc[f][g];
            }
        }
    if (lane == 0) box[cell] = e0 | e1 << 2;
}

template <int N>
__device__ __forceinline__ void load_rw_blk(const double *p, double v[N]) {
    if constexpr (N % 2 == 0) {
#pragma unroll
        for (int q = 0; q < N / 2; ++q) {
            const double2 t = reinterpret_cast<const double2 *>(p)[q];
            v[2 * q] = t.x; v[2 * q + 1] = t.y;
        }
    } else {
#pragma unroll
        for (int q = 0; q < N; ++q) v[q] = p[q];
    }
}

// Pass 3: a warp per block row.  Lane t < 25 sums the block at stencil bit t, lanes
// 25 .. 25 + NF - 1 the residual fields, over the cells that reach the node.  Rows of
// the nodes with ny0 <= y < ny1; cell0 as in pass 2.
constexpr int kGatherRows = 8;  // rows per CTA
template <int KIND, bool WANT_K, typename VT>
__global__ void __launch_bounds__(32 * kGatherRows) k_row_gather(gw_grid_t grid, int by_cell,
                                                                 int cell0, int ny0, int ny1,
                                                                 const int *__restrict__ cstart,
                                                                 const int *__restrict__ box,
                                                                 const double *__restrict__ sums,
                                                                 const uint8_t *__restrict__ free_mask, PtrsA A,
                                                                 double *__restrict__ R) {
    typedef CellSums<KIND> CS;
    constexpr int NF = CS::NF, BB = NF * NF;
    const int lane = threadIdx.x & 31;
    const int r = blockIdx.x * kGatherRows + (threadIdx.x >> 5);
    const int ncx = grid.n_grid[0], ncy = grid.n_grid[1];
    if (r >= A.n_rows) return;  // whole warps
    const int node = A.row2node[r];
    if (!in_range(node, grid.n_nodes, GS_ASSEMBLE)) return;
    const int nx = node % (ncx + 1), ny = node / (ncx + 1);
    if (ny < ny0 || ny >= ny1) return;  // whole warps
    const unsigned fa = free_mask[node];
    // lanes 0-8: the cell of each (cx mod 3, cy mod 3) that reaches this node, in the order of the sums
    int slot = 0, info = 0;  // info: box extents, and this node's slot (ax, ay)
    if (lane < 9) {
        const int kx = lane % 3, ky = lane / 3;
        const int cx = nx - (nx - kx + 3) % 3, cy = ny - (ny - ky + 3) % 3;
        if (cx >= 0 && cx < ncx && cy >= 0 && cy < ncy) {
            const int cell = cx + cy * ncx, b = box[cell], ax = nx - cx, ay = ny - cy;
            if (ax < (b & 3) && ay < (b >> 2)) {
                info = b | ax << 4 | ay << 6;
                slot = by_cell ? cell - cell0 : cstart[cell];
            }
        }
    }
    const int ox = lane % 5 - 2, oy = lane / 5 - 2;
    // what the end needs, loaded ahead of the sums
    const unsigned st = WANT_K ? A.stencil[node] : 0u;
    const int base = WANT_K ? A.row_ptr[r] : 0;
    const int jx = nx + ox, jy = ny + oy;
    unsigned fb = 0u;
    if (WANT_K && lane < 25 && jx >= 0 && jx <= ncx && jy >= 0 && jy <= ncy) fb = free_mask[jx + jy * (ncx + 1)];
    VT blk[WANT_K ? BB : 1];
#pragma unroll
    for (int q = 0; q < (WANT_K ? BB : 1); ++q) blk[q] = (VT)0;
    double rsum = 0.0;
    bool touched = false;  // a cell holds this lane's block
    // the cells that reach the node (four where particles stay inside their cells, up
    // to nine), four at a time with their values in flight
    unsigned left = __ballot_sync(0xffffffffu, info != 0);
    while (left) {
        constexpr int M = 4;
        double v[M][WANT_K ? BB : 1], rv[M];
        bool on[M];
#pragma unroll
        for (int o = 0; o < M; ++o) {
            on[o] = false;
            rv[o] = 0.0;
            const int from = left ? __ffs(left) - 1 : 0;
            const int in = __shfl_sync(0xffffffffu, info, from), sl = __shfl_sync(0xffffffffu, slot, from);
            if (!left) continue;  // uniform
            left &= left - 1u;
            const int ax = in >> 4 & 3, ay = in >> 6, bx = ax + ox, by = ay + oy;
            const int e0 = in & 3, e1 = in >> 2 & 3, ns = e0 * e1, a = ax + e0 * ay;
            const double *src = sums + (size_t)sl * CS::ND;
            if (lane >= 25) {
                if (lane < 25 + NF) rv[o] = src[ns * ns * BB + a * NF + lane - 25];
            } else if (WANT_K && bx >= 0 && by >= 0 && bx < e0 && by < e1) {
                on[o] = true;
                load_rw_blk<WANT_K ? BB : 1>(src + (a * ns + bx + e0 * by) * BB, v[o]);
            }
        }
#pragma unroll
        for (int o = 0; o < M; ++o) {
            rsum += rv[o];
            if (WANT_K && on[o]) {
                touched = true;
#pragma unroll
                for (int q = 0; q < (WANT_K ? BB : 1); ++q) blk[q] = (VT)((double)blk[q] + v[o][q]);
            }
        }
    }
    if (lane >= 25) {
        if (lane < 25 + NF) {
            const int f = lane - 25;
            const bool free = (fa >> f) & 1u;
            if (free && !isfinite(rsum)) atomicOr(&g_status, ST_NAN);
            R[(size_t)r * NF + f] = free ? rsum : 0.0;
        }
        return;
    }
    if (!WANT_K) return;
    if (!((st >> lane) & 1u)) {
        // no diagonal block, or a cell that couples two free nodes outside the pattern (a
        // node without free DOFs may lie inside a particle's span and have no row: u-p
        // nodes below the activation weight)
        if (lane == 12 || (touched && fa && fb)) atomicOr(&g_status, ST_RANGE);
        return;
    }
    const long long jb = (long long)base + __popc(st & ((1u << lane) - 1u));
    if (!in_range(jb, A.nnzb, GS_ASSEMBLE)) return;
    VT *dst = (VT *)A.vals + (size_t)jb * BB;
#pragma unroll
    for (int f = 0; f < NF; ++f)
#pragma unroll
        for (int g = 0; g < NF; ++g) {
            VT v = (((fa >> f) & 1u) && ((fb >> g) & 1u)) ? blk[WANT_K ? f * NF + g : 0] : (VT)0;
            if (lane == 12 && f == g && !((fa >> f) & 1u)) v = (VT)1;  // Dirichlet DOF: identity row
            dst[f * NF + g] = v;
        }
}

}  // namespace
}  // namespace gw
