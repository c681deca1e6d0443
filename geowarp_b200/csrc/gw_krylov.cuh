// Preconditioned Krylov solvers on the node-block CSR matrix.
//
// Replaces wp.optim.linear.bicgstab + preconditioner(ptype='diag') and the
// host solvers of solvers/quasi_static_solver_2d.py:236-256.  Every iteration
// is a fixed sequence of fused kernels; inner products are FP64 block
// partials summed in block order by the last block to finish (deterministic),
// which also derives the iteration scalars on the device.  Kernels return
// immediately once the device "done" flag is set, so the host can enqueue
// iterations in chunks and poll the flag once per chunk.
#pragma once
#include <cuda_bf16.h>
#include <stddef.h>

#include "gw_kernels.cuh"

namespace gw {
namespace {  // internal linkage: each translation unit compiles the kernels it launches

// Programmatic dependent launch: pdl_wait() returns once every earlier kernel of
// the chain has completed (at once in a kernel launched without the attribute);
// pdl_release() lets the next kernel of the chain start.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

constexpr int kRedBlocks = 148 * 8;  // grid size of reduction kernels (multiple of the B200 SM count)

struct KScalars {
    double rho, rho_old, alpha, omega, beta;
    double rr, bb, tol2;
    double tmp0, tmp1;
    int done, status, iters, max_iter;
    unsigned ticket;
};

// ---------------------------------------------------------------- block reduction helpers
template <int NV>
__device__ __forceinline__ void block_reduce(double v[NV]) {
    __shared__ double sh[NV][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        double x = v[k];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
        if (lane == 0) sh[k][w] = x;
    }
    __syncthreads();
    if (w == 0) {
#pragma unroll
        for (int k = 0; k < NV; ++k) {
            double x = lane < nw ? sh[k][lane] : 0.0;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
            v[k] = x;
        }
    }
    __syncthreads();
}

// Writes this block's partials; returns true in the last block, whose v[] then
// holds the grid totals (summed in block order).
template <int NV>
__device__ __forceinline__ bool grid_reduce(double v[NV], double *partials, unsigned *ticket) {
    block_reduce<NV>(v);
    __shared__ bool last;
    if (threadIdx.x == 0) {
#pragma unroll
        for (int k = 0; k < NV; ++k) partials[blockIdx.x * NV + k] = v[k];
        __threadfence();
        const unsigned t = atomicAdd(ticket, 1u);
        last = (t == gridDim.x - 1);
    }
    __syncthreads();
    if (!last) return false;
    __threadfence();
    double acc[NV];
#pragma unroll
    for (int k = 0; k < NV; ++k) acc[k] = 0.0;
    // fixed-order sum: thread t sums partials t, t+B, ... then a block tree
    for (int b = threadIdx.x; b < gridDim.x; b += blockDim.x)
#pragma unroll
        for (int k = 0; k < NV; ++k) acc[k] += ((volatile double *)partials)[b * NV + k];
    block_reduce<NV>(acc);
#pragma unroll
    for (int k = 0; k < NV; ++k) v[k] = acc[k];
    if (threadIdx.x == 0) *ticket = 0u;
    return true;
}

// ---------------------------------------------------------------- SpMV
// Vectorised gathers of one NF x NF block and one NF-vector: 16-byte loads
// for NF = 2 and 4 (block values and vectors 16-byte aligned; the entry
// points check it), scalar loads otherwise.  The values and the order they
// are used in are the same either way.
template <int NF, typename VT>
__device__ __forceinline__ void load_block(const VT *__restrict__ p, double out[NF * NF]) {
#pragma unroll
    for (int i = 0; i < NF * NF; ++i) out[i] = (double)p[i];
}
// BF16 blocks (the multigrid's preconditioner copy of a mixed-precision fine
// level): 2x2 blocks in one 8-byte load, otherwise element by element
template <int NF>
__device__ __forceinline__ void load_block_bf16(const __nv_bfloat16 *__restrict__ p, double out[NF * NF]) {
    if constexpr (NF == 2) {
        const uint2 u = *reinterpret_cast<const uint2 *>(p);
        const __nv_bfloat162 a = *reinterpret_cast<const __nv_bfloat162 *>(&u.x);
        const __nv_bfloat162 b = *reinterpret_cast<const __nv_bfloat162 *>(&u.y);
        out[0] = __low2float(a); out[1] = __high2float(a); out[2] = __low2float(b); out[3] = __high2float(b);
    } else {
#pragma unroll
        for (int i = 0; i < NF * NF; ++i) out[i] = __bfloat162float(p[i]);
    }
}
template <> __device__ __forceinline__ void load_block<1, __nv_bfloat16>(const __nv_bfloat16 *__restrict__ p, double out[1]) { load_block_bf16<1>(p, out); }
template <> __device__ __forceinline__ void load_block<2, __nv_bfloat16>(const __nv_bfloat16 *__restrict__ p, double out[4]) { load_block_bf16<2>(p, out); }
template <> __device__ __forceinline__ void load_block<3, __nv_bfloat16>(const __nv_bfloat16 *__restrict__ p, double out[9]) { load_block_bf16<3>(p, out); }
template <> __device__ __forceinline__ void load_block<4, __nv_bfloat16>(const __nv_bfloat16 *__restrict__ p, double out[16]) { load_block_bf16<4>(p, out); }
template <>
__device__ __forceinline__ void load_block<2, float>(const float *__restrict__ p, double out[4]) {
    const float4 v = *reinterpret_cast<const float4 *>(p);
    out[0] = v.x; out[1] = v.y; out[2] = v.z; out[3] = v.w;
}
template <>
__device__ __forceinline__ void load_block<2, double>(const double *__restrict__ p, double out[4]) {
    const double2 a = reinterpret_cast<const double2 *>(p)[0], b = reinterpret_cast<const double2 *>(p)[1];
    out[0] = a.x; out[1] = a.y; out[2] = b.x; out[3] = b.y;
}
template <>
__device__ __forceinline__ void load_block<4, float>(const float *__restrict__ p, double out[16]) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const float4 v = reinterpret_cast<const float4 *>(p)[q];
        out[4 * q] = v.x; out[4 * q + 1] = v.y; out[4 * q + 2] = v.z; out[4 * q + 3] = v.w;
    }
}
template <>
__device__ __forceinline__ void load_block<4, double>(const double *__restrict__ p, double out[16]) {
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const double2 v = reinterpret_cast<const double2 *>(p)[q];
        out[2 * q] = v.x; out[2 * q + 1] = v.y;
    }
}
template <int NF>
__device__ __forceinline__ void load_vec(const double *__restrict__ p, double out[NF]) {
    if constexpr (NF == 2 || NF == 4) {
#pragma unroll
        for (int q = 0; q < NF / 2; ++q) {
            const double2 v = reinterpret_cast<const double2 *>(p)[q];
            out[2 * q] = v.x; out[2 * q + 1] = v.y;
        }
    } else {
#pragma unroll
        for (int g = 0; g < NF; ++g) out[g] = p[g];
    }
}

// one row's vector through the ordinary (coherent) path: 16-byte accesses where
// the row starts are aligned (NF = 2, 4: buffers are; a basis vector of n
// unknowns is when n is even, and n is a multiple of NF)
template <int NF>
__device__ __forceinline__ void load_rw(const double *p, double out[NF]) {
    if constexpr (NF == 2 || NF == 4) {
#pragma unroll
        for (int q = 0; q < NF / 2; ++q) {
            const double2 v = reinterpret_cast<const double2 *>(p)[q];
            out[2 * q] = v.x; out[2 * q + 1] = v.y;
        }
    } else {
#pragma unroll
        for (int g = 0; g < NF; ++g) out[g] = p[g];
    }
}
template <int NF>
__device__ __forceinline__ void store_rw(double *p, const double v[NF]) {
    if constexpr (NF == 2 || NF == 4) {
#pragma unroll
        for (int q = 0; q < NF / 2; ++q) reinterpret_cast<double2 *>(p)[q] = make_double2(v[2 * q], v[2 * q + 1]);
    } else {
#pragma unroll
        for (int g = 0; g < NF; ++g) p[g] = v[g];
    }
}

// Block rows are processed by groups of kLPR lanes, kRowsPerWarp rows per
// warp in flight: the lanes of a group take consecutive blocks of their row
// (kLPR x 16 bytes per step for 2x2 FP32 blocks: one 128-byte line) and a
// warp keeps four independent row_ptr -> cols -> x load chains going.  Every
// lane of a warp runs the same number of row sweeps (rows at or past n_rows
// are idle groups), so the group shuffles can use the full mask.
constexpr int kLPR = 8;
constexpr int kRowsPerWarp = 32 / kLPR;

// acc = (A x)_r summed over the group (valid in the group's first lane); an
// idle group (r >= n_rows) returns zeros.
template <int NF, typename VT>
__device__ __forceinline__ void row_mv(const PtrsA &A, int r, const double *__restrict__ x, double acc[NF]) {
    const int lane = threadIdx.x & (kLPR - 1);
#pragma unroll
    for (int f = 0; f < NF; ++f) acc[f] = 0.0;
    const int s = r < A.n_rows ? A.row_ptr[r] : 0, e = r < A.n_rows ? A.row_ptr[r + 1] : 0;
    const VT *vals = (const VT *)A.vals;
#pragma unroll 2
    for (int j = s + lane; j < e; j += kLPR) {
        const int col = A.cols[j];
        if (!in_range(col, A.n_rows, GS_ROW_MV)) continue;
        double xv[NF], bv[NF * NF];
        load_vec<NF>(x + (size_t)col * NF, xv);
        load_block<NF, VT>(vals + (size_t)j * NF * NF, bv);
#pragma unroll
        for (int f = 0; f < NF; ++f)
#pragma unroll
            for (int g = 0; g < NF; ++g) acc[f] += bv[f * NF + g] * xv[g];
    }
#pragma unroll
    for (int f = 0; f < NF; ++f)
#pragma unroll
        for (int o = kLPR / 2; o > 0; o >>= 1) acc[f] += __shfl_down_sync(0xffffffffu, acc[f], o, kLPR);
}

template <int NF, typename VT>
__global__ void k_spmv(PtrsA A, const double *__restrict__ x, double *__restrict__ y) {
    const int nw = gridDim.x * (blockDim.x >> 5) * kRowsPerWarp;
    for (int rb = (blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * kRowsPerWarp; rb < A.n_rows; rb += nw) {
        const int r = rb + (threadIdx.x & 31) / kLPR;
        double acc[NF];
        row_mv<NF, VT>(A, r, x, acc);
        if (r < A.n_rows && (threadIdx.x & (kLPR - 1)) == 0)
#pragma unroll
            for (int f = 0; f < NF; ++f) y[(size_t)r * NF + f] = acc[f];
    }
}

// y = A^T x (atomic scatter; used by the adjoint)
template <int NF, typename VT>
__global__ void k_spmv_t(PtrsA A, const double *__restrict__ x, double *__restrict__ y) {
    const int nw = gridDim.x * (blockDim.x >> 5) * kRowsPerWarp;
    const int lane = threadIdx.x & (kLPR - 1);
    const VT *vals = (const VT *)A.vals;
    for (int rb = (blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * kRowsPerWarp; rb < A.n_rows; rb += nw) {
        const int r = rb + (threadIdx.x & 31) / kLPR;
        if (r >= A.n_rows) continue;  // no shuffles below
        double xr[NF];
#pragma unroll
        for (int f = 0; f < NF; ++f) xr[f] = x[(size_t)r * NF + f];
        for (int j = A.row_ptr[r] + lane; j < A.row_ptr[r + 1]; j += kLPR) {
            const int col = A.cols[j];
            if (!in_range(col, A.n_rows, GS_ROW_MV)) continue;
            const VT *blk = vals + (size_t)j * NF * NF;
#pragma unroll
            for (int g = 0; g < NF; ++g) {
                double v = 0.0;
#pragma unroll
                for (int f = 0; f < NF; ++f) v += (double)blk[f * NF + g] * xr[f];
                atomicAdd(&y[(size_t)col * NF + g], v);
            }
        }
    }
}

// ---------------------------------------------------------------- preconditioner
// Inverse of one NF x NF block by Gauss-Jordan with partial pivoting, into
// out (row-major).  A singular block falls back to the inverse of its
// diagonal (zero diagonal entries -> 1).
template <int NF>
__device__ __forceinline__ void invert_block(const double Min[NF][NF], double *__restrict__ out) {
    double M[NF][NF], I[NF][NF];
    for (int i = 0; i < NF; ++i)
        for (int j = 0; j < NF; ++j) { M[i][j] = Min[i][j]; I[i][j] = (i == j) ? 1.0 : 0.0; }
    bool ok = true;
    for (int cidx = 0; cidx < NF; ++cidx) {
        int piv = cidx;
        for (int i = cidx + 1; i < NF; ++i)
            if (fabs(M[i][cidx]) > fabs(M[piv][cidx])) piv = i;
        if (M[piv][cidx] == 0.0) { ok = false; break; }
        for (int j = 0; j < NF; ++j) {
            double t = M[cidx][j]; M[cidx][j] = M[piv][j]; M[piv][j] = t;
            t = I[cidx][j]; I[cidx][j] = I[piv][j]; I[piv][j] = t;
        }
        const double d = 1.0 / M[cidx][cidx];
        for (int j = 0; j < NF; ++j) { M[cidx][j] *= d; I[cidx][j] *= d; }
        for (int i = 0; i < NF; ++i) {
            if (i == cidx) continue;
            const double f = M[i][cidx];
            for (int j = 0; j < NF; ++j) { M[i][j] -= f * M[cidx][j]; I[i][j] -= f * I[cidx][j]; }
        }
    }
    for (int i = 0; i < NF; ++i)
        for (int j = 0; j < NF; ++j) {
            if (ok) out[i * NF + j] = I[i][j];
            else out[i * NF + j] = (i == j) ? (Min[i][i] != 0.0 ? 1.0 / Min[i][i] : 1.0) : 0.0;
        }
}

// Minv: per row an NF x NF block.  mode 0: inverse of the scalar diagonal
// (zero diagonal -> 1, as a Jacobi guard), mode 1: inverse of the diagonal block.
template <int NF, typename VT>
__global__ void k_precond_setup(PtrsA A, int D, int mode, double *__restrict__ Minv) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= A.n_rows) return;
    const int node = A.row2node[r];
    const int off[3] = {0, 0, 0};
    const int bit = D == 2 ? offset_bit<2>(off) : offset_bit<3>(off);
    const int slot = stencil_slot(A.stencil, A.mw, node, bit);
    double *out = Minv + (size_t)r * NF * NF;
    if (slot < 0) {  // no diagonal block: identity preconditioner on this row
        for (int i = 0; i < NF; ++i)
            for (int j = 0; j < NF; ++j) out[i * NF + j] = (i == j) ? 1.0 : 0.0;
        return;
    }
    const VT *blk = (const VT *)A.vals + ((size_t)A.row_ptr[r] + slot) * NF * NF;
    double M[NF][NF];
    for (int i = 0; i < NF; ++i)
        for (int j = 0; j < NF; ++j) M[i][j] = (double)blk[i * NF + j];
    if (mode == 0) {
        for (int i = 0; i < NF; ++i)
            for (int j = 0; j < NF; ++j) out[i * NF + j] = (i == j) ? (M[i][i] != 0.0 ? 1.0 / M[i][i] : 1.0) : 0.0;
        return;
    }
    invert_block<NF>(M, out);
}

template <int NF>
__device__ __forceinline__ void apply_minv(const double *__restrict__ Minv, int r, const double in[NF], double out[NF]) {
    const double *M = Minv + (size_t)r * NF * NF;
#pragma unroll
    for (int i = 0; i < NF; ++i) {
        double v = 0.0;
#pragma unroll
        for (int j = 0; j < NF; ++j) v += M[i * NF + j] * in[j];
        out[i] = v;
    }
}

// ---------------------------------------------------------------- BiCGSTAB
struct BicgVecs {
    double *x, *r, *rh, *p, *v, *y, *s, *z, *t;
    const double *b;
    double *Minv, *partials;
    KScalars *sc;
};

// r = b - A x ; rh = r ; p = v = 0 ; dots (r,r), (b,b)
template <int NF, typename VT>
__global__ void k_bicg_init(PtrsA A, BicgVecs V, double rtol) {
    const int nw = gridDim.x * (blockDim.x >> 5) * kRowsPerWarp;
    double d[2] = {0.0, 0.0};
    for (int rb = (blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * kRowsPerWarp; rb < A.n_rows; rb += nw) {
        const int r = rb + (threadIdx.x & 31) / kLPR;
        double acc[NF];
        row_mv<NF, VT>(A, r, V.x, acc);
        if (r < A.n_rows && (threadIdx.x & (kLPR - 1)) == 0) {
#pragma unroll
            for (int f = 0; f < NF; ++f) {
                const size_t i = (size_t)r * NF + f;
                const double rv = V.b[i] - acc[f];
                V.r[i] = rv; V.rh[i] = rv; V.p[i] = 0.0; V.v[i] = 0.0;
                d[0] += rv * rv;
                d[1] += V.b[i] * V.b[i];
            }
        }
    }
    if (grid_reduce<2>(d, V.partials, &V.sc->ticket) && threadIdx.x == 0) {
        KScalars *sc = V.sc;
        sc->rr = d[0]; sc->bb = d[1];
        sc->rho = d[0]; sc->rho_old = 1.0; sc->alpha = 1.0; sc->omega = 1.0;
        sc->tol2 = rtol * rtol * d[1];
        sc->iters = 0; sc->status = 0;
        sc->done = (d[0] <= sc->tol2 || d[1] == 0.0) ? 1 : 0;
        sc->beta = 0.0;
    }
}

// p = r + beta (p - omega v) ; y = Minv p
template <int NF>
__global__ void k_bicg_p(int n_rows, BicgVecs V) {
    if (V.sc->done) return;
    const double beta = V.sc->beta, omega = V.sc->omega;
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < n_rows; r += gridDim.x * blockDim.x) {
        double pv[NF], yv[NF];
#pragma unroll
        for (int f = 0; f < NF; ++f) {
            const size_t i = (size_t)r * NF + f;
            pv[f] = V.r[i] + beta * (V.p[i] - omega * V.v[i]);
            V.p[i] = pv[f];
        }
        apply_minv<NF>(V.Minv, r, pv, yv);
#pragma unroll
        for (int f = 0; f < NF; ++f) V.y[(size_t)r * NF + f] = yv[f];
    }
}

// v = A y ; alpha = rho / (rh, v)
template <int NF, typename VT>
__global__ void k_bicg_v(PtrsA A, BicgVecs V) {
    if (V.sc->done) return;
    const int nw = gridDim.x * (blockDim.x >> 5) * kRowsPerWarp;
    double d[1] = {0.0};
    for (int rb = (blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * kRowsPerWarp; rb < A.n_rows; rb += nw) {
        const int r = rb + (threadIdx.x & 31) / kLPR;
        double acc[NF];
        row_mv<NF, VT>(A, r, V.y, acc);
        if (r < A.n_rows && (threadIdx.x & (kLPR - 1)) == 0)
#pragma unroll
            for (int f = 0; f < NF; ++f) {
                const size_t i = (size_t)r * NF + f;
                V.v[i] = acc[f];
                d[0] += V.rh[i] * acc[f];
            }
    }
    if (grid_reduce<1>(d, V.partials, &V.sc->ticket) && threadIdx.x == 0) {
        KScalars *sc = V.sc;
        if (d[0] == 0.0 || !isfinite(d[0])) { sc->status = ST_BREAKDOWN; sc->done = 1; return; }
        sc->alpha = sc->rho / d[0];
    }
}

// s = r - alpha v ; z = Minv s
template <int NF>
__global__ void k_bicg_s(int n_rows, BicgVecs V) {
    if (V.sc->done) return;
    const double alpha = V.sc->alpha;
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < n_rows; r += gridDim.x * blockDim.x) {
        double sv[NF], zv[NF];
#pragma unroll
        for (int f = 0; f < NF; ++f) {
            const size_t i = (size_t)r * NF + f;
            sv[f] = V.r[i] - alpha * V.v[i];
            V.s[i] = sv[f];
        }
        apply_minv<NF>(V.Minv, r, sv, zv);
#pragma unroll
        for (int f = 0; f < NF; ++f) V.z[(size_t)r * NF + f] = zv[f];
    }
}

// t = A z ; omega = (t,s)/(t,t)
template <int NF, typename VT>
__global__ void k_bicg_t(PtrsA A, BicgVecs V) {
    if (V.sc->done) return;
    const int nw = gridDim.x * (blockDim.x >> 5) * kRowsPerWarp;
    double d[3] = {0.0, 0.0, 0.0};
    for (int rb = (blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * kRowsPerWarp; rb < A.n_rows; rb += nw) {
        const int r = rb + (threadIdx.x & 31) / kLPR;
        double acc[NF];
        row_mv<NF, VT>(A, r, V.z, acc);
        if (r < A.n_rows && (threadIdx.x & (kLPR - 1)) == 0)
#pragma unroll
            for (int f = 0; f < NF; ++f) {
                const size_t i = (size_t)r * NF + f;
                V.t[i] = acc[f];
                d[0] += acc[f] * V.s[i];
                d[1] += acc[f] * acc[f];
                d[2] += V.s[i] * V.s[i];
            }
    }
    if (grid_reduce<3>(d, V.partials, &V.sc->ticket) && threadIdx.x == 0) {
        KScalars *sc = V.sc;
        sc->omega = (d[1] != 0.0) ? d[0] / d[1] : 0.0;
        sc->tmp0 = d[2];  // ||s||^2: converged already when below tolerance
    }
}

// x += alpha y + omega z ; r = s - omega t ; rho = (rh, r) ; rr = (r, r)
template <int NF>
__global__ void k_bicg_xr(int n_rows, BicgVecs V) {
    if (V.sc->done) return;
    const double alpha = V.sc->alpha, omega = V.sc->omega;
    double d[2] = {0.0, 0.0};
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < n_rows; r += gridDim.x * blockDim.x) {
#pragma unroll
        for (int f = 0; f < NF; ++f) {
            const size_t i = (size_t)r * NF + f;
            V.x[i] += alpha * V.y[i] + omega * V.z[i];
            const double rv = V.s[i] - omega * V.t[i];
            V.r[i] = rv;
            d[0] += V.rh[i] * rv;
            d[1] += rv * rv;
        }
    }
    if (grid_reduce<2>(d, V.partials, &V.sc->ticket) && threadIdx.x == 0) {
        KScalars *sc = V.sc;
        sc->iters += 1;
        sc->rr = d[1];
        if (!isfinite(d[1])) { sc->status = ST_NAN; sc->done = 1; return; }
        if (d[1] <= sc->tol2) { sc->done = 1; return; }
        if (sc->iters >= sc->max_iter) { sc->done = 1; return; }
        if (d[0] == 0.0 || omega == 0.0) { sc->status = ST_BREAKDOWN; sc->done = 1; return; }
        sc->beta = (d[0] / sc->rho) * (sc->alpha / omega);
        sc->rho_old = sc->rho;
        sc->rho = d[0];
    }
}

// ---------------------------------------------------------------- CG (SPD; consistent mass)
// init: r = b - A x ; z = Minv r ; p = z ; rz = (r,z)
template <int NF, typename VT>
__global__ void k_cg_init(PtrsA A, BicgVecs V, double rtol) {
    const int nw = gridDim.x * (blockDim.x >> 5) * kRowsPerWarp;
    double d[3] = {0.0, 0.0, 0.0};
    for (int rb = (blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * kRowsPerWarp; rb < A.n_rows; rb += nw) {
        const int r = rb + (threadIdx.x & 31) / kLPR;
        double acc[NF];
        row_mv<NF, VT>(A, r, V.x, acc);
        if (r < A.n_rows && (threadIdx.x & (kLPR - 1)) == 0) {
            double rv[NF], zv[NF];
#pragma unroll
            for (int f = 0; f < NF; ++f) rv[f] = V.b[(size_t)r * NF + f] - acc[f];
            apply_minv<NF>(V.Minv, r, rv, zv);
#pragma unroll
            for (int f = 0; f < NF; ++f) {
                const size_t i = (size_t)r * NF + f;
                V.r[i] = rv[f]; V.z[i] = zv[f]; V.p[i] = zv[f];
                d[0] += rv[f] * zv[f];
                d[1] += rv[f] * rv[f];
                d[2] += V.b[i] * V.b[i];
            }
        }
    }
    if (grid_reduce<3>(d, V.partials, &V.sc->ticket) && threadIdx.x == 0) {
        KScalars *sc = V.sc;
        sc->rho = d[0]; sc->rr = d[1]; sc->bb = d[2];
        sc->tol2 = rtol * rtol * d[2];
        sc->iters = 0; sc->status = 0; sc->beta = 0.0;
        sc->done = (d[1] <= sc->tol2 || d[2] == 0.0) ? 1 : 0;
    }
}

// p = z + beta p (skipped on the first iteration: beta = 0 and p = z already)
template <int NF>
__global__ void k_cg_p(int n_rows, BicgVecs V) {
    if (V.sc->done) return;
    const double beta = V.sc->beta;
    if (beta == 0.0) return;
    for (size_t i = blockIdx.x * blockDim.x + threadIdx.x; i < (size_t)n_rows * NF; i += gridDim.x * blockDim.x)
        V.p[i] = V.z[i] + beta * V.p[i];
}

// q(=v) = A p ; alpha = rz / (p, q)
template <int NF, typename VT>
__global__ void k_cg_q(PtrsA A, BicgVecs V) {
    if (V.sc->done) return;
    const int nw = gridDim.x * (blockDim.x >> 5) * kRowsPerWarp;
    double d[1] = {0.0};
    for (int rb = (blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * kRowsPerWarp; rb < A.n_rows; rb += nw) {
        const int r = rb + (threadIdx.x & 31) / kLPR;
        double acc[NF];
        row_mv<NF, VT>(A, r, V.p, acc);
        if (r < A.n_rows && (threadIdx.x & (kLPR - 1)) == 0)
#pragma unroll
            for (int f = 0; f < NF; ++f) {
                const size_t i = (size_t)r * NF + f;
                V.v[i] = acc[f];
                d[0] += V.p[i] * acc[f];
            }
    }
    if (grid_reduce<1>(d, V.partials, &V.sc->ticket) && threadIdx.x == 0) {
        KScalars *sc = V.sc;
        if (d[0] == 0.0 || !isfinite(d[0])) { sc->status = ST_BREAKDOWN; sc->done = 1; return; }
        sc->alpha = sc->rho / d[0];
    }
}

// x += alpha p ; r -= alpha q ; z = Minv r ; beta = (r,z)_new / (r,z)
template <int NF>
__global__ void k_cg_xr(int n_rows, BicgVecs V) {
    if (V.sc->done) return;
    const double alpha = V.sc->alpha;
    double d[2] = {0.0, 0.0};
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < n_rows; r += gridDim.x * blockDim.x) {
        double rv[NF], zv[NF];
#pragma unroll
        for (int f = 0; f < NF; ++f) {
            const size_t i = (size_t)r * NF + f;
            V.x[i] += alpha * V.p[i];
            rv[f] = V.r[i] - alpha * V.v[i];
            V.r[i] = rv[f];
        }
        apply_minv<NF>(V.Minv, r, rv, zv);
#pragma unroll
        for (int f = 0; f < NF; ++f) {
            V.z[(size_t)r * NF + f] = zv[f];
            d[0] += rv[f] * zv[f];
            d[1] += rv[f] * rv[f];
        }
    }
    if (grid_reduce<2>(d, V.partials, &V.sc->ticket) && threadIdx.x == 0) {
        KScalars *sc = V.sc;
        sc->iters += 1;
        sc->rr = d[1];
        if (!isfinite(d[1])) { sc->status = ST_NAN; sc->done = 1; return; }
        if (d[1] <= sc->tol2 || sc->iters >= sc->max_iter) { sc->done = 1; return; }
        sc->beta = d[0] / sc->rho;
        sc->rho = d[0];
    }
}

// ---------------------------------------------------------------- misc vector kernels
__global__ void k_norm2(const double *__restrict__ v, int n, double *__restrict__ partials, unsigned *ticket,
                        double *__restrict__ out) {
    double d[1] = {0.0};
    for (size_t i = blockIdx.x * blockDim.x + threadIdx.x; i < (size_t)n; i += gridDim.x * blockDim.x) d[0] += v[i] * v[i];
    if (grid_reduce<1>(d, partials, ticket) && threadIdx.x == 0) *out = ::sqrt(d[0]);
}

__global__ void k_apply_increment(int n_rows, int nf, const int *__restrict__ row2node, const double *__restrict__ delta,
                                  double *__restrict__ u) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n_rows) return;
    const int node = row2node[r];
    for (int f = 0; f < nf; ++f) u[(size_t)node * nf + f] += delta[(size_t)r * nf + f];
}

// u[node*nf+f] = u_prev[node*nf+f] on the free DOFs of the active rows (bit f
// of free_mask[node]), 0 on their Dirichlet DOFs; other nodes are not written
__global__ void k_predict_increment(int n_rows, int nf, const int *__restrict__ row2node,
                                    const uint8_t *__restrict__ free_mask, const double *__restrict__ u_prev,
                                    double *__restrict__ u) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n_rows) return;
    const int node = row2node[r];
    const unsigned m = free_mask[node];
    for (int f = 0; f < nf; ++f) {
        const size_t i = (size_t)node * nf + f;
        u[i] = ((m >> f) & 1u) ? u_prev[i] : 0.0;
    }
}

}  // namespace
}  // namespace gw

namespace gw {
namespace {  // internal linkage: each translation unit compiles the kernels it launches

// ---------------------------------------------------------------- restarted GMRES(m)
// Right-preconditioned GMRES with classical Gram-Schmidt and a
// re-orthogonalisation pass when needed.  Column k of the Arnoldi process is
// four kernels:
//   spmv:  w = A z_k                       (z_k = Minv v_k, or a V-cycle)
//   dots:  block partials of (v_i, w), i <= k, and (w, w)
//   upd:   every block sums the partials to h; w -= V h; block partials of
//          ||w||^2; block 0 stores h.  ||w - V h||^2 = (w, w) - sum h_i^2 below
//          gs_eta2 (w, w) (by default 1/100: the projection removed more than
//          90% of w's norm) means V h lost more than ~10 ulp of orthogonality and
//          a second pass (dots and upd with pass = 1) is needed
//   next:  every block sums ||w||; v_{k+1} = w / ||w||, z_{k+1}; meanwhile block 0
//          closes the column: Givens rotation, residual estimate, cycle /
//          convergence flags, k += 1
// No kernel ends in a grid-wide reduction: its consumer sums the partials in
// block order (deterministic).  The second pass is queued with every column and
// returns at once where the first one is enough.
// Robust for the nonsymmetric, indefinite Jacobians of the penalty footing
// and the u-p saddle-point systems, on which BiCGSTAB breaks down.
constexpr int kGmresMaxRestart = 128;

struct GScalars {
    // scalar header first: the host polls only this prefix
    double beta, bnorm, tol, resid;
    double gs_eta2;  // second Gram-Schmidt pass below this fraction of ||w||^2 left
    int k;           // completed Arnoldi columns in the current cycle
    int cycle_done, done, status, iters, max_iter, restart;
    unsigned ticket;
    int reorth;      // column k takes the second Gram-Schmidt pass
    int kn;          // basis vector `next` forms (its own copy: block 0 advances k meanwhile)
    int reorths;     // second passes taken in this solve
    int guard;       // first failed index guard up to the last residual
    double H[kGmresMaxRestart + 1][kGmresMaxRestart];
    double cs[kGmresMaxRestart], sn[kGmresMaxRestart];
    double g[kGmresMaxRestart + 1];
    double y[kGmresMaxRestart];
};

struct GmresVecs {
    double *x, *w, *V, *Minv, *partials, *z;
    const double *b;
    GScalars *sc;
    size_t n;  // n_rows * NF (stride of V)
};

// start of a solve: the header cleared, the limits set (one launch for a memset
// and two host copies)
__global__ void k_gm_begin(GScalars *sc, int max_iter, int restart, double eta2) {
    constexpr int head = offsetof(GScalars, H) / 4;
    for (int i = threadIdx.x; i < head; i += blockDim.x) ((int *)sc)[i] = 0;
    __syncthreads();
    if (threadIdx.x == 0) {
        sc->max_iter = max_iter;
        sc->restart = restart;
        sc->gs_eta2 = eta2;
    }
}

// w = r = b - A x ; beta = ||r|| ; first cycle also ||b|| and the tolerance
template <int NF, typename VT>
__global__ void k_gm_residual(PtrsA A, GmresVecs G, int first, double rtol) {
    if (G.sc->done) return;
    const int nw = gridDim.x * (blockDim.x >> 5) * kRowsPerWarp;
    double d[2] = {0.0, 0.0};
    for (int rb = (blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * kRowsPerWarp; rb < A.n_rows; rb += nw) {
        const int r = rb + (threadIdx.x & 31) / kLPR;
        double acc[NF];
        row_mv<NF, VT>(A, r, G.x, acc);
        if (r < A.n_rows && (threadIdx.x & (kLPR - 1)) == 0)
#pragma unroll
            for (int f = 0; f < NF; ++f) {
                const size_t i = (size_t)r * NF + f;
                const double rv = G.b[i] - acc[f];
                G.w[i] = rv;
                d[0] += rv * rv;
                d[1] += G.b[i] * G.b[i];
            }
    }
    if (grid_reduce<2>(d, G.partials, &G.sc->ticket) && threadIdx.x == 0) {
        GScalars *sc = G.sc;
        sc->beta = ::sqrt(d[0]);
        if (first) {
            sc->bnorm = ::sqrt(d[1]);
            sc->tol = rtol * sc->bnorm;
            sc->iters = 0;
            sc->status = 0;
        }
        sc->resid = sc->beta;
        sc->k = 0;
        sc->cycle_done = 0;
        sc->reorth = sc->kn = 0;
        sc->guard = *(volatile int *)&g_guard_site;
        sc->g[0] = sc->beta;
        for (int i = 1; i <= kGmresMaxRestart; ++i) sc->g[i] = 0.0;
        if (!isfinite(sc->beta)) { sc->status = ST_NAN; sc->done = 1; sc->cycle_done = 1; }
        else if (sc->beta <= sc->tol || sc->bnorm == 0.0 || sc->iters >= sc->max_iter) { sc->done = 1; sc->cycle_done = 1; }
    }
}

// w = A z_k
template <int NF, typename VT>
__global__ void k_gm_spmv(PtrsA A, GmresVecs G) {
    pdl_wait();
    pdl_release();
    if (G.sc->cycle_done) return;
    const int nw = gridDim.x * (blockDim.x >> 5) * kRowsPerWarp;
    for (int rb = (blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * kRowsPerWarp; rb < A.n_rows; rb += nw) {
        const int r = rb + (threadIdx.x & 31) / kLPR;
        double acc[NF];
        row_mv<NF, VT>(A, r, G.z, acc);
        if (r < A.n_rows && (threadIdx.x & (kLPR - 1)) == 0)
#pragma unroll
            for (int f = 0; f < NF; ++f) G.w[(size_t)r * NF + f] = acc[f];
    }
}

// The same with a warp per row, for small systems of long rows (3D: up to 125
// blocks): eight lanes per row leave 216 rows on 7 CTAs and eight dependent trips
// per lane (12.8 us for 13,824 4 x 4 FP64 blocks).  The first PF trips' columns and
// blocks are loaded ahead of the wait; the state is tested before the store.
template <int NF, typename VT>
__global__ void __launch_bounds__(128) k_gm_spmv_wide(PtrsA A, GmresVecs G) {
    const int r = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (r >= A.n_rows) return;  // whole warps
    constexpr int PF = NF * NF * (int)sizeof(VT) > 64 ? 2 : 3;
    const VT *vals = (const VT *)A.vals;
    const int s = __ldg(A.row_ptr + r), e = __ldg(A.row_ptr + r + 1);
    int col[PF];
    double bv[PF][NF * NF], acc[NF], xv[NF];
#pragma unroll
    for (int t = 0; t < PF; ++t) {
        const int j = s + lane + 32 * t;
        col[t] = -1;
        if (j < e) {
            col[t] = __ldg(A.cols + j);
            if (!in_range(col[t], A.n_rows, GS_ROW_MV)) col[t] = -1;
            load_block<NF, VT>(vals + (size_t)j * NF * NF, bv[t]);
        }
    }
    pdl_wait();
    pdl_release();
    const bool off = G.sc->cycle_done;
#pragma unroll
    for (int f = 0; f < NF; ++f) acc[f] = 0.0;
#pragma unroll
    for (int t = 0; t < PF; ++t)
        if (col[t] >= 0) {
            load_rw<NF>(G.z + (size_t)col[t] * NF, xv);
#pragma unroll
            for (int f = 0; f < NF; ++f)
#pragma unroll
                for (int g = 0; g < NF; ++g) acc[f] += bv[t][f * NF + g] * xv[g];
        }
    for (int j = s + lane + 32 * PF; j < e; j += 32) {
        const int c = __ldg(A.cols + j);
        if (!in_range(c, A.n_rows, GS_ROW_MV)) continue;
        double b[NF * NF];
        load_rw<NF>(G.z + (size_t)c * NF, xv);
        load_block<NF, VT>(vals + (size_t)j * NF * NF, b);
#pragma unroll
        for (int f = 0; f < NF; ++f)
#pragma unroll
            for (int g = 0; g < NF; ++g) acc[f] += b[f * NF + g] * xv[g];
    }
#pragma unroll
    for (int f = 0; f < NF; ++f)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) acc[f] += __shfl_down_sync(0xffffffffu, acc[f], o);
    if (lane == 0 && !off) store_rw<NF>(G.w + (size_t)r * NF, acc);
}

// ---------------------------------------------------------------- Gram-Schmidt
// What bounds these kernels: the basis, read once by dots and once by upd (8 (k + 1) n
// bytes each), and on systems below ~50k unknowns the latency of the reduction.
// Dots and update of column 8, B200: 532k unknowns 49 us as one kernel each with a
// last-block reduction -> 12 + 11 us; 52k unknowns 20 -> 2 + 4 us; 864 unknowns with a
// 100-vector basis (3D node-block GMRES): one iteration 90 -> 46 us.
constexpr int kGsThreads = 256;
constexpr int kGsBlocks = 296;                    // element blocks: two per SM
constexpr int kGsItems = kGmresMaxRestart + 1;    // (v_i, w), i <= k < restart, and (w, w)
constexpr int kGsGroup = 8;                       // items per block of k_gm_dots
// Unknowns up to which k_gm_update splits the basis over warps.  A solve of 100 columns,
// never split -> always: 8,788 unknowns 2,988 -> 2,683 us, 16,384: 3,397 -> 3,148, 23,328:
// 3,764 -> 3,865, 32,000: 4,136 -> 4,291, 108,000: 9,425 -> 10,478.
constexpr int kGsSplitMax = 16384;
// partials: dots item i of element block b at [i * kGsBlocks + b]; ||w||^2 after them
constexpr int kGsPartials = (kGsItems + 1) * kGsBlocks;

// element blocks of k_gm_dots (gridDim.x) and of k_gm_update for n unknowns
__host__ __device__ inline int gs_dots_blocks(size_t n) {
    const size_t b = (n / 2 + kGsThreads - 1) / kGsThreads;
    return b < 1 ? 1 : (b > (size_t)kGsBlocks ? kGsBlocks : (int)b);
}
__host__ __device__ inline int gs_update_blocks(size_t n) {
    const size_t per = n <= (size_t)kGsSplitMax ? 64 : 2 * kGsThreads;
    const size_t b = (n + per - 1) / per;
    return b < 1 ? 1 : (b > (size_t)kGsBlocks ? kGsBlocks : (int)b);
}
// a warp's sum in a fixed tree, valid in every lane
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// one thread's share of inner products g .. g + CNT - 1 (CNT = 0: cnt of them, at
// run time); item k + 1 is (w, w)
template <bool PAIR, int CNT>
__device__ __forceinline__ void gs_dots_body(const GmresVecs &G, int g, int cnt, int k, double acc[kGsGroup]) {
    const size_t n = G.n, nv = PAIR ? n / 2 : n;
    const size_t T = (size_t)gridDim.x * kGsThreads;
    constexpr int M = CNT ? CNT : kGsGroup;
#pragma unroll 2
    for (size_t e = (size_t)blockIdx.x * kGsThreads + threadIdx.x; e < nv; e += T) {
        if (PAIR) {
            const double2 w = reinterpret_cast<const double2 *>(G.w)[e];
            double2 x[M];
#pragma unroll
            for (int v = 0; v < M; ++v)
                if (CNT || v < cnt)
                    x[v] = reinterpret_cast<const double2 *>((CNT || g + v <= k) ? G.V + (size_t)(g + v) * n : G.w)[e];
#pragma unroll
            for (int v = 0; v < M; ++v)
                if (CNT || v < cnt) acc[v] += x[v].x * w.x + x[v].y * w.y;
        } else {
            const double w = G.w[e];
            double x[M];
#pragma unroll
            for (int v = 0; v < M; ++v)
                if (CNT || v < cnt) x[v] = ((CNT || g + v <= k) ? G.V + (size_t)(g + v) * n : G.w)[e];
#pragma unroll
            for (int v = 0; v < M; ++v)
                if (CNT || v < cnt) acc[v] += x[v] * w;
        }
    }
}

// Block (bx, by): elements of block bx against the eight items from 8 by on, so a
// thread has eight independent loads per element in flight and small systems
// still spread over the basis.  The eight sums of a warp are reduced together
// (each exchange halves what a lane keeps: 9 shuffles instead of 40).
__global__ void __launch_bounds__(kGsThreads) k_gm_dots(GmresVecs G, int pass) {
    pdl_wait();
    pdl_release();
    if (G.sc->cycle_done) return;
    if (pass == 1 && !G.sc->reorth) return;  // uniform over the grid
    const int k = G.sc->k;
    if (!in_range(k, G.sc->restart, GS_KRYLOV_K)) return;
    const int items = pass == 0 ? k + 2 : k + 1;  // k < restart <= kGmresMaxRestart
    const int g = blockIdx.y * kGsGroup;
    if (g >= items) return;
    const int cnt = min(kGsGroup, items - g);
    double a[kGsGroup];
#pragma unroll
    for (int v = 0; v < kGsGroup; ++v) a[v] = 0.0;
    const bool full = g + kGsGroup <= k + 1;  // eight basis vectors
    if (G.n & 1) {
        if (full) gs_dots_body<false, kGsGroup>(G, g, cnt, k, a);
        else gs_dots_body<false, 0>(G, g, cnt, k, a);
    } else {
        if (full) gs_dots_body<true, kGsGroup>(G, g, cnt, k, a);
        else gs_dots_body<true, 0>(G, g, cnt, k, a);
    }
    __shared__ double sh[kGsThreads / 32][kGsGroup];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int h = kGsGroup / 2, o = 16; h > 0; h >>= 1, o >>= 1) {
        const bool up = lane & o;
#pragma unroll
        for (int j = 0; j < h; ++j) {
            const double keep = up ? a[j + h] : a[j], send = up ? a[j] : a[j + h];
            a[j] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
    }
    a[0] += __shfl_xor_sync(0xffffffffu, a[0], 2);
    a[0] += __shfl_xor_sync(0xffffffffu, a[0], 1);
    // lane bits 4, 3, 2 now select the item's bits 2, 1, 0
    if ((lane & 3) == 0) sh[warp][(lane >> 4 & 1) * 4 + (lane >> 3 & 1) * 2 + (lane >> 2 & 1)] = a[0];
    __syncthreads();
    if (threadIdx.x < cnt) {
        double s = 0.0;
#pragma unroll
        for (int w = 0; w < kGsThreads / 32; ++w) s += sh[w][threadIdx.x];
        G.partials[(size_t)(g + threadIdx.x) * kGsBlocks + blockIdx.x] = s;
    }
}

// w -= V c (c = the first pass's h, or the second's correction), block partials of
// ||w||^2.  SPLIT (small systems): a block takes 64 elements (32 for odd n) and
// its warps every eighth basis vector each, so a column of 100 vectors is a
// chain of 13 loads; otherwise a thread runs over the basis with eight loads in
// flight.
template <bool SPLIT, bool PAIR>
__device__ __forceinline__ double gs_update_body(const GmresVecs &G, int k, const double *coef) {
    const size_t n = G.n;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr int NW = kGsThreads / 32;
    constexpr int E = PAIR ? 2 : 1;
    double d = 0.0;
    if (SPLIT) {
        __shared__ double part[NW][64];
        const size_t tiles = (n + 32 * E - 1) / (32 * E);
        for (size_t t = blockIdx.x; t < tiles; t += gridDim.x) {
            const size_t q = t * 32 * E + lane * E;
            double s0 = 0.0, s1 = 0.0;
            if (q < n) {
#pragma unroll 8
                for (int i = warp; i <= k; i += NW) {
                    const double c = coef[i];
                    if (PAIR) {
                        const double2 v = *reinterpret_cast<const double2 *>(G.V + (size_t)i * n + q);
                        s0 += c * v.x;
                        s1 += c * v.y;
                    } else {
                        s0 += c * G.V[(size_t)i * n + q];
                    }
                }
            }
            part[warp][lane * E] = s0;
            if (PAIR) part[warp][lane * E + 1] = s1;
            __syncthreads();
            const size_t p = t * 32 * E + threadIdx.x;
            if (threadIdx.x < 32 * E && p < n) {
                double s = 0.0;
#pragma unroll
                for (int w = 0; w < NW; ++w) s += part[w][threadIdx.x];
                const double w = G.w[p] - s;
                G.w[p] = w;
                d += w * w;
            }
            __syncthreads();
        }
    } else {
        const size_t nv = n / E, T = (size_t)gridDim.x * kGsThreads;
#pragma unroll 2
        for (size_t e = (size_t)blockIdx.x * kGsThreads + threadIdx.x; e < nv; e += T) {
            if (PAIR) {
                double2 w = reinterpret_cast<const double2 *>(G.w)[e];
#pragma unroll 8
                for (int i = 0; i <= k; ++i) {
                    const double2 v = reinterpret_cast<const double2 *>(G.V + (size_t)i * n)[e];
                    w.x -= coef[i] * v.x;
                    w.y -= coef[i] * v.y;
                }
                reinterpret_cast<double2 *>(G.w)[e] = w;
                d += w.x * w.x + w.y * w.y;
            } else {
                double w = G.w[e];
#pragma unroll 8
                for (int i = 0; i <= k; ++i) w -= coef[i] * G.V[(size_t)i * n + e];
                G.w[e] = w;
                d += w * w;
            }
        }
    }
    return d;
}

__global__ void __launch_bounds__(kGsThreads) k_gm_update(GmresVecs G, int pass) {
    pdl_wait();
    pdl_release();
    GScalars *sc = G.sc;
    if (sc->cycle_done) return;
    if (pass == 1 && !sc->reorth) return;  // uniform over the grid
    const int k = sc->k;
    if (!in_range(k, sc->restart, GS_KRYLOV_K)) return;  // uniform over the grid
    __shared__ double coef[kGsItems + 1];
    __shared__ double red[kGsThreads / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int items = pass == 0 ? k + 2 : k + 1, nb = gs_dots_blocks(G.n);
    if (nb <= 8) {  // a thread per item, all of its partials in flight
        if (threadIdx.x < items) {
            double p[8], s = 0.0;
#pragma unroll
            for (int b = 0; b < 8; ++b) p[b] = b < nb ? G.partials[(size_t)threadIdx.x * kGsBlocks + b] : 0.0;
#pragma unroll
            for (int b = 0; b < 8; ++b) s += p[b];
            coef[threadIdx.x] = s;
        }
    } else {
        for (int i0 = warp; i0 < items; i0 += 4 * kGsThreads / 32) {  // four items of a warp in flight
            double s[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 2
            for (int b = lane; b < nb; b += 32)
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    if (i0 + q * kGsThreads / 32 < items)
                        s[q] += G.partials[(size_t)(i0 + q * kGsThreads / 32) * kGsBlocks + b];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                s[q] = warp_sum(s[q]);
                if (lane == 0 && i0 + q * kGsThreads / 32 < items) coef[i0 + q * kGsThreads / 32] = s[q];
            }
        }
    }
    __syncthreads();
    if (blockIdx.x == 0 && warp == 0) {
        if (pass == 0) {
            double q = 0.0;
            for (int i = lane; i <= k; i += 32) {
                sc->H[i][k] = coef[i];
                q += coef[i] * coef[i];
            }
            q = warp_sum(q);
            if (lane == 0) {
                const double wsq = coef[k + 1];
                const int re = !(wsq - q >= sc->gs_eta2 * wsq);  // also when not finite
                sc->reorth = re;
                sc->reorths += re;
                sc->kn = k + 1;
            }
        } else {
            for (int i = lane; i <= k; i += 32) sc->H[i][k] += coef[i];
        }
    }
    const bool split = G.n <= (size_t)kGsSplitMax, odd = G.n & 1;
    double d;
    if (split) d = odd ? gs_update_body<true, false>(G, k, coef) : gs_update_body<true, true>(G, k, coef);
    else d = odd ? gs_update_body<false, false>(G, k, coef) : gs_update_body<false, true>(G, k, coef);
    d = warp_sum(d);
    if (lane == 0) red[warp] = d;
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = 0.0;
#pragma unroll
        for (int w = 0; w < kGsThreads / 32; ++w) s += red[w];
        G.partials[(size_t)kGsItems * kGsBlocks + blockIdx.x] = s;
    }
}

// Closes column k with ||w|| = hn (one warp): rotations of the earlier columns,
// the new one, residual estimate and flags.
__device__ __forceinline__ void gs_close(GScalars *sc, int k, double hn) {
    __shared__ double h[kGmresMaxRestart + 1], cs[kGmresMaxRestart], sn[kGmresMaxRestart];
    const int lane = threadIdx.x & 31;
    for (int i = lane; i <= k; i += 32) {
        h[i] = sc->H[i][k];
        if (i < k) { cs[i] = sc->cs[i]; sn[i] = sc->sn[i]; }
    }
    __syncwarp();
    if (lane == 0) {
        double a = h[0];
#pragma unroll 8
        for (int i = 0; i < k; ++i) {  // previous rotations
            const double b2 = h[i + 1];
            h[i] = cs[i] * a + sn[i] * b2;
            a = -sn[i] * a + cs[i] * b2;
        }
        const double rr = ::sqrt(a * a + hn * hn);
        double c = 1.0, s = 0.0;
        if (rr > 0.0) { c = a / rr; s = hn / rr; }
        h[k] = rr;
        const double gk = sc->g[k], next = -s * gk;
        sc->cs[k] = c;
        sc->sn[k] = s;
        sc->H[k + 1][k] = 0.0;
        sc->g[k + 1] = next;
        sc->g[k] = c * gk;
        sc->resid = fabs(next);
        const int it = sc->iters + 1;
        sc->iters = it;
        sc->k = k + 1;
        if (!isfinite(next)) { sc->status = ST_NAN; sc->cycle_done = 1; sc->done = 1; }
        else if (fabs(next) <= sc->tol || hn == 0.0 || k + 1 >= sc->restart || it >= sc->max_iter) sc->cycle_done = 1;
    }
    __syncwarp();
    for (int i = lane; i <= k; i += 32) sc->H[i][k] = h[i];
}

// v_{k+1} = w / ||w|| (v_0 = w / beta at a cycle start) -> V, and
//   zout = scale Minv v   (node-block preconditioner, or a smoother's zero-start sweep), or
//   zout = v              (Minv nullptr: a V-cycle's right-hand side), or nothing (zout nullptr).
// Block 0 closes the column (one warp; not at a start) while the others work:
// they read kn, which the close leaves alone, and a
// cycle_done that appears under them only spares them a vector no one reads.
template <int NF>
__global__ void __launch_bounds__(kGsThreads) k_gm_next(int n_rows, GmresVecs G, int start, const double *Minv,
                                                        double *zout, double scale) {
    GScalars *sc = G.sc;
    const int r = ((int)blockIdx.x - 1) * kGsThreads + threadIdx.x;
    const bool own = blockIdx.x > 0 && r < n_rows;
    double M[NF * NF];  // written before this solve's Arnoldi steps: loaded ahead of the wait
    if (Minv && own)
#pragma unroll
        for (int i = 0; i < NF * NF; ++i) M[i] = __ldg(Minv + (size_t)r * NF * NF + i);
    pdl_wait();
    pdl_release();
    double v[NF];
    if (own) load_rw<NF>(G.w + (size_t)r * NF, v);
    if (sc->cycle_done) return;
    const int kn = sc->kn;
    if (!in_range(kn, sc->restart + 1, GS_KRYLOV_K)) return;  // V holds restart + 1 vectors
    double hn;
    __shared__ double red[kGsThreads / 32];
    if (start) {
        hn = sc->beta;
    } else {
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nb = gs_update_blocks(G.n);
        double s = 0.0;
        for (int b = threadIdx.x; b < nb; b += kGsThreads) s += G.partials[(size_t)kGsItems * kGsBlocks + b];
        s = warp_sum(s);
        if (lane == 0) red[warp] = s;
        __syncthreads();
        s = 0.0;
#pragma unroll
        for (int w = 0; w < kGsThreads / 32; ++w) s += red[w];
        hn = ::sqrt(s);
    }
    if (blockIdx.x == 0) {
        if (!start && threadIdx.x < 32) gs_close(sc, kn - 1, hn);
        return;
    }
    if (!own) return;
    const double ih = 1.0 / hn;
#pragma unroll
    for (int f = 0; f < NF; ++f) v[f] *= ih;
    store_rw<NF>(G.V + (size_t)kn * G.n + (size_t)r * NF, v);
    if (!zout) return;
    if (Minv) {
        double z[NF];
#pragma unroll
        for (int i = 0; i < NF; ++i) {
            double t = 0.0;
#pragma unroll
            for (int j = 0; j < NF; ++j) t += M[i * NF + j] * v[j];
            z[i] = scale * t;
        }
        store_rw<NF>(zout + (size_t)r * NF, z);
    } else {
        store_rw<NF>(zout + (size_t)r * NF, v);
    }
}

// End of a cycle: y = H^{-1} g by back substitution, one warp, by columns: a
// lane keeps the right-hand sides of rows lane, lane + 32, ... and the loads of
// the next column do not wait for this one's y.
__global__ void k_gm_solve_y(GScalars *sc) {
    if (sc->done) return;
    const int k = sc->k, lane = threadIdx.x;
    if (!in_range(k, sc->restart + 1, GS_KRYLOV_K)) return;
    constexpr int R = kGmresMaxRestart / 32;
    double g[R], h[R];
#pragma unroll
    for (int q = 0; q < R; ++q) {
        const int r = lane + 32 * q;
        g[q] = r < k ? sc->g[r] : 0.0;
        h[q] = r < k ? sc->H[r][k - 1] : 0.0;
    }
    for (int i = k - 1; i >= 0; --i) {
        double hn[R];
#pragma unroll
        for (int q = 0; q < R; ++q) hn[q] = (i > 0 && lane + 32 * q < i) ? sc->H[lane + 32 * q][i - 1] : 0.0;
        double gi = 0.0, hi = 0.0;
#pragma unroll
        for (int q = 0; q < R; ++q)
            if (i >> 5 == q) { gi = g[q]; hi = h[q]; }
        gi = __shfl_sync(0xffffffffu, gi, i & 31);
        hi = __shfl_sync(0xffffffffu, hi, i & 31);
        const double y = hi != 0.0 ? gi / hi : 0.0;
        if (lane == 0) sc->y[i] = y;
#pragma unroll
        for (int q = 0; q < R; ++q) {
            g[q] -= h[q] * y;
            h[q] = hn[q];
        }
    }
}

// x += Minv (V y)
template <int NF>
__global__ void k_gm_update_x(int n_rows, GmresVecs G) {
    const GScalars *sc = G.sc;
    if (sc->done) return;
    const int k = sc->k;
    if (!in_range(k, sc->restart + 1, GS_KRYLOV_K)) return;
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < n_rows; r += gridDim.x * blockDim.x) {
        double u[NF], z[NF];
#pragma unroll
        for (int f = 0; f < NF; ++f) {
            double s = 0.0;
            for (int i = 0; i < k; ++i) s += sc->y[i] * G.V[(size_t)i * G.n + (size_t)r * NF + f];
            u[f] = s;
        }
        apply_minv<NF>(G.Minv, r, u, z);
#pragma unroll
        for (int f = 0; f < NF; ++f) G.x[(size_t)r * NF + f] += z[f];
    }
}

}  // namespace
}  // namespace gw
