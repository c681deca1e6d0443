// Row kernels of the 2D multigrid-preconditioned GMRES on a sliced layout.
//
// What bounds them: on levels of a few thousand rows, the chain of dependent
// loads (row_ptr -> cols -> x) and the kernel boundary; on the finest level of
// a large batch, the bytes of the matrix.  Block-CSR rows served neither: a
// 3 x 3-node row holds 9 blocks, so a group of 8 lanes ran two trips with one
// lane of the second at work, and every lane waited for row_ptr, then cols,
// then x.
//
// Layout: rows go in chunks of 32 / LPR, one warp per chunk, LPR lanes per
// row; trip t of a chunk holds slots t * LPR .. t * LPR + LPR - 1 of each row (the
// block-CSR order of the row), one block per lane, so every load of columns and
// values is coalesced and needs no row pointer.  A chunk takes kSellTrips<LPR>
// trips of storage at a fixed stride and runs trips[c] of them; slots past a row's
// length hold zeros and the row's own column.  Column indices are checked once,
// when the pattern is laid out.
//
// LPR = 1 where the rows alone fill the device (no padding beyond the longest
// row of 32, no shuffles), 4 on small levels (a quarter of the chain per lane);
// see sell_lpr.
//
// Kernels of one Arnoldi step are launched with programmatic dependent launch:
// a kernel starts while its predecessor runs, loads what no kernel of the
// solve writes (columns, values, smoother blocks, transfer lists) and then waits
// (griddepcontrol.wait) before it touches a vector.  It releases its successor
// after that wait, so when a kernel starts, everything before its predecessor
// has completed.  Vectors are read through plain pointers: never __restrict__
// const, whose read-only path may be hoisted above the wait.
//
// One Arnoldi step, B200 at 1965 MHz, with block-CSR rows and plain launches -> with
// this layout and dependent launch alone: 26k rows FP64 125 -> 91 us, 267k rows FP32
// 297 -> 189 us.
#pragma once
#include <algorithm>

#include "gw_mg.cuh"

namespace gw {
namespace {  // internal linkage: each translation unit compiles the kernels it launches

constexpr int kSellSlots = 25;  // blocks of a 2D row: the 5 x 5 stencil
template <int LPR>
constexpr int kSellTrips = (kSellSlots + LPR - 1) / LPR;
__host__ __device__ inline int sell_trips(int lpr) { return (kSellSlots + lpr - 1) / lpr; }

// Lanes per row of a level, by its rows alone (both the separate kernels and
// the fused tail follow it, so their sums are the same).  Few rows with a lane each
// are less than 6 warps per SM, and too few loads in flight; above, four lanes load a
// quarter more (9 blocks in 12 slots).  30 Arnoldi steps with the finest level at four
// lanes -> one, 2 x 2 blocks FP64 / FP32: 10,000 rows 2.01 -> 2.04 / 2.01 -> 2.01 ms, 15,129:
// 2.15 -> 2.17 / 2.17 -> 2.16, 19,881: 2.32 -> 2.26 / 2.29 -> 2.20, 24,964: 2.36 -> 2.27 /
// 2.37 -> 2.24, 40,000: 2.92 -> 2.74 / 2.85 -> 2.64, 90,000: 4.26 -> 3.84 / 4.00 -> 3.54; 3 x 3
// blocks alike.  Below the finest level, 19k FP32 rows got slower with one lane (solves on
// 72k and 267k rows 14.40 -> 14.59 and 51.3 -> 52.1 ms), so the line lies above them.
constexpr int kSellOneLane = 24576;
inline int sell_lpr(int n_rows) { return n_rows >= kSellOneLane ? 1 : 4; }

__host__ __device__ inline int sell_chunks(int n_rows, int lpr) { return (n_rows + 32 / lpr - 1) / (32 / lpr); }

// One block is NU units of one load each: 16-byte units for even NF in FP32 and
// FP64, a 4 x BF16 unit for NF = 2, else scalars.  Unit u of trip t of chunk c
// is at ((c * trips + t) * NU + u) * 32 + lane.
template <int NF, typename VT> struct SellUnit { typedef VT U; static const int NU = NF * NF; };
template <> struct SellUnit<2, float> { typedef float4 U; static const int NU = 1; };
template <> struct SellUnit<2, double> { typedef double2 U; static const int NU = 2; };
template <> struct SellUnit<4, float> { typedef float4 U; static const int NU = 4; };
template <> struct SellUnit<4, double> { typedef double2 U; static const int NU = 8; };
template <> struct SellUnit<2, __nv_bfloat16> { typedef uint2 U; static const int NU = 1; };

struct SellA {
    int n_rows, n_chunks;
    const int *cols;
    const void *vals;
    const int *trips;
};

// block slots of a level of at most n_rows rows, whatever its lanes per row
inline int64_t sell_elems(int64_t n_rows) {
    const int64_t four = std::min<int64_t>(n_rows, kSellOneLane - 1), one = n_rows >= kSellOneLane ? n_rows : 0;
    return 32 * std::max((four + 7) / 8 * kSellTrips<4>, (one + 31) / 32 * kSellTrips<1>);
}

__device__ __forceinline__ void unit_get(float v, double *o) { o[0] = (double)v; }
__device__ __forceinline__ void unit_get(double v, double *o) { o[0] = v; }
__device__ __forceinline__ void unit_get(__nv_bfloat16 v, double *o) { o[0] = (double)__bfloat162float(v); }
__device__ __forceinline__ void unit_get(const float4 &v, double *o) { o[0] = v.x; o[1] = v.y; o[2] = v.z; o[3] = v.w; }
__device__ __forceinline__ void unit_get(const double2 &v, double *o) { o[0] = v.x; o[1] = v.y; }
__device__ __forceinline__ void unit_get(const uint2 &v, double *o) {
    const __nv_bfloat162 a = *reinterpret_cast<const __nv_bfloat162 *>(&v.x);
    const __nv_bfloat162 b = *reinterpret_cast<const __nv_bfloat162 *>(&v.y);
    o[0] = __low2float(a); o[1] = __high2float(a); o[2] = __low2float(b); o[3] = __high2float(b);
}
template <typename T> __device__ __forceinline__ T sell_ld(const T *p) { return __ldg(p); }

// The columns and values of a chunk's first PF trips in registers, the rest
// streamed; PF keeps the prefetched values within about 72 registers.
template <int NF, typename VT, int LPR>
struct SellRow {
    typedef typename SellUnit<NF, VT>::U U;
    static const int NU = SellUnit<NF, VT>::NU;
    static const int T = kSellTrips<LPR>;
    static const int COST = 1 + (int)(NU * sizeof(U) / 4);
    static const int FIT = (LPR == 1 ? 48 : 72) / COST;
    static const int PF = FIT < 1 ? 1 : (FIT > T ? T : FIT);
    int trips;
    int col[PF];
    U val[PF][NU];

    __device__ __forceinline__ void load(const SellA &A, int c, int lane) {
        trips = sell_ld(A.trips + c);
        const int *cp = A.cols + (size_t)c * T * 32 + lane;
        const U *vp = (const U *)A.vals + (size_t)c * T * NU * 32 + lane;
#pragma unroll
        for (int t = 0; t < PF; ++t)
            if (t < trips) {
                col[t] = sell_ld(cp + t * 32);
#pragma unroll
                for (int u = 0; u < NU; ++u) val[t][u] = sell_ld(vp + (t * NU + u) * 32);
            }
    }
    static __device__ __forceinline__ void mad(const U v[NU], const double xv[NF], double acc[NF]) {
        double b[NF * NF];
#pragma unroll
        for (int u = 0; u < NU; ++u) unit_get(v[u], b + u * (NF * NF / NU));
#pragma unroll
        for (int f = 0; f < NF; ++f)
#pragma unroll
            for (int g = 0; g < NF; ++g) acc[f] += b[f * NF + g] * xv[g];
    }
    // acc = (A x)_r, valid in the first lane of the row's group
    __device__ __forceinline__ void mul(const SellA &A, int c, int lane, const double *x, double acc[NF]) const {
#pragma unroll
        for (int f = 0; f < NF; ++f) acc[f] = 0.0;
        double xv[NF];
#pragma unroll
        for (int t = 0; t < PF; ++t)
            if (t < trips) {
                load_rw<NF>(x + (size_t)col[t] * NF, xv);
                mad(val[t], xv, acc);
            }
        if (PF < T) {
            const int *cp = A.cols + (size_t)c * T * 32 + lane;
            const U *vp = (const U *)A.vals + (size_t)c * T * NU * 32 + lane;
#pragma unroll 2
            for (int t = PF; t < trips; ++t) {
                U v[NU];
#pragma unroll
                for (int u = 0; u < NU; ++u) v[u] = sell_ld(vp + (t * NU + u) * 32);
                load_rw<NF>(x + (size_t)sell_ld(cp + t * 32) * NF, xv);
                mad(v, xv, acc);
            }
        }
        if (LPR > 1) {
#pragma unroll
            for (int f = 0; f < NF; ++f)
#pragma unroll
                for (int o = LPR / 2; o > 0; o >>= 1) acc[f] += __shfl_down_sync(0xffffffffu, acc[f], o, LPR);
        }
    }
};
// ---------------------------------------------------------------- laying a matrix out
// One warp per chunk: trips and columns (pattern), or the values.
__global__ void k_sell_pattern(PtrsA A, int lpr, int *__restrict__ trips, int *__restrict__ cols) {
    const int c = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    const int rpc = 32 / lpr, T = sell_trips(lpr);
    if (c >= (A.n_rows + rpc - 1) / rpc) return;  // whole warps
    const int r = c * rpc + lane / lpr, q = lane % lpr;
    const int s = r < A.n_rows ? A.row_ptr[r] : 0;
    int len = r < A.n_rows ? A.row_ptr[r + 1] - s : 0;
    if (len > kSellSlots) len = in_range(len, kSellSlots + 1, GS_ROW_MV) ? len : kSellSlots;
    int m = len;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
    const int nt = (m + lpr - 1) / lpr;
    if (lane == 0) trips[c] = nt;
    const int self = r < A.n_rows ? r : A.n_rows - 1;
    for (int t = 0; t < nt; ++t) {
        const int k = t * lpr + q;
        int col = self;
        if (k < len && in_range((long long)s + k, A.nnzb, GS_ROW_MV)) {
            const int j = A.cols[s + k];
            if (in_range(j, A.n_rows, GS_ROW_MV)) col = j;
        }
        cols[((size_t)c * T + t) * 32 + lane] = col;
    }
}

template <typename U, int N, typename VT>
__device__ __forceinline__ U unit_put(const VT *p);
template <> __device__ __forceinline__ float unit_put<float, 1, float>(const float *p) { return p[0]; }
template <> __device__ __forceinline__ double unit_put<double, 1, double>(const double *p) { return p[0]; }
template <> __device__ __forceinline__ __nv_bfloat16 unit_put<__nv_bfloat16, 1, float>(const float *p) { return __float2bfloat16_rn(p[0]); }
template <> __device__ __forceinline__ float4 unit_put<float4, 4, float>(const float *p) { return *reinterpret_cast<const float4 *>(p); }
template <> __device__ __forceinline__ double2 unit_put<double2, 2, double>(const double *p) { return *reinterpret_cast<const double2 *>(p); }
template <> __device__ __forceinline__ uint2 unit_put<uint2, 4, float>(const float *p) {
    const float4 v = *reinterpret_cast<const float4 *>(p);
    uint2 o;
    *reinterpret_cast<__nv_bfloat162 *>(&o.x) = __floats2bfloat162_rn(v.x, v.y);
    *reinterpret_cast<__nv_bfloat162 *>(&o.y) = __floats2bfloat162_rn(v.z, v.w);
    return o;
}

struct SellJob {
    PtrsA A;
    int lpr, first_warp;  // warps [first_warp, next job's first_warp) lay this level out
    const int *trips, *cols;
    void *vals;
};
struct SellJobs {
    int n, warps;
    SellJob j[kMgMaxLevels];
};

// Values of every listed level in one launch.  A slot whose stored column is
// not the matrix's (refused when the pattern was laid out) keeps a zero block.
template <int NF, typename VT, typename OT>
__global__ void k_sell_values(SellJobs js) {
    typedef typename SellUnit<NF, OT>::U U;
    constexpr int NU = SellUnit<NF, OT>::NU, PU = NF * NF / NU;
    const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (w >= js.warps) return;
    int q = 0;
    while (q + 1 < js.n && w >= js.j[q + 1].first_warp) ++q;
    const SellJob &J = js.j[q];
    const PtrsA &A = J.A;
    const int c = w - J.first_warp, rpc = 32 / J.lpr, T = sell_trips(J.lpr);
    const int r = c * rpc + lane / J.lpr, sub = lane % J.lpr;
    const int s = r < A.n_rows ? A.row_ptr[r] : 0, len = r < A.n_rows ? A.row_ptr[r + 1] - s : 0;
    const VT *src = (const VT *)A.vals;
    U *out = (U *)J.vals + (size_t)c * T * NU * 32 + lane;
    const int *cols = J.cols + (size_t)c * T * 32 + lane;
    const int nt = J.trips[c];
    for (int t = 0; t < nt; ++t) {
        const int k = t * J.lpr + sub;
        const bool on = k < len && k < kSellSlots && s + k < A.nnzb && A.cols[s + k] == cols[t * 32];
#pragma unroll
        for (int u = 0; u < NU; ++u) {
            if (on) {
                out[(t * NU + u) * 32] = unit_put<U, PU, VT>(src + (size_t)(s + k) * NF * NF + u * PU);
            } else {
                U z;
                memset(&z, 0, sizeof(U));
                out[(t * NU + u) * 32] = z;
            }
        }
    }
}

// ---------------------------------------------------------------- Arnoldi-step kernels
// A vector of the Arnoldi basis at the current column k, or a fixed buffer (stride 0).
struct VecRef {
    double *p;
    size_t stride;
    // a fixed buffer's address does not wait for k
    __device__ __forceinline__ double *at(int k) const { return stride ? p + (size_t)k * stride : p; }
};

// Whether this step's kernel has work: the state is read here, and on small
// levels (LPR > 1) tested only before the stores, so that the vector loads do not
// wait for it (a step queued past convergence computes on stale vectors and
// stores nothing); on large ones such a step must not move the matrix.
struct StepState {
    int k;
    bool off;
};
__device__ __forceinline__ StepState step_state(const GScalars *sc) {
    StepState st;
    st.k = sc->k;
    st.off = sc->cycle_done || (unsigned)st.k >= (unsigned)sc->restart;  // Z holds restart vectors
    if (st.off) st.k = 0;
    return st;
}
// one row's smoother block
template <int NF>
__device__ __forceinline__ void minv_ld(const double *Minv, int r, double M[NF * NF]) {
    if constexpr (NF == 2 || NF == 4) {
#pragma unroll
        for (int q = 0; q < NF * NF / 2; ++q) {
            const double2 v = __ldg(reinterpret_cast<const double2 *>(Minv + (size_t)r * NF * NF) + q);
            M[2 * q] = v.x; M[2 * q + 1] = v.y;
        }
    } else {
#pragma unroll
        for (int i = 0; i < NF * NF; ++i) M[i] = __ldg(Minv + (size_t)r * NF * NF + i);
    }
}
template <int NF>
__device__ __forceinline__ void minv_mul(const double M[NF * NF], const double v[NF], double z[NF]) {
#pragma unroll
    for (int i = 0; i < NF; ++i) {
        z[i] = 0.0;
#pragma unroll
        for (int j = 0; j < NF; ++j) z[i] += M[i * NF + j] * v[j];
    }
}

// x_out = x_in + omega Minv (b - A x_in)
template <int NF, typename VT, int LPR>
__global__ void __launch_bounds__(256) k_sell_jacobi(SellA A, const double *Minv, VecRef b, const double *x_in,
                                                     VecRef x_out, double omega, const GScalars *sc) {
    const int lane = threadIdx.x & 31, sub = lane % LPR;
    const int nw = gridDim.x * (blockDim.x >> 5);
    int c = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    SellRow<NF, VT, LPR> row;
    double M[NF * NF];
    auto fetch = [&]() {
        row.load(A, c, lane);
        const int r = c * (32 / LPR) + lane / LPR;
        if (r < A.n_rows && sub == 0) minv_ld<NF>(Minv, r, M);
    };
    if (c < A.n_chunks) fetch();
    pdl_wait();
    pdl_release();
    const StepState st = step_state(sc);
    if (LPR == 1 && st.off) return;
    const double *bp = b.at(st.k);
    double *xo = x_out.at(st.k);
    while (c < A.n_chunks) {
        const int r = c * (32 / LPR) + lane / LPR;
        const bool own = r < A.n_rows && sub == 0;
        double t[NF], z[NF], xi[NF], acc[NF];
        if (own) {
            load_rw<NF>(bp + (size_t)r * NF, t);
            load_rw<NF>(x_in + (size_t)r * NF, xi);
        }
        row.mul(A, c, lane, x_in, acc);
        if (LPR > 1 && st.off) return;
        if (own) {
#pragma unroll
            for (int f = 0; f < NF; ++f) t[f] -= acc[f];
            minv_mul<NF>(M, t, z);
#pragma unroll
            for (int f = 0; f < NF; ++f) z[f] = xi[f] + omega * z[f];
            store_rw<NF>(xo + (size_t)r * NF, z);
        }
        c += nw;
        if (c < A.n_chunks) fetch();
    }
}

// r = b - A x
template <int NF, typename VT, int LPR>
__global__ void __launch_bounds__(256) k_sell_residual(SellA A, VecRef b, const double *x, double *r_out,
                                                       const GScalars *sc) {
    const int lane = threadIdx.x & 31, sub = lane % LPR;
    const int nw = gridDim.x * (blockDim.x >> 5);
    int c = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    SellRow<NF, VT, LPR> row;
    if (c < A.n_chunks) row.load(A, c, lane);
    pdl_wait();
    pdl_release();
    const StepState st = step_state(sc);
    if (LPR == 1 && st.off) return;
    const double *bp = b.at(st.k);
    while (c < A.n_chunks) {
        const int r = c * (32 / LPR) + lane / LPR;
        const bool own = r < A.n_rows && sub == 0;
        double t[NF], acc[NF];
        if (own) load_rw<NF>(bp + (size_t)r * NF, t);
        row.mul(A, c, lane, x, acc);
        if (LPR > 1 && st.off) return;
        if (own) {
#pragma unroll
            for (int f = 0; f < NF; ++f) t[f] -= acc[f];
            store_rw<NF>(r_out + (size_t)r * NF, t);
        }
        c += nw;
        if (c < A.n_chunks) row.load(A, c, lane);
    }
}

// w = A z_k, z_k = Z[k] (the V-cycle's output)
template <int NF, typename VT, int LPR>
__global__ void __launch_bounds__(256) k_sell_spmv(SellA A, VecRef z, double *w, const GScalars *sc) {
    const int lane = threadIdx.x & 31, sub = lane % LPR;
    const int nw = gridDim.x * (blockDim.x >> 5);
    int c = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    SellRow<NF, VT, LPR> row;
    if (c < A.n_chunks) row.load(A, c, lane);
    pdl_wait();
    pdl_release();
    const StepState st = step_state(sc);
    if (st.off) return;
    const double *zp = z.at(st.k);
    while (c < A.n_chunks) {
        const int r = c * (32 / LPR) + lane / LPR;
        double acc[NF];
        row.mul(A, c, lane, zp, acc);
        if (r < A.n_rows && sub == 0) store_rw<NF>(w + (size_t)r * NF, acc);
        c += nw;
        if (c < A.n_chunks) row.load(A, c, lane);
    }
}

// b_c = P^T r_f through the child lists, and the coarse level's zero-start sweep
// x_1 = omega Minv b_c (Minv nullptr on the dense level)
template <int NF>
__global__ void k_sell_restrict(int nc, int nf_rows, const int *child, const uint8_t *ffixed, const double *rf,
                                double *bc, const double *Minv, double *x1, double omega, const GScalars *sc) {
    const int R = blockIdx.x * blockDim.x + threadIdx.x;
    int fr[9];
    uint8_t fx[9];
    double M[NF * NF];
    if (R < nc) {
#pragma unroll
        for (int q = 0; q < 9; ++q) fr[q] = __ldg(child + (size_t)q * nc + R);
#pragma unroll
        for (int q = 0; q < 9; ++q) {
            if (fr[q] >= 0 && !in_range(fr[q], nf_rows, GS_RESTRICT)) fr[q] = -1;
            fx[q] = fr[q] >= 0 ? __ldg(ffixed + fr[q]) : 0;
        }
        if (Minv) minv_ld<NF>(Minv, R, M);
    }
    pdl_wait();
    pdl_release();
    if (R >= nc) return;
    const bool off = sc->cycle_done;  // tested before the stores: the loads do not wait for it
    double acc[NF];
#pragma unroll
    for (int f = 0; f < NF; ++f) acc[f] = 0.0;
#pragma unroll
    for (int q = 0; q < 9; ++q) {
        if (fr[q] < 0) continue;
        const double w = (q % 3 == 1 ? 1.0 : 0.5) * (q / 3 == 1 ? 1.0 : 0.5);
        double v[NF];
        load_rw<NF>(rf + (size_t)fr[q] * NF, v);
#pragma unroll
        for (int f = 0; f < NF; ++f)
            if (!((fx[q] >> f) & 1)) acc[f] += w * v[f];
    }
    if (off) return;
    store_rw<NF>(bc + (size_t)R * NF, acc);
    if (!Minv) return;
    double z[NF];
    minv_mul<NF>(M, acc, z);
#pragma unroll
    for (int f = 0; f < NF; ++f) z[f] *= omega;
    store_rw<NF>(x1 + (size_t)R * NF, z);
}

// x = Inv b on the dense level (one warp per row)
__global__ void k_sell_dense_apply(const double *Inv, VecRef b, VecRef x, int n, const GScalars *sc) {
    pdl_wait();
    pdl_release();
    const StepState st = step_state(sc);
    const double *bp = b.at(st.k);
    double *xp = x.at(st.k);
    const int nw = gridDim.x * (blockDim.x >> 5), lane = threadIdx.x & 31;
    for (int i = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); i < n; i += nw) {
        double s = 0.0;
        for (int j = lane; j < n; j += 32) s += Inv[(size_t)i * n + j] * bp[j];
        for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
        if (lane == 0 && !st.off) xp[i] = s;
    }
}

// x_f += P x_c through the parent lists
template <int NF>
__global__ void k_sell_prolong(int n_rows, int nc, const int *parent, const uint8_t *ffixed, const double *xc,
                               double *xf, const GScalars *sc) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    int R[4];
    uint8_t fx = 0;
    if (r < n_rows) {
#pragma unroll
        for (int q = 0; q < 4; ++q) R[q] = __ldg(parent + (size_t)q * n_rows + r);
        fx = __ldg(ffixed + r);
    }
    pdl_wait();
    pdl_release();
    if (r >= n_rows) return;
    const bool off = sc->cycle_done;  // tested before the store: the loads do not wait for it
    int cnt = 0;
#pragma unroll
    for (int q = 0; q < 4; ++q) cnt += R[q] != -2;
    const double w = cnt == 1 ? 1.0 : (cnt == 2 ? 0.5 : 0.25);
    double acc[NF], x[NF];
    load_rw<NF>(xf + (size_t)r * NF, x);
#pragma unroll
    for (int f = 0; f < NF; ++f) acc[f] = 0.0;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        if (R[q] < 0 || !in_range(R[q], nc, GS_PROLONG)) continue;
        double v[NF];
        load_rw<NF>(xc + (size_t)R[q] * NF, v);
#pragma unroll
        for (int f = 0; f < NF; ++f) acc[f] += w * v[f];
    }
#pragma unroll
    for (int f = 0; f < NF; ++f)
        if (!((fx >> f) & 1)) x[f] += acc[f];
    if (off) return;
    store_rw<NF>(xf + (size_t)r * NF, x);
}

}  // namespace
}  // namespace gw
