// Fused coarse tail of the 2D multigrid V-cycle.
//
// Below a few thousand rows a V-cycle phase (smoothing, residual, transfer) is a
// kernel boundary and a chain of two or three L2 loads: 1.7-2.0 us each even with
// programmatic dependent launch, 25 of them per V-cycle on 26k rows.  k_sell_tail
// runs every level from l0 down to the dense one and back up as ONE thread-block
// cluster.  The vectors of its levels live in the cluster's shared memory, split by
// rows (row r of a level belongs to CTA r >> sh); a gather is a load from
// distributed shared memory and a phase boundary a hardware cluster barrier.
// What the phases read besides (matrix rows, smoother blocks, transfer lists,
// rows of the dense inverse) is laid out once per solve as an image of each CTA's
// shared memory (k_tail_image), every column, child and parent turned into CTA
// and byte offset of its row, and copied in with cp.async before the wait for the
// predecessor.  (Read from global memory in each phase, the same data costs what
// the fusion saves: an acquire at cluster scope drops the L1 and a phase is an L2
// chain again, 1.7 us; gathered into shared memory by the cluster itself, 25,000
// cycles a V-cycle.)  A row's gathers are issued together: one distributed
// shared-memory latency per phase.
//
// Rows, lanes and sums are those of the separate kernels (SellRow, the same
// formulas in the same order), so the V-cycle is bitwise the same with or without
// the tail and wherever it starts.
#pragma once
#include <type_traits>

#include "gw_sell.cuh"

namespace gw {
namespace {  // internal linkage: each translation unit compiles the kernels it launches

constexpr int kTailThreads = 512;
constexpr int kTailWarps = kTailThreads / 32;
constexpr int kTailMaxCluster = 16;
constexpr int kTailT = kSellTrips<4>;
constexpr uint32_t kNoRow = 0xffffffffu;

struct TailLevel {
    SellA A;
    const double *Minv;
    const uint8_t *fixed;
    const int *child;   // of this level's rows: rows of the level above (levels past l0)
    const int *parent;  // of this level's rows: rows of the level below
    int sh;             // rows per CTA: 1 << sh (at least one chunk of 8)
    int off;            // byte offset of this level's vectors in shared memory
    int sweeps;
};
struct TailArgs {
    int l0, last;  // levels l0 .. last-1 are smoothed, level last is solved with the dense inverse
    int cluster;
    TailLevel lv[kMgMaxLevels];
    const double *dInv;
    int dn, n_last;     // unknowns and rows of the dense level
    const int *child_last;
    int off_last;       // its b and x (dn doubles each, whole in every CTA)
    int off_img;        // where the image starts, after the vectors
    unsigned char *img;
    int img_stride;     // bytes per CTA
    double omega;
    VecRef b, out;      // level l0: right-hand side in, result out
    const double *x1;   // its zero-start sweep
    const GScalars *sc;
};
// vectors of a level in one CTA: x, x2, b, r
template <int NF>
__host__ __device__ inline int tail_vec(int sh) { return 8 * NF << sh; }
// Image of one CTA: head, then per level inverse blocks, children (9 per row),
// parents (4 per row and a word of flags), columns and values of T trips; then the
// dense level's inverse rows and children.
struct TailHead {
    int bytes, dense, pad[2];
    int off[kMgMaxLevels], T[kMgMaxLevels];  // a level's part and its trips (3 or 7)
};
template <int NF, typename VT>
struct TailPart {
    typedef typename SellUnit<NF, VT>::U U;
    static const int NU = SellUnit<NF, VT>::NU;
    int rows, T;
    __host__ __device__ TailPart(int sh, int t) : rows(1 << sh), T(t) {}
    __host__ __device__ int child() const { return 8 * NF * NF * rows; }
    __host__ __device__ int parent() const { return child() + 9 * 4 * rows; }
    __host__ __device__ int cols() const { return parent() + 5 * 4 * rows; }
    __host__ __device__ int vals() const { return cols() + rows / 8 * T * 32 * 4; }
    __host__ __device__ int bytes() const { return vals() + rows / 8 * T * 32 * NU * (int)sizeof(U); }  // a multiple of 16: rows >= 8
};
__host__ __device__ inline int tail_dense_rows(int dn, int cluster) { return (dn + cluster - 1) / cluster; }
__host__ __device__ inline int tail_dense_bytes(int dn, int n_last, int cluster) {
    return (8 * dn * tail_dense_rows(dn, cluster) + 9 * 4 * n_last + 15) / 16 * 16;
}

__device__ __forceinline__ uint32_t cl_rank() { uint32_t r; asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
__device__ __forceinline__ uint32_t cl_size() { uint32_t r; asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(r)); return r; }
__device__ __forceinline__ void cl_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t cl_map(uint32_t a, uint32_t rank) {
    uint32_t d;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(rank));
    return d;
}
template <int NF>
__device__ __forceinline__ void cl_ld(uint32_t a, double v[NF]) {
    if constexpr (NF == 2 || NF == 4) {
#pragma unroll
        for (int q = 0; q < NF / 2; ++q)
            asm volatile("ld.shared::cluster.v2.f64 {%0, %1}, [%2];" : "=d"(v[2 * q]), "=d"(v[2 * q + 1]) : "r"(a + 16 * q) : "memory");
    } else {
#pragma unroll
        for (int g = 0; g < NF; ++g) asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v[g]) : "r"(a + 8 * g) : "memory");
    }
}
// CTA and byte offset of row r of a vector that starts at byte `off` in every CTA
template <int NF>
__device__ __forceinline__ uint32_t tail_ref(int off, int r, int sh) {
    return ((uint32_t)r >> sh) << 20 | (uint32_t)(off + 8 * NF * (r & ((1 << sh) - 1)));
}

// grid (cluster, levels + 1): block (rank, q) fills level l0 + q of that CTA's image
template <int NF, typename VT>
__global__ void __launch_bounds__(256) k_tail_image(const __grid_constant__ TailArgs a) {
    typedef TailPart<NF, VT> Part;
    typedef typename Part::U U;
    constexpr int NU = Part::NU;
    __shared__ TailHead head;
    const int rank = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned char *const img = a.img + (size_t)rank * a.img_stride;
    for (int l = a.l0 + warp; l < a.last; l += 8) {
        const TailLevel &v = a.lv[l];
        const int c0 = rank << (v.sh - 3);
        int m = 0;
        for (int i = lane; i < 1 << (v.sh - 3); i += 32)
            if (c0 + i < v.A.n_chunks) m = max(m, v.A.trips[c0 + i]);
        m = __reduce_max_sync(0xffffffffu, m);
        if (lane == 0) head.T[l] = m <= 3 ? 3 : kTailT;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        int o = (int)sizeof(TailHead);
        for (int l = a.l0; l < a.last; ++l) {
            head.off[l] = o;
            o += Part(a.lv[l].sh, head.T[l]).bytes();
        }
        head.dense = o;
        head.bytes = o + tail_dense_bytes(a.dn, a.n_last, a.cluster);
    }
    __syncthreads();
    auto child_ref = [&](const TailLevel &f, int fr) {  // the finer level's r, its fixed DOFs in the low bits
        return (fr >= 0 && in_range(fr, f.A.n_rows, GS_RESTRICT))
                   ? tail_ref<NF>(f.off + 3 * tail_vec<NF>(f.sh), fr, f.sh) | f.fixed[fr]
                   : kNoRow;
    };
    const int l = a.l0 + blockIdx.y;
    if (l == a.last) {
        const int dr = tail_dense_rows(a.dn, a.cluster), d0 = rank * dr, d1 = min(a.dn, d0 + dr);
        double *const inv = (double *)(img + head.dense);
        for (int q = threadIdx.x; q < (d1 - d0) * a.dn; q += blockDim.x) inv[q] = a.dInv[(size_t)d0 * a.dn + q];
        uint32_t *const ch = (uint32_t *)(inv + (size_t)dr * a.dn);
        for (int q = threadIdx.x; q < 9 * a.n_last; q += blockDim.x) ch[q] = child_ref(a.lv[a.last - 1], a.child_last[q]);
        for (int q = threadIdx.x; q < (int)sizeof(TailHead) / 4; q += blockDim.x) ((int *)img)[q] = ((const int *)&head)[q];
        return;
    }
    const TailLevel &v = a.lv[l];
    const Part P(v.sh, head.T[l]);
    unsigned char *const sp = img + head.off[l];
    const int c0 = rank << (v.sh - 3), r0 = rank << v.sh;
    for (int i = warp; i < P.rows / 8 && c0 + i < v.A.n_chunks; i += 8) {
        const int c = c0 + i, trips = v.A.trips[c];
        const int self = min(c * 8 + (lane >> 2), v.A.n_rows - 1);
        uint32_t *const cp = (uint32_t *)(sp + P.cols()) + i * P.T * 32 + lane;
        U *const vp = (U *)(sp + P.vals()) + (size_t)i * P.T * NU * 32 + lane;
        const int *sc = v.A.cols + (size_t)c * kTailT * 32 + lane;
        const U *sv = (const U *)v.A.vals + (size_t)c * kTailT * NU * 32 + lane;
        for (int t = 0; t < P.T; ++t) {  // trips past the chunk's own: its rows, zero blocks
            cp[t * 32] = tail_ref<NF>(v.off, t < trips ? sc[t * 32] : self, v.sh);
            for (int u = 0; u < NU; ++u) {
                U z;
                memset(&z, 0, sizeof(U));
                vp[(t * NU + u) * 32] = t < trips ? sv[(t * NU + u) * 32] : z;
            }
        }
    }
    const bool dense = l + 1 == a.last;
    const TailLevel &w = a.lv[l + 1];
    for (int q = threadIdx.x; q < P.rows && r0 + q < v.A.n_rows; q += blockDim.x) {
        const int r = r0 + q;
        for (int i = 0; i < NF * NF; ++i) ((double *)sp)[q * NF * NF + i] = v.Minv[(size_t)r * NF * NF + i];
        uint32_t *const pa = (uint32_t *)(sp + P.parent());
        int cnt = 0;
        for (int t = 0; t < 4; ++t) {
            const int R = v.parent[(size_t)t * v.A.n_rows + r];
            cnt += R != -2;
            uint32_t ad = kNoRow;
            if (R >= 0 && in_range(R, dense ? a.n_last : w.A.n_rows, GS_PROLONG))
                ad = dense ? (uint32_t)rank << 20 | (uint32_t)(a.off_last + 8 * (a.dn + R * NF))
                           : tail_ref<NF>(w.off + tail_vec<NF>(w.sh), R, w.sh);  // a level's result is in x2
            pa[t * P.rows + q] = ad;
        }
        pa[4 * P.rows + q] = (uint32_t)v.fixed[r] | (cnt == 1 ? 0u : (cnt == 2 ? 16u : 32u));
        if (l == a.l0) continue;
        uint32_t *const ch = (uint32_t *)(sp + P.child());
        for (int t = 0; t < 9; ++t) ch[t * P.rows + q] = child_ref(a.lv[l - 1], v.child[(size_t)t * v.A.n_rows + r]);
    }
}

template <int NF, typename VT>
__global__ void __launch_bounds__(kTailThreads, 1) k_sell_tail(const __grid_constant__ TailArgs a) {
    typedef TailPart<NF, VT> Part;
    typedef typename Part::U U;
    constexpr int NU = Part::NU;
    extern __shared__ __align__(16) unsigned char sm[];
    const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(sm);
    const uint32_t rank = cl_rank(), nct = cl_size();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, sub = lane & 3;
    unsigned char *const im = sm + a.off_img;
    {
        const unsigned char *src = a.img + (size_t)rank * a.img_stride;
        const int n = min(__ldg((const int *)src), a.img_stride);
        for (int q = threadIdx.x * 16; q < n; q += kTailThreads * 16)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(sbase + (uint32_t)(a.off_img + q)), "l"(src + q) : "memory");
    }
    pdl_wait();
    pdl_release();
    const StepState st = step_state(a.sc);
    if (!st.off) {
        const TailLevel &v = a.lv[a.l0];
        const int r0 = (int)(rank << v.sh), m = min(1 << v.sh, v.A.n_rows - r0) * NF;
        const double *bp = a.b.at(st.k);
        for (int q = threadIdx.x; q < m; q += kTailThreads) {
            ((double *)(sm + v.off))[q] = a.x1[(size_t)r0 * NF + q];
            ((double *)(sm + v.off + 2 * tail_vec<NF>(v.sh)))[q] = bp[(size_t)r0 * NF + q];
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    if (st.off) return;  // the same in every CTA: no barrier is left waiting
    cl_sync();
    const TailHead &head = *(const TailHead *)im;
    auto ref = [&](uint32_t e) { return cl_map(sbase + (e & 0xfffffu), e >> 20); };

    // what = 0: x_out = x_in + omega Minv (b - A x_in), 1: r = b - A x_in, over this CTA's rows
    auto sweep_t = [&](auto TT, int l, int xin, int xout, int what, double *gout) {
        constexpr int T = decltype(TT)::value;
        const TailLevel &v = a.lv[l];
        const Part P(v.sh, T);
        const unsigned char *const ip = im + head.off[l];
        unsigned char *const vp0 = sm + v.off;
        const int n1 = tail_vec<NF>(v.sh);
        const uint32_t dx = (uint32_t)(xin * n1);
        const int c0 = (int)(rank << (v.sh - 3));
        for (int i = warp; i < P.rows / 8 && c0 + i < v.A.n_chunks; i += kTailWarps) {
            const int lr = i * 8 + (lane >> 2), r = c0 * 8 + lr;
            const bool own = r < v.A.n_rows && sub == 0;
            const U *const vp = (const U *)(ip + P.vals()) + (size_t)i * T * NU * 32 + lane;
            const uint32_t *const cp = (const uint32_t *)(ip + P.cols()) + i * T * 32 + lane;
            double acc[NF], xv[T][NF];
#pragma unroll
            for (int t = 0; t < T; ++t) cl_ld<NF>(ref(cp[t * 32] + dx), xv[t]);
#pragma unroll
            for (int f = 0; f < NF; ++f) acc[f] = 0.0;
#pragma unroll
            for (int t = 0; t < T; ++t) {
                U val[NU];
#pragma unroll
                for (int u = 0; u < NU; ++u) val[u] = vp[(t * NU + u) * 32];
                SellRow<NF, VT, 4>::mad(val, xv[t], acc);
            }
#pragma unroll
            for (int f = 0; f < NF; ++f)
#pragma unroll
                for (int o = 2; o > 0; o >>= 1) acc[f] += __shfl_down_sync(0xffffffffu, acc[f], o, 4);
            if (!own) continue;
            double t[NF], xi[NF], z[NF], M[NF * NF];
            load_rw<NF>((const double *)(vp0 + 2 * n1) + lr * NF, t);
#pragma unroll
            for (int f = 0; f < NF; ++f) t[f] -= acc[f];
            if (what == 1) {
                store_rw<NF>((double *)(vp0 + 3 * n1) + lr * NF, t);
                continue;
            }
            load_rw<NF>((const double *)(vp0 + dx) + lr * NF, xi);
#pragma unroll
            for (int q = 0; q < NF * NF; ++q) M[q] = ((const double *)ip)[lr * NF * NF + q];
            minv_mul<NF>(M, t, z);
#pragma unroll
            for (int f = 0; f < NF; ++f) z[f] = xi[f] + a.omega * z[f];
            if (gout) store_rw<NF>(gout + (size_t)r * NF, z);
            else store_rw<NF>((double *)(vp0 + xout * n1) + lr * NF, z);
        }
    };
    auto sweep = [&](int l, int xin, int xout, int what, double *gout) {
        if (head.T[l] == 3) sweep_t(std::integral_constant<int, 3>(), l, xin, xout, what, gout);
        else sweep_t(std::integral_constant<int, kTailT>(), l, xin, xout, what, gout);
    };
    auto restricted = [&](const uint32_t *ch, int stride, double acc[NF]) {  // P^T r of one coarse row
        constexpr uint32_t mask = (1u << NF) - 1u;  // fixed DOFs, below the row's alignment
        uint32_t e[9];
        double t[9][NF];
#pragma unroll
        for (int q = 0; q < 9; ++q) e[q] = ch[q * stride];
#pragma unroll
        for (int q = 0; q < 9; ++q) cl_ld<NF>(e[q] == kNoRow ? sbase : ref(e[q] & ~mask), t[q]);
#pragma unroll
        for (int f = 0; f < NF; ++f) acc[f] = 0.0;
#pragma unroll
        for (int q = 0; q < 9; ++q) {
            const double wt = (q % 3 == 1 ? 1.0 : 0.5) * (q / 3 == 1 ? 1.0 : 0.5);
#pragma unroll
            for (int f = 0; f < NF; ++f)
                if (e[q] != kNoRow && !((e[q] >> f) & 1u)) acc[f] += wt * t[q][f];
        }
    };

    double *const db = (double *)(sm + a.off_last);  // dense level: b, then x
    const double *const dinv = (const double *)(im + head.dense);
    const int dr = tail_dense_rows(a.dn, (int)nct), d0 = (int)rank * dr, d1 = min(a.dn, d0 + dr);
    for (int l = a.l0; l < a.last; ++l) {
        const TailLevel &v = a.lv[l];
        int x = 0;
        for (int it = 1; it < v.sweeps; ++it) {
            sweep(l, x, 1 - x, 0, nullptr);
            x = 1 - x;
            cl_sync();
        }
        sweep(l, x, 0, 1, nullptr);
        cl_sync();
        if (l + 1 == a.last) {  // the dense level's whole right-hand side in every CTA
            const uint32_t *const ch = (const uint32_t *)(dinv + (size_t)dr * a.dn);
            for (int R = threadIdx.x; R < a.n_last; R += kTailThreads) {
                double acc[NF];
                restricted(ch + R, a.n_last, acc);
#pragma unroll
                for (int f = 0; f < NF; ++f) db[R * NF + f] = acc[f];
            }
            __syncthreads();
            break;
        }
        // b_c = P^T r, and the coarse level's zero-start sweep
        const TailLevel &w = a.lv[l + 1];
        const Part P(w.sh, head.T[l + 1]);
        const unsigned char *const ip = im + head.off[l + 1];
        const int n1 = tail_vec<NF>(w.sh), m = min(P.rows, w.A.n_rows - (int)(rank << w.sh));
        for (int q = threadIdx.x; q < m; q += kTailThreads) {
            double acc[NF], z[NF], M[NF * NF];
            restricted((const uint32_t *)(ip + P.child()) + q, P.rows, acc);
#pragma unroll
            for (int i = 0; i < NF * NF; ++i) M[i] = ((const double *)ip)[q * NF * NF + i];
            store_rw<NF>((double *)(sm + w.off + 2 * n1) + q * NF, acc);
            minv_mul<NF>(M, acc, z);
#pragma unroll
            for (int f = 0; f < NF; ++f) z[f] *= a.omega;
            store_rw<NF>((double *)(sm + w.off) + q * NF, z);
        }
        cl_sync();
    }
    // dense level: a warp takes a row and leaves its result in every CTA
    for (int i = d0 + warp; i < d1; i += kTailWarps) {
        const double *inv = dinv + (size_t)(i - d0) * a.dn;
        double s = 0.0;
#pragma unroll 5
        for (int j = lane; j < a.dn; j += 32) s += inv[j] * db[j];
        for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
        s = __shfl_sync(0xffffffffu, s, 0);
        if ((uint32_t)lane < nct) {
            const uint32_t d = cl_map(sbase + (uint32_t)a.off_last + 8u * (uint32_t)(a.dn + i), (uint32_t)lane);
            asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(d), "d"(s) : "memory");
        }
    }
    cl_sync();
    for (int l = a.last - 1; l >= a.l0; --l) {
        const TailLevel &v = a.lv[l];
        const Part P(v.sh, head.T[l]);
        const int m = min(P.rows, v.A.n_rows - (int)(rank << v.sh));
        int x = (v.sweeps - 1) & 1;
        const uint32_t *const pa = (const uint32_t *)(im + head.off[l] + P.parent());
        for (int q = threadIdx.x; q < m; q += kTailThreads) {
            const uint32_t info = pa[4 * P.rows + q];
            const double wt = info < 16u ? 1.0 : (info < 32u ? 0.5 : 0.25);
            uint32_t e[4];
            double acc[NF], xv[NF], c[4][NF];
            double *xp = (double *)(sm + v.off + x * tail_vec<NF>(v.sh)) + q * NF;
#pragma unroll
            for (int t = 0; t < 4; ++t) e[t] = pa[t * P.rows + q];
#pragma unroll
            for (int t = 0; t < 4; ++t) cl_ld<NF>(e[t] == kNoRow ? sbase : ref(e[t]), c[t]);
            load_rw<NF>(xp, xv);
#pragma unroll
            for (int f = 0; f < NF; ++f) acc[f] = 0.0;
#pragma unroll
            for (int t = 0; t < 4; ++t)
#pragma unroll
                for (int f = 0; f < NF; ++f)
                    if (e[t] != kNoRow) acc[f] += wt * c[t][f];
#pragma unroll
            for (int f = 0; f < NF; ++f)
                if (!((info >> f) & 1u)) xv[f] += acc[f];
            store_rw<NF>(xp, xv);
        }
        cl_sync();
        for (int it = 0; it < v.sweeps; ++it) {
            const bool out = l == a.l0 && it + 1 == v.sweeps;
            sweep(l, x, 1 - x, 0, out ? a.out.at(st.k) : nullptr);
            x = 1 - x;
            cl_sync();  // also the last one: no CTA leaves while its rows are read
        }
    }
}

}  // namespace
}  // namespace gw
