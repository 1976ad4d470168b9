// Reference engine: the reference PDHG (CPUFirstOrderSolver::solve,
// src/first_order_solver.cpp:103-279) on the GPU, iterate for iterate.
//
// Compiled with --fmad=false and with every sum taken in the reference's order
// (rows ascending inside each column for A^T y, columns ascending inside each
// row for A x), so x^k, y^k, the convergence checks, the iteration count and
// the status are bit-identical to the compiled reference.
//
// Layout: one thread per column (primal step over A^T) and one thread per row
// (dual step over A), each over a copy of the matrix in slices of 32 rows, entry q
// of the slice's lanes side by side (Sell below): a warp reads 32 consecutive values
// and indices per step while every lane still sums its own row in order.
// An LP small enough for one cluster of CTAs runs whole in one launch
// (k_ref_cluster): its vectors live in shared memory, and the convergence checks are
// decided on the device.  A larger one takes two kernels per iteration, captured in a CUDA
// graph of kGraphIters iterations; the host reads back four doubles per check.
#include <cub/cub.cuh>

#include <cmath>
#include <cstring>
#include <type_traits>

#include "b2p_internal.cuh"
#include "cluster.cuh"
#include "pdl.cuh"

namespace b2p {

namespace {

// bharatopt::clamp (include/bharatopt/config.hpp:25-28): NaN passes through.
__device__ __forceinline__ double ref_clamp(double v, double lo, double hi) {
    return (v < lo) ? lo : ((hi < v) ? hi : v);
}

constexpr int kBatch = 16;       // entries in flight per row: the two-kernel form (few warps per SM)
constexpr int kBatchSmall = 8;   // ... and the cluster form
constexpr int kGraphIters = 20;  // plain iterations per captured graph
// LPs of at most this many entries (and whose vectors fit shared memory) run on one cluster
constexpr int64_t kClusterNnz = 49152;
// ... and of at most this many on one CTA: 1.50 us against 1.64 on eight at 2,500 entries, 2.6 against
// 1.8 at 5,000
constexpr int64_t kOneCtaNnz = 3072;
// ... and their long rows (of at least kLongRow entries each)
constexpr int kLongRow = 128;
constexpr int kMostLong = kClusterNnz / kLongRow;

// Slots of the per-check reduction block.
enum { R_DPRIMAL = 0, R_DDUAL, R_VIOL_X, R_VIOL_AVG, R_BOUND, R_COUNT };

struct RefState {
    double *tau, *sigma, *x, *y, *x_hat, *x_sum, *x_avg;
    unsigned long long* red;  // R_COUNT slots (bit patterns of non-negative doubles)
    long long* iter;          // device iteration counter (== avg_count)
};

// One orientation of the matrix by slices of 32 rows in their natural order: entry q of
// row 32 s + l at off[s] + 32 q + l, slices padded to their longest row and to a multiple
// of kPad entries.  A padding entry has value 0 and the index one past the gathered vector, where
// a 0 is stored: it adds +0 to a sum that started from +0, which leaves every sum as it was
// (such a sum is never -0), whatever the iterates hold.  off null: the CSR arrays (slices whose rows
// differ too much in length).  Rows of more than `limit` entries are not in the slices but in `longs`:
// a whole warp sums each over the CSR arrays (long_row_sum).
struct Sell {
    const int64_t* off;
    const int32_t* ptr;  // CSR row pointers
    const int32_t* idx;
    const double* val;
    const int32_t* csr_idx;
    const double* csr_val;
    const int32_t* longs;
    int nlong, limit;
    __device__ __forceinline__ bool is_long(int i) const { return ptr[i + 1] - ptr[i] > limit; }
};
constexpr int kPad = 2;
// Entries from which a row is long, kLongRow at least: a lane takes 64 ns an entry there (a thread on the CSR
// arrays 50), a warp 7 to 10; rows of a usual length, which 32 lanes sum side by side, stay in the slices.
int long_limit(int64_t nnz, int rows) { return (int)std::max<int64_t>(kLongRow, 8 * nnz / rows); }

// Sum over row i in entry order, products and sums rounded separately.  The products of a
// batch are independent; only the additions are a chain.
template <int B, bool SLICED>
__device__ __forceinline__ double row_sum(const Sell& S, int i, const double* g) {
    double w = 0.0;
    if constexpr (!SLICED) {
        for (int k = S.ptr[i]; k < S.ptr[i + 1]; ++k) w += S.val[k] * g[S.idx[k]];
        return w;
    }
    const int64_t p0 = __ldg(S.off + (i >> 5));
    int len = (int)((__ldg(S.off + (i >> 5) + 1) - p0) >> 5);
    const double* v = S.val + p0 + (i & 31);
    const int32_t* ix = S.idx + p0 + (i & 31);
    auto batch = [&](auto size) {
        constexpr int N = decltype(size)::value;
        double vv[N], gg[N];
        int ii[N];
#pragma unroll
        for (int u = 0; u < N; ++u) {
            vv[u] = __ldg(v + u * 32);
            ii[u] = __ldg(ix + u * 32);
        }
#pragma unroll
        for (int u = 0; u < N; ++u) gg[u] = g[ii[u]];
#pragma unroll
        for (int u = 0; u < N; ++u) w += vv[u] * gg[u];
        v += N * 32;
        ix += N * 32;
        len -= N;
    };
#pragma unroll 1
    while (len >= B) batch(std::integral_constant<int, B>());
    if constexpr (B > 8)
        if (len >= 8) batch(std::integral_constant<int, 8>());
    if (len >= 4) batch(std::integral_constant<int, 4>());
    if (len >= kPad) batch(std::integral_constant<int, kPad>());
    return w;
}

// Sum over row i in entry order by a whole warp: the lanes load, gather and multiply 128 entries side by
// side, the next 128 on their way, and every lane adds the products up in order.
__device__ __noinline__ double long_row_sum(const double* __restrict__ val, const int32_t* __restrict__ idx, int e0, int e1,
                                            const double* g) {
    constexpr int U = 4;
    const int lane = threadIdx.x & 31;
    double w = 0.0, v[U];
    int c[U];
    auto load = [&](int64_t e) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const bool h = e + 32 * u + lane < e1;
            v[u] = h ? __ldg(val + e + 32 * u + lane) : 0.0;
            c[u] = h ? __ldg(idx + e + 32 * u + lane) : -1;
        }
    };
    load(e0);
    for (int64_t e = e0; e < e1; e += 32 * U) {
        double p[U];
#pragma unroll
        for (int u = 0; u < U; ++u) p[u] = c[u] >= 0 ? v[u] * g[c[u]] : 0.0;
        load(e + 32 * U);
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int n = (int)min((int64_t)32, e1 - (e + 32 * u));
            if (n == 32) {
#pragma unroll
                for (int l = 0; l < 32; ++l) w += __shfl_sync(0xffffffffu, p[u], l);
            } else {
                for (int l = 0; l < n; ++l) w += __shfl_sync(0xffffffffu, p[u], l);
            }
        }
    }
    return w;
}

// update(i, sum) of every long row, by one lane; all warps of the grid take part
template <typename F>
__device__ __forceinline__ void for_long_rows(const Sell& S, const double* g, F update) {
    const int warps = (gridDim.x * blockDim.x) >> 5;
    for (int q = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; q < S.nlong; q += warps) {
        const int i = S.longs[q];
        const double w = long_row_sum(S.csr_val, S.csr_idx, S.ptr[i], S.ptr[i + 1], g);
        if ((threadIdx.x & 31) == 0) update(i, w);
    }
}

// padded length of every slice, x 32 lanes (the offsets are their sums), without the long rows; those
// into `longs`, their number into off[number of slices + 1] (zeroed by the caller)
__global__ void k_ref_slice_len(int rows, int limit, const int32_t* __restrict__ ptr, int64_t* __restrict__ off,
                                int32_t* __restrict__ longs) {
    const int nsl = (rows + 31) >> 5;
    for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < nsl; s += gridDim.x * blockDim.x) {
        int mx = 0;
        for (int i = s << 5; i < min(rows, (s + 1) << 5); ++i) {
            const int len = ptr[i + 1] - ptr[i];
            if (len <= limit) mx = max(mx, len);
            else longs[atomicAdd(reinterpret_cast<unsigned long long*>(off + nsl + 1), 1ull)] = i;
        }
        off[s + 1] = 32ll * ((mx + kPad - 1) / kPad * kPad);
        if (s == 0) off[0] = 0;
    }
}

// every lane slot of every slice; `other`: the length of the gathered vector
__global__ void k_ref_slice_fill(int rows, int limit, int other, const int32_t* __restrict__ ptr, const int32_t* __restrict__ idx,
                                 const double* __restrict__ val, const int64_t* __restrict__ off,
                                 int32_t* __restrict__ oidx, double* __restrict__ oval) {
    const int padded = (rows + 31) & ~31;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < padded; i += gridDim.x * blockDim.x) {
        const int64_t base = off[i >> 5] + (i & 31);
        const int slen = (int)((off[(i >> 5) + 1] - off[i >> 5]) >> 5);
        const int p0 = i < rows ? ptr[i] : 0, all = i < rows ? ptr[i + 1] - p0 : 0, len = all <= limit ? all : 0;
        for (int q = 0; q < slen; ++q) {
            oidx[base + 32ll * q] = q < len ? idx[p0 + q] : other;
            oval[base + 32ll * q] = q < len ? val[p0 + q] : 0.0;
        }
    }
}

// first_order_solver.cpp:103-128
__global__ void k_ref_steps(int m, int n, const int32_t* __restrict__ rowptr, const double* __restrict__ vals,
                            const int32_t* __restrict__ t_rowptr, const double* __restrict__ t_vals, int adaptive,
                            double pstep, double dstep, double* __restrict__ tau, double* __restrict__ sigma) {
    int tid = blockIdx.x * blockDim.x + threadIdx.x, stride = gridDim.x * blockDim.x;
    for (int j = tid; j < n; j += stride) {
        double s = 0.0;
        for (int k = t_rowptr[j]; k < t_rowptr[j + 1]; ++k) s += fabs(t_vals[k]);
        tau[j] = adaptive ? ((s > 1e-12) ? (0.95 / s) : 1.0) : pstep;
    }
    for (int i = tid; i < m; i += stride) {
        double s = 0.0;
        for (int k = rowptr[i]; k < rowptr[i + 1]; ++k) s += fabs(vals[k]);
        sigma[i] = adaptive ? ((s > 1e-12) ? (0.95 / s) : 1.0) : dstep;
    }
}

// first_order_solver.cpp:130-151
__global__ void k_ref_init(int m, int n, const double* __restrict__ lb, const double* __restrict__ ub,
                           double* __restrict__ x, double* __restrict__ y, double* __restrict__ x_sum,
                           double* __restrict__ x_hat, double* __restrict__ x_avg, long long* iter, unsigned long long* red) {
    int tid = blockIdx.x * blockDim.x + threadIdx.x, stride = gridDim.x * blockDim.x;
    const double inf = INFINITY;
    for (int j = tid; j < n; j += stride) {
        double target = 0.0;
        if (lb[j] > -inf && ub[j] < inf) target = 0.5 * (lb[j] + ub[j]);
        else if (lb[j] > -inf) target = lb[j];
        else if (ub[j] < inf) target = ub[j];
        x[j] = ref_clamp(target, lb[j], ub[j]);
        x_sum[j] = 0.0;
    }
    for (int i = tid; i < m; i += stride) y[i] = 0.0;
    if (tid == 0) {
        y[m] = 0.0;  // where the padding of the sliced copies points
        x[n] = x_hat[n] = x_avg[n] = 0.0;
        *iter = 0;
        for (int r = 0; r < R_COUNT; ++r) red[r] = 0ull;
    }
}

// Steps A-C (first_order_solver.cpp:163-180): A^T y, projected primal step,
// ergodic sum, extrapolation.  x_prev == x at entry, so x_hat = 2 x_new - x.
template <bool CHECK, bool SLICED, bool LONG>
__global__ void __launch_bounds__(128) k_ref_primal(int n, Sell At, const double* __restrict__ c,
                                                    const double* __restrict__ lb, const double* __restrict__ ub,
                                                    RefState st) {
    pdl_wait();
    pdl_trigger();
    auto update = [&](int j, double w) {
        double xj = st.x[j];
        double grad = c[j] + w;
        double next_x = xj - st.tau[j] * grad;
        double new_x = ref_clamp(next_x, lb[j], ub[j]);
        if (CHECK) atomic_max_nonneg(&st.red[R_DPRIMAL], fabs(new_x - xj));
        st.x_sum[j] += new_x;
        st.x_hat[j] = 2.0 * new_x - xj;
        st.x[j] = new_x;
    };
    if (LONG) for_long_rows(At, st.y, update);
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x)
        if (!LONG || !At.is_long(j)) update(j, row_sum<kBatch, SLICED>(At, j, st.y));
}

// Steps D-E (first_order_solver.cpp:183-192): A x_hat, dual step, sign projection.
template <bool CHECK, bool SLICED, bool LONG>
__global__ void __launch_bounds__(128) k_ref_dual(int m, Sell A, const double* __restrict__ b,
                                                  const uint8_t* __restrict__ is_eq, RefState st) {
    int tid = blockIdx.x * blockDim.x + threadIdx.x;
    pdl_wait();
    pdl_trigger();
    auto update = [&](int i, double v) {
        double yi = st.y[i];
        double next_y = yi + st.sigma[i] * (v - b[i]);
        // std::max(0.0, next_y) == (0.0 < next_y) ? next_y : 0.0
        double new_y = (!is_eq[i]) ? ((0.0 < next_y) ? next_y : 0.0) : next_y;
        if (CHECK) atomic_max_nonneg(&st.red[R_DDUAL], fabs(new_y - yi));
        st.y[i] = new_y;
    };
    if (LONG) for_long_rows(A, st.x_hat, update);
    for (int i = tid; i < m; i += gridDim.x * blockDim.x)
        if (!LONG || !A.is_long(i)) update(i, row_sum<kBatch, SLICED>(A, i, st.x_hat));
    if (tid == 0) *st.iter += 1;
}

// Step F, column part (first_order_solver.cpp:208-218): bound violation of x and the
// clamped ergodic average x_avg = clamp(x_sum / avg_count).
__global__ void k_ref_check_cols(int n, const double* __restrict__ lb, const double* __restrict__ ub, RefState st) {
    long long cnt = *st.iter;
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
        double xj = st.x[j];
        if (xj < lb[j] - 1e-12) atomic_max_nonneg(&st.red[R_BOUND], lb[j] - xj);
        if (xj > ub[j] + 1e-12) atomic_max_nonneg(&st.red[R_BOUND], xj - ub[j]);
        st.x_avg[j] = (cnt > 0) ? ref_clamp(st.x_sum[j] / (double)cnt, lb[j], ub[j]) : xj;
    }
}

// Step F, row part (first_order_solver.cpp:199-206, 219-225): max row violation of x and x_avg.
template <bool SLICED>
__global__ void __launch_bounds__(128) k_ref_check_rows(int m, Sell A, const double* __restrict__ b,
                                                        const uint8_t* __restrict__ is_eq, RefState st) {
    auto violation = [&](int i, int slot, double v) {
        const double d = v - b[i];
        atomic_max_nonneg(&st.red[slot], (!is_eq[i]) ? ((0.0 < d) ? d : 0.0) : fabs(d));
    };
    for_long_rows(A, st.x, [&](int i, double v) { violation(i, R_VIOL_X, v); });
    for_long_rows(A, st.x_avg, [&](int i, double v) { violation(i, R_VIOL_AVG, v); });
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < m; i += gridDim.x * blockDim.x) {
        if (A.nlong > 0 && A.is_long(i)) continue;
        violation(i, R_VIOL_X, row_sum<kBatch, SLICED>(A, i, st.x));
        violation(i, R_VIOL_AVG, row_sum<kBatch, SLICED>(A, i, st.x_avg));
    }
}

__global__ void k_ref_clear(unsigned long long* red) {
    if (threadIdx.x < R_COUNT) red[threadIdx.x] = 0ull;
}

double bits_to_double(unsigned long long b) {
    double d;
    std::memcpy(&d, &b, sizeof(d));
    return d;
}

// The whole run of an LP whose vectors fit shared memory, on one cluster: each CTA owns a
// range of column and row slices with their vectors, copies of y and x_hat (which at a check
// hold x and then x_avg) are in every CTA, and the owned part of the matrix is in shared
// memory too where it fits (MAT_SMEM, 16-bit indices).  The check of every interval (steps F,
// :195-246) is decided here by the host loop's own comparisons.  Runs until convergence,
// failure, or iteration `stop`.
//
// Bound: latency -- the additions of a row (8.6 cycles each), shared-memory gathers, and the
// posts to the peers with the wait for theirs.  us per iteration: two kernels in a graph -> this
// with cluster barriers -> now: 60 x 200 7.9 -> 0.95 (one CTA), 300 x 1,000 9.0 -> 2.7 -> 1.8,
// 1,000 x 3,000 10.0 -> 3.9 -> 2.6, 2,000 x 6,000 10.1 -> 5.2 -> 4.3.  From 3,000 x 9,000 on
// (54,000 entries) the posts to eight copies cost more than kernel boundaries: 8.4 here, 7.2
// with two kernels (12.2 before, over CSR and without their overlap), so the line is drawn at
// 49,152 entries.
struct RefOutcome {
    long long iter;
    int converged, failed, wait_failed;
    double viol_x, viol_avg, bound, dprimal, ddual;
};

// Shared memory of one CTA (bytes from the start of the dynamic array), the same in all.
struct RefLayout {
    int cols, rows;      // most owned columns / rows of any CTA
    int y, xh, x, xsum, tau, c, lb, ub, sigma, b, eq, cval, rval, cidx, ridx, coff, roff, cmask, rmask, total;
};

// entries in shared memory by slices: entry q of lane l of the CTA's slice s at off + 32 q + l
template <bool MAT_SMEM>
struct SliceView {
    const double* val;
    const void* idx;  // uint16_t in shared memory, int32_t in global memory
    __device__ __forceinline__ double sum(int64_t p0, int len, int lane, const double* g) const {
        double w = 0.0;
        const double* v = val + p0 + lane;
        const uint16_t* i16 = (const uint16_t*)idx + p0 + lane;
        const int32_t* i32 = (const int32_t*)idx + p0 + lane;
        auto batch = [&](auto size) {
            constexpr int N = decltype(size)::value;
            double vv[N], gg[N];
            int ii[N];
#pragma unroll
            for (int u = 0; u < N; ++u) {
                vv[u] = MAT_SMEM ? v[u * 32] : __ldg(v + u * 32);
                ii[u] = MAT_SMEM ? (int)i16[u * 32] : __ldg(i32 + u * 32);
            }
#pragma unroll
            for (int u = 0; u < N; ++u) gg[u] = g[ii[u]];
#pragma unroll
            for (int u = 0; u < N; ++u) w += vv[u] * gg[u];
            v += N * 32;
            i16 += N * 32;
            i32 += N * 32;
            len -= N;
        };
#pragma unroll 1
        while (len >= kBatchSmall) batch(std::integral_constant<int, kBatchSmall>());
        if (len >= 4) batch(std::integral_constant<int, 4>());
        if (len >= kPad) batch(std::integral_constant<int, kPad>());
        return w;
    }
};

// LONG: some rows or columns are long; the warps of the CTA that owns them take them before its slices.
template <int NC, bool MAT_SMEM, bool LONG>
__global__ void __launch_bounds__(kClusterThreads, 1)
k_ref_cluster(int m, int n, Sell A, Sell At, const double* __restrict__ c, const double* __restrict__ lb,
              const double* __restrict__ ub, const double* __restrict__ b, const uint8_t* __restrict__ is_eq, RefState st,
              RefLayout lay, long long stop, long long max_it, long long cf, double tol, RefOutcome* out) {
    namespace cg = cooperative_groups;
    cg::cluster_group cl = cg::this_cluster();
    extern __shared__ __align__(16) unsigned char sh[];
    __shared__ unsigned long long red[R_COUNT];
    __shared__ uint64_t bar[2];  // arrivals of x_hat, of y
    __shared__ double token;     // where CTAs without columns post
    __shared__ int longs[2][LONG ? kMostLong : 1], nlong[2];  // owned long columns, rows
    auto at = [&](int off) { return reinterpret_cast<double*>(sh + off); };
    double *ys = at(lay.y), *xh = at(lay.xh), *xs = at(lay.x), *sums = at(lay.xsum), *ts = at(lay.tau), *cs = at(lay.c);
    double *ls = at(lay.lb), *us = at(lay.ub), *ss = at(lay.sigma), *bs = at(lay.b);
    uint8_t* eq = sh + lay.eq;
    const int rank = (int)cl.block_rank(), tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5;
    const int ncs = (n + 31) >> 5, nrs = (m + 31) >> 5;
    const int c0 = cluster_slice<NC>(ncs, rank), c1 = cluster_slice<NC>(ncs, rank + 1);
    const int r0 = cluster_slice<NC>(nrs, rank), r1 = cluster_slice<NC>(nrs, rank + 1);
    const ClusterPeers<NC> peers(sh);
    const ClusterPost<double, NC> xv(peers, xh, bar), yv(peers, ys, bar + 1), tv(peers, &token, bar);
    // a CTA without columns posts a token, so that no iteration passes it by
    int empty = 0;
    for (int r = 0; r < NC; ++r) empty += cluster_slice<NC>(ncs, r) == cluster_slice<NC>(ncs, r + 1);
    const uint32_t x_bytes = 8u * (uint32_t)(n + empty), y_bytes = 8u * (uint32_t)m;
    if (NC > 1 && tid == 0) {
        tx_init(bar);
        tx_init(bar + 1);
        tx_expect(bar, x_bytes);
        tx_expect(bar + 1, y_bytes);
    }
    // the first entries of the owned slices, from the CTA's first
    int *co = reinterpret_cast<int*>(sh + lay.coff), *ro = reinterpret_cast<int*>(sh + lay.roff);
    for (int q = tid; q <= c1 - c0; q += blockDim.x) co[q] = (int)(At.off[c0 + q] - At.off[c0]);
    for (int q = tid; q <= r1 - r0; q += blockDim.x) ro[q] = (int)(A.off[r0 + q] - A.off[r0]);
    // owned long columns and rows, and per slice the lanes that have one
    unsigned *cmask = reinterpret_cast<unsigned*>(sh + lay.cmask), *rmask = reinterpret_cast<unsigned*>(sh + lay.rmask);
    if (LONG) {
        for (int q = tid; q < c1 - c0; q += blockDim.x) cmask[q] = 0;
        for (int q = tid; q < r1 - r0; q += blockDim.x) rmask[q] = 0;
        if (tid < 2) nlong[tid] = 0;
        __syncthreads();
        auto own = [&](const Sell& S, int s0, int s1, int side, unsigned* mask) {
            for (int q = tid; q < S.nlong; q += blockDim.x) {
                const int i = S.longs[q];
                if ((i >> 5) < s0 || (i >> 5) >= s1) continue;
                longs[side][atomicAdd(&nlong[side], 1)] = i;
                atomicOr(&mask[(i >> 5) - s0], 1u << (i & 31));
            }
        };
        own(At, c0, c1, 0, cmask);
        own(A, r0, r1, 1, rmask);
    }
    // full copies, owned vectors, owned part of the matrix
    for (int i = tid; i <= m; i += blockDim.x) ys[i] = st.y[i];
    if (tid == 0) xh[n] = 0.0;
    for (int j = (c0 << 5) + tid; j < min(n, c1 << 5); j += blockDim.x) {
        const int o = j - (c0 << 5);
        xs[o] = st.x[j];
        sums[o] = st.x_sum[j];
        ts[o] = st.tau[j];
        cs[o] = c[j];
        ls[o] = lb[j];
        us[o] = ub[j];
    }
    for (int i = (r0 << 5) + tid; i < min(m, r1 << 5); i += blockDim.x) {
        const int o = i - (r0 << 5);
        ss[o] = st.sigma[i];
        bs[o] = b[i];
        eq[o] = is_eq[i];
    }
    const int64_t cb = At.off[c0], rb = A.off[r0];
    SliceView<MAT_SMEM> cv{At.val, At.idx}, rv{A.val, A.idx};
    if (MAT_SMEM) {
        double *vc = at(lay.cval), *vr = at(lay.rval);
        uint16_t *ic = (uint16_t*)(sh + lay.cidx), *ir = (uint16_t*)(sh + lay.ridx);
        for (int e = tid; e < (int)(At.off[c1] - cb); e += blockDim.x) {
            vc[e] = At.val[cb + e];
            ic[e] = (uint16_t)At.idx[cb + e];
        }
        for (int e = tid; e < (int)(A.off[r1] - rb); e += blockDim.x) {
            vr[e] = A.val[rb + e];
            ir[e] = (uint16_t)A.idx[rb + e];
        }
        cv = SliceView<MAT_SMEM>{vc - cb, ic - cb};
        rv = SliceView<MAT_SMEM>{vr - rb, ir - rb};
    }
    cluster_phase<NC>(cl);
    // End of a phase: this CTA's copy is complete.  A thread that gave up once waits no more and
    // runs on, so that barriers still meet.
    bool ok = true;
    uint32_t parity = 0;
    auto phase_end = [&](int v, uint32_t bytes) {
        if constexpr (NC == 1) {
            __syncthreads();
        } else {
            if (ok) ok = tx_wait(bar + v, parity);
            if (tid == 0) tx_expect(bar + v, bytes);
            if (v == 1) __syncthreads();
        }
    };
    long long it = out->iter;
    bool finished = out->converged || out->failed;
    // update(i, sum) for the owned long rows of one orientation
    auto long_rows = [&](const Sell& S, int side, const double* g, auto update) {
        for (int q = warp; LONG && q < nlong[side]; q += nw) {
            const int i = longs[side][q];
            const double w = long_row_sum(S.csr_val, S.csr_idx, S.ptr[i], S.ptr[i + 1], g);
            if (lane == 0) update(i, w);
        }
    };
    auto in_slices = [&](const unsigned* mask, int sl) { return !LONG || !(mask[sl] >> lane & 1u); };
    // max row violation of the vector whose copies are in xh, into slot
    auto violation = [&](int slot) {
        auto row = [&](int i, double v) {
            const int o = i - (r0 << 5);
            const double d = v - bs[o];
            atomic_max_nonneg(&red[slot], (!eq[o]) ? ((0.0 < d) ? d : 0.0) : fabs(d));
        };
        long_rows(A, 1, xh, row);
        for (int sl = r0 + warp; sl < r1; sl += nw) {
            const int p0 = ro[sl - r0];
            const double v = rv.sum(rb + p0, (ro[sl - r0 + 1] - p0) >> 5, lane, xh);
            const int i = (sl << 5) + lane;
            if (i < m && in_slices(rmask, sl - r0)) row(i, v);
        }
    };
    while (it < stop && !finished) {
        const long long check_at = min(it - it % cf + cf, max_it);  // the interval ends on a check
        for (; it < check_at; ++it) {
            const bool check = it + 1 == check_at;
            if (check) {
                if (tid < R_COUNT) red[tid] = 0ull;
                __syncthreads();
            }
            auto column = [&](int j, double w) {
                const int o = j - (c0 << 5);
                double xj = xs[o];
                double grad = cs[o] + w;
                double next_x = xj - ts[o] * grad;
                double new_x = ref_clamp(next_x, ls[o], us[o]);
                if (check) atomic_max_nonneg(&red[R_DPRIMAL], fabs(new_x - xj));
                sums[o] += new_x;
                xv.store(peers, j, 2.0 * new_x - xj);
                xs[o] = new_x;
            };
            long_rows(At, 0, ys, column);
            for (int sl = c0 + warp; sl < c1; sl += nw) {
                const int p0 = co[sl - c0];
                const double w = cv.sum(cb + p0, (co[sl - c0 + 1] - p0) >> 5, lane, ys);
                const int j = (sl << 5) + lane;
                if (j < n && in_slices(cmask, sl - c0)) column(j, w);
            }
            if (NC > 1 && c0 == c1 && tid == 0) tv.store(peers, 0, 0.0);
            phase_end(0, x_bytes);
            auto row = [&](int i, double v) {
                const int o = i - (r0 << 5);
                double yi = ys[i];
                double next_y = yi + ss[o] * (v - bs[o]);
                double new_y = (!eq[o]) ? ((0.0 < next_y) ? next_y : 0.0) : next_y;
                if (check) atomic_max_nonneg(&red[R_DDUAL], fabs(new_y - yi));
                yv.store(peers, i, new_y);
            };
            long_rows(A, 1, xh, row);
            for (int sl = r0 + warp; sl < r1; sl += nw) {
                const int p0 = ro[sl - r0];
                const double v = rv.sum(rb + p0, (ro[sl - r0 + 1] - p0) >> 5, lane, xh);
                const int i = (sl << 5) + lane;
                if (i < m && in_slices(rmask, sl - r0)) row(i, v);
            }
            phase_end(1, y_bytes);
            parity ^= 1;
        }
        const ClusterVec<double, NC> xc(cl, xh);
        for (int j = (c0 << 5) + tid; j < min(n, c1 << 5); j += blockDim.x) {
            const int o = j - (c0 << 5);
            const double xj = xs[o];
            if (xj < ls[o] - 1e-12) atomic_max_nonneg(&red[R_BOUND], ls[o] - xj);
            if (xj > us[o] + 1e-12) atomic_max_nonneg(&red[R_BOUND], xj - us[o]);
            xc.store(j, xj);
        }
        cluster_phase<NC>(cl);
        violation(R_VIOL_X);
        cluster_phase<NC>(cl);
        for (int j = (c0 << 5) + tid; j < min(n, c1 << 5); j += blockDim.x) {
            const int o = j - (c0 << 5);
            const double a = ref_clamp(sums[o] / (double)it, ls[o], us[o]);
            st.x_avg[j] = a;
            xc.store(j, a);
        }
        cluster_phase<NC>(cl);
        violation(R_VIOL_AVG);
        cluster_phase<NC>(cl);
        double v[R_COUNT];
#pragma unroll
        for (int q = 0; q < R_COUNT; ++q) {
            unsigned long long mx = 0ull;
            for (int r = 0; r < NC; ++r) mx = max(mx, *cl.map_shared_rank(&red[q], r));
            v[q] = __longlong_as_double((long long)mx);
        }
        const double best = (v[R_VIOL_AVG] < v[R_VIOL_X]) ? v[R_VIOL_AVG] : v[R_VIOL_X];
        const bool failed = isnan(best) || best > 1e15;
        const bool converged =
            !failed && best <= tol && v[R_BOUND] <= tol && v[R_DPRIMAL] <= 1e-7 && v[R_DDUAL] <= 1e-7 && it >= 100;
        finished = failed || converged;
        cluster_phase<NC>(cl);  // every CTA has read the others' maxima
        if (rank == 0 && tid == 0) {
            out->iter = it;
            out->failed = failed;
            out->converged = converged;
            out->viol_x = v[R_VIOL_X];
            out->viol_avg = v[R_VIOL_AVG];
            out->bound = v[R_BOUND];
            out->dprimal = v[R_DPRIMAL];
            out->ddual = v[R_DDUAL];
        }
    }
    for (int i = (r0 << 5) + tid; i < min(m, r1 << 5); i += blockDim.x) st.y[i] = ys[i];
    for (int j = (c0 << 5) + tid; j < min(n, c1 << 5); j += blockDim.x) {
        st.x[j] = xs[j - (c0 << 5)];
        st.x_sum[j] = sums[j - (c0 << 5)];
    }
    if (!ok) {
        out->wait_failed = 1;
        __nanosleep(1000000);  // late elements land before the CTA they go to leaves
    }
    cluster_phase<NC>(cl);  // no CTA leaves while another may still store into its copies
}

// Shared-memory layout for an m x n LP whose largest owned parts hold `ce` / `re` padded entries
// (0: the matrix stays in global memory).
template <int NC>
RefLayout ref_layout(int m, int n, int64_t ce, int64_t re) {
    RefLayout L;
    const int ncs = (n + 31) >> 5, nrs = (m + 31) >> 5;
    L.cols = L.rows = 0;
    for (int r = 0; r < NC; ++r) {
        L.cols = std::max(L.cols, 32 * (cluster_slice<NC>(ncs, r + 1) - cluster_slice<NC>(ncs, r)));
        L.rows = std::max(L.rows, 32 * (cluster_slice<NC>(nrs, r + 1) - cluster_slice<NC>(nrs, r)));
    }
    int64_t o = 0;
    auto take = [&](int64_t bytes) {
        const int64_t at = o;
        o = (o + bytes + 15) & ~15ll;
        return (int)std::min<int64_t>(at, 1 << 30);
    };
    L.y = take(8ll * (m + 1));
    L.xh = take(8ll * (n + 1));
    for (int* f : {&L.x, &L.xsum, &L.tau, &L.c, &L.lb, &L.ub}) *f = take(8ll * L.cols);
    for (int* f : {&L.sigma, &L.b}) *f = take(8ll * L.rows);
    L.eq = take(L.rows);
    L.cval = take(8 * ce);
    L.rval = take(8 * re);
    L.cidx = take(2 * ce);
    L.ridx = take(2 * re);
    L.coff = take(4 * (L.cols / 32 + 1));
    L.roff = take(4 * (L.rows / 32 + 1));
    L.cmask = take(4 * (L.cols / 32));
    L.rmask = take(4 * (L.rows / 32));
    L.total = (int)std::min<int64_t>(o, 1 << 30);
    return L;
}

// Device buffers of the engine, kept by the context between solves of LPs of at most kKeepEntries
// entries and as many rows and columns (up to 72 bytes an entry of sliced copies).
constexpr int64_t kKeepEntries = 1 << 20;
struct RefBuffers {
    DBuf<double> tau, sigma, x, y, x_hat, x_sum, x_avg;
    DBuf<unsigned long long> red;
    DBuf<long long> iter;
    DBuf<RefOutcome> outcome;
    DBuf<int64_t> off, t_off;
    DBuf<int32_t> idx, t_idx, longs, t_longs;
    DBuf<double> val, t_val;
};

// The sliced copy of one orientation, or the CSR arrays where padding would cost more than
// three times the entries.
int build_sell(Ctx* ctx, int rows, int other, int64_t nnz, const int32_t* ptr, const int32_t* idx, const double* val,
               DBuf<int64_t>& off, DBuf<int32_t>& longs, DBuf<int32_t>& oidx, DBuf<double>& oval, Sell* S,
               std::vector<int64_t>* h_off) {
    cudaStream_t s = ctx->stream;
    const int nsl = (rows + 31) >> 5, limit = long_limit(nnz, rows);
    B2P_CUDA(ctx, off.reserve(nsl + 2));
    B2P_CUDA(ctx, longs.reserve(nnz / limit + 1));
    B2P_CUDA(ctx, cudaMemsetAsync(off.p + nsl + 1, 0, sizeof(int64_t), s));
    k_ref_slice_len<<<grid_for(nsl, 128, ctx->sm_count), 128, 0, s>>>(rows, limit, ptr, off.p, longs.p);
    B2P_LAUNCH(ctx);
    size_t tmp = 0;
    B2P_CUDA(ctx, cub::DeviceScan::InclusiveSum(nullptr, tmp, off.p + 1, off.p + 1, nsl, s));
    B2P_CUDA(ctx, ctx->cub_tmp.reserve(tmp));
    tmp = ctx->cub_tmp.bytes();
    B2P_CUDA(ctx, cub::DeviceScan::InclusiveSum(ctx->cub_tmp.p, tmp, off.p + 1, off.p + 1, nsl, s));
    // the offsets of an LP that may run on a cluster are wanted on the host, else only the total; the number
    // of long rows lies behind them
    const size_t want = nnz <= kClusterNnz ? (size_t)nsl + 2 : 2;
    h_off->resize(want);
    B2P_CUDA(ctx, cudaMemcpyAsync(h_off->data(), off.p + nsl + 2 - want, sizeof(int64_t) * want, cudaMemcpyDeviceToHost, s));
    B2P_CUDA(ctx, cudaStreamSynchronize(s));
    *S = Sell{nullptr, ptr, idx, val, idx, val, longs.p, (int)h_off->back(), limit};
    h_off->pop_back();
    const int64_t total = h_off->back();
    ctx->launches += 2;
    if (total > 3 * nnz + 4096) return B2P_OK;
    B2P_CUDA(ctx, oidx.reserve(total));
    B2P_CUDA(ctx, oval.reserve(total));
    k_ref_slice_fill<<<grid_for(rows + 31, 128, ctx->sm_count), 128, 0, s>>>(rows, limit, other, ptr, idx, val, off.p, oidx.p,
                                                                            oval.p);
    B2P_LAUNCH(ctx);
    ctx->launches += 1;
    S->off = off.p;
    S->idx = oidx.p;
    S->val = oval.p;
    return B2P_OK;
}

}  // namespace

struct RefWork {
    RefBuffers b;
};

void ref_free(Ctx* ctx) {
    delete ctx->rw;
    ctx->rw = nullptr;
}

int ref_engine_solve(Ctx* ctx, const b2p_params* p, b2p_result* r, double* x_out, double* y_out) {
    DevLP& L = ctx->lp;
    const int m = L.m, n = L.n;
    cudaStream_t s = ctx->stream;
    if (!ctx->rw) ctx->rw = new RefWork();
    // a large LP's buffers go back when the solve ends (freeing waits for what is in flight)
    struct Keep {
        Ctx* ctx;
        bool keep;
        ~Keep() {
            if (!keep) ref_free(ctx);
        }
    } keep{ctx, L.nnz <= kKeepEntries && (int64_t)m + n <= kKeepEntries};
    RefBuffers& B = ctx->rw->b;
    B2P_CUDA(ctx, B.tau.reserve(n));
    B2P_CUDA(ctx, B.sigma.reserve(m));
    B2P_CUDA(ctx, B.x.reserve((size_t)n + 1));
    B2P_CUDA(ctx, B.y.reserve((size_t)m + 1));
    B2P_CUDA(ctx, B.x_hat.reserve((size_t)n + 1));
    B2P_CUDA(ctx, B.x_sum.reserve(n));
    B2P_CUDA(ctx, B.x_avg.reserve((size_t)n + 1));
    B2P_CUDA(ctx, B.red.reserve(R_COUNT));
    B2P_CUDA(ctx, B.iter.reserve(1));
    RefState st{B.tau.p, B.sigma.p, B.x.p, B.y.p, B.x_hat.p, B.x_sum.p, B.x_avg.p, B.red.p, B.iter.p};

    const int TB = 128;
    unsigned gn = grid_for(n, TB, ctx->sm_count), gm = grid_for(m, TB, ctx->sm_count);
    unsigned gmn = grid_for(std::max(m, n), TB, ctx->sm_count);
    k_ref_steps<<<gmn, TB, 0, s>>>(m, n, L.rowptr.p, L.vals.p, L.t_rowptr.p, L.t_vals.p, p->adaptive_step_size,
                                   p->primal_step_size, p->dual_step_size, st.tau, st.sigma);
    k_ref_init<<<gmn, TB, 0, s>>>(m, n, L.lb.p, L.ub.p, st.x, st.y, st.x_sum, st.x_hat, st.x_avg, st.iter, st.red);
    B2P_LAUNCH(ctx);
    ctx->launches += 2;
    Sell A, At;
    std::vector<int64_t> h_off, h_toff;
    int bst = build_sell(ctx, m, n, L.nnz, L.rowptr.p, L.colidx.p, L.vals.p, B.off, B.longs, B.idx, B.val, &A, &h_off);
    if (bst) return bst;
    bst = build_sell(ctx, n, m, L.nnz, L.t_rowptr.p, L.t_colidx.p, L.t_vals.p, B.t_off, B.t_longs, B.t_idx, B.t_val, &At,
                     &h_toff);
    if (bst) return bst;

    auto primal = [&](auto check) {
        constexpr bool C = decltype(check)::value;
        const auto fn = At.nlong ? (At.off ? k_ref_primal<C, true, true> : k_ref_primal<C, false, true>)
                                 : (At.off ? k_ref_primal<C, true, false> : k_ref_primal<C, false, false>);
        pdl_launch(fn, gn, TB, 0, s, n, At, L.c.p, L.lb.p, L.ub.p, st);
    };
    auto dual = [&](auto check) {
        constexpr bool C = decltype(check)::value;
        const auto fn = A.nlong ? (A.off ? k_ref_dual<C, true, true> : k_ref_dual<C, false, true>)
                                : (A.off ? k_ref_dual<C, true, false> : k_ref_dual<C, false, false>);
        pdl_launch(fn, gm, TB, 0, s, m, A, L.b.p, L.is_eq.p, st);
    };
    auto check_xs = [&]() {
        k_ref_check_cols<<<gn, TB, 0, s>>>(n, L.lb.p, L.ub.p, st);
        if (A.off) k_ref_check_rows<true><<<gm, TB, 0, s>>>(m, A, L.b.p, L.is_eq.p, st);
        else k_ref_check_rows<false><<<gm, TB, 0, s>>>(m, A, L.b.p, L.is_eq.p, st);
    };
    auto plain_iter = [&]() {
        primal(std::false_type());
        dual(std::false_type());
    };
    auto check_iter = [&]() {
        k_ref_clear<<<1, 32, 0, s>>>(st.red);
        primal(std::true_type());
        dual(std::true_type());
        check_xs();
    };

    const int64_t max_it = p->max_iterations;
    const int64_t cf = std::min<int64_t>(p->check_frequency, 100);  // first_order_solver.cpp:156
    // One CTA for up to kOneCtaNnz entries that fit its shared memory with the vectors, else a
    // cluster where the vectors do, with the owned parts of the matrix in shared memory if
    // they fit as well.
    RefLayout lay{};
    const bool longs = A.nlong > 0 || At.nlong > 0;
    decltype(&k_ref_cluster<1, true, false>) small_fn = nullptr;
    int ctas = 1;
    if (A.off && At.off && L.nnz <= kClusterNnz && m < 65535 && n < 65535) {
        const int ncs = (n + 31) >> 5, nrs = (m + 31) >> 5;
        // the form `fn` with the layout `l` if its CTAs have the shared memory and the device the clusters
        auto take = [&](auto fn, int nc, const RefLayout& l) -> int {
            int most = 0;
            B2P_CUDA(ctx, open_smem(ctx, fn, &most));
            if (l.total > most || (nc > 1 && clusters_resident(fn, nc, kClusterThreads, l.total) < 1)) return B2P_OK;
            small_fn = fn;
            ctas = nc;
            lay = l;
            return B2P_OK;
        };
        if (L.nnz <= kOneCtaNnz) {
            const int tst = take(longs ? k_ref_cluster<1, true, true> : k_ref_cluster<1, true, false>, 1,
                                 ref_layout<1>(m, n, h_toff[ncs], h_off[nrs]));
            if (tst) return tst;
        }
        if (!small_fn) {
            int64_t ce = 0, re = 0;
            for (int r = 0; r < kClusterCtas; ++r) {
                ce = std::max(ce, h_toff[cluster_slice<kClusterCtas>(ncs, r + 1)] - h_toff[cluster_slice<kClusterCtas>(ncs, r)]);
                re = std::max(re, h_off[cluster_slice<kClusterCtas>(nrs, r + 1)] - h_off[cluster_slice<kClusterCtas>(nrs, r)]);
            }
            const int tst = take(longs ? k_ref_cluster<kClusterCtas, true, true> : k_ref_cluster<kClusterCtas, true, false>,
                                 kClusterCtas, ref_layout<kClusterCtas>(m, n, ce, re));
            if (tst) return tst;
        }
        if (!small_fn) {
            const int tst = take(longs ? k_ref_cluster<kClusterCtas, false, true> : k_ref_cluster<kClusterCtas, false, false>,
                                 kClusterCtas, ref_layout<kClusterCtas>(m, n, 0, 0));
            if (tst) return tst;
        }
    }
    const bool small = small_fn != nullptr;
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    if (!small && max_it >= kGraphIters && cf > kGraphIters) {
        B2P_CUDA(ctx, cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
        for (int k = 0; k < kGraphIters; ++k) plain_iter();
        cudaError_t ce = cudaStreamEndCapture(s, &graph);
        if (ce != cudaSuccess) {
            ctx->err = std::string("graph capture: ") + cudaGetErrorString(ce);
            return B2P_EXECUTION_FAILED;
        }
        ce = cudaGraphInstantiate(&exec, graph, 0);
        if (ce != cudaSuccess) {
            cudaGraphDestroy(graph);
            ctx->err = std::string("graph instantiate: ") + cudaGetErrorString(ce);
            return B2P_EXECUTION_FAILED;
        }
    }
    struct GraphGuard {
        cudaGraph_t g;
        cudaGraphExec_t e;
        ~GraphGuard() {
            if (e) cudaGraphExecDestroy(e);
            if (g) cudaGraphDestroy(g);
        }
    } guard{graph, exec};

    unsigned long long host_red[R_COUNT];
    int64_t iter = 0;
    bool converged = false, failed = false;
    double cons_viol = 0.0, bound_viol = 0.0, dpr = 0.0, ddu = 0.0;
    cudaEventRecord(ctx->ev0, s);
    if (small) {
        B2P_CUDA(ctx, B.outcome.reserve(1));
        B2P_CUDA(ctx, cudaMemsetAsync(B.outcome.p, 0, sizeof(RefOutcome), s));
        cudaLaunchAttribute dims;
        const cudaLaunchConfig_t lc = cluster_config(ctas, ctas, kClusterThreads, lay.total, s, &dims);
        // one launch runs up to 100,000 iterations (a fraction of a second)
        while (iter < max_it && !converged && !failed) {
            const int64_t stop = std::min<int64_t>(iter + 100000, max_it);
            B2P_CUDA(ctx, cudaLaunchKernelEx(&lc, small_fn, m, n, A, At, (const double*)L.c.p, (const double*)L.lb.p,
                                             (const double*)L.ub.p, (const double*)L.b.p, (const uint8_t*)L.is_eq.p, st, lay,
                                             (long long)stop, (long long)max_it, (long long)cf, p->feasibility_tolerance,
                                             B.outcome.p));
            B2P_LAUNCH(ctx);
            ctx->launches += 1;
            RefOutcome o;
            B2P_CUDA(ctx, cudaMemcpyAsync(&o, B.outcome.p, sizeof(o), cudaMemcpyDeviceToHost, s));
            B2P_CUDA(ctx, cudaStreamSynchronize(s));
            if (o.wait_failed) {
                ctx->err = "the cluster's exchange did not complete";
                return B2P_EXECUTION_FAILED;
            }
            iter = o.iter;
            converged = o.converged != 0;
            failed = o.failed != 0;
            cons_viol = (o.viol_avg < o.viol_x) ? o.viol_avg : o.viol_x;
            bound_viol = o.bound;
            dpr = o.dprimal;
            ddu = o.ddual;
        }
        B2P_CUDA(ctx, cudaMemcpyAsync(st.iter, &iter, sizeof(iter), cudaMemcpyHostToDevice, s));
    }
    while (!small && iter < max_it) {
        int64_t next_check = std::min<int64_t>((iter / cf + 1) * cf, max_it);
        int64_t span = next_check - iter;
        int64_t k = 0;
        for (; exec && k + kGraphIters <= span - 1; k += kGraphIters) B2P_CUDA(ctx, cudaGraphLaunch(exec, s));
        for (; k < span - 1; ++k) plain_iter();
        check_iter();
        B2P_LAUNCH(ctx);
        ctx->launches += 2 * span + 3;
        iter = next_check;
        B2P_CUDA(ctx, cudaMemcpyAsync(host_red, st.red, sizeof(host_red), cudaMemcpyDeviceToHost, s));
        B2P_CUDA(ctx, cudaStreamSynchronize(s));
        double vx = bits_to_double(host_red[R_VIOL_X]), va = bits_to_double(host_red[R_VIOL_AVG]);
        double best = (va < vx) ? va : vx;  // std::min(max_viol, avg_viol)
        bound_viol = bits_to_double(host_red[R_BOUND]);
        dpr = bits_to_double(host_red[R_DPRIMAL]);
        ddu = bits_to_double(host_red[R_DDUAL]);
        cons_viol = best;
        if (std::isnan(best) || best > 1e15) {  // first_order_solver.cpp:232-236
            failed = true;
            break;
        }
        bool feasible = best <= p->feasibility_tolerance && bound_viol <= p->feasibility_tolerance;
        bool stationary = dpr <= 1e-7 && ddu <= 1e-7;
        if (feasible && stationary && iter >= 100) {
            converged = true;
            break;
        }
    }
    cudaEventRecord(ctx->ev1, s);
    r->iterations = iter;
    r->constraint_violation = cons_viol;
    r->bound_violation = bound_viol;
    r->max_primal_delta = dpr;
    r->max_dual_delta = ddu;
    if (failed) {
        r->status = B2P_STATUS_NUMERICAL_FAILURE;
    } else {
        r->status = converged ? B2P_STATUS_OPTIMAL : B2P_STATUS_MAX_ITERATIONS;
        // first_order_solver.cpp:261-279: the ergodic average replaces x only when the
        // loop did not converge and its violation is no worse than the last check's.
        k_ref_clear<<<1, 32, 0, s>>>(st.red);
        check_xs();
        B2P_LAUNCH(ctx);
        ctx->launches += 3;
        B2P_CUDA(ctx, cudaMemcpyAsync(host_red, st.red, sizeof(host_red), cudaMemcpyDeviceToHost, s));
        B2P_CUDA(ctx, cudaStreamSynchronize(s));
        double avg_viol = bits_to_double(host_red[R_VIOL_AVG]);
        r->used_average = (!converged && avg_viol <= cons_viol) ? 1 : 0;
    }
    float kms = 0.f;
    cudaEventElapsedTime(&kms, ctx->ev0, ctx->ev1);
    r->kernel_time_ms = kms;
    double t0 = now_ms();
    if (x_out) B2P_CUDA(ctx, cudaMemcpyAsync(x_out, r->used_average ? st.x_avg : st.x, sizeof(double) * n,
                                             cudaMemcpyDeviceToHost, s));
    if (y_out) B2P_CUDA(ctx, cudaMemcpyAsync(y_out, st.y, sizeof(double) * m, cudaMemcpyDeviceToHost, s));
    B2P_CUDA(ctx, cudaStreamSynchronize(s));
    r->transfer_time_ms = now_ms() - t0;
    return B2P_OK;
}

}  // namespace b2p
