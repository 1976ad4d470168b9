// Batched engine: thousands of independent LPs in one persistent launch.
//
// Layout in HBM
//   * `nmat` constraint matrices concatenated into one block-diagonal CSR with
//     GLOBAL row/column indices (row_off[k], col_off[k] per matrix) plus its
//     stable transpose (FP64 originals and scaled copies: the restart-check KKT
//     and the re-centring read these).  Rows and columns of every matrix are
//     renumbered at upload by decreasing length (stable), so that consecutive
//     32-row / 32-column slices hold rows of nearly equal length.
//   * the iteration SpMVs read SELL-32 copies of the scaled matrix, one per
//     orientation: per slice of 32 rows (columns), `len` = the longest row of the
//     slice, entries stored column-major inside the slice (entry q of lane l at
//     slice_ptr + 32 q + l, zero-padded), values in the solve's precision and
//     16-bit LOCAL indices (an instance whose iterates fit in shared memory has
//     m, n < 65536).  A warp reads 32 consecutive values and 32 consecutive
//     indices per step: coalesced, no per-row pointers, no divergence.
//   * `count` instances, each naming a matrix; b, c, l, u in FP64 (internal
//     order; KKT and re-centring); column and row records of the scaled problem in
//     the solve's precision, one 32-column (row) block after another (col_rec,
//     row_rec); iterates x, y and the check-point copies xt, yt.  All
//     concatenated at per-instance offsets; warm starts and answers are mapped
//     between external and internal order on the device.
// Execution
//   * one CTA owns a group of NI instances at a time (persistent grid, work queue
//     sorted by nnz descending = longest-first): NI = 1 for any batch, 2 or 4 for
//     batches whose instances share one matrix, iterated in lockstep so that each
//     SELL load feeds all of them.  When a CTA takes a group it copies its matrix's
//     slice pointers into a shared-memory table.  The gathered operands of both SpMVs --
//     y (also the dual iterate) for A^T y and xh for A xh -- live in shared
//     memory, interleaved over the group; x follows from xh, so a plain iteration
//     reads only the records and the matrix.  A PDHG iteration is: primal phase (one thread per
//     column, one warp per column slice) | barrier | dual phase (one thread per
//     row) | barrier.  Rows longer than kLongSlice are summed by whole warps over
//     the CSR copy instead (one dense row cannot stall its slice).  Control scalars
//     and step sizes live in shared memory; restart checks are out of line.
//   * precision MT (float = mixed, double = FP64) is the type of the scaled
//     matrix values, the packed records, the iterates and the SpMV sums.  FP64 is
//     kept for the scaling factors, the squared-residual sums, the KKT of the
//     original instance every K iterations, and the re-centring: the mixed
//     engine starts every restart epoch at an FP64 centre (xbar, ybar) and
//     solves the shifted problem rhs b - A xbar, cost c + A^T ybar, bounds
//     l - xbar, u - xbar, dual bound -ybar, rebuilt from the FP64 matrix, so
//     the FP32 iterates only carry the correction (iterative refinement).
//   * per instance: own step size (from its matrix), primal weight, Halpern
//     counter, restart state, FP64 KKT every K iterations (over FP64 SELL copies
//     with the checked vectors staged in shared memory; block reductions in a
//     fixed order: deterministic), own termination.
//   * a launch runs every active instance for up to `chunk` iterations; a
//     compaction kernel drops finished instances; [chunk, compact] x 2 is
//     captured as a CUDA graph and replayed until no instance is active.
//   * CTA size, SELL entry order (one entry or a pair per lane load), instances per
//     CTA and chunk length come from an autotuner that times the candidates on a
//     sample of the batch (cached on disk); between replays the host picks the form
//     with the least rounds of resident CTAs x time per round for the instances
//     still active, and a wide single form for the tail.
#include <cooperative_groups.h>
#include <cub/cub.cuh>

#include <algorithm>
#include <type_traits>
#include <climits>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <fstream>
#include <numeric>
#include <sstream>
#include <string>

#include "b2p_internal.cuh"
#include "cluster.cuh"

namespace b2p {

// per-instance control scalars (device)
struct InstCtrl {
    double omega, r0, rprev;
    double rel_p, rel_d, rel_g, pobj, dobj;
    double obj_err;  // FP64 bound on |c.x - optimum| / max(1, |c.x|) at the last check
    long long k, total, restarts;
    long long base;  // iterations spent on the instance before this run (cold fallback after a warm run)
    int status, done, first;
    int pad;
};

// A tuned launch shape of the chunk kernel.
struct TuneCfg {
    int threads = 256, chunk = 2048, w = 1;  // CTA size, iterations per chunk launch, SELL entries per lane load (1 or 2)
    int ni = 1;                              // instances per CTA: 1, or 2 or 4 (groups, batches of one shared matrix)
    // the forms a solve chooses between by the number of instances still active: instances
    // per CTA 1, 2, 4 with their CTA sizes (0: not available) and microseconds per iteration
    // of one round of resident CTAs
    int form_th[3] = {0, 0, 0};
    double form_us[3] = {0, 0, 0};
    bool pinned = false;  // B2P_BATCH_SHAPE named the shape: no other form runs
};
constexpr int kFormNi[3] = {1, 2, 4};

struct BatchWork {
    int nmat = 0, count = 0;
    int64_t tot_m = 0, tot_n = 0, nnz = 0, inst_m = 0, inst_n = 0;
    // matrices (internal numbering)
    DBuf<int32_t> rowptr, colidx, t_rowptr, t_colidx;
    DBuf<double> vals, t_vals, sv64, stv64, dr, dc, pv, pu;
    DBuf<float> sv32, stv32;
    DBuf<int32_t> mat_m, mat_n;
    DBuf<int64_t> mat_row_off, mat_col_off;
    DBuf<double> mat_eta;
    // SELL-32 copies: slice pointers (per matrix nslices + 1, at mat_*s_off), local
    // indices, scaled values in both precisions; internal -> external local index
    DBuf<int64_t> r_sptr, c_sptr, mat_rs_off, mat_cs_off;
    DBuf<uint16_t> r_eidx, c_eidx;
    DBuf<double> r_ev64, c_ev64;
    DBuf<float> r_ev32, c_ev32;
    DBuf<int32_t> r_ext, c_ext;
    std::vector<int32_t> h_mat_m, h_mat_n;
    // instances
    DBuf<int32_t> inst_mat;
    DBuf<int64_t> x_off, y_off;    // of an instance's vectors
    DBuf<int64_t> xp_off, yp_off;  // of its column / row records (whole slices), in values
    DBuf<double> b, c, lb, ub, bnorm, cnorm;
    DBuf<uint8_t> is_eq;
    // packed records and iterates, sized for FP64 and reinterpreted for FP32; dx, dy hold
    // the fixed-point displacement T(z) - z of the last check (infeasibility certificates)
    DBuf<double> colp, rowp, x, xt, y, yt, dx, dy;
    bool recenter = false;
    DBuf<double> xbar, atybar, ybar, axbar;  // re-centring state (per instance, original space)
    DBuf<InstCtrl> ictrl;
    DBuf<int32_t> active, active2, counters;  // counters[0]=head, [1]=active count
    std::vector<int32_t> h_inst_mat, order;
    int max_m = 0, max_n = 0;
    int max_len = 0;  // longest row or column of any matrix
    // results of the last solve: per-instance control blocks (host) and the answers
    // in the original space, external order (device, FP64), with the primal weights
    std::vector<InstCtrl> hc;
    DBuf<double> ox, oy, oom;
    bool solved = false;
    bool tuned[2] = {false, false};
    TuneCfg tuned_cfg[2];           // per precision
    int ell_w = 1;                  // entry order the SELL copies hold now
    DBuf<int32_t> list;             // instances re-initialised by a subset solve
    // active-instance trace of the last solve: host time (ms from the first graph launch of
    // the solve) and instances still active after each graph launch (a fallback run continues
    // the same trace)
    std::vector<double> trace_ms;
    std::vector<int32_t> trace_active;
};

void batch_free(Ctx* ctx) {
    delete ctx->bw;
    ctx->bw = nullptr;
}

namespace {

constexpr int kPowerCluster = 16384;  // entries from which a matrix's power iteration runs on a cluster
constexpr int kPowerCtas = 8;
constexpr int kLongSlice = 128;  // entries per lane above which a slice is summed warp-cooperatively

// Column and row records of the scaled (and, when re-centred, shifted) problem in the
// solve's precision, in blocks of one 32-column / 32-row slice: cost, lower bound, upper
// bound, Halpern anchor (4 x 32 values) per column slice; rhs, lower bound of the dual
// (-inf on equality rows), anchor (3 x 32) per row slice.  A warp reads each part it
// needs as one contiguous 128- or 256-byte run, and a re-centred solve, whose anchors are
// 0, does not read that part at all.
__host__ __device__ __forceinline__ size_t col_rec(int j) { return (size_t)(j >> 5) * 128 + (j & 31); }
__host__ __device__ __forceinline__ size_t row_rec(int i) { return (size_t)(i >> 5) * 96 + (i & 31); }

struct BArgs {
    // matrices
    const int32_t *rowptr, *colidx, *t_rowptr, *t_colidx;
    const double *sv64, *stv64, *dr, *dc, *mat_eta;
    const void *sv, *stv;  // MT-typed scaled values (CSR)
    const int32_t *mat_m, *mat_n;
    const int64_t *mat_row_off, *mat_col_off;
    // SELL-32 copies
    const int64_t *r_sptr, *c_sptr, *mat_rs_off, *mat_cs_off;
    const uint16_t *r_eidx, *c_eidx;
    const void *r_ev, *c_ev;  // MT-typed
    const double *r_ev64, *c_ev64;  // FP64 values in the same order (restart-check KKT)
    const int32_t *r_ext, *c_ext;
    // instances
    const int32_t* inst_mat;
    const int64_t *x_off, *y_off;    // vectors
    const int64_t *xp_off, *yp_off;  // column / row records
    const double *b, *c, *lb, *ub;
    double *bnorm, *cnorm;  // written by the init kernel
    const uint8_t* is_eq;
    void *colp, *rowp, *x, *xt, *y, *yt;  // MT-typed
    void *dx, *dy;                        // MT-typed: T(z) - z at check iterations (eps_inf > 0)
    InstCtrl* ictrl;
    const int32_t* active;
    int32_t* counters;
    // parameters
    double eps, beta_s, beta_n, beta_a, rho;
    double eps_obj, eps_inf;  // objective-accuracy stop (0 = off), certificate tolerance (0 = off)
    // FP64 re-centring: per-instance centre in the original space, A xbar, A^T ybar;
    // original FP64 values in both orientations
    int recenter;
    const double *vals, *t_vals;
    double *xbar, *ybar, *axbar, *atybar;
    long long max_iter;
    int K;
};

template <typename T>
__device__ __forceinline__ T clampT(T v, T lo, T hi) { return v < lo ? lo : (v > hi ? hi : v); }

// Block-wide FP64 sum of NV values (sh holds 32 * NV), fixed reduction order (deterministic).
template <int NV>
__device__ __forceinline__ void block_sums(double (&v)[NV], double* sh /* [32*NV] */) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
    for (int q = 0; q < NV; ++q) v[q] = warp_sum(v[q]);
    __syncthreads();
    if (lane == 0)
#pragma unroll
        for (int q = 0; q < NV; ++q) sh[w * NV + q] = v[q];
    __syncthreads();
    if (threadIdx.x == 0) {
#pragma unroll
        for (int q = 0; q < NV; ++q) {
            double t = 0.0;
            for (int i = 0; i < nw; ++i) t += sh[i * NV + q];
            v[q] = t;
        }
    }
}

// One lane's row of a SELL-32 slice (len entries per lane, even).  W = 1: v / ix point at
// the lane's first entry and entry q sits 32 q further.  W = 2: entries are stored in
// pairs -- pair t of lane l at slice + 64 t + 2 l -- so one 8- (FP32) or 16-byte (FP64)
// value load and one 4-byte index load fetch two entries; v / ix point at the lane's
// first pair.  Sequential sum in entry order in both layouts (bit-identical results).
// Entries are taken in batches of B (8 in FP32, 4 in FP64, the most the register
// budget of two 512-thread CTAs per SM holds without spilling in the loop): every
// value and index load of a batch (the last batch predicated on the row's length)
// is issued before the first gather that needs one, so a slice of up to B entries
// per lane costs one L2 round trip and a longer one a round trip per batch.
template <typename VT, typename GT, int W>
__device__ __forceinline__ VT ell_dot_vg(const VT* __restrict__ v, const uint16_t* __restrict__ ix, int len,
                                        const GT* __restrict__ g) {
    constexpr int B = sizeof(VT) == 4 ? 8 : 4;
    VT s = (VT)0;
    if constexpr (W == 1) {
        for (int q = 0; q < len; q += B) {
            VT vv[B];
            unsigned ii[B];
#pragma unroll
            for (int u = 0; u < B; ++u) {
                const bool h = q + u < len;
                vv[u] = h ? v[(q + u) * 32] : (VT)0;
                ii[u] = h ? (unsigned)ix[(q + u) * 32] : 0u;
            }
#pragma unroll
            for (int u = 0; u < B; ++u)
                if (q + u < len) s += vv[u] * (VT)g[ii[u]];
        }
    } else {
        typedef typename std::conditional<sizeof(VT) == 4, float2, double2>::type VT2;
        constexpr int P = B / 2;  // pairs per batch
        const int np = len >> 1;
        for (int t = 0; t < np; t += P) {
            VT2 vv[P];
            unsigned ii[P];
#pragma unroll
            for (int u = 0; u < P; ++u) {
                const bool h = t + u < np;
                vv[u] = h ? *reinterpret_cast<const VT2*>(v + (t + u) * 64) : VT2{(VT)0, (VT)0};
                ii[u] = h ? *reinterpret_cast<const unsigned*>(ix + (t + u) * 64) : 0u;
            }
#pragma unroll
            for (int u = 0; u < P; ++u)
                if (t + u < np) {
                    s += vv[u].x * (VT)g[ii[u] & 0xFFFFu];
                    s += vv[u].y * (VT)g[ii[u] >> 16];
                }
        }
    }
    return s;
}

// Entries of a CTA's slice table (column slices, then row slices; even, so what follows
// it in shared memory stays 16-byte aligned).
__host__ __device__ __forceinline__ int slice_tab_len(int nrs, int ncs) { return (nrs + ncs + 1) & ~1; }

// The slice table of one matrix in shared memory, built when a CTA takes an instance:
// per slice {first entry, entries per lane}.  The iterations then read one 8-byte shared
// word per slice instead of two slice pointers from L2 in front of every value load.
// Entry offsets fit 32 bits (the upload refuses batches whose SELL copies do not).
__device__ __forceinline__ void fill_slice_tab(int2* tab, const int64_t* __restrict__ csp, int ncs,
                                               const int64_t* __restrict__ rsp, int nrs) {
    for (int i = threadIdx.x; i < ncs; i += blockDim.x)
        tab[i] = make_int2((int)csp[i], (int)((csp[i + 1] - csp[i]) >> 5));
    for (int i = threadIdx.x; i < nrs; i += blockDim.x)
        tab[ncs + i] = make_int2((int)rsp[i], (int)((rsp[i + 1] - rsp[i]) >> 5));
}

// Slice of round r for warp w of nw: rounds alternate the direction in which the
// (length-sorted) slices are dealt, w then nw - 1 - w, so every warp's share of long
// and short slices is even.  Increasing in r for a fixed warp.
__device__ __forceinline__ int snake_slice(int r, int w, int nw) { return r * nw + ((r & 1) ? nw - 1 - w : w); }

// The 32 rows of one slice summed by the whole warp over the CSR copy (rows
// first .. first+cnt-1, global numbering; `off` localises the column index).
// Lane r returns the sum of row first + r.
template <typename MT, typename GT = MT>
__device__ MT long_slice_dot(const MT* __restrict__ vals, const int32_t* __restrict__ ptr,
                             const int32_t* __restrict__ idx, int64_t first, int cnt, int64_t off,
                             const GT* __restrict__ g, int lane) {
    MT mine = (MT)0;
    for (int r = 0; r < cnt; ++r) {
        MT s = (MT)0;
        for (int e = ptr[first + r] + lane; e < ptr[first + r + 1]; e += 32) s += vals[e] * (MT)g[idx[e] - off];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == r) mine = s;
    }
    return mine;
}

// Re-centring, an exact change of variables in FP64: rewrite the scaled problem of
// one instance around its centre (xbar, ybar) -- rhs dr*(b - A xbar), cost
// dc*(c + A^T ybar), bounds (l - xbar)/dc, (u - xbar)/dc, dual lower bound -ybar/dr
// on inequality rows -- from the original FP64 matrix, with zero anchors (the
// iterates restart at the centre).  Called by every thread of the owning CTA.
template <typename MT>
__device__ void rebuild_shifted(const BArgs& a, int m, int n, int64_t ro, int64_t co, int64_t xo, int64_t yo,
                                int64_t xp, int64_t yp) {
    for (int i = threadIdx.x; i < m; i += blockDim.x) {
        const int64_t gi = ro + i;
        double s = 0.0;
        for (int e = a.rowptr[gi]; e < a.rowptr[gi + 1]; ++e) s += a.vals[e] * a.xbar[xo + a.colidx[e] - co];
        const double dri = a.dr[gi];
        a.axbar[yo + i] = s;
        MT* r = (MT*)a.rowp + yp + row_rec(i);
        r[0] = (MT)(dri * (a.b[yo + i] - s));
        r[32] = a.is_eq[yo + i] ? (MT)(-INFINITY) : (MT)(-a.ybar[yo + i] / dri);
        r[64] = (MT)0;
    }
    for (int j = threadIdx.x; j < n; j += blockDim.x) {
        const int64_t gj = co + j;
        double s = 0.0;
        for (int e = a.t_rowptr[gj]; e < a.t_rowptr[gj + 1]; ++e) s += a.t_vals[e] * a.ybar[yo + a.t_colidx[e] - ro];
        const double dcj = a.dc[gj], xb = a.xbar[xo + j];
        a.atybar[xo + j] = s;
        MT* p = (MT*)a.colp + xp + col_rec(j);
        p[0] = (MT)(dcj * (a.c[xo + j] + s));
        p[32] = (MT)((a.lb[xo + j] - xb) / dcj);
        p[64] = (MT)((a.ub[xo + j] - xb) / dcj);
        p[96] = (MT)0;
    }
}

// Restart of one instance after its check decided so, by every thread of the owning
// CTA (ys: its dual iterate in shared memory): z <- anchor <- T(z), or, re-centred,
// T(z) becomes the new FP64 centre and the shifted problem is rebuilt around it.
// Element i of the dual iterate is ys[YS i].
template <typename MT, int YS>
__device__ __noinline__ void restart_instance(const BArgs& a, int m, int n, int64_t ro, int64_t co, int64_t xo,
                                              int64_t yo, int64_t xp, int64_t yp, MT* ys) {
    const int tid = threadIdx.x, nt = blockDim.x;
    MT *xg = (MT*)a.x, *xtg = (MT*)a.xt, *ytg = (MT*)a.yt;
    if (!a.recenter) {
        for (int j = tid; j < n; j += nt) {
            const MT v = xtg[xo + j];
            xg[xo + j] = v;
            ((MT*)a.colp)[xp + col_rec(j) + 96] = v;
        }
        for (int i = tid; i < m; i += nt) {
            const MT v = ytg[yo + i];
            ys[YS * i] = v;
            ((MT*)a.rowp)[yp + row_rec(i) + 64] = v;
        }
    } else {
        for (int j = tid; j < n; j += nt) {
            a.xbar[xo + j] += a.dc[co + j] * (double)xtg[xo + j];
            xg[xo + j] = (MT)0;
            xtg[xo + j] = (MT)0;
        }
        for (int i = tid; i < m; i += nt) {
            a.ybar[yo + i] += a.dr[ro + i] * (double)ytg[yo + i];
            ys[YS * i] = (MT)0;
            ytg[yo + i] = (MT)0;
        }
        __syncthreads();
        rebuild_shifted<MT>(a, m, n, ro, co, xo, yo, xp, yp);
    }
}

// Restart-check iteration of one instance, run by every thread of the owning CTA
// after T(z) (xt, yt) and, with certificates on, the displacement (dx, dy) are in
// global memory: the FP64 KKT of T(z) on the original instance, the objective-error
// bound, the certificates (every fourth check) and the decisions -- termination,
// restart, primal weight -- which thread 0 writes to `sc` and `s_flags` (0: done,
// 1: restart).  The products A xt, A^T yt (and A dx, A^T dy) run over the FP64 SELL
// copies of the scaled matrix with the slice table `tab`, one lane per row / column as
// in the iterations, gathering from `buf` -- the instance's xh region of shared memory,
// free at a check (the dual phase has consumed xh, the next primal phase rewrites it) --
// into which each gathered vector is staged first.  Kept out of line: its FP64
// accumulators would otherwise raise the register demand of the iteration loop.
template <typename MT, int W>
__device__ __noinline__ void check_instance(const BArgs& a, int inst, int m, int n, int64_t ro, int64_t co,
                                            int64_t xo, int64_t yo, long long total, long long kk, double om,
                                            double r_now, double dxa, double dya, InstCtrl& sc, int* s_flags,
                                            double* red, const int2* tab, MT* buf) {
    const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, warp = tid >> 5, nwarps = nt >> 5;
    const int ncs = (n + 31) >> 5, nrs = (m + 31) >> 5;
    const MT *xtg = (const MT*)a.xt, *ytg = (const MT*)a.yt;
    const MT *dxg = (const MT*)a.dx, *dyg = (const MT*)a.dy;
    const bool rays = a.eps_inf > 0.0;
    // (A v)_i in the scaled space for lane `lane` of row slice sl, v staged in buf
    auto row_dot = [&](int sl) -> double {
        const int2 t = tab[ncs + sl];
        return t.y <= kLongSlice
                   ? ell_dot_vg<double, MT, W>(a.r_ev64 + t.x + W * lane, a.r_eidx + t.x + W * lane, t.y, buf)
                   : long_slice_dot<double, MT>(a.sv64, a.rowptr, a.colidx, ro + (sl << 5), min(32, m - (sl << 5)),
                                                co, buf, lane);
    };
    auto col_dot = [&](int sl) -> double {
        const int2 t = tab[sl];
        return t.y <= kLongSlice
                   ? ell_dot_vg<double, MT, W>(a.c_ev64 + t.x + W * lane, a.c_eidx + t.x + W * lane, t.y, buf)
                   : long_slice_dot<double, MT>(a.stv64, a.t_rowptr, a.t_colidx, co + (sl << 5),
                                                min(32, n - (sl << 5)), ro, buf, lane);
    };
    // ---- FP64 KKT of T(z) on the original instance and the objective-error bound
    double kk2[6] = {0, 0, 0, 0, 0, 0};
    // |primal residual|^2, b.y, |dual residual|^2, c.x, bound term, sum |y| viol
    for (int j = tid; j < n; j += nt) buf[j] = xtg[xo + j];
    __syncthreads();
    for (int sl = warp; sl < nrs; sl += nwarps) {
        const int i = (sl << 5) + lane;
        const double s = row_dot(sl);
        if (i < m) {
            const double dri = a.dr[ro + i];
            const double ax = (a.recenter ? a.axbar[yo + i] : 0.0) + s / dri;
            double rp = ax - a.b[yo + i];
            if (!a.is_eq[yo + i]) rp = fmax(rp, 0.0);
            kk2[0] += rp * rp;
            const double yv = (a.recenter ? a.ybar[yo + i] : 0.0) + dri * (double)ytg[yo + i];
            kk2[1] += a.b[yo + i] * yv;
            kk2[5] += fabs(yv) * fabs(rp);
            if (!a.is_eq[yo + i] && yv < 0.0) kk2[2] += yv * yv;  // y >= 0 on <= rows (dual residual)
        }
    }
    __syncthreads();  // every warp is done with xt
    for (int i = tid; i < m; i += nt) buf[i] = ytg[yo + i];
    __syncthreads();
    for (int sl = warp; sl < ncs; sl += nwarps) {
        const int j = (sl << 5) + lane;
        const double s = col_dot(sl);
        if (j < n) {
            const double dcj = a.dc[co + j];
            const double cj = a.c[xo + j], lj = a.lb[xo + j], uj = a.ub[xo + j];
            const double g = cj + (a.recenter ? a.atybar[xo + j] : 0.0) + s / dcj;
            const bool fl = isfinite(lj), fu = isfinite(uj);
            const double lam = (fl && fu) ? g : (fl ? fmax(g, 0.0) : (fu ? fmin(g, 0.0) : 0.0));
            const double rd = g - lam;
            kk2[2] += rd * rd;
            kk2[3] += cj * ((a.recenter ? a.xbar[xo + j] : 0.0) + dcj * (double)xtg[xo + j]);
            if (lam > 0.0) kk2[4] += lam * lj;
            else if (lam < 0.0) kk2[4] += lam * uj;
        }
    }
    block_sums<6>(kk2, red);
    // ---- certificates of the displacement dx, dy = T(z) - z (every fourth check): primal
    // ray dx -- 0 |viol of A dx and of the bounds' recession cone|^2, 1 c.dx, 2 sum |c dx|;
    // dual ray dy -- 3 b.dy, 4 bound term of a = A^T dy, 5 sum of |terms|, 6 |viol of a|^2
    double ry[7] = {0, 0, 0, 0, 0, 0, 0};
    const bool ray_check = rays && ((total / a.K) & 3) == 0;
    if (ray_check) {
        for (int j = tid; j < n; j += nt) buf[j] = dxg[xo + j];
        __syncthreads();
        for (int sl = warp; sl < nrs; sl += nwarps) {
            const int i = (sl << 5) + lane;
            const double s = row_dot(sl);
            if (i < m) {
                const double dri = a.dr[ro + i];
                const double adx = s / dri;  // (A dx)_i in the original space
                const double v = a.is_eq[yo + i] ? adx : fmax(adx, 0.0);
                ry[0] += v * v;
                const double dyo = dri * (double)dyg[yo + i];
                ry[3] += a.b[yo + i] * dyo;
                ry[5] += fabs(a.b[yo + i] * dyo);
            }
        }
        __syncthreads();
        for (int i = tid; i < m; i += nt) buf[i] = dyg[yo + i];
        __syncthreads();
        for (int sl = warp; sl < ncs; sl += nwarps) {
            const int j = (sl << 5) + lane;
            const double s = col_dot(sl);
            if (j < n) {
                const double dcj = a.dc[co + j];
                const double cj = a.c[xo + j], lj = a.lb[xo + j], uj = a.ub[xo + j];
                const bool fl = isfinite(lj), fu = isfinite(uj);
                const double dxo = dcj * (double)dxg[xo + j];
                ry[1] += cj * dxo;
                ry[2] += fabs(cj * dxo);
                const double bv = (fl && dxo < 0.0 ? -dxo : 0.0) + (fu && dxo > 0.0 ? dxo : 0.0);
                ry[0] += bv * bv;
                const double at = s / dcj;  // (A^T dy)_j in the original space
                const double t = at > 0.0 ? (fl ? at * lj : 0.0) : (at < 0.0 ? (fu ? at * uj : 0.0) : 0.0);
                ry[4] += t;
                ry[5] += fabs(t);
                const double av = (!fl && at > 0.0 ? at : 0.0) + (!fu && at < 0.0 ? -at : 0.0);
                ry[6] += av * av;
            }
        }
        block_sums<7>(ry, red);
    }
    if (tid == 0) {
        const double pres = sqrt(kk2[0]), dres = sqrt(kk2[2]);
        const double pobj = kk2[3], dobj = -kk2[1] + kk2[4];
        sc.rel_p = pres / (1.0 + a.bnorm[inst]);
        sc.rel_d = dres / (1.0 + a.cnorm[inst]);
        sc.rel_g = fabs(pobj - dobj) / (1.0 + fabs(pobj) + fabs(dobj));
        sc.pobj = pobj;
        sc.dobj = dobj;
        sc.obj_err = fmax(fmax(pobj - dobj, kk2[5]), 0.0) / fmax(1.0, fabs(pobj));
        const bool finite = isfinite(pres) && isfinite(dres) && isfinite(pobj) && isfinite(dobj) && isfinite(r_now);
        const bool obj_ok = a.eps_obj <= 0.0 || sc.obj_err <= a.eps_obj;
        // certificates (ratio tests of PDLP; the 1e-9 floors keep rounding noise of a
        // vanishing displacement from passing for a ray)
        const double dray = -ry[3] + ry[4], pray = ry[1];
        const bool infeas = ray_check && dray > 0.0 && dray > 1e-9 * ry[5] && sqrt(ry[6]) <= a.eps_inf * dray;
        const bool unbnd = ray_check && pray < 0.0 && -pray > 1e-9 * ry[2] && sqrt(ry[0]) <= a.eps_inf * -pray;
        if (!finite) {
            sc.done = 1;
            sc.status = B2P_STATUS_NUMERICAL_FAILURE;
        } else if (sc.rel_p <= a.eps && sc.rel_d <= a.eps && sc.rel_g <= a.eps && obj_ok) {
            sc.done = 1;
            sc.status = B2P_STATUS_OPTIMAL;
        } else if (infeas) {
            sc.done = 1;
            sc.status = B2P_STATUS_INFEASIBLE_DETECTED;
        } else if (unbnd) {
            sc.done = 1;
            sc.status = B2P_STATUS_UNBOUNDED_DETECTED;
        } else if (total + sc.base >= a.max_iter) {
            sc.done = 1;
            sc.status = B2P_STATUS_MAX_ITERATIONS;
        }
        s_flags[1] = 0;
        if (!sc.done) {
            const bool rs = (r_now <= a.beta_s * sc.r0) || (r_now <= a.beta_n * sc.r0 && r_now > sc.rprev) ||
                            ((double)kk >= a.beta_a * (double)total);
            sc.rprev = r_now;
            if (rs) {
                if (dxa > 1e-10 && dya > 1e-10) {
                    const double nw = exp(0.5 * log(dya / dxa) + 0.5 * log(om));
                    if (isfinite(nw) && nw > 0.0) sc.omega = nw;
                }
                sc.restarts += 1;
                s_flags[1] = 1;
            }
        }
        s_flags[0] = sc.done;
    }
}

// The NI operands of gather index i: element i of instance k is stored at NI i + k, so one
// 4-, 8- or 16-byte shared-memory load serves all NI instances.
template <typename MT, int NI>
__device__ __forceinline__ void ld_group(const MT* __restrict__ g, unsigned i, MT (&t)[NI]) {
    if constexpr (NI == 1) {
        t[0] = g[i];
    } else if constexpr (sizeof(MT) == 4 && NI == 4) {
        const float4 q = reinterpret_cast<const float4*>(g)[i];
        t[0] = q.x; t[1] = q.y; t[2] = q.z; t[3] = q.w;
    } else if constexpr (sizeof(MT) == 4) {
        static_assert(NI == 2, "a group holds 1, 2 or 4 instances");
        const float2 q = reinterpret_cast<const float2*>(g)[i];
        t[0] = q.x; t[1] = q.y;
    } else {
        static_assert(NI == 2, "an FP64 group holds 1 or 2 instances");
        const double2 q = reinterpret_cast<const double2*>(g)[i];
        t[0] = q.x; t[1] = q.y;
    }
}
template <typename MT, int NI>
__device__ __forceinline__ void st_group(MT* g, int i, const MT (&t)[NI]) {
    if constexpr (NI == 1)
        g[i] = t[0];
    else if constexpr (sizeof(MT) == 4 && NI == 4)
        reinterpret_cast<float4*>(g)[i] = make_float4(t[0], t[1], t[2], t[3]);
    else if constexpr (sizeof(MT) == 4)
        reinterpret_cast<float2*>(g)[i] = make_float2(t[0], t[1]);
    else
        reinterpret_cast<double2*>(g)[i] = make_double2(t[0], t[1]);
}

// One row summed by the whole warp over the CSR copy, for the NI interleaved operands of a
// group (each entry is read once); every lane returns the sums.
template <typename MT, int NI>
__device__ __forceinline__ void long_row_group(const MT* __restrict__ vals, const int32_t* __restrict__ idx, int e0,
                                               int e1, int64_t off, const MT* __restrict__ g, int lane, MT (&s)[NI]) {
#pragma unroll
    for (int k = 0; k < NI; ++k) s[k] = (MT)0;
#pragma unroll 4
    for (int e = e0 + lane; e < e1; e += 32) {
        const MT v = vals[e];
        MT t[NI];
        ld_group<MT, NI>(g, (unsigned)(idx[e] - off), t);
#pragma unroll
        for (int k = 0; k < NI; ++k) s[k] += v * t[k];
    }
#pragma unroll
    for (int k = 0; k < NI; ++k)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s[k] += __shfl_xor_sync(0xffffffffu, s[k], o);
}

// The rows of one slice (long_slice_dot for a group): lane r returns the sums of row first + r.
template <typename MT, int NI>
__device__ __forceinline__ void long_slice_group(const MT* __restrict__ vals, const int32_t* __restrict__ ptr,
                                                 const int32_t* __restrict__ idx, int64_t first, int cnt, int64_t off,
                                                 const MT* __restrict__ g, int lane, MT (&mine)[NI]) {
#pragma unroll 1
    for (int r = 0; r < cnt; ++r) {
        MT s[NI];
        long_row_group<MT, NI>(vals, idx, ptr[first + r], ptr[first + r + 1], off, g, lane, s);
#pragma unroll
        for (int k = 0; k < NI; ++k)
            if (lane == r) mine[k] = s[k];
    }
}

// One batch of a lane's entries of a slice (entries q .. q + B - 1 of its len), loaded
// before it is needed: the iteration loop issues the next batch (of this slice, or the
// first one of the warp's next slice) before it gathers for the current one, so the L2
// round trip of the matrix stream overlaps the gathers.
template <typename VT, int W, int B>
struct EllBatch {
    VT v[B];
    unsigned i[W == 1 ? B : B / 2];
    __device__ __forceinline__ void load_at(const VT* __restrict__ pv, const uint16_t* __restrict__ pi, int u) {
        if constexpr (W == 1) {
            v[u] = pv[u * 32];
            i[u] = pi[u * 32];
        } else if (!(u & 1)) {
            typedef typename std::conditional<sizeof(VT) == 4, float2, double2>::type VT2;
            const VT2 t = *reinterpret_cast<const VT2*>(pv + u * 32);
            v[u] = t.x;
            v[u + 1] = t.y;
            i[u / 2] = *reinterpret_cast<const unsigned*>(pi + u * 32);
        }
    }
    // pv, pi: the lane's first entry; lengths are even
    __device__ __forceinline__ void load(const VT* __restrict__ pv, const uint16_t* __restrict__ pi, int q, int len) {
        pv += q * 32;
        pi += q * 32;
        if (q + B <= len) {
#pragma unroll
            for (int u = 0; u < B; ++u) load_at(pv, pi, u);
        } else {
#pragma unroll
            for (int u = 0; u < B; ++u)
                if (q + (u & ~1) < len) load_at(pv, pi, u);
        }
    }
    template <int NI>
    __device__ __forceinline__ void add_at(int u, const VT* __restrict__ g, VT (&s)[NI]) const {
        const unsigned idx = W == 1 ? i[u] : ((u & 1) ? i[u / 2] >> 16 : i[u / 2] & 0xFFFFu);
        VT t[NI];
        ld_group<VT, NI>(g, idx, t);
#pragma unroll
        for (int k = 0; k < NI; ++k) s[k] += v[u] * t[k];
    }
    // s[k] += entry * g[NI index + k], in entry order
    template <int NI>
    __device__ __forceinline__ void add(int q, int len, const VT* __restrict__ g, VT (&s)[NI]) const {
        if (q + B <= len) {
#pragma unroll
            for (int u = 0; u < B; ++u) add_at<NI>(u, g, s);
        } else {
#pragma unroll
            for (int u = 0; u < B; u += 2) {
                if (q + u >= len) break;
                add_at<NI>(u, g, s);
                add_at<NI>(u + 1, g, s);
            }
        }
    }
};

// One instance of a group: what the iterations need of it, in shared memory.
template <typename MT>
struct alignas(16) GroupInst {
    MT par[2][4];  // tau, sigma and the Halpern weights wk, wa of the even / odd iterations
    long long xo, yo, xp, yp;  // offsets of its vectors and of its column / row records
    int inst;                  // -1: an empty slot of the last group
    int stat;                  // this iteration gives its restart reference residual (1) or is its check (2)
};

// Parameters of an instance's next iteration (one thread per instance).
template <typename MT>
__device__ __forceinline__ void group_params(GroupInst<MT>& g, const InstCtrl& sc, int slot, double eta) {
    g.par[slot][0] = (MT)(eta / sc.omega);
    g.par[slot][1] = (MT)(eta * sc.omega);
    g.par[slot][2] = (MT)((sc.k + 1.0) / (sc.k + 2.0));
    g.par[slot][3] = (MT)(1.0 / (sc.k + 2.0));
}

// Iteration (counted within this launch, from `it` on) of the next reference residual or
// check of any live instance; INT_MAX when none is live.
template <typename MT, int NI>
__device__ __forceinline__ int group_next_stat(const GroupInst<MT>* gi, const InstCtrl* sc, int it, int K) {
    int nx = INT_MAX;
#pragma unroll
    for (int k = 0; k < NI; ++k)
        if (gi[k].inst >= 0 && !sc[k].done) nx = min(nx, sc[k].first ? it : it + (K - 1) - (int)(sc[k].total % K));
    return nx;
}

// The matrix a CTA iterates on.  Dynamic shared memory holds the slice table (column slices,
// then row slices), the interleaved dual iterates ys and the extrapolated primal points xh;
// they are addressed from the array itself, by offsets, so that every access is known to be
// to shared memory.
struct GroupView {
    int m, n, ncs, nrs;
    int ys_off, xh_off;  // bytes
    int nlc, nlr;        // long column / row slices (they come first)
    int64_t ro, co;
    double eta;
};
// Bytes of the per-instance blocks in front of the slice table.
template <typename MT>
__host__ __device__ constexpr int group_head(int ni) {
    return (int)((ni * (sizeof(GroupInst<MT>) + sizeof(InstCtrl)) + 15) & ~(size_t)15);
}
template <typename T>
__device__ __forceinline__ T* smem_at(int off) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    return reinterpret_cast<T*>(smem_raw + off);
}

// x of the next iteration from this one's extrapolation h = 2 T(x) - x (reflection 1):
// wk h + wa anchor.
template <typename MT>
__device__ __forceinline__ MT halpern_point(MT wk, MT h, MT wa, MT anchor) {
    if constexpr (sizeof(MT) == 4) return __fmaf_rn(wk, h, __fmul_rn(wa, anchor));
    else return __fma_rn(wk, h, __dmul_rn(wa, anchor));
}

// What a plain iteration reads of the launch's arguments, passed by value.
template <typename MT>
struct IterPtrs {
    const MT *c_ev, *r_ev, *colp, *rowp;
    const uint16_t *c_eidx, *r_eidx;
    const BArgs* a;  // everything else (long slices, general iterations)
    MT rho, one_rho;
    bool anchors;  // re-centred iterates restart at 0: no anchors
};

// The slices with rows (columns) longer than kLongSlice in a plain iteration: their rows are
// dealt to all warps of the CTA, each summed by a whole warp over the CSR copy, so a dense
// row stalls neither its slice nor one warp.  Out of line and outside the slice loop, which
// then holds no call.
template <typename MT, int NI, bool PRIMAL>
__device__ __noinline__ void long_slices(const IterPtrs<MT> ip, int slot, const GroupView gv) {
    const BArgs& a = *ip.a;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    const GroupInst<MT>* gi = smem_at<GroupInst<MT>>(0);
    MT *ys = smem_at<MT>(gv.ys_off), *xh = smem_at<MT>(gv.xh_off);
    const int rows = PRIMAL ? min(gv.n, gv.nlc << 5) : min(gv.m, gv.nlr << 5);
#pragma unroll 1
    for (int i = warp; i < rows; i += nwarps) {
        MT s[NI], v[NI];
        if (PRIMAL)
            long_row_group<MT, NI>((const MT*)a.stv, a.t_colidx, a.t_rowptr[gv.co + i], a.t_rowptr[gv.co + i + 1], gv.ro,
                                   ys, lane, s);
        else
            long_row_group<MT, NI>((const MT*)a.sv, a.colidx, a.rowptr[gv.ro + i], a.rowptr[gv.ro + i + 1], gv.co, xh,
                                   lane, s);
        if (lane != 0) continue;
        ld_group<MT, NI>(PRIMAL ? xh : ys, i, v);
#pragma unroll
        for (int k = 0; k < NI; ++k) {
            const MT* par = gi[k].par[slot];
            if (PRIMAL) {
                const MT* q = ip.colp + gi[k].xp + col_rec(i);
                const MT x0 = halpern_point<MT>(gi[k].par[slot ^ 1][2], v[k], gi[k].par[slot ^ 1][3],
                                                ip.anchors ? q[96] : (MT)0);
                v[k] = (MT)2 * clampT(x0 - par[0] * (q[0] + s[k]), q[32], q[64]) - x0;
            } else {
                const MT* q = ip.rowp + gi[k].yp + row_rec(i);
                MT yt = v[k] + par[1] * (s[k] - q[0]);
                if (yt < q[32]) yt = q[32];
                v[k] = halpern_point<MT>(par[2], ip.one_rho * yt - ip.rho * v[k], par[3], ip.anchors ? q[64] : (MT)0);
            }
        }
        st_group<MT, NI>(PRIMAL ? xh : ys, i, v);
    }
}

// One PDHG iteration of a group of NI instances of one matrix.
// GEN = false: a plain iteration with reflection 1.  x is not in memory: it is
// wk h + wa anchor of the previous iteration's xh, which is still in shared memory, so a
// column costs its record (c, l, u; the anchor only where it is not 0) and no more.
// GEN = true: any iteration.  ldx / stx: x is read from / written to memory (around a
// check, which overwrites xh, at the ends of a launch, and always when the reflection is
// not 1); gi[].stat names the instances whose residual sums are taken (into acc, per warp)
// and whose T(z) and displacement are stored for the check.
template <typename MT, int W, int NI, int B, bool GEN, bool PIPE, bool LONG>
__device__ __forceinline__ void iteration_body(const IterPtrs<MT> ip, int slot, const GroupView gv,
                                               double (*acc)[NI][4], bool ldx, bool stx) {
    const BArgs& a = *ip.a;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;
    const MT rho = ip.rho, one_rho = ip.one_rho;
    const bool rays = GEN && a.eps_inf > 0.0;
    GroupInst<MT>* gi = smem_at<GroupInst<MT>>(0);
    InstCtrl* sc = smem_at<InstCtrl>(NI * (int)sizeof(GroupInst<MT>));
    const int2* tab = smem_at<const int2>(group_head<MT>(NI));
    MT* ys = smem_at<MT>(gv.ys_off);
    MT* xh = smem_at<MT>(gv.xh_off);
    double st[NI][2];
    if (GEN)
#pragma unroll
        for (int k = 0; k < NI; ++k) st[k][0] = st[k][1] = 0.0;
    if (LONG && gv.nlc > 0) long_slices<MT, NI, true>(ip, slot, gv);
    // ---- primal phase: one thread per column, gathers y.  Slices (longest first) are dealt
    // to the warps boustrophedon-wise, which evens out their work before the barrier.
    {
        const MT* ev = ip.c_ev + W * lane;
        const uint16_t* ei = ip.c_eidx + W * lane;
        const MT* rec[NI];
        MT tau[NI], wk[NI], wa[NI];
#pragma unroll
        for (int k = 0; k < NI; ++k) {
            rec[k] = ip.colp + gi[k].xp + lane;
            tau[k] = gi[k].par[slot][0];
            wk[k] = gi[k].par[slot ^ 1][2];  // of the previous iteration
            wa[k] = gi[k].par[slot ^ 1][3];
        }
        EllBatch<MT, W, B> cur, nxt;
        int r = 0, sl = warp;
        if (LONG)
            while (sl < gv.nlc) sl = snake_slice(++r, warp, nwarps);  // done by long_slices
        int2 t = sl < gv.ncs ? tab[sl] : make_int2(0, 0);
        if (PIPE) cur.load(ev + t.x, ei + t.x, 0, t.y);
#pragma unroll 1
        for (; sl < gv.ncs; ++r) {
            const int j = (sl << 5) + lane;
            const bool valid = j < gv.n;
            MT c[NI], l[NI], u[NI], an[NI];
#pragma unroll
            for (int k = 0; k < NI; ++k) {  // records are padded to whole slices
                const MT* q = rec[k] + (size_t)sl * 128;
                c[k] = q[0];
                l[k] = q[32];
                u[k] = q[64];
                an[k] = ip.anchors ? q[96] : (MT)0;
            }
            const int sl2 = snake_slice(r + 1, warp, nwarps);
            const int2 t2 = sl2 < gv.ncs ? tab[sl2] : make_int2(0, 0);
            MT s[NI];
#pragma unroll
            for (int k = 0; k < NI; ++k) s[k] = (MT)0;
            if (!GEN || t.y <= kLongSlice) {
                int q = 0;
                if (PIPE) {
#pragma unroll 1
                    for (; q + B < t.y; q += B) {
                        nxt.load(ev + t.x, ei + t.x, q + B, t.y);
                        cur.template add<NI>(q, t.y, ys, s);
                        cur = nxt;
                    }
                    nxt.load(ev + t2.x, ei + t2.x, 0, t2.y);
                    cur.template add<NI>(q, t.y, ys, s);
                } else {
#pragma unroll 1
                    for (; q < t.y; q += B) {
                        cur.load(ev + t.x, ei + t.x, q, t.y);
                        cur.template add<NI>(q, t.y, ys, s);
                    }
                }
            } else {
                long_slice_group<MT, NI>((const MT*)a.stv, a.t_rowptr, a.t_colidx, gv.co + (sl << 5),
                                         min(32, gv.n - (sl << 5)), gv.ro, ys, lane, s);
            }
            if (valid) {
                MT h[NI];
                if (!GEN || !ldx) ld_group<MT, NI>(xh, j, h);
#pragma unroll
                for (int k = 0; k < NI; ++k) {
                    const MT x0 = (GEN && ldx) ? ((const MT*)a.x)[gi[k].xo + j]
                                               : halpern_point<MT>(wk[k], h[k], wa[k], an[k]);
                    const MT xt = clampT(x0 - tau[k] * (c[k] + s[k]), l[k], u[k]);
                    h[k] = (MT)2 * xt - x0;
                    if (GEN) {
                        const int stat = gi[k].stat;
                        if (stx && gi[k].inst >= 0 && !sc[k].done)
                            ((MT*)a.x)[gi[k].xo + j] = halpern_point<MT>(gi[k].par[slot][2], one_rho * xt - rho * x0,
                                                                         gi[k].par[slot][3], an[k]);
                        if (stat) {
                            const double d = (double)x0 - (double)xt;
                            st[k][0] += d * d;
                        }
                        if (stat == 2) {
                            ((MT*)a.xt)[gi[k].xo + j] = xt;
                            if (rays) ((MT*)a.dx)[gi[k].xo + j] = xt - x0;
                            const double e = (double)xt - (double)an[k];
                            st[k][1] += e * e;
                        }
                    }
                }
                st_group<MT, NI>(xh, j, h);
            }
            if (PIPE) cur = nxt;
            t = t2;
            sl = sl2;
        }
    }
    if (GEN)
#pragma unroll
        for (int k = 0; k < NI; ++k) {
            st[k][0] = warp_sum(st[k][0]);
            st[k][1] = warp_sum(st[k][1]);
            if (lane == 0) {
                acc[warp][k][0] = st[k][0];
                acc[warp][k][1] = st[k][1];
            }
            st[k][0] = st[k][1] = 0.0;
        }
    __syncthreads();
    if (LONG && gv.nlr > 0) long_slices<MT, NI, false>(ip, slot, gv);
    // ---- dual phase: one thread per row, gathers xh
    {
        const MT* ev = ip.r_ev + W * lane;
        const uint16_t* ei = ip.r_eidx + W * lane;
        const MT* rec[NI];
        MT sigma[NI], wk[NI], wa[NI];
#pragma unroll
        for (int k = 0; k < NI; ++k) {
            rec[k] = ip.rowp + gi[k].yp + lane;
            sigma[k] = gi[k].par[slot][1];
            wk[k] = gi[k].par[slot][2];
            wa[k] = gi[k].par[slot][3];
        }
        // the next iteration's parameters, in the slot whose last reads are behind the barrier
        if (tid < NI && !sc[tid].done) {
            sc[tid].k += 1;
            sc[tid].total += 1;
            group_params<MT>(gi[tid], sc[tid], slot ^ 1, gv.eta);
        }
        EllBatch<MT, W, B> cur, nxt;
        int r = 0, sl = warp;
        if (LONG)
            while (sl < gv.nlr) sl = snake_slice(++r, warp, nwarps);
        int2 t = sl < gv.nrs ? tab[gv.ncs + sl] : make_int2(0, 0);
        if (PIPE) cur.load(ev + t.x, ei + t.x, 0, t.y);
#pragma unroll 1
        for (; sl < gv.nrs; ++r) {
            const int i = (sl << 5) + lane;
            const bool valid = i < gv.m;
            MT b[NI], lo[NI], an[NI];
#pragma unroll
            for (int k = 0; k < NI; ++k) {
                const MT* q = rec[k] + (size_t)sl * 96;
                b[k] = q[0];
                lo[k] = q[32];
                an[k] = ip.anchors ? q[64] : (MT)0;
            }
            const int sl2 = snake_slice(r + 1, warp, nwarps);
            const int2 t2 = sl2 < gv.nrs ? tab[gv.ncs + sl2] : make_int2(0, 0);
            MT s[NI];
#pragma unroll
            for (int k = 0; k < NI; ++k) s[k] = (MT)0;
            if (!GEN || t.y <= kLongSlice) {
                int q = 0;
                if (PIPE) {
#pragma unroll 1
                    for (; q + B < t.y; q += B) {
                        nxt.load(ev + t.x, ei + t.x, q + B, t.y);
                        cur.template add<NI>(q, t.y, xh, s);
                        cur = nxt;
                    }
                    nxt.load(ev + t2.x, ei + t2.x, 0, t2.y);
                    cur.template add<NI>(q, t.y, xh, s);
                } else {
#pragma unroll 1
                    for (; q < t.y; q += B) {
                        cur.load(ev + t.x, ei + t.x, q, t.y);
                        cur.template add<NI>(q, t.y, xh, s);
                    }
                }
            } else {
                long_slice_group<MT, NI>((const MT*)a.sv, a.rowptr, a.colidx, gv.ro + (sl << 5),
                                         min(32, gv.m - (sl << 5)), gv.co, xh, lane, s);
            }
            if (valid) {
                MT y0[NI], h[NI];
                ld_group<MT, NI>(ys, i, y0);
#pragma unroll
                for (int k = 0; k < NI; ++k) {
                    MT yt = y0[k] + sigma[k] * (s[k] - b[k]);
                    if (yt < lo[k]) yt = lo[k];  // NaN stays NaN
                    h[k] = halpern_point<MT>(wk[k], one_rho * yt - rho * y0[k], wa[k], an[k]);
                    if (GEN) {
                        const int stat = gi[k].stat;
                        if (stat) {
                            const double d = (double)y0[k] - (double)yt;
                            st[k][0] += d * d;
                        }
                        if (stat == 2) {
                            ((MT*)a.yt)[gi[k].yo + i] = yt;
                            if (rays) {  // a dual ray candidate keeps y >= 0 on <= rows (lo = -inf on = rows)
                                MT d = yt - y0[k];
                                if (lo[k] != (MT)(-INFINITY) && d < (MT)0) d = (MT)0;
                                ((MT*)a.dy)[gi[k].yo + i] = d;
                            }
                            const double e = (double)yt - (double)an[k];
                            st[k][1] += e * e;
                        }
                    }
                }
                st_group<MT, NI>(ys, i, h);
            }
            if (PIPE) cur = nxt;
            t = t2;
            sl = sl2;
        }
    }
    if (GEN)
#pragma unroll
        for (int k = 0; k < NI; ++k) {
            st[k][0] = warp_sum(st[k][0]);
            st[k][1] = warp_sum(st[k][1]);
            if (lane == 0) {
                acc[warp][k][2] = st[k][0];
                acc[warp][k][3] = st[k][1];
            }
        }
    __syncthreads();
}

// The general one is out of line: its FP64 sums stay out of the plain loop's registers.
template <typename MT, int W, int NI, int B, bool PIPE, bool LONG>
__device__ __forceinline__ void plain_iteration(const IterPtrs<MT> ip, int slot, const GroupView gv) {
    iteration_body<MT, W, NI, B, false, PIPE, LONG>(ip, slot, gv, nullptr, false, false);
}
template <typename MT, int W, int NI, int B>
__device__ __noinline__ void general_iteration(const IterPtrs<MT> ip, int slot, const GroupView gv,
                                               double (*acc)[NI][4], bool ldx, bool stx) {
    iteration_body<MT, W, NI, B, true, false, false>(ip, slot, gv, acc, ldx, stx);
}

// The chunk kernel: a CTA takes NI consecutive entries of the active list at a time and
// iterates them in lockstep for up to `chunk` iterations.  NI = 1 serves any batch.
// NI = 2 or 4 serve a batch whose instances all share one matrix (a parametric family, the
// nodes of a branch-and-bound search): every SELL value and index load feeds NI instances,
// and one vector gather reads the operands of all of them.  Per instance the arithmetic and
// the thread-to-column/row assignment do not depend on NI, so at one CTA size the
// iterates, statuses and iteration counts are the same bit for bit in every form.  An
// instance that finishes leaves its slot idle until the chunk ends; the compaction between
// chunks regroups the survivors.
// MAXT, MINB: the largest CTA size of this instantiation and the CTAs per SM it leaves
// registers for.  PIPE: the next batch of entries is loaded ahead (groups: one CTA per SM,
// 128 registers; a single instance at 64 registers is faster without).  LONG: the batch has
// rows longer than kLongSlice (kept apart because a call in the plain loop costs registers).
//
// Bound: shared-memory wavefronts of the random gathers (16-byte gathers of 4 instances: 8.7
// wavefronts per 32 entries against 4 without conflicts) and the L2 latency in front of
// them.  2,000 x 8,000, 47,984 nonzeros, 1,184 instances, checks every 256 iterations, ns per
// instance-iteration (before: one scalar gather per instance, x and 16-byte records in
// memory): FP32 NI = 1 118 -> 92, NI = 2 103 -> 64, NI = 4 49 (10.6 k of 14.4 k SM cycles are
// L1 wavefronts; L2 hit rate 94 % because the records without x and anchors fit); FP64 NI = 1
// 182 -> 139, NI = 2 160 -> 114.
template <typename MT, int W, int NI, int MAXT, int MINB, bool PIPE, bool LONG>
__global__ void __launch_bounds__(MAXT, MINB) k_batch_chunk(const __grid_constant__ BArgs a, int chunk) {
    constexpr int B = sizeof(MT) == 4 ? 8 : 4;
    constexpr int kWarps = MAXT / 32;
    __shared__ double red[kWarps * 7];
    __shared__ double acc[kWarps][NI][4];
    __shared__ int s_q;
    __shared__ int s_flags[2];  // 0: done, 1: restart
    const int tid = threadIdx.x, nt = blockDim.x, nwarps = nt >> 5;
    MT* yg = (MT*)a.y;
    const int active_count = a.counters[1];
    const bool plain_x = a.rho == 1.0;  // x follows from xh
    GroupInst<MT>* gi = smem_at<GroupInst<MT>>(0);
    InstCtrl* sc = smem_at<InstCtrl>(NI * (int)sizeof(GroupInst<MT>));
    int2* tab = smem_at<int2>(group_head<MT>(NI));
    const IterPtrs<MT> ip{(const MT*)a.c_ev, (const MT*)a.r_ev, (const MT*)a.colp, (const MT*)a.rowp, a.c_eidx,
                          a.r_eidx, &a, (MT)a.rho, (MT)(1.0 + a.rho), !a.recenter};
    GroupView gv;
    int cur_mat = -1;
    while (true) {
        if (tid == 0) s_q = atomicAdd(&a.counters[0], NI);
        __syncthreads();
        const int q = s_q;
        if (q >= active_count) break;
        const int mat = NI > 1 ? 0 : a.inst_mat[a.active[q]];
        if (mat != cur_mat) {
            cur_mat = mat;
            gv.m = a.mat_m[mat];
            gv.n = a.mat_n[mat];
            gv.ro = a.mat_row_off[mat];
            gv.co = a.mat_col_off[mat];
            gv.nrs = (gv.m + 31) >> 5;
            gv.ncs = (gv.n + 31) >> 5;
            gv.eta = a.mat_eta[mat];
            gv.ys_off = group_head<MT>(NI) + (int)sizeof(int2) * slice_tab_len(gv.nrs, gv.ncs);
            gv.xh_off = gv.ys_off + (int)sizeof(MT) * NI * ((gv.m + 3) & ~3);  // at a check: stages max(n, m) elements
            fill_slice_tab(tab, a.c_sptr + a.mat_cs_off[mat], gv.ncs, a.r_sptr + a.mat_rs_off[mat], gv.nrs);
        }
        if (tid < NI) {
            GroupInst<MT>& g = gi[tid];
            const bool real = q + tid < active_count;
            const int inst = a.active[real ? q + tid : q];
            sc[tid] = a.ictrl[inst];
            g.inst = real ? inst : -1;
            g.xo = a.x_off[inst];  // an empty slot reads the first instance's vectors and writes nothing
            g.yo = a.y_off[inst];
            g.xp = a.xp_off[inst];
            g.yp = a.yp_off[inst];
            group_params<MT>(g, sc[tid], 0, gv.eta);
        }
        MT* ys = smem_at<MT>(gv.ys_off);
        __syncthreads();
#pragma unroll
        for (int k = 0; k < NI; ++k)
            for (int i = tid; i < gv.m; i += nt) ys[NI * i + k] = gi[k].inst >= 0 ? yg[gi[k].yo + i] : (MT)0;
        if (LONG) {
            gv.nlc = gv.nlr = 0;
            while (gv.nlc < gv.ncs && tab[gv.nlc].y > kLongSlice) ++gv.nlc;
            while (gv.nlr < gv.nrs && tab[gv.ncs + gv.nlr].y > kLongSlice) ++gv.nlr;
        }
        int next_stat = group_next_stat<MT, NI>(gi, sc, 0, a.K);
        bool ldx = true;
        __syncthreads();
        for (int it = 0; it < chunk && next_stat != INT_MAX; ++it) {
            if (!ldx && plain_x)
                for (const int stop = min(next_stat, chunk - 1); it < stop; ++it)
                    plain_iteration<MT, W, NI, B, PIPE, LONG>(ip, it & 1, gv);
            const int slot = it & 1;
            const bool stats = it == next_stat;
            if (tid < NI) {
                const InstCtrl& c = sc[tid];
                gi[tid].stat = (!stats || gi[tid].inst < 0 || c.done) ? 0 : ((c.total + 1) % a.K == 0 ? 2 : (c.first ? 1 : 0));
            }
            __syncthreads();
            bool check = false;
#pragma unroll
            for (int k = 0; k < NI; ++k) check |= gi[k].stat == 2;
            const bool stx = check || !plain_x || it + 1 == chunk;
            general_iteration<MT, W, NI, B>(ip, slot, gv, acc, ldx, stx);
            ldx = check || !plain_x;
            if (!stats) continue;
            // the sums of every instance, over the warps in order
            if (tid < 4 * NI) {
                double t = 0.0;
                for (int w = 0; w < nwarps; ++w) t += acc[w][tid >> 2][tid & 3];
                acc[0][tid >> 2][tid & 3] = t;
            }
            __syncthreads();
            // ---- per instance: restart reference residual, or the check and its decisions
            for (int k = 0; k < NI; ++k) {
                const int stat = gi[k].stat;
                if (!stat) continue;
                double r_now = 0, dxa = 0, dya = 0;
                const double om = sc[k].omega;
                const long long kk = sc[k].k, total = sc[k].total;
                __syncthreads();  // every thread holds its copy of the instance's state
                if (tid == 0) {
                    r_now = sqrt(om * acc[0][k][0] + acc[0][k][2] / om);
                    if (sc[k].first) {
                        sc[k].r0 = r_now;
                        sc[k].rprev = r_now;
                        sc[k].first = 0;
                    }
                    dxa = sqrt(acc[0][k][1]);
                    dya = sqrt(acc[0][k][3]);
                }
                if (stat == 2) {
                    check_instance<MT, W>(a, gi[k].inst, gv.m, gv.n, gv.ro, gv.co, gi[k].xo, gi[k].yo, total, kk, om,
                                          r_now, dxa, dya, sc[k], s_flags, red, tab, smem_at<MT>(gv.xh_off));
                    __syncthreads();
                    const bool restart = s_flags[1] != 0;
                    if (tid == 0) {
                        if (restart) {
                            sc[k].k = 0;
                            sc[k].first = 1;
                        }
                        group_params<MT>(gi[k], sc[k], slot ^ 1, gv.eta);
                    }
                    if (restart)
                        restart_instance<MT, NI>(a, gv.m, gv.n, gv.ro, gv.co, gi[k].xo, gi[k].yo, gi[k].xp, gi[k].yp,
                                                 ys + k);
                    __syncthreads();
                }
            }
            __syncthreads();
            next_stat = group_next_stat<MT, NI>(gi, sc, it + 1, a.K);
        }
        // store the dual iterates and the control blocks
#pragma unroll
        for (int k = 0; k < NI; ++k)
            if (gi[k].inst >= 0)
                for (int i = tid; i < gv.m; i += nt) yg[gi[k].yo + i] = ys[NI * i + k];
        if (tid < NI && gi[tid].inst >= 0) a.ictrl[gi[tid].inst] = sc[tid];
        __syncthreads();
    }
}

// Order-preserving compaction of the active list (one CTA).
__global__ void k_batch_compact(const InstCtrl* __restrict__ ictrl, const int32_t* __restrict__ in,
                                int32_t* __restrict__ out, int32_t* counters) {
    typedef cub::BlockScan<int, 1024> Scan;
    __shared__ typename Scan::TempStorage tmp;
    __shared__ int base;
    const int count = counters[1];
    if (threadIdx.x == 0) base = 0;
    __syncthreads();
    for (int start = 0; start < count; start += 1024) {
        int idx = start + threadIdx.x;
        int keep = (idx < count && !ictrl[in[idx]].done) ? 1 : 0;
        int pos, tot;
        Scan(tmp).ExclusiveSum(keep, pos, tot);
        if (keep) out[base + pos] = in[idx];
        __syncthreads();
        if (threadIdx.x == 0) base += tot;
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        counters[1] = base;
        counters[0] = 0;
    }
}

// ------------------------------------------------------------------ setup kernels (CTA per matrix, FP64)
__global__ void k_batch_scaling(int nmat, const int32_t* __restrict__ mat_m, const int32_t* __restrict__ mat_n,
                                const int64_t* __restrict__ row_off, const int64_t* __restrict__ col_off,
                                const int32_t* __restrict__ rowptr, const int32_t* __restrict__ colidx,
                                const double* __restrict__ vals, const int32_t* __restrict__ t_rowptr,
                                const int32_t* __restrict__ t_colidx, const double* __restrict__ t_vals,
                                int ruiz_iters, double* __restrict__ dr, double* __restrict__ dc,
                                double* __restrict__ tmp_r, double* __restrict__ tmp_c) {
    for (int k = blockIdx.x; k < nmat; k += gridDim.x) {
        const int m = mat_m[k], n = mat_n[k];
        const int64_t ro = row_off[k], co = col_off[k];
        for (int i = threadIdx.x; i < m; i += blockDim.x) dr[ro + i] = 1.0;
        for (int j = threadIdx.x; j < n; j += blockDim.x) dc[co + j] = 1.0;
        __syncthreads();
        for (int pass = 0; pass <= ruiz_iters; ++pass) {
            const bool pc = pass == ruiz_iters;  // last pass: Pock-Chambolle sums
            for (int i = threadIdx.x; i < m; i += blockDim.x) {
                double acc = 0.0, di = dr[ro + i];
                for (int e = rowptr[ro + i]; e < rowptr[ro + i + 1]; ++e) {
                    double v = fabs(vals[e]) * di * dc[colidx[e]];
                    acc = pc ? acc + v : fmax(acc, v);
                }
                tmp_r[ro + i] = acc;
            }
            for (int j = threadIdx.x; j < n; j += blockDim.x) {
                double acc = 0.0, dj = dc[co + j];
                for (int e = t_rowptr[co + j]; e < t_rowptr[co + j + 1]; ++e) {
                    double v = fabs(t_vals[e]) * dj * dr[t_colidx[e]];
                    acc = pc ? acc + v : fmax(acc, v);
                }
                tmp_c[co + j] = acc;
            }
            __syncthreads();
            for (int i = threadIdx.x; i < m; i += blockDim.x)
                if (tmp_r[ro + i] > 0.0) dr[ro + i] /= sqrt(tmp_r[ro + i]);
            for (int j = threadIdx.x; j < n; j += blockDim.x)
                if (tmp_c[co + j] > 0.0) dc[co + j] /= sqrt(tmp_c[co + j]);
            __syncthreads();
        }
    }
}

__global__ void k_batch_scale_vals(int64_t tot_m, int64_t tot_n, const int32_t* __restrict__ rowptr,
                                   const int32_t* __restrict__ colidx, const double* __restrict__ vals,
                                   const int32_t* __restrict__ t_rowptr, const int32_t* __restrict__ t_colidx,
                                   const double* __restrict__ t_vals, const double* __restrict__ dr,
                                   const double* __restrict__ dc, double* sv64, float* sv32, double* stv64,
                                   float* stv32) {
    int64_t tid = blockIdx.x * (int64_t)blockDim.x + threadIdx.x, st = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = tid; i < tot_m; i += st) {
        double di = dr[i];
        for (int e = rowptr[i]; e < rowptr[i + 1]; ++e) {
            double v = vals[e] * di * dc[colidx[e]];
            sv64[e] = v;
            sv32[e] = (float)v;
        }
    }
    for (int64_t j = tid; j < tot_n; j += st) {
        double dj = dc[j];
        for (int e = t_rowptr[j]; e < t_rowptr[j + 1]; ++e) {
            double v = t_vals[e] * dj * dr[t_colidx[e]];
            stv64[e] = v;
            stv32[e] = (float)v;
        }
    }
}

// Start entry j of the power iteration: in (0.5, 1.5), splitmix64 of j.
__device__ __forceinline__ double power_start(int j) {
    unsigned long long z = (unsigned long long)j * 0x9E3779B97F4A7C15ull + 0x1234567ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    z ^= z >> 31;
    return 0.5 + (double)(z >> 11) * (1.0 / 9007199254740992.0);
}

// sigma_max(A_s)^2 per matrix by power iteration (stops at rel change 1e-7).  Two kernels
// share the matrices: this one takes one CTA each, all of them or (SMALL) those of fewer than
// kPowerCluster entries -- a batch of many matrices fills the GPU that way.
template <bool SMALL>
__global__ void k_batch_power(int nmat, const int32_t* __restrict__ mat_m, const int32_t* __restrict__ mat_n,
                              const int64_t* __restrict__ row_off, const int64_t* __restrict__ col_off,
                              const int32_t* __restrict__ rowptr, const int32_t* __restrict__ colidx,
                              const double* __restrict__ sv64, const int32_t* __restrict__ t_rowptr,
                              const int32_t* __restrict__ t_colidx, const double* __restrict__ stv64, double* pv,
                              double* pu, double safety, double* __restrict__ eta_out) {
    __shared__ double red[32];
    __shared__ double s_norm, s_prev;
    __shared__ int s_stop;
    for (int k = blockIdx.x; k < nmat; k += gridDim.x) {
        const int m = mat_m[k], n = mat_n[k];
        const int64_t ro = row_off[k], co = col_off[k];
        if (SMALL && rowptr[ro + m] - rowptr[ro] >= kPowerCluster) continue;
        double part = 0.0;
        for (int j = threadIdx.x; j < n; j += blockDim.x) {
            const double v = power_start(j);
            pv[co + j] = v;
            part += v * v;
        }
        double vv[1] = {part};
        block_sums<1>(vv, red);
        if (threadIdx.x == 0) {
            s_norm = sqrt(vv[0]);
            s_prev = 0.0;
            s_stop = 0;
        }
        __syncthreads();
        for (int t = 0; t < 1000 && !s_stop; ++t) {
            const double inv = 1.0 / s_norm;
            for (int i = threadIdx.x; i < m; i += blockDim.x) {
                double s = 0.0;
                for (int e = rowptr[ro + i]; e < rowptr[ro + i + 1]; ++e) s += sv64[e] * pv[colidx[e]];
                pu[ro + i] = s * inv;
            }
            __syncthreads();
            double p2 = 0.0;
            for (int j = threadIdx.x; j < n; j += blockDim.x) {
                double s = 0.0;
                for (int e = t_rowptr[co + j]; e < t_rowptr[co + j + 1]; ++e) s += stv64[e] * pu[t_colidx[e]];
                pv[co + j] = s;
                p2 += s * s;
            }
            double w[1] = {p2};
            block_sums<1>(w, red);
            if (threadIdx.x == 0) {
                double nn = sqrt(w[0]);
                if (nn <= 0.0 || fabs(nn - s_prev) <= 1e-7 * nn) s_stop = 1;
                s_prev = nn;
                s_norm = nn > 0.0 ? nn : 1.0;
            }
            __syncthreads();
        }
        if (threadIdx.x == 0) {
            double sig = sqrt(fmax(s_prev, 0.0));
            eta_out[k] = sig > 0.0 ? safety / sig : 1.0;
        }
        __syncthreads();
    }
}

// Sum of one row by a whole warp over the CSR arrays (`off` localises the index), eight entries a lane
// in flight; every lane returns it.  L2: the vector is read past L1.
template <bool L2>
__device__ __noinline__ double power_row(const double* __restrict__ val, const int32_t* __restrict__ idx, int64_t e, int64_t e1,
                                         int64_t off, const double* g, int lane) {
    constexpr int U = 8;
    double s = 0.0;
    for (e += lane; e < e1; e += 32 * U) {
        double v[U], a[U];
        int c[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const bool h = e + 32 * u < e1;
            v[u] = h ? val[e + 32 * u] : 0.0;
            c[u] = h ? (int)(idx[e + 32 * u] - off) : -1;
        }
#pragma unroll
        for (int u = 0; u < U; ++u) a[u] = c[u] < 0 ? 0.0 : (L2 ? __ldcg(g + c[u]) : g[c[u]]);
#pragma unroll
        for (int u = 0; u < U; ++u) s += v[u] * a[u];
    }
    return __shfl_sync(0xffffffffu, warp_sum(s), 0);
}

// The matrices of at least kPowerCluster entries, where a batch has few of them: a cluster of
// kPowerCtas CTAs each.  One CTA's step is a chain of dependent loads over its whole share of
// rows and columns (41 us a step on a 2,000 x 8,000 matrix of 47,984 entries, up to 1,000
// steps); eight CTAs walk an eighth of it.  Rows and columns are summed over the FP64 SELL
// copies (entry order W = 1), one lane each, in the order of the one-CTA kernel; the rows of slices of more
// than kLongSlice entries are dealt to all warps of the cluster instead, a whole warp each over the CSR
// arrays (upload of 2,000 x 8,000 with one full row: 1,357 ms with a lane on it, 526 with one thread of
// a single CTA, now 41).  SM: every CTA
// holds whole copies of both vectors in shared memory, into which the owners post
// (ClusterPost), and its share of the matrix where `room` bytes are left for it (4.6 us a
// step on that matrix); otherwise the vectors lie in L2 (loads bypass L1, which other CTAs'
// stores do not reach) and a cluster barrier ends each half step (9 us).  The `nbig`
// matrices to take (`bigs`) are dealt to the kernel's clusters in turn: by their place among all
// matrices, 36 large ones of 648 that lay 18 apart met on two clusters (upload 99 ms with one
// CTA each, 239 ms; now 65).  Every CTA of a cluster makes the same decisions from the same sums.  Every step ends with a cluster barrier, so no thread falls a phase behind.
template <bool SM>
__global__ void __cluster_dims__(kPowerCtas, 1, 1) __launch_bounds__(512)
k_batch_power_cluster(int nbig, const int32_t* __restrict__ bigs, const int32_t* __restrict__ mat_m,
                      const int32_t* __restrict__ mat_n,
                      const int64_t* __restrict__ row_off, const int64_t* __restrict__ col_off,
                      const int32_t* __restrict__ rowptr, const int32_t* __restrict__ colidx,
                      const double* __restrict__ sv64, const int32_t* __restrict__ t_rowptr,
                      const int32_t* __restrict__ t_colidx, const double* __restrict__ stv64,
                      const int64_t* __restrict__ rs_off, const int64_t* __restrict__ cs_off,
                      const int64_t* __restrict__ r_sptr, const int64_t* __restrict__ c_sptr, const uint16_t* __restrict__ r_eidx,
                      const uint16_t* __restrict__ c_eidx, const double* __restrict__ r_ev,
                      const double* __restrict__ c_ev, double* pv, double* pu, double safety, int max_m, int max_n,
                      int room, int* __restrict__ wait_failed, double* __restrict__ eta_out) {
    namespace cg = cooperative_groups;
    cg::cluster_group cl = cg::this_cluster();
    __shared__ double red[32];
    __shared__ double part[2];  // this CTA's share of ||v||^2, by step parity
    __shared__ uint64_t bar[2];  // arrivals of v, of u
    __shared__ int s_fits;
    __shared__ int s_long[2];  // slices of more than kLongSlice entries a lane (they come first): columns, rows
    double* vs = smem_at<double>(0);
    double* us = smem_at<double>(8 * max_n);
    int2* tab = smem_at<int2>(8 * (max_n + max_m));  // per owned slice {first entry, entries per lane}
    const int tabs = (((max_n + 31) >> 5) + kPowerCtas - 1) / kPowerCtas + (((max_m + 31) >> 5) + kPowerCtas - 1) / kPowerCtas;
    double* sv = smem_at<double>(8 * (max_n + max_m + tabs));
    const int rank = (int)cl.block_rank(), tid = threadIdx.x;
    const int lane = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5;
    const ClusterPeers<SM ? kPowerCtas : 1> peers(smem_at<double>(0));
    const ClusterPost<double, SM ? kPowerCtas : 1> vp(peers, vs, bar), up(peers, us, bar + 1);
    uint32_t parity = 0;
    bool ok = true;
    if (SM && tid == 0) {
        tx_init(bar);
        tx_init(bar + 1);
    }
    // the whole cluster's ||v||^2 from the CTAs' shares, in rank order
    auto total = [&](double share, int slot) -> double {
        double w[1] = {share};
        block_sums<1>(w, red);
        if (threadIdx.x == 0) part[slot] = w[0];
        cl.sync();
        double t = 0.0;
        for (int r = 0; r < kPowerCtas; ++r) t += *cl.map_shared_rank(&part[slot], r);
        return t;
    };
    // entries of one row (column) of a slice, 8 in flight
    auto dot = [&](const double* v, const uint16_t* ix, int len, auto g) -> double {
        double s = 0.0;
        for (int q = 0; q < len; q += 8) {
            double vv[8];
            unsigned ii[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const bool h = q + u < len;
                vv[u] = h ? v[(q + u) * 32] : 0.0;
                ii[u] = h ? (unsigned)ix[(q + u) * 32] : 0u;
            }
            double gg[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) gg[u] = q + u < len ? g(ii[u]) : 0.0;
#pragma unroll
            for (int u = 0; u < 8; ++u)
                if (q + u < len) s += vv[u] * gg[u];
        }
        return s;
    };
    for (int q = blockIdx.x / kPowerCtas; q < nbig; q += gridDim.x / kPowerCtas) {
        const int k = bigs[q];
        const int m = mat_m[k], n = mat_n[k];
        const int64_t ro = row_off[k], co = col_off[k];
        const int64_t* rsp = r_sptr + rs_off[k];
        const int64_t* csp = c_sptr + cs_off[k];
        const int nrs = (m + 31) >> 5, ncs = (n + 31) >> 5;
        // this CTA's slices: rank, rank + kPowerCtas, ...; those of the columns first
        const int ncl = (ncs - rank + kPowerCtas - 1) / kPowerCtas, nrl = (nrs - rank + kPowerCtas - 1) / kPowerCtas;
        if (tid < 2) s_long[tid] = 0;
        __syncthreads();
        for (int sl = tid; sl < ncs + nrs; sl += blockDim.x) {
            const int64_t* o = sl < ncs ? csp + sl : rsp + (sl - ncs);
            if (o[1] - o[0] > 32 * kLongSlice) atomicAdd(&s_long[sl < ncs ? 0 : 1], 1);
        }
        __syncthreads();
        const int lcs = s_long[0], lrs = s_long[1];
        bool fits = false;
        uint16_t* si = nullptr;
        if constexpr (SM) {
            for (int l = tid; l < ncl + nrl; l += blockDim.x) {
                const int64_t* o = l < ncl ? csp + rank + kPowerCtas * l : rsp + rank + kPowerCtas * (l - ncl);
                const bool is_long = l < ncl ? rank + kPowerCtas * l < lcs : rank + kPowerCtas * (l - ncl) < lrs;
                tab[l] = make_int2(0, is_long ? 0 : (int)((o[1] - o[0]) >> 5));
            }
            __syncthreads();
            if (tid == 0) {
                int64_t e = 0;
                for (int l = 0; l < ncl + nrl; ++l) {
                    tab[l].x = (int)min(e, (int64_t)INT_MAX);
                    e += 32 * (int64_t)tab[l].y;
                }
                s_fits = 10 * e <= room ? (int)e : -1;
            }
            __syncthreads();
            fits = s_fits >= 0;
            if (fits) {
                si = reinterpret_cast<uint16_t*>(sv + s_fits);
                for (int l = warp; l < ncl + nrl; l += nw) {
                    const int2 t = tab[l];
                    const int64_t p0 = l < ncl ? csp[rank + kPowerCtas * l] : rsp[rank + kPowerCtas * (l - ncl)];
                    const double* v = (l < ncl ? c_ev : r_ev) + p0;
                    const uint16_t* ix = (l < ncl ? c_eidx : r_eidx) + p0;
                    for (int e = lane; e < 32 * t.y; e += 32) {
                        sv[t.x + e] = v[e];
                        si[t.x + e] = ix[e];
                    }
                }
            }
            for (int j = tid; j < n; j += blockDim.x) vs[j] = power_start(j);
        }
        double sum = 0.0;
        for (int l = warp; l < ncl; l += nw) {
            const int j = (rank + kPowerCtas * l) * 32 + lane;
            if (j < n) {
                const double v = power_start(j);
                if (!SM) pv[co + j] = v;
                sum += v * v;
            }
        }
        // the sum of slice l's rows (columns) over the gathered vector
        auto slice = [&](int l, int64_t p0, int64_t p1, const double* gv, const uint16_t* gi, auto g) -> double {
            if (SM && fits) {
                const int2 t = tab[l];
                return dot(sv + t.x + lane, si + t.x + lane, t.y, g);
            }
            return dot(gv + p0 + lane, gi + p0 + lane, (int)((p1 - p0) >> 5), g);
        };
        double norm = sqrt(total(sum, 0)), prev = 0.0;
        for (int t = 0; t < 1000; ++t) {
            const double inv = 1.0 / norm;
            if (SM && tid == 0) {
                tx_expect(bar, 8u * (uint32_t)n);
                tx_expect(bar + 1, 8u * (uint32_t)m);
            }
            for (int i = rank + kPowerCtas * warp; i < min(m, 32 * lrs); i += kPowerCtas * nw) {
                const double s = power_row<!SM>(sv64, colidx, rowptr[ro + i], rowptr[ro + i + 1], co, SM ? vs : pv + co, lane);
                if (lane == 0) {
                    if constexpr (SM) up.store(peers, i, s * inv);
                    else pu[ro + i] = s * inv;
                }
            }
            for (int l = warp; l < nrl; l += nw) {
                const int sl = rank + kPowerCtas * l, i = (sl << 5) + lane;
                if (sl < lrs) continue;
                const double s = slice(ncl + l, rsp[sl], rsp[sl + 1], r_ev, r_eidx,
                                       [&](unsigned c) { return SM ? vs[c] : __ldcg(pv + co + c); });
                if (i < m) {
                    if constexpr (SM) up.store(peers, i, s * inv);
                    else pu[ro + i] = s * inv;
                }
            }
            if constexpr (SM) {
                if (ok) ok = tx_wait(bar + 1, parity);
            } else {
                cl.sync();
            }
            sum = 0.0;
            for (int j = rank + kPowerCtas * warp; j < min(n, 32 * lcs); j += kPowerCtas * nw) {
                const double s = power_row<!SM>(stv64, t_colidx, t_rowptr[co + j], t_rowptr[co + j + 1], ro, SM ? us : pu + ro, lane);
                if (lane == 0) {
                    if constexpr (SM) vp.store(peers, j, s);
                    else pv[co + j] = s;
                    sum += s * s;
                }
            }
            for (int l = warp; l < ncl; l += nw) {
                const int sl = rank + kPowerCtas * l, j = (sl << 5) + lane;
                if (sl < lcs) continue;
                const double s = slice(l, csp[sl], csp[sl + 1], c_ev, c_eidx,
                                       [&](unsigned c) { return SM ? us[c] : __ldcg(pu + ro + c); });
                if (j < n) {
                    if constexpr (SM) vp.store(peers, j, s);
                    else pv[co + j] = s;
                    sum += s * s;
                }
            }
            const double nn = sqrt(total(sum, (t + 1) & 1));
            if constexpr (SM) {
                if (ok) ok = tx_wait(bar, parity);
                parity ^= 1;
                __syncthreads();  // the copies are whole for every warp before tid 0 opens the next phases
            }
            const bool stop = nn <= 0.0 || fabs(nn - prev) <= 1e-7 * nn;
            prev = nn;
            norm = nn > 0.0 ? nn : 1.0;
            if (stop) break;
        }
        if (!ok) {
            *wait_failed = 1;
            __nanosleep(1000000);  // late elements land before the CTA they go to leaves
        }
        if (rank == 0 && threadIdx.x == 0) {
            const double sig = sqrt(fmax(prev, 0.0));
            eta_out[k] = sig > 0.0 ? safety / sig : 1.0;
        }
        cl.sync();  // every CTA has read the shares before the next matrix writes them
    }
    cl.sync();  // no CTA leaves while another may still read its shares
}

// SELL-32 copy of one orientation, CTA per matrix: every lane slot of every slice
// (rows past the matrix end and entries past a row's end are zero padding with
// local index 0), in the W = 1 or W = 2 (pairs) order of ell_dot.  ptr / idx / v64 /
// v32 are the CSR of that orientation in global numbering; `other_off` localises its
// indices.
__global__ void k_fill_ell(int W, int nmat, const int32_t* __restrict__ dim, const int64_t* __restrict__ off,
                           const int64_t* __restrict__ other_off, const int64_t* __restrict__ s_off,
                           const int64_t* __restrict__ sptr, const int32_t* __restrict__ ptr,
                           const int32_t* __restrict__ idx, const double* __restrict__ v64,
                           const float* __restrict__ v32, uint16_t* __restrict__ eidx, double* __restrict__ ev64,
                           float* __restrict__ ev32) {
    for (int k = blockIdx.x; k < nmat; k += gridDim.x) {
        const int d = dim[k];
        const int padded = (d + 31) & ~31;
        const int64_t base = off[k], ob = other_off[k];
        const int64_t* sp = sptr + s_off[k];
        for (int li = threadIdx.x; li < padded; li += blockDim.x) {
            const int s = li >> 5, lane = li & 31;
            const int64_t p0 = sp[s];
            const int len = (int)((sp[s + 1] - p0) >> 5);
            int e = 0, e1 = 0;
            if (li < d) {
                e = ptr[base + li];
                e1 = ptr[base + li + 1];
            }
            for (int q = 0; q < len; ++q) {
                const int64_t pos = W == 1 ? p0 + 32 * (int64_t)q + lane : p0 + 64 * (int64_t)(q >> 1) + 2 * lane + (q & 1);
                if (e + q < e1) {
                    eidx[pos] = (uint16_t)(idx[e + q] - ob);
                    ev64[pos] = v64[e + q];
                    ev32[pos] = v32[e + q];
                } else {
                    eidx[pos] = 0;
                    ev64[pos] = 0.0;
                    ev32[pos] = 0.0f;
                }
            }
        }
    }
}

// Per-instance b, c, l, u, row kinds from external to internal order (CTA per instance).
__global__ void k_permute_inst(int count, const int32_t* __restrict__ inst_mat, const int32_t* __restrict__ mat_m,
                               const int32_t* __restrict__ mat_n, const int64_t* __restrict__ row_off,
                               const int64_t* __restrict__ col_off, const int64_t* __restrict__ x_off,
                               const int64_t* __restrict__ y_off, const int32_t* __restrict__ r_ext,
                               const int32_t* __restrict__ c_ext, const double* __restrict__ sb,
                               const double* __restrict__ sc, const double* __restrict__ sl,
                               const double* __restrict__ su, const uint8_t* __restrict__ seq, double* __restrict__ b,
                               double* __restrict__ c, double* __restrict__ lb, double* __restrict__ ub,
                               uint8_t* __restrict__ is_eq) {
    for (int inst = blockIdx.x; inst < count; inst += gridDim.x) {
        const int k = inst_mat[inst];
        const int m = mat_m[k], n = mat_n[k];
        const int64_t ro = row_off[k], co = col_off[k], xo = x_off[inst], yo = y_off[inst];
        for (int j = threadIdx.x; j < n; j += blockDim.x) {
            const int64_t src = xo + c_ext[co + j];
            c[xo + j] = sc[src];
            lb[xo + j] = sl[src];
            ub[xo + j] = su[src];
        }
        for (int i = threadIdx.x; i < m; i += blockDim.x) {
            const int64_t src = yo + r_ext[ro + i];
            b[yo + i] = sb[src];
            is_eq[yo + i] = seq[src];
        }
    }
}

// Per-instance norms, initial point, packed records and control block (CTA per
// instance; all `count` instances, or those named by `list`).  Warm starts arrive
// in external order.  With re-centring the initial
// point (warm start, else the bound projection of 0) becomes the first FP64
// centre and the iterates start at 0.
template <typename MT>
__global__ void k_batch_init(BArgs a, int count, const int32_t* __restrict__ list, const double* __restrict__ x0,
                             const double* __restrict__ y0, const double* __restrict__ omega0,
                             const long long* __restrict__ base0) {
    __shared__ double red[32 * 4];
    MT *xg = (MT*)a.x, *xtg = (MT*)a.xt, *yg = (MT*)a.y, *ytg = (MT*)a.yt;
    for (int q = blockIdx.x; q < count; q += gridDim.x) {
        const int inst = list ? list[q] : q;
        const int k = a.inst_mat[inst];
        const int m = a.mat_m[k], n = a.mat_n[k];
        const int64_t ro = a.mat_row_off[k], co = a.mat_col_off[k], xo = a.x_off[inst], yo = a.y_off[inst];
        const int64_t xp = a.xp_off[inst], yp = a.yp_off[inst];
        double acc[4] = {0, 0, 0, 0};  // ||b||^2, ||c||^2, ||b_s||^2, ||c_s||^2
        for (int j = threadIdx.x; j < n; j += blockDim.x) {
            const double d = a.dc[co + j];
            const double cj = a.c[xo + j], lj = a.lb[xo + j], uj = a.ub[xo + j];
            const double v = clampT(x0 ? x0[xo + a.c_ext[co + j]] : 0.0, lj, uj);
            if (a.recenter) {
                a.xbar[xo + j] = v;
                xg[xo + j] = (MT)0;
                xtg[xo + j] = (MT)0;
            } else {
                const MT vs = (MT)(v / d);
                xg[xo + j] = vs;
                xtg[xo + j] = vs;
                MT* p = (MT*)a.colp + xp + col_rec(j);
                p[0] = (MT)(cj * d);
                p[32] = (MT)(lj / d);
                p[64] = (MT)(uj / d);
                p[96] = vs;
            }
            acc[1] += cj * cj;
            acc[3] += (cj * d) * (cj * d);
        }
        for (int i = threadIdx.x; i < m; i += blockDim.x) {
            const double d = a.dr[ro + i];
            const double bi = a.b[yo + i];
            const bool eq = a.is_eq[yo + i] != 0;
            double v = y0 ? y0[yo + a.r_ext[ro + i]] : 0.0;
            if (!eq && v < 0.0) v = 0.0;
            if (a.recenter) {
                a.ybar[yo + i] = v;
                yg[yo + i] = (MT)0;
                ytg[yo + i] = (MT)0;
            } else {
                const MT vs = (MT)(v / d);
                yg[yo + i] = vs;
                ytg[yo + i] = vs;
                MT* r = (MT*)a.rowp + yp + row_rec(i);
                r[0] = (MT)(bi * d);
                r[32] = eq ? (MT)(-INFINITY) : (MT)0;
                r[64] = vs;
            }
            acc[0] += bi * bi;
            acc[2] += (bi * d) * (bi * d);
        }
        block_sums<4>(acc, red);
        if (threadIdx.x == 0) {
            a.bnorm[inst] = sqrt(acc[0]);
            a.cnorm[inst] = sqrt(acc[1]);
            const double bn = sqrt(acc[2]), cn = sqrt(acc[3]);
            InstCtrl s;
            memset(&s, 0, sizeof(s));
            s.omega = (omega0 && omega0[inst] > 0.0) ? omega0[inst] : ((bn > 1e-10 && cn > 1e-10) ? cn / bn : 1.0);
            s.first = 1;
            s.base = base0 ? base0[q] : 0;
            s.status = B2P_STATUS_MAX_ITERATIONS;
            a.ictrl[inst] = s;
        }
        if (a.recenter) {
            __syncthreads();  // the centre of this instance is complete
            rebuild_shifted<MT>(a, m, n, ro, co, xo, yo, xp, yp);
        }
        __syncthreads();
    }
}

// Answers in the original space and external order: x = xbar + dc * xt, y = ybar + dr * yt.
template <typename T>
__global__ void k_batch_unscale(BArgs a, int count, const double* __restrict__ xbar, const double* __restrict__ ybar,
                                double* __restrict__ xo_, double* __restrict__ yo_) {
    const T* xt = (const T*)a.xt;
    const T* yt = (const T*)a.yt;
    for (int inst = blockIdx.x; inst < count; inst += gridDim.x) {
        const int k = a.inst_mat[inst];
        const int m = a.mat_m[k], n = a.mat_n[k];
        const int64_t ro = a.mat_row_off[k], co = a.mat_col_off[k], xo = a.x_off[inst], yo = a.y_off[inst];
        for (int j = threadIdx.x; j < n; j += blockDim.x)
            xo_[xo + a.c_ext[co + j]] = (xbar ? xbar[xo + j] : 0.0) + a.dc[co + j] * (double)xt[xo + j];
        for (int i = threadIdx.x; i < m; i += blockDim.x)
            yo_[yo + a.r_ext[ro + i]] = (ybar ? ybar[yo + i] : 0.0) + a.dr[ro + i] * (double)yt[yo + i];
    }
}

// ------------------------------------------------------------------ host side

// Candidate shapes of the autotuner: CTA sizes, SELL entry orders and instances per CTA
// (more than 1 only when every instance shares one matrix; 4 only in FP32).
// B2P_BATCH_SHAPE="threads,w,ni" pins all three for the whole solve (the chunk length is still
// tuned); a pinned group on a batch of several matrices falls back to one instance per CTA.
struct ShapeChoices {
    std::vector<int> threads{128, 256, 512}, w{1, 2}, ni{1, 2, 4};
    bool pinned = false;
};

ShapeChoices shape_choices(BatchWork* w) {
    ShapeChoices c;
    const bool can_pair = w->nmat == 1 && w->count > 1;
    if (!can_pair) c.ni = {1};
    const char* e = std::getenv("B2P_BATCH_SHAPE");
    int th = 0, ww = 0, ni = 0;
    if (e && std::sscanf(e, "%d,%d,%d", &th, &ww, &ni) == 3 && (th == 128 || th == 256 || th == 512 || th == 1024) &&
        (ww == 1 || ww == 2) && (ni == 1 || ni == 2 || ni == 4)) {
        c.threads = {th};
        c.w = {ww};
        c.ni = {can_pair ? ni : 1};
        c.pinned = true;
    }
    return c;
}

std::string cache_path() {
    const char* p = std::getenv("B2P_AUTOTUNE_CACHE");
    if (p && *p) return p;
    const char* h = std::getenv("HOME");
    return std::string(h ? h : "/tmp") + "/.cache/b2p_autotune.txt";
}

std::string batch_key(BatchWork* w, int precision) {
    // signature: kernel version, precision, size classes of the batch
    double mean_m = (double)w->inst_m / w->count, mean_n = (double)w->inst_n / w->count;
    double nnz_col = (double)w->nnz / std::max<int64_t>(w->tot_n, 1);
    std::ostringstream os;
    const char* f = std::getenv("B2P_BATCH_SHAPE");
    os << "batch7" << (f && *f ? std::string("_s") + f : std::string()) << "_p" << precision << "_c" << (int)std::log2(std::max(1, w->count)) << "_m"
       << (int)std::log2(mean_m + 1) << "_n" << (int)std::log2(mean_n + 1) << "_k" << (int)std::lround(nnz_col) << "_M"
       << w->max_m << "_N" << w->max_n << "_shared" << (w->nmat == 1 && w->count > 1);
    return os.str();
}

bool cache_lookup(const std::string& key, TuneCfg* out) {
    std::ifstream f(cache_path());
    std::string line;
    while (std::getline(f, line)) {
        std::istringstream is(line);
        std::string k;
        TuneCfg c;
        if (!(is >> k) || k != key) continue;
        if (is >> c.threads >> c.chunk >> c.w >> c.ni >> c.form_th[0] >> c.form_us[0] >> c.form_th[1] >> c.form_us[1] >>
            c.form_th[2] >> c.form_us[2]) {
            *out = c;
            return true;
        }
    }
    return false;
}

void cache_store(const std::string& key, const TuneCfg& c) {
    std::string p = cache_path();
    std::string dir = p.substr(0, p.find_last_of('/'));
    if (!dir.empty()) {
        std::string cmd = "mkdir -p '" + dir + "'";
        if (std::system(cmd.c_str()) != 0) return;
    }
    std::ofstream f(p, std::ios::app);
    f << key << " " << c.threads << " " << c.chunk << " " << c.w << " " << c.ni;
    for (int i = 0; i < 3; ++i) f << " " << c.form_th[i] << " " << c.form_us[i];
    f << "\n";
}

template <typename MT>
BArgs make_args(BatchWork* w, const b2p_params* p, const int32_t* active) {
    const bool f64 = sizeof(MT) == 8;
    BArgs a;
    a.rowptr = w->rowptr.p;
    a.colidx = w->colidx.p;
    a.t_rowptr = w->t_rowptr.p;
    a.t_colidx = w->t_colidx.p;
    a.sv64 = w->sv64.p;
    a.stv64 = w->stv64.p;
    a.dr = w->dr.p;
    a.dc = w->dc.p;
    a.mat_eta = w->mat_eta.p;
    a.sv = f64 ? (const void*)w->sv64.p : (const void*)w->sv32.p;
    a.stv = f64 ? (const void*)w->stv64.p : (const void*)w->stv32.p;
    a.mat_m = w->mat_m.p;
    a.mat_n = w->mat_n.p;
    a.mat_row_off = w->mat_row_off.p;
    a.mat_col_off = w->mat_col_off.p;
    a.r_sptr = w->r_sptr.p;
    a.c_sptr = w->c_sptr.p;
    a.mat_rs_off = w->mat_rs_off.p;
    a.mat_cs_off = w->mat_cs_off.p;
    a.r_eidx = w->r_eidx.p;
    a.c_eidx = w->c_eidx.p;
    a.r_ev = f64 ? (const void*)w->r_ev64.p : (const void*)w->r_ev32.p;
    a.c_ev = f64 ? (const void*)w->c_ev64.p : (const void*)w->c_ev32.p;
    a.r_ev64 = w->r_ev64.p;
    a.c_ev64 = w->c_ev64.p;
    a.r_ext = w->r_ext.p;
    a.c_ext = w->c_ext.p;
    a.inst_mat = w->inst_mat.p;
    a.x_off = w->x_off.p;
    a.y_off = w->y_off.p;
    a.xp_off = w->xp_off.p;
    a.yp_off = w->yp_off.p;
    a.b = w->b.p;
    a.c = w->c.p;
    a.lb = w->lb.p;
    a.ub = w->ub.p;
    a.bnorm = w->bnorm.p;
    a.cnorm = w->cnorm.p;
    a.is_eq = w->is_eq.p;
    a.colp = w->colp.p;
    a.rowp = w->rowp.p;
    a.x = w->x.p;
    a.xt = w->xt.p;
    a.y = w->y.p;
    a.yt = w->yt.p;
    a.dx = w->dx.p;
    a.dy = w->dy.p;
    a.ictrl = w->ictrl.p;
    a.active = active;
    a.counters = w->counters.p;
    a.eps = p->eps_rel_kkt;
    a.beta_s = p->restart_sufficient;
    a.beta_n = p->restart_necessary;
    a.beta_a = p->restart_artificial;
    a.rho = p->reflection;
    a.eps_obj = p->eps_objective;
    a.eps_inf = (w->dx.p && w->dy.p) ? p->eps_infeasible : 0.0;
    a.max_iter = p->max_iterations;
    a.K = p->check_every;
    a.recenter = w->recenter ? 1 : 0;
    a.vals = w->vals.p;
    a.t_vals = w->t_vals.p;
    a.xbar = w->xbar.p;
    a.ybar = w->ybar.p;
    a.axbar = w->axbar.p;
    a.atybar = w->atybar.p;
    return a;
}

// dynamic shared memory of one CTA: per-instance blocks, slice table, y and xh (MT) of the largest
// instance, or of ni instances of the shared matrix
size_t smem_bytes(BatchWork* w, size_t mt_size, int ni = 1) {
    const size_t tab = sizeof(int2) * slice_tab_len((w->max_m + 31) >> 5, (w->max_n + 31) >> 5);
    const size_t m4 = (size_t)((w->max_m + 3) & ~3), n4 = (size_t)((w->max_n + 3) & ~3);
    const size_t head = mt_size == 4 ? group_head<float>(ni) : group_head<double>(ni);
    return head + tab + mt_size * ni * (m4 + std::max(n4, m4)) + 16;  // y, then xh (which also stages y at checks)
}

// CTA size of the tail form: two warps per slice of the largest instance, a power of two from 128 to
// 1024 threads.  The second warp shares the checks' and restarts' passes over single elements.  ms for
// 4,096 iterations of 48 instances, checks every 64, FP32 / FP64 by CTA size: 30 x 70 (3 slices)
// 128: 6.7 / 6.7, 256: 6.2 / 6.3, 1024: 6.7 / 6.7; 100 x 251 (8) 256: 10.7 / 11.1, 512: 9.4 / 9.8, 1024:
// 9.6 / 9.8; 200 x 500 (16) 256: 18.9 / 24.3, 512: 13.6 / 15.5, 1024: 12.5 / 14.6.
int tail_threads(BatchWork* w) {
    const int slices = (std::max(w->max_m, w->max_n) + 31) >> 5;
    int th = 128;
    while (th < 1024 && th / 32 < 2 * slices) th *= 2;
    return th;
}

// The chunk kernel of a shape (null: there is none).
template <typename MT, int W, bool LONG>
void (*chunk_kernel_w(int ni, int threads))(const BArgs, int) {
    const bool wide = threads > 512;
    if (ni == 1) return wide ? k_batch_chunk<MT, W, 1, 1024, 1, false, LONG> : k_batch_chunk<MT, W, 1, 512, 2, false, LONG>;
    if (wide) return nullptr;
    if (ni == 2) return k_batch_chunk<MT, W, 2, 512, 1, true, LONG>;
    if constexpr (sizeof(MT) == 4)
        if (ni == 4) return k_batch_chunk<MT, W, 4, 512, 1, true, LONG>;
    return nullptr;
}
template <typename MT>
void (*chunk_kernel(const BatchWork* bw, int w, int ni, int threads))(const BArgs, int) {
    if (bw->max_len > kLongSlice)
        return w == 2 ? chunk_kernel_w<MT, 2, true>(ni, threads) : chunk_kernel_w<MT, 1, true>(ni, threads);
    return w == 2 ? chunk_kernel_w<MT, 2, false>(ni, threads) : chunk_kernel_w<MT, 1, false>(ni, threads);
}

template <typename MT>
int init_instances(Ctx* ctx, BatchWork* w, const b2p_params* p, const double* x0_dev, const double* y0_dev,
                   const double* om_dev, const int32_t* list_dev = nullptr, int list_count = 0,
                   const long long* base_dev = nullptr) {
    const int cnt = list_dev ? list_count : w->count;
    int grid = std::min(cnt, ctx->sm_count * 8);
    BArgs a = make_args<MT>(w, p, w->active.p);
    k_batch_init<MT><<<grid, 256, 0, ctx->stream>>>(a, cnt, list_dev, x0_dev, y0_dev, om_dev, base_dev);
    B2P_LAUNCH(ctx);
    ctx->launches += 1;
    return B2P_OK;
}

// Rewrites both SELL copies in entry order W (1 or 2); the slice pointers (even lengths)
// serve both orders.
int refill_ell(Ctx* ctx, BatchWork* w, int W) {
    if (w->ell_w == W) return B2P_OK;
    cudaStream_t s = ctx->stream;
    const unsigned gmat = (unsigned)std::min(w->nmat, ctx->sm_count * 8);
    k_fill_ell<<<gmat, 256, 0, s>>>(W, w->nmat, w->mat_m.p, w->mat_row_off.p, w->mat_col_off.p, w->mat_rs_off.p,
                                     w->r_sptr.p, w->rowptr.p, w->colidx.p, w->sv64.p, w->sv32.p, w->r_eidx.p,
                                     w->r_ev64.p, w->r_ev32.p);
    k_fill_ell<<<gmat, 256, 0, s>>>(W, w->nmat, w->mat_n.p, w->mat_col_off.p, w->mat_row_off.p, w->mat_cs_off.p,
                                     w->c_sptr.p, w->t_rowptr.p, w->t_colidx.p, w->stv64.p, w->stv32.p, w->c_eidx.p,
                                     w->c_ev64.p, w->c_ev32.p);
    B2P_LAUNCH(ctx);
    ctx->launches += 2;
    w->ell_w = W;
    return B2P_OK;
}

// Times each shape on a size-stratified sample of the batch (no termination, 4a
// iterations -- long enough that the restart checks weigh as in a real solve -- no
// re-centring), then the chunk length: with the chosen shape, launches of a and 4a
// iterations give the per-iteration cost p and the fixed cost o of a chunk (launch, loading and storing every instance's state, plus the
// compaction that follows); the chunk is the shortest power of two from 256 to 8192
// whose fixed cost is at most 2 % of its iterations -- shorter chunks drop finished
// instances sooner, so the tail of an uneven batch is cut finer.  Each block size is
// tried with one instance per CTA and both SELL entry orders (one entry or a pair per lane
// load), and, when every instance shares one matrix, with groups of 2 and 4 instances (pair
// order only: their gathers are vectors, so fewer loads always won).  Of the chosen entry
// order the fastest size of every form is kept with its time per round of resident CTAs.
// Instance state is re-initialised afterwards by the caller.
template <typename MT>
int autotune(Ctx* ctx, BatchWork* w, const b2p_params* p, TuneCfg* best) {
    std::string key = batch_key(w, sizeof(MT) == 8 ? 0 : 1);
    if (cache_lookup(key, best)) return B2P_OK;
    cudaStream_t s = ctx->stream;
    int sample = std::min(w->count, ctx->sm_count * 4);
    std::vector<int32_t> ids(sample);
    for (int i = 0; i < sample; ++i) ids[i] = w->order[(int64_t)i * w->count / sample];
    DBuf<int32_t> dids;
    B2P_CUDA(ctx, dids.reserve(sample));
    B2P_CUDA(ctx, cudaMemcpyAsync(dids.p, ids.data(), sizeof(int32_t) * sample, cudaMemcpyHostToDevice, s));
    b2p_params tp = *p;
    tp.max_iterations = 1LL << 40;
    tp.eps_rel_kkt = 0.0;  // never terminates inside the trial
    tp.eps_infeasible = 0.0;
    const int trial_iters = 128;
    float best_ms = 1e30f;
    *best = TuneCfg();
    // one trial launch of `iters` iterations over the sample with `th` threads, entry order W
    // and ni instances per CTA (ms; < 0: the shape does not fit)
    auto trial = [&](int th, int W, int ni, int iters, float* ms, int* rounds) -> int {
        *ms = -1.0f;
        auto fn = chunk_kernel<MT>(w, W, ni, th);
        if (!fn) return B2P_OK;
        const size_t sm = smem_bytes(w, sizeof(MT), ni);
        int most = 0;
        B2P_CUDA(ctx, open_smem(ctx, fn, &most));
        if (sm > (size_t)most) return B2P_OK;
        int st = refill_ell(ctx, w, W);
        if (st) return st;
        st = init_instances<MT>(ctx, w, &tp, nullptr, nullptr, nullptr);
        if (st) return st;
        int32_t cnt[2] = {0, sample};
        B2P_CUDA(ctx, cudaMemcpyAsync(w->counters.p, cnt, sizeof(cnt), cudaMemcpyHostToDevice, s));
        BArgs a = make_args<MT>(w, &tp, dids.p);
        int per_sm = 0;
        B2P_CUDA(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, th, sm));
        if (per_sm < 1) return B2P_OK;
        const int groups = (sample + ni - 1) / ni, slots = ctx->sm_count * per_sm;
        const int grid = std::min(groups, slots);
        *rounds = (groups + slots - 1) / slots;
        cudaEventRecord(ctx->ev0, s);
        fn<<<grid, th, sm, s>>>(a, iters);
        k_batch_compact<<<1, 1024, 0, s>>>(w->ictrl.p, dids.p, w->active2.p, w->counters.p);
        cudaEventRecord(ctx->ev1, s);
        B2P_LAUNCH(ctx);
        B2P_CUDA(ctx, cudaEventSynchronize(ctx->ev1));
        ctx->launches += 2;
        cudaEventElapsedTime(ms, ctx->ev0, ctx->ev1);
        return B2P_OK;
    };
    const ShapeChoices choices = shape_choices(w);
    int rounds = 1;
    int form_th[3][3] = {};  // [form][entry order]
    float form_ms[3][3], form_us[3][3] = {};
    for (auto& r : form_ms)
        for (float& v : r) v = 1e30f;
    for (int f = 0; f < 3; ++f) {
        const int ni = kFormNi[f];
        if (std::find(choices.ni.begin(), choices.ni.end(), ni) == choices.ni.end()) continue;
        for (int W : choices.w) {
            if (ni > 1 && W == 1 && !choices.pinned) continue;
            for (int th : choices.threads) {
                float ms = 0.0f;
                int st = trial(th, W, ni, 4 * trial_iters, &ms, &rounds);
                if (st) return st;
                if (ms >= 0.0f && ms < form_ms[f][W]) {
                    form_ms[f][W] = ms;
                    form_us[f][W] = 1e3f * ms / (4 * trial_iters * rounds);
                    form_th[f][W] = th;
                }
                if (ms >= 0.0f && ms < best_ms) {
                    best_ms = ms;
                    best->threads = th;
                    best->w = W;
                    best->ni = ni;
                }
            }
        }
    }
    for (int f = 0; f < 3; ++f) {
        best->form_th[f] = form_th[f][best->w];
        best->form_us[f] = form_us[f][best->w];
    }
    if (best_ms >= 1e30f) {
        ctx->err = "batch: no chunk-kernel shape fits this batch";
        return B2P_INVALID_ARGUMENT;
    }
    float t1 = 0.0f;
    int st = trial(best->threads, best->w, best->ni, trial_iters, &t1, &rounds);
    if (st) return st;
    const double per_iter = std::max(1e-9, (double)(best_ms - t1) / (3.0 * trial_iters));
    const double fixed = std::max(0.0, (double)t1 - trial_iters * per_iter);
    int chunk = 256;
    while (chunk < 8192 && fixed > 0.02 * chunk * per_iter) chunk *= 2;
    best->chunk = chunk;
    cache_store(key, *best);
    return B2P_OK;
}

template <typename MT>
int batch_run(Ctx* ctx, BatchWork* w, const b2p_params* p, const double* x0_dev, const double* y0_dev,
              const double* om_dev, const std::vector<int32_t>* subset, bool* timed_out_out, float* kms_out,
              TuneCfg* cfg_out, const std::vector<long long>* base = nullptr) {
    cudaStream_t s = ctx->stream;
    double t_start = now_ms();
    const int64_t IN = w->inst_n, IM = w->inst_m;
    const int prec = sizeof(MT) == 8 ? 0 : 1;
    {
        // y and xh of the largest instance must fit one CTA's shared memory
        int max_smem = 0;
        B2P_CUDA(ctx, cudaDeviceGetAttribute(&max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, ctx->device));
        const size_t need = smem_bytes(w, sizeof(MT));
        if (need > (size_t)max_smem) {
            ctx->err = "batch instance too large for one CTA's shared memory: needs " + std::to_string(need) +
                       " bytes (" + std::to_string(w->max_m) + " rows + " + std::to_string(w->max_n) +
                       " columns), the device allows " + std::to_string(max_smem) +
                       "; solve it with b2p_solve";
            return B2P_INVALID_ARGUMENT;
        }
    }
    w->recenter = false;  // autotune trials run without re-centring
    TuneCfg cfg;
    if (w->tuned[prec]) {
        cfg = w->tuned_cfg[prec];
    } else {
        if (subset) {
            ctx->err = "subset solve before a full solve of this precision";
            return B2P_INVALID_ARGUMENT;
        }
        int st = autotune<MT>(ctx, w, p, &cfg);
        if (st) return st;
        cfg.pinned = shape_choices(w).pinned;
        w->tuned[prec] = true;
        w->tuned_cfg[prec] = cfg;
    }
    {
        int st = refill_ell(ctx, w, cfg.w);
        if (st) return st;
    }
    // displacement buffers of the infeasibility certificates (sized for FP64, read as MT)
    if (p->eps_infeasible > 0.0) {
        B2P_CUDA(ctx, w->dx.reserve(IN));
        B2P_CUDA(ctx, w->dy.reserve(IM));
    }
    // re-centring: on by default for the mixed engine (refinement_rounds < 0), forced by > 0
    w->recenter = p->refinement_rounds > 0 || (p->refinement_rounds < 0 && sizeof(MT) == 4);
    if (w->recenter) {
        for (auto* b : {&w->xbar, &w->atybar}) B2P_CUDA(ctx, b->reserve(IN));
        for (auto* b : {&w->ybar, &w->axbar}) B2P_CUDA(ctx, b->reserve(IM));
    }
    // instances to run, longest first
    std::vector<int32_t> act;
    if (subset) {
        std::vector<uint8_t> in_set(w->count, 0);
        for (int32_t i : *subset) in_set[i] = 1;
        for (int32_t i : w->order)
            if (in_set[i]) act.push_back(i);
        if (act.empty()) {
            if (timed_out_out) *timed_out_out = false;
            if (kms_out) *kms_out = 0.0f;
            if (cfg_out) *cfg_out = cfg;
            return B2P_OK;
        }
        B2P_CUDA(ctx, w->list.reserve(act.size()));
        B2P_CUDA(ctx, cudaMemcpyAsync(w->list.p, act.data(), sizeof(int32_t) * act.size(), cudaMemcpyHostToDevice, s));
        DBuf<long long> dbase;
        if (base) {  // per listed instance, in list order
            std::vector<long long> b(act.size());
            for (size_t q = 0; q < act.size(); ++q) b[q] = (*base)[act[q]];
            B2P_CUDA(ctx, dbase.reserve(act.size()));
            B2P_CUDA(ctx, cudaMemcpyAsync(dbase.p, b.data(), sizeof(long long) * b.size(), cudaMemcpyHostToDevice, s));
        }
        int st = init_instances<MT>(ctx, w, p, x0_dev, y0_dev, om_dev, w->list.p, (int)act.size(),
                                    base ? dbase.p : nullptr);
        if (st) return st;
        B2P_CUDA(ctx, cudaStreamSynchronize(s));  // dbase is released at scope end
    } else {
        act = w->order;
        int st = init_instances<MT>(ctx, w, p, x0_dev, y0_dev, om_dev);
        if (st) return st;
    }
    const int n_act = (int)act.size();
    B2P_CUDA(ctx, cudaMemcpyAsync(w->active.p, act.data(), sizeof(int32_t) * n_act, cudaMemcpyHostToDevice, s));
    int32_t cnt[2] = {0, n_act};
    B2P_CUDA(ctx, cudaMemcpyAsync(w->counters.p, cnt, sizeof(cnt), cudaMemcpyHostToDevice, s));
    BArgs a1 = make_args<MT>(w, p, w->active.p);
    BArgs a2 = make_args<MT>(w, p, w->active2.p);
    // The forms of this solve: the tuned ones by instances per CTA, and for the tail, when no
    // more than one instance per SM is left, one CTA per SM, as wide as the largest instance
    // can occupy (tail_threads).  A pinned shape is the only one: the tail form adds the FP64 sums of a
    // check in another order, and where a solve goes over to it depends on the chunk.
    struct Form {
        void (*fn)(const BArgs, int) = nullptr;
        int ni = 1, threads = 0, slots = 0;  // instances per CTA, CTA size, resident CTAs
        size_t smem = 0;
        double us = 0.0;
        cudaGraph_t graph = nullptr;
        cudaGraphExec_t exec = nullptr;
    };
    // the graphs, their executables and the pinned counter copy are released on every way out
    struct Owned {
        Form form[4];
        int32_t* host_cnt = nullptr;
        ~Owned() {
            for (Form& f : form) {
                if (f.exec) cudaGraphExecDestroy(f.exec);
                if (f.graph) cudaGraphDestroy(f.graph);
            }
            if (host_cnt) cudaFreeHost(host_cnt);
        }
    } own;
    auto open_form = [&](Form& f, int ni, int threads, double us) -> int {
        auto fn = chunk_kernel<MT>(w, cfg.w, ni, threads);
        const size_t sm = smem_bytes(w, sizeof(MT), ni);
        if (!fn) return B2P_OK;
        int most = 0;
        B2P_CUDA(ctx, open_smem(ctx, fn, &most));
        if (sm > (size_t)most) return B2P_OK;
        int per_sm = 0;
        B2P_CUDA(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, threads, sm));
        if (per_sm < 1) return B2P_OK;
        f.fn = fn;
        f.ni = ni;
        f.threads = threads;
        f.slots = ctx->sm_count * per_sm;
        f.smem = sm;
        f.us = us;
        return B2P_OK;
    };
    for (int f = 0; f < 3; ++f)
        if (cfg.form_th[f] > 0) {
            int st = open_form(own.form[f], kFormNi[f], cfg.form_th[f], cfg.form_us[f]);
            if (st) return st;
        }
    if (!cfg.pinned) {
        int st = open_form(own.form[3], 1, tail_threads(w), 0.0);
        if (st) return st;
    }
    bool any = false;
    for (const Form& f : own.form) any = any || f.fn != nullptr;
    if (!any) {
        ctx->err = "batch instance too large for one CTA's shared memory";
        return B2P_INVALID_ARGUMENT;
    }
    // the form for `n` active instances: the tail form for up to one instance per SM, else the
    // one with the least rounds x time per round
    auto pick_form = [&](int n) -> Form& {
        if (own.form[3].fn && n <= ctx->sm_count) return own.form[3];
        Form* best = nullptr;
        double best_us = 0.0;
        for (int i = 0; i < 3; ++i) {
            Form& f = own.form[i];
            if (!f.fn) continue;
            const int groups = (n + f.ni - 1) / f.ni;
            const double us = ((groups + f.slots - 1) / f.slots) * std::max(f.us, 1e-3);
            if (!best || us < best_us) {
                best = &f;
                best_us = us;
            }
        }
        return best ? *best : own.form[3];
    };
    // one graph = two chunk launches with compaction (ping-pong active lists), captured when
    // the form is first picked
    auto capture = [&](Form& f) -> int {
        if (f.exec) return B2P_OK;
        B2P_CUDA(ctx, cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
        f.fn<<<f.slots, f.threads, f.smem, s>>>(a1, cfg.chunk);
        k_batch_compact<<<1, 1024, 0, s>>>(w->ictrl.p, w->active.p, w->active2.p, w->counters.p);
        f.fn<<<f.slots, f.threads, f.smem, s>>>(a2, cfg.chunk);
        k_batch_compact<<<1, 1024, 0, s>>>(w->ictrl.p, w->active2.p, w->active.p, w->counters.p);
        cudaError_t ce = cudaStreamEndCapture(s, &f.graph);
        if (ce != cudaSuccess) {
            f.graph = nullptr;
            ctx->err = std::string("batch graph capture: ") + cudaGetErrorString(ce);
            return B2P_EXECUTION_FAILED;
        }
        ce = cudaGraphInstantiate(&f.exec, f.graph, 0);
        if (ce != cudaSuccess) {
            f.exec = nullptr;
            ctx->err = std::string("batch graph instantiate: ") + cudaGetErrorString(ce);
            return B2P_EXECUTION_FAILED;
        }
        return B2P_OK;
    };
    int32_t*& host_cnt = own.host_cnt;
    B2P_CUDA(ctx, cudaMallocHost(&host_cnt, 2 * sizeof(int32_t)));
    host_cnt[1] = n_act;
    const int first_ni = pick_form(n_act).ni;  // instances per CTA of the first launch
    const int64_t max_graphs = p->max_iterations / (2LL * cfg.chunk) + 3;
    int64_t graphs = 0;
    bool timed_out = false;
    const double tl = p->time_limit_s * 1000.0;
    cudaEventRecord(ctx->ev0, s);
    const double trace_base = subset && !w->trace_ms.empty() ? w->trace_ms.back() : 0.0;
    if (!subset) {
        w->trace_ms.clear();
        w->trace_active.clear();
    }
    const double t_loop = now_ms();
    w->trace_ms.push_back(trace_base);
    w->trace_active.push_back(n_act);
    while (graphs < max_graphs) {
        Form& form = pick_form(host_cnt[1]);
        {
            int st = capture(form);
            if (st) return st;
        }
        B2P_CUDA(ctx, cudaGraphLaunch(form.exec, s));
        graphs++;
        B2P_CUDA(ctx, cudaMemcpyAsync(host_cnt, w->counters.p, 2 * sizeof(int32_t), cudaMemcpyDeviceToHost, s));
        B2P_CUDA(ctx, cudaStreamSynchronize(s));
        w->trace_ms.push_back(trace_base + now_ms() - t_loop);
        w->trace_active.push_back(host_cnt[1]);
        if (host_cnt[1] == 0) break;
        if (tl > 0 && now_ms() - t_start > tl) {
            timed_out = true;
            break;
        }
    }
    cudaEventRecord(ctx->ev1, s);
    B2P_CUDA(ctx, cudaStreamSynchronize(s));
    ctx->launches += graphs * 4;
    float kms = 0;
    cudaEventElapsedTime(&kms, ctx->ev0, ctx->ev1);
    // results of every instance: control blocks to the host, answers (original space,
    // external order) and primal weights kept on the device
    w->hc.resize(w->count);
    B2P_CUDA(ctx, cudaMemcpyAsync(w->hc.data(), w->ictrl.p, sizeof(InstCtrl) * w->count, cudaMemcpyDeviceToHost, s));
    B2P_CUDA(ctx, w->ox.reserve(IN));
    B2P_CUDA(ctx, w->oy.reserve(IM));
    B2P_CUDA(ctx, w->oom.reserve(w->count));
    k_batch_unscale<MT><<<std::min(w->count, ctx->sm_count * 8), 256, 0, s>>>(
        a1, w->count, w->recenter ? w->xbar.p : nullptr, w->recenter ? w->ybar.p : nullptr, w->ox.p, w->oy.p);
    B2P_LAUNCH(ctx);
    ctx->launches += 1;
    B2P_CUDA(ctx, cudaStreamSynchronize(s));
    std::vector<double> om(w->count);
    for (int i = 0; i < w->count; ++i) om[i] = w->hc[i].omega;
    B2P_CUDA(ctx, cudaMemcpyAsync(w->oom.p, om.data(), sizeof(double) * w->count, cudaMemcpyHostToDevice, s));
    B2P_CUDA(ctx, cudaStreamSynchronize(s));
    w->solved = true;
    if (timed_out_out) *timed_out_out = timed_out;
    if (kms_out) *kms_out = kms;
    if (cfg_out) {
        *cfg_out = cfg;
        cfg_out->ni = first_ni;
    }
    return B2P_OK;
}

// Per-instance outputs of the last solve (any pointer may be null).
int collect_outputs(Ctx* ctx, BatchWork* w, bool timed_out, int32_t* status_out, int64_t* iters_out, double* kkt_out,
                    double* omega_out, double* x_out, double* y_out, int64_t* tot_it, int64_t* maxit, int64_t* opt,
                    double* worst) {
    cudaStream_t s = ctx->stream;
    *tot_it = 0;
    *maxit = 0;
    *opt = 0;
    *worst = 0.0;
    for (int i = 0; i < w->count; ++i) {
        const InstCtrl& c = w->hc[i];
        int stt = c.done ? c.status : (timed_out ? B2P_STATUS_INTERRUPTED : B2P_STATUS_MAX_ITERATIONS);
        double kk = std::max(c.rel_p, std::max(c.rel_d, c.rel_g));
        if (status_out) status_out[i] = stt;
        if (iters_out) iters_out[i] = c.total + c.base;
        if (kkt_out) kkt_out[i] = kk;
        if (omega_out) omega_out[i] = c.omega;
        *tot_it += c.total + c.base;
        *maxit = std::max<int64_t>(*maxit, c.total + c.base);
        *opt += (stt == B2P_STATUS_OPTIMAL);
        *worst = std::max(*worst, kk);
    }
    if (x_out) B2P_CUDA(ctx, cudaMemcpyAsync(x_out, w->ox.p, sizeof(double) * w->inst_n, cudaMemcpyDeviceToHost, s));
    if (y_out) B2P_CUDA(ctx, cudaMemcpyAsync(y_out, w->oy.p, sizeof(double) * w->inst_m, cudaMemcpyDeviceToHost, s));
    B2P_CUDA(ctx, cudaStreamSynchronize(s));
    return B2P_OK;
}

void fill_summary(b2p_result* sum, int count, bool timed_out, int64_t tot_it, int64_t maxit, int64_t opt, double worst,
                  float kms, const TuneCfg& cfg) {
    if (!sum) return;
    sum->status = (opt == count) ? B2P_STATUS_OPTIMAL : (timed_out ? B2P_STATUS_INTERRUPTED : B2P_STATUS_MAX_ITERATIONS);
    sum->iterations = tot_it;  // sum over instances
    sum->restarts = maxit;     // longest instance
    sum->rel_kkt = worst;
    sum->kernel_time_ms = kms;
    sum->primal_weight = 0.0;
    sum->step_size = cfg.threads * 100000.0 + cfg.chunk;  // tuned block size * 1e5 + chunk length
    sum->used_average = 10 * cfg.ni + cfg.w;                // 10 * instances per CTA at first + SELL entries per lane load
}

// All instances of the batch share one shape (required by the learned warm start).
bool uniform_shape(BatchWork* w, int* n, int* m) {
    *n = w->h_mat_n[w->h_inst_mat[0]];
    *m = w->h_mat_m[w->h_inst_mat[0]];
    for (int i = 1; i < w->count; ++i)
        if (w->h_mat_n[w->h_inst_mat[i]] != *n || w->h_mat_m[w->h_inst_mat[i]] != *m) return false;
    return true;
}

}  // namespace
}  // namespace b2p

using namespace b2p;

extern "C" {

int b2p_batch_upload(void* p, int nmat, const int32_t* mat_m, const int32_t* mat_n, const int64_t* mat_nnz_off,
                     const int32_t* rowptr, const int32_t* colidx, const double* vals, int count,
                     const int32_t* inst_mat, const double* b, const double* c, const double* lb, const double* ub,
                     const uint8_t* is_eq) {
    Ctx* ctx = static_cast<Ctx*>(p);
    if (!ctx) return B2P_GPU_UNINITIALIZED;
    if (nmat <= 0 || count <= 0 || !mat_m || !mat_n || !mat_nnz_off || !rowptr || !inst_mat || !b || !c || !lb || !ub ||
        !is_eq) {
        ctx->err = "b2p_batch_upload: empty batch or null argument";
        return B2P_INVALID_ARGUMENT;
    }
    cudaSetDevice(ctx->device);
    batch_free(ctx);
    BatchWork* w = new BatchWork();
    ctx->bw = w;
    w->nmat = nmat;
    w->count = count;
    std::vector<int64_t> row_off(nmat), col_off(nmat);
    int64_t tm = 0, tn = 0;
    for (int k = 0; k < nmat; ++k) {
        if (mat_m[k] <= 0 || mat_n[k] <= 0) {
            ctx->err = "b2p_batch_upload: empty matrix";
            return B2P_INVALID_ARGUMENT;
        }
        if (mat_m[k] > 65535 || mat_n[k] > 65535) {
            ctx->err = "b2p_batch_upload: a batched instance has at most 65535 rows and columns";
            return B2P_INVALID_ARGUMENT;
        }
        row_off[k] = tm;
        col_off[k] = tn;
        tm += mat_m[k];
        tn += mat_n[k];
        w->max_m = std::max(w->max_m, mat_m[k]);
        w->max_n = std::max(w->max_n, mat_n[k]);
    }
    const int64_t nnz = mat_nnz_off[nmat];
    std::vector<int32_t> bigs{0};  // the wait status of the cluster kernel, then the matrices worth a cluster
    for (int k = 0; k < nmat; ++k)
        if (mat_nnz_off[k + 1] - mat_nnz_off[k] >= kPowerCluster) bigs.push_back(k);
    const int big = (int)bigs.size() - 1;
    if (nnz > INT32_MAX || tm > INT32_MAX || tn > INT32_MAX) {
        ctx->err = "b2p_batch_upload: batch exceeds 32-bit index range";
        return B2P_INVALID_ARGUMENT;
    }
    w->tot_m = tm;
    w->tot_n = tn;
    w->nnz = nnz;
    // validate, then renumber rows and columns of each matrix by decreasing length
    // (stable) and build the internal CSR (global indices) and the SELL-32 slice
    // pointers of both orientations
    std::vector<int32_t> grp(tm + 1), gci(nnz), r_ext(tm), c_ext(tn);
    std::vector<double> gval(nnz);
    std::vector<int64_t> rs_off(nmat), cs_off(nmat), r_sptr, c_sptr;
    r_sptr.reserve(tm / 32 + 2 * nmat);
    c_sptr.reserve(tn / 32 + 2 * nmat);
    int64_t rp_base = 0, r_pad = 0, c_pad = 0, pos = 0;
    grp[0] = 0;
    std::vector<int32_t> rlen, clen, rord, cord, cinv;
    for (int k = 0; k < nmat; ++k) {
        const int32_t* rp = rowptr + rp_base;
        const int m = mat_m[k], n = mat_n[k];
        const int64_t e0 = mat_nnz_off[k], e1 = mat_nnz_off[k + 1];
        if (rp[0] != 0 || rp[m] != e1 - e0) {
            ctx->err = "b2p_batch_upload: matrix " + std::to_string(k) + " row pointers do not match its nnz";
            return B2P_INVALID_ARGUMENT;
        }
        rlen.assign(m, 0);
        clen.assign(n, 0);
        for (int i = 0; i < m; ++i) {
            if (rp[i + 1] < rp[i]) {
                ctx->err = "b2p_batch_upload: decreasing row pointer";
                return B2P_INVALID_ARGUMENT;
            }
            int prev = -1;
            for (int e = rp[i]; e < rp[i + 1]; ++e) {
                int cidx = colidx[e0 + e];
                if (cidx < 0 || cidx >= n || cidx <= prev) {
                    ctx->err = "b2p_batch_upload: matrix " + std::to_string(k) + " row " + std::to_string(i) +
                               ": column indices out of range or not strictly ascending";
                    return B2P_INVALID_ARGUMENT;
                }
                prev = cidx;
                clen[cidx]++;
            }
            rlen[i] = rp[i + 1] - rp[i];
            w->max_len = std::max(w->max_len, rlen[i]);
        }
        for (int j = 0; j < n; ++j) w->max_len = std::max(w->max_len, clen[j]);
        rord.resize(m);
        cord.resize(n);
        std::iota(rord.begin(), rord.end(), 0);
        std::iota(cord.begin(), cord.end(), 0);
        std::stable_sort(rord.begin(), rord.end(), [&](int x, int y) { return rlen[x] > rlen[y]; });
        std::stable_sort(cord.begin(), cord.end(), [&](int x, int y) { return clen[x] > clen[y]; });
        cinv.resize(n);
        for (int j = 0; j < n; ++j) {
            cinv[cord[j]] = j;
            c_ext[col_off[k] + j] = cord[j];
        }
        for (int i = 0; i < m; ++i) {
            const int old = rord[i];
            r_ext[row_off[k] + i] = old;
            for (int e = rp[old]; e < rp[old + 1]; ++e) {
                gci[pos] = (int32_t)(cinv[colidx[e0 + e]] + col_off[k]);
                gval[pos] = vals[e0 + e];
                ++pos;
            }
            grp[row_off[k] + i + 1] = (int32_t)pos;
        }
        // slice pointers: matrix k owns nslices + 1 entries
        rs_off[k] = (int64_t)r_sptr.size();
        for (int s0 = 0; s0 < m; s0 += 32) {
            r_sptr.push_back(r_pad);
            r_pad += 32LL * ((rlen[rord[s0]] + 1) & ~1);  // even: both entry orders (W = 1, 2) fit
        }
        r_sptr.push_back(r_pad);
        cs_off[k] = (int64_t)c_sptr.size();
        for (int s0 = 0; s0 < n; s0 += 32) {
            c_sptr.push_back(c_pad);
            c_pad += 32LL * ((clen[cord[s0]] + 1) & ~1);
        }
        c_sptr.push_back(c_pad);
        if (r_pad > INT32_MAX || c_pad > INT32_MAX) {  // the kernels' slice tables hold 32-bit offsets
            ctx->err = "b2p_batch_upload: the batch's padded matrices exceed 2^31 entries; split the batch";
            return B2P_INVALID_ARGUMENT;
        }
        rp_base += m + 1;
    }
    w->h_mat_m.assign(mat_m, mat_m + nmat);
    w->h_mat_n.assign(mat_n, mat_n + nmat);
    // instances
    std::vector<int64_t> xoff(count), yoff(count), xpoff(count), ypoff(count);
    int64_t IN = 0, IM = 0, IC = 0, IR = 0;
    std::vector<int64_t> inst_nnz(count);
    for (int i = 0; i < count; ++i) {
        int k = inst_mat[i];
        if (k < 0 || k >= nmat) {
            ctx->err = "b2p_batch_upload: instance names a matrix out of range";
            return B2P_INVALID_ARGUMENT;
        }
        xoff[i] = IN;
        yoff[i] = IM;
        xpoff[i] = IC;
        ypoff[i] = IR;
        IN += mat_n[k];
        IM += mat_m[k];
        IC += (int64_t)col_rec((mat_n[k] + 31) & ~31);
        IR += (int64_t)row_rec((mat_m[k] + 31) & ~31);
        inst_nnz[i] = mat_nnz_off[k + 1] - mat_nnz_off[k];
    }
    w->inst_n = IN;
    w->inst_m = IM;
    for (int64_t j = 0; j < IN; ++j)
        if (std::isnan(c[j]) || std::isnan(lb[j]) || std::isnan(ub[j])) {
            ctx->err = "b2p_batch_upload: NaN in c / lb / ub";
            return B2P_INVALID_ARGUMENT;
        }
    w->h_inst_mat.assign(inst_mat, inst_mat + count);
    w->order.resize(count);
    std::iota(w->order.begin(), w->order.end(), 0);
    std::stable_sort(w->order.begin(), w->order.end(),
                     [&](int a, int b2) { return inst_nnz[a] > inst_nnz[b2]; });
    cudaStream_t s = ctx->stream;
    B2P_CUDA(ctx, w->rowptr.reserve(tm + 1));
    B2P_CUDA(ctx, w->t_rowptr.reserve(tn + 1));
    for (auto* bf : {&w->colidx, &w->t_colidx}) B2P_CUDA(ctx, bf->reserve(nnz));
    for (auto* bf : {&w->vals, &w->t_vals, &w->sv64, &w->stv64}) B2P_CUDA(ctx, bf->reserve(nnz));
    for (auto* bf : {&w->sv32, &w->stv32}) B2P_CUDA(ctx, bf->reserve(nnz));
    for (auto* bf : {&w->dr, &w->pu}) B2P_CUDA(ctx, bf->reserve(tm));
    for (auto* bf : {&w->dc, &w->pv}) B2P_CUDA(ctx, bf->reserve(tn));
    B2P_CUDA(ctx, w->r_ext.reserve(tm));
    B2P_CUDA(ctx, w->c_ext.reserve(tn));
    for (auto* bf : {&w->mat_m, &w->mat_n}) B2P_CUDA(ctx, bf->reserve(nmat));
    for (auto* bf : {&w->mat_row_off, &w->mat_col_off, &w->mat_rs_off, &w->mat_cs_off}) B2P_CUDA(ctx, bf->reserve(nmat));
    B2P_CUDA(ctx, w->r_sptr.reserve(r_sptr.size()));
    B2P_CUDA(ctx, w->c_sptr.reserve(c_sptr.size()));
    B2P_CUDA(ctx, w->r_eidx.reserve(r_pad));
    B2P_CUDA(ctx, w->c_eidx.reserve(c_pad));
    B2P_CUDA(ctx, w->r_ev64.reserve(r_pad));
    B2P_CUDA(ctx, w->c_ev64.reserve(c_pad));
    B2P_CUDA(ctx, w->r_ev32.reserve(r_pad));
    B2P_CUDA(ctx, w->c_ev32.reserve(c_pad));
    B2P_CUDA(ctx, w->mat_eta.reserve(nmat));
    B2P_CUDA(ctx, w->inst_mat.reserve(count));
    for (auto* bf : {&w->x_off, &w->y_off, &w->xp_off, &w->yp_off}) B2P_CUDA(ctx, bf->reserve(count));
    for (auto* bf : {&w->c, &w->lb, &w->ub, &w->x, &w->xt}) B2P_CUDA(ctx, bf->reserve(IN));
    for (auto* bf : {&w->b, &w->y, &w->yt}) B2P_CUDA(ctx, bf->reserve(IM));
    B2P_CUDA(ctx, w->colp.reserve(IC));
    B2P_CUDA(ctx, w->rowp.reserve(IR));
    B2P_CUDA(ctx, w->is_eq.reserve(IM));
    for (auto* bf : {&w->bnorm, &w->cnorm}) B2P_CUDA(ctx, bf->reserve(count));
    B2P_CUDA(ctx, w->ictrl.reserve(count));
    for (auto* bf : {&w->active, &w->active2}) B2P_CUDA(ctx, bf->reserve(count));
    B2P_CUDA(ctx, w->counters.reserve(2));
    B2P_CUDA(ctx, cudaMemcpyAsync(w->rowptr.p, grp.data(), sizeof(int32_t) * (tm + 1), cudaMemcpyHostToDevice, s));
    B2P_CUDA(ctx, cudaMemcpyAsync(w->colidx.p, gci.data(), sizeof(int32_t) * nnz, cudaMemcpyHostToDevice, s));
    B2P_CUDA(ctx, cudaMemcpyAsync(w->vals.p, gval.data(), sizeof(double) * nnz, cudaMemcpyHostToDevice, s));
    B2P_CUDA(ctx, cudaMemcpyAsync(w->r_ext.p, r_ext.data(), sizeof(int32_t) * tm, cudaMemcpyHostToDevice, s));
    B2P_CUDA(ctx, cudaMemcpyAsync(w->c_ext.p, c_ext.data(), sizeof(int32_t) * tn, cudaMemcpyHostToDevice, s));
    B2P_CUDA(ctx, cudaMemcpyAsync(w->r_sptr.p, r_sptr.data(), sizeof(int64_t) * r_sptr.size(), cudaMemcpyHostToDevice, s));
    B2P_CUDA(ctx, cudaMemcpyAsync(w->c_sptr.p, c_sptr.data(), sizeof(int64_t) * c_sptr.size(), cudaMemcpyHostToDevice, s));
    B2P_CUDA(ctx, cudaMemcpyAsync(w->mat_rs_off.p, rs_off.data(), sizeof(int64_t) * nmat, cudaMemcpyHostToDevice, s));
    B2P_CUDA(ctx, cudaMemcpyAsync(w->mat_cs_off.p, cs_off.data(), sizeof(int64_t) * nmat, cudaMemcpyHostToDevice, s));
    B2P_CUDA(ctx, cudaMemcpyAsync(w->mat_m.p, mat_m, sizeof(int32_t) * nmat, cudaMemcpyHostToDevice, s));
    B2P_CUDA(ctx, cudaMemcpyAsync(w->mat_n.p, mat_n, sizeof(int32_t) * nmat, cudaMemcpyHostToDevice, s));
    B2P_CUDA(ctx, cudaMemcpyAsync(w->mat_row_off.p, row_off.data(), sizeof(int64_t) * nmat, cudaMemcpyHostToDevice, s));
    B2P_CUDA(ctx, cudaMemcpyAsync(w->mat_col_off.p, col_off.data(), sizeof(int64_t) * nmat, cudaMemcpyHostToDevice, s));
    B2P_CUDA(ctx, cudaMemcpyAsync(w->inst_mat.p, inst_mat, sizeof(int32_t) * count, cudaMemcpyHostToDevice, s));
    B2P_CUDA(ctx, cudaMemcpyAsync(w->x_off.p, xoff.data(), sizeof(int64_t) * count, cudaMemcpyHostToDevice, s));
    B2P_CUDA(ctx, cudaMemcpyAsync(w->y_off.p, yoff.data(), sizeof(int64_t) * count, cudaMemcpyHostToDevice, s));
    B2P_CUDA(ctx, cudaMemcpyAsync(w->xp_off.p, xpoff.data(), sizeof(int64_t) * count, cudaMemcpyHostToDevice, s));
    B2P_CUDA(ctx, cudaMemcpyAsync(w->yp_off.p, ypoff.data(), sizeof(int64_t) * count, cudaMemcpyHostToDevice, s));
    {
        // per-instance vectors arrive in external order: stage, then permute on the device
        DBuf<double> sb, scv, sl, su;
        DBuf<uint8_t> seq;
        for (auto* bf : {&scv, &sl, &su}) B2P_CUDA(ctx, bf->reserve(IN));
        B2P_CUDA(ctx, sb.reserve(IM));
        B2P_CUDA(ctx, seq.reserve(IM));
        B2P_CUDA(ctx, cudaMemcpyAsync(scv.p, c, sizeof(double) * IN, cudaMemcpyHostToDevice, s));
        B2P_CUDA(ctx, cudaMemcpyAsync(sl.p, lb, sizeof(double) * IN, cudaMemcpyHostToDevice, s));
        B2P_CUDA(ctx, cudaMemcpyAsync(su.p, ub, sizeof(double) * IN, cudaMemcpyHostToDevice, s));
        B2P_CUDA(ctx, cudaMemcpyAsync(sb.p, b, sizeof(double) * IM, cudaMemcpyHostToDevice, s));
        B2P_CUDA(ctx, cudaMemcpyAsync(seq.p, is_eq, IM, cudaMemcpyHostToDevice, s));
        k_permute_inst<<<std::min(count, ctx->sm_count * 8), 256, 0, s>>>(
            count, w->inst_mat.p, w->mat_m.p, w->mat_n.p, w->mat_row_off.p, w->mat_col_off.p, w->x_off.p, w->y_off.p,
            w->r_ext.p, w->c_ext.p, sb.p, scv.p, sl.p, su.p, seq.p, w->b.p, w->c.p, w->lb.p, w->ub.p, w->is_eq.p);
        B2P_LAUNCH(ctx);
        ctx->launches += 1;
        B2P_CUDA(ctx, cudaStreamSynchronize(s));  // staging buffers are released at scope end
    }
    int st = build_transpose(ctx, (int)tm, (int)tn, nnz, w->rowptr.p, w->colidx.p, w->vals.p, w->t_rowptr.p,
                             w->t_colidx.p, w->t_vals.p);
    if (st) return st;
    // scaling + scaled values + step sizes (per matrix, FP64), then the SELL-32 copies
    DBuf<double> tr, tc;
    B2P_CUDA(ctx, tr.reserve(tm));
    B2P_CUDA(ctx, tc.reserve(tn));
    int ruiz = 10;
    int gmat = std::min(nmat, ctx->sm_count * 8);
    k_batch_scaling<<<gmat, 256, 0, s>>>(nmat, w->mat_m.p, w->mat_n.p, w->mat_row_off.p, w->mat_col_off.p, w->rowptr.p,
                                          w->colidx.p, w->vals.p, w->t_rowptr.p, w->t_colidx.p, w->t_vals.p, ruiz,
                                          w->dr.p, w->dc.p, tr.p, tc.p);
    k_batch_scale_vals<<<grid_for(std::max(tm, tn), 256, ctx->sm_count), 256, 0, s>>>(
        tm, tn, w->rowptr.p, w->colidx.p, w->vals.p, w->t_rowptr.p, w->t_colidx.p, w->t_vals.p, w->dr.p, w->dc.p,
        w->sv64.p, w->sv32.p, w->stv64.p, w->stv32.p);
    k_fill_ell<<<gmat, 256, 0, s>>>(1, nmat, w->mat_m.p, w->mat_row_off.p, w->mat_col_off.p, w->mat_rs_off.p, w->r_sptr.p,
                                     w->rowptr.p, w->colidx.p, w->sv64.p, w->sv32.p, w->r_eidx.p, w->r_ev64.p,
                                     w->r_ev32.p);
    k_fill_ell<<<gmat, 256, 0, s>>>(1, nmat, w->mat_n.p, w->mat_col_off.p, w->mat_row_off.p, w->mat_cs_off.p, w->c_sptr.p,
                                     w->t_rowptr.p, w->t_colidx.p, w->stv64.p, w->stv32.p, w->c_eidx.p, w->c_ev64.p,
                                     w->c_ev32.p);
    // clusters for up to two large matrices per 8 SMs -- the L2 form's clusters are then resident at once,
    // the shared-memory form's take two or three turns of a fifth of the time -- beyond that one CTA each
    // fills the GPU as well: 304 large matrices of 1,024 take 130 ms longer on clusters
    const int clusters = 2 * ctx->sm_count / kPowerCtas;
    int max_smem = 0;
    B2P_CUDA(ctx, open_smem(ctx, k_batch_power_cluster<true>, &max_smem));
    const int tabs = (((w->max_n + 31) >> 5) + kPowerCtas - 1) / kPowerCtas + (((w->max_m + 31) >> 5) + kPowerCtas - 1) / kPowerCtas;
    const int64_t vec = 8ll * ((int64_t)w->max_n + w->max_m + tabs);
    const bool sm = vec <= max_smem;  // both vectors fit a CTA's shared memory
    const auto power_fn = sm ? k_batch_power_cluster<true> : k_batch_power_cluster<false>;
    const int resident = big > 0 && big <= clusters ? clusters_resident(power_fn, kPowerCtas, 512, sm ? max_smem : 0) : 0;
    const bool use_clusters = resident > 0;
    const auto one_cta_fn = use_clusters ? k_batch_power<true> : k_batch_power<false>;
    one_cta_fn<<<gmat, 256, 0, s>>>(nmat, w->mat_m.p, w->mat_n.p, w->mat_row_off.p, w->mat_col_off.p, w->rowptr.p,
                                    w->colidx.p, w->sv64.p, w->t_rowptr.p, w->t_colidx.p, w->stv64.p, w->pv.p, w->pu.p,
                                    0.998, w->mat_eta.p);
    int wait_failed = 0;
    DBuf<int32_t> dbigs;
    if (use_clusters) {
        B2P_CUDA(ctx, dbigs.reserve(bigs.size()));
        B2P_CUDA(ctx, cudaMemcpyAsync(dbigs.p, bigs.data(), sizeof(int32_t) * bigs.size(), cudaMemcpyHostToDevice, s));
        power_fn<<<std::min(big, resident) * kPowerCtas, 512, sm ? max_smem : 0, s>>>(
            big, dbigs.p + 1, w->mat_m.p, w->mat_n.p, w->mat_row_off.p, w->mat_col_off.p, w->rowptr.p, w->colidx.p,
            w->sv64.p, w->t_rowptr.p, w->t_colidx.p, w->stv64.p, w->mat_rs_off.p, w->mat_cs_off.p, w->r_sptr.p,
            w->c_sptr.p, w->r_eidx.p, w->c_eidx.p, w->r_ev64.p, w->c_ev64.p, w->pv.p, w->pu.p, 0.998, w->max_m, w->max_n,
            (int)(max_smem - vec), dbigs.p, w->mat_eta.p);
        ctx->launches += 1;
        B2P_CUDA(ctx, cudaMemcpyAsync(&wait_failed, dbigs.p, sizeof(int), cudaMemcpyDeviceToHost, s));
    }
    B2P_LAUNCH(ctx);
    ctx->launches += 5;
    B2P_CUDA(ctx, cudaStreamSynchronize(s));
    if (wait_failed) {
        ctx->err = "batch upload: the power iteration's cluster exchange did not complete";
        return B2P_EXECUTION_FAILED;
    }
    return B2P_OK;
}

int b2p_batch_solve(void* p, const b2p_params* params, const double* x0, const double* y0, const double* omega0,
                    int32_t* status_out, int64_t* iters_out, double* kkt_out, double* omega_out, double* x_out,
                    double* y_out, b2p_result* summary) {
    Ctx* ctx = static_cast<Ctx*>(p);
    if (!ctx) return B2P_GPU_UNINITIALIZED;
    BatchWork* w = ctx->bw;
    if (!w) {
        ctx->err = "b2p_batch_solve: no batch uploaded";
        return B2P_NO_LP;
    }
    b2p_params def;
    b2p_params_default(&def);
    def.engine = B2P_ENGINE_HALPERN;
    const b2p_params* pp = params ? params : &def;
    if (pp->check_every < 2 || pp->max_iterations < 0) {
        ctx->err = "b2p_batch_solve: check_every must be >= 2";
        return B2P_INVALID_ARGUMENT;
    }
    cudaSetDevice(ctx->device);
    if (summary) std::memset(summary, 0, sizeof(*summary));
    int64_t l0 = ctx->launches;
    double t0 = now_ms();
    cudaStream_t s = ctx->stream;
    // warm starts / weights to the device
    DBuf<double> dx0, dy0, dom;
    if (x0) {
        B2P_CUDA(ctx, dx0.reserve(w->inst_n));
        B2P_CUDA(ctx, cudaMemcpyAsync(dx0.p, x0, sizeof(double) * w->inst_n, cudaMemcpyHostToDevice, s));
    }
    if (y0) {
        B2P_CUDA(ctx, dy0.reserve(w->inst_m));
        B2P_CUDA(ctx, cudaMemcpyAsync(dy0.p, y0, sizeof(double) * w->inst_m, cudaMemcpyHostToDevice, s));
    }
    if (omega0) {
        B2P_CUDA(ctx, dom.reserve(w->count));
        B2P_CUDA(ctx, cudaMemcpyAsync(dom.p, omega0, sizeof(double) * w->count, cudaMemcpyHostToDevice, s));
    }
    bool timed_out = false;
    float kms = 0.0f;
    TuneCfg cfg;
    int st = pp->precision == B2P_FP64
                 ? batch_run<double>(ctx, w, pp, x0 ? dx0.p : nullptr, y0 ? dy0.p : nullptr, omega0 ? dom.p : nullptr,
                                     nullptr, &timed_out, &kms, &cfg)
                 : batch_run<float>(ctx, w, pp, x0 ? dx0.p : nullptr, y0 ? dy0.p : nullptr, omega0 ? dom.p : nullptr,
                                    nullptr, &timed_out, &kms, &cfg);
    if (st) return st;
    int64_t tot_it, maxit, opt;
    double worst;
    st = collect_outputs(ctx, w, timed_out, status_out, iters_out, kkt_out, omega_out, x_out, y_out, &tot_it, &maxit,
                         &opt, &worst);
    if (st) return st;
    fill_summary(summary, w->count, timed_out, tot_it, maxit, opt, worst, kms, cfg);
    if (summary) {
        summary->solve_time_ms = now_ms() - t0;
        summary->kernel_launches = ctx->launches - l0;
    }
    return B2P_OK;
}

int b2p_batch_trace(void* p, int capacity, int* count, double* t_ms, int32_t* active) {
    Ctx* ctx = static_cast<Ctx*>(p);
    if (!ctx) return B2P_GPU_UNINITIALIZED;
    BatchWork* w = ctx->bw;
    if (!w || !w->solved) {
        ctx->err = "b2p_batch_trace: no batched solve to report";
        return B2P_NO_LP;
    }
    const int n = (int)w->trace_ms.size();
    if (count) *count = n;
    const int k = std::min(n, std::max(capacity, 0));
    for (int i = 0; i < k; ++i) {
        if (t_ms) t_ms[i] = w->trace_ms[i];
        if (active) active[i] = w->trace_active[i];
    }
    return B2P_OK;
}

int b2p_batch_objectives(void* p, double* pobj_out, double* dobj_out, double* obj_err_out) {
    Ctx* ctx = static_cast<Ctx*>(p);
    if (!ctx) return B2P_GPU_UNINITIALIZED;
    BatchWork* w = ctx->bw;
    if (!w || !w->solved || (int)w->hc.size() != w->count) {
        ctx->err = "b2p_batch_objectives: no batched solve to report";
        return B2P_NO_LP;
    }
    for (int i = 0; i < w->count; ++i) {
        if (pobj_out) pobj_out[i] = w->hc[i].pobj;
        if (dobj_out) dobj_out[i] = w->hc[i].dobj;
        if (obj_err_out) obj_err_out[i] = w->hc[i].obj_err;
    }
    return B2P_OK;
}

int b2p_batch_solve_learned(void* p, const b2p_params* params, const float* features, int fallback,
                            int32_t* status_out, int64_t* iters_out, double* kkt_out, uint8_t* warm_used_out,
                            double* x_out, double* y_out, b2p_result* summary) {
    Ctx* ctx = static_cast<Ctx*>(p);
    if (!ctx) return B2P_GPU_UNINITIALIZED;
    BatchWork* w = ctx->bw;
    if (!w) {
        ctx->err = "b2p_batch_solve_learned: no batch uploaded";
        return B2P_NO_LP;
    }
    if (!features) {
        ctx->err = "b2p_batch_solve_learned: null parameter vectors";
        return B2P_INVALID_ARGUMENT;
    }
    int n = 0, m = 0;
    if (!uniform_shape(w, &n, &m)) {
        ctx->err = "b2p_batch_solve_learned: the instances of the batch differ in shape";
        return B2P_INVALID_ARGUMENT;
    }
    b2p_params def;
    b2p_params_default(&def);
    def.engine = B2P_ENGINE_HALPERN;
    def.precision = B2P_FP32;
    const b2p_params* pp = params ? params : &def;
    if (pp->check_every < 2 || pp->max_iterations < 0) {
        ctx->err = "b2p_batch_solve_learned: check_every must be >= 2";
        return B2P_INVALID_ARGUMENT;
    }
    cudaSetDevice(ctx->device);
    if (summary) std::memset(summary, 0, sizeof(*summary));
    int64_t l0 = ctx->launches;
    double t0 = now_ms();
    // warm start from the MLP, on the device
    DBuf<double> dx0, dy0, dom;
    B2P_CUDA(ctx, dx0.reserve(w->inst_n));
    B2P_CUDA(ctx, dy0.reserve(w->inst_m));
    B2P_CUDA(ctx, dom.reserve(w->count));
    int st = mlp_predict_warm(ctx, features, w->count, n, m, dx0.p, dy0.p, dom.p);
    if (st) return st;
    const bool f64 = pp->precision == B2P_FP64;
    bool timed_out = false;
    float kms = 0.0f, kms2 = 0.0f;
    TuneCfg cfg;
    st = f64 ? batch_run<double>(ctx, w, pp, dx0.p, dy0.p, dom.p, nullptr, &timed_out, &kms, &cfg)
             : batch_run<float>(ctx, w, pp, dx0.p, dy0.p, dom.p, nullptr, &timed_out, &kms, &cfg);
    if (st) return st;
    // cold-start fallback for every instance the warm-started run did not solve and
    // that has iterations left: the cold run continues the instance's iteration count,
    // so warm + cold together stay within max_iterations (an instance that spent its
    // whole budget warm is reported MAX_ITERATIONS, as a cold run would be)
    std::vector<long long> warm_iters(w->count);
    std::vector<int32_t> failed;
    for (int i = 0; i < w->count; ++i) {
        warm_iters[i] = w->hc[i].total;
        // an answer, or a certificate of infeasibility / unboundedness (which holds
        // whatever the starting point), ends the instance
        const int sti = w->hc[i].status;
        const bool ok = w->hc[i].done && (sti == B2P_STATUS_OPTIMAL || sti == B2P_STATUS_INFEASIBLE_DETECTED ||
                                          sti == B2P_STATUS_UNBOUNDED_DETECTED);
        if (!ok && warm_iters[i] < pp->max_iterations) failed.push_back(i);
    }
    if (fallback && !failed.empty() && !timed_out) {
        // the summary names the shape of the warm run
        st = f64 ? batch_run<double>(ctx, w, pp, nullptr, nullptr, nullptr, &failed, &timed_out, &kms2, nullptr,
                                     &warm_iters)
                 : batch_run<float>(ctx, w, pp, nullptr, nullptr, nullptr, &failed, &timed_out, &kms2, nullptr,
                                    &warm_iters);
        if (st) return st;
    }
    int64_t tot_it, maxit, opt;
    double worst;
    // iterations per instance: the warm run, plus the cold run when it fell back
    st = collect_outputs(ctx, w, timed_out, status_out, iters_out, kkt_out, nullptr, x_out, y_out, &tot_it, &maxit,
                         &opt, &worst);
    if (st) return st;
    std::vector<uint8_t> is_failed(w->count, 0);
    if (fallback)
        for (int32_t i : failed) is_failed[i] = 1;
    if (warm_used_out)
        for (int i = 0; i < w->count; ++i) warm_used_out[i] = is_failed[i] ? 0 : 1;
    fill_summary(summary, w->count, timed_out, tot_it, maxit, opt, worst, kms + kms2, cfg);
    if (summary) {
        summary->solve_time_ms = now_ms() - t0;
        summary->kernel_launches = ctx->launches - l0;
        summary->refinement_rounds_done = fallback ? (int)failed.size() : 0;  // instances that fell back
    }
    return B2P_OK;
}

int b2p_mlp_dataset_from_batch(void* p, const float* features, int count) {
    Ctx* ctx = static_cast<Ctx*>(p);
    if (!ctx) return B2P_GPU_UNINITIALIZED;
    BatchWork* w = ctx->bw;
    if (!w || !w->solved) {
        ctx->err = "b2p_mlp_dataset_from_batch: no solved batch";
        return B2P_NO_LP;
    }
    if (!features || count != w->count) {
        ctx->err = "b2p_mlp_dataset_from_batch: one parameter vector per instance of the batch is required";
        return B2P_INVALID_ARGUMENT;
    }
    int n = 0, m = 0;
    if (!uniform_shape(w, &n, &m)) {
        ctx->err = "b2p_mlp_dataset_from_batch: the instances of the batch differ in shape";
        return B2P_INVALID_ARGUMENT;
    }
    cudaSetDevice(ctx->device);
    return mlp_set_dataset(ctx, features, count, n, m, w->ox.p, w->oy.p, w->oom.p);
}

}  // extern "C"
