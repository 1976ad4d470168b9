// libb2p: device/context management, LP upload, and the GpuBackend primitives.
//
// Compiled with --fmad=false: the FP64 SpMV and vector primitives here round
// every multiply and add separately, as the reference host loops do
// (src/gpu_backend.cpp:60-69, 135-327), so results agree bit for bit with
// CSRMatrix::multiply (src/sparse_matrix.cpp:153-163).
#include <cub/cub.cuh>

#include <chrono>
#include <cmath>
#include <cstring>
#include <new>

#include "b2p_internal.cuh"

namespace b2p {

int map_cuda_error(cudaError_t e) {
    switch (e) {
        case cudaSuccess: return B2P_OK;
        case cudaErrorMemoryAllocation: return B2P_OUT_OF_MEMORY;
        case cudaErrorNoDevice:
        case cudaErrorInsufficientDriver:
        case cudaErrorInvalidDevice: return B2P_GPU_UNAVAILABLE;
        case cudaErrorInvalidValue: return B2P_INVALID_ARGUMENT;
        default: return B2P_EXECUTION_FAILED;
    }
}

double now_ms() {
    using namespace std::chrono;
    return duration<double, std::milli>(steady_clock::now().time_since_epoch()).count();
}

// ---------------------------------------------------------------- transpose (setup only)
// Entries up to which the context keeps the scratch of a transpose (16 bytes each) for the next one.
constexpr int64_t kKeepTranspose = 1 << 20;

__global__ void k_row_of(int m, const int32_t* __restrict__ rowptr, int32_t* __restrict__ row_of) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < m; i += gridDim.x * blockDim.x)
        for (int k = rowptr[i]; k < rowptr[i + 1]; ++k) row_of[k] = i;
}

__global__ void k_iota(int64_t nnz, int32_t* __restrict__ v) {
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < nnz; k += (int64_t)gridDim.x * blockDim.x)
        v[k] = (int32_t)k;
}

__global__ void k_count(int64_t nnz, const int32_t* __restrict__ colidx, int32_t* __restrict__ counts) {
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < nnz; k += (int64_t)gridDim.x * blockDim.x)
        atomicAdd(&counts[colidx[k]], 1);
}

__global__ void k_gather_t(int64_t nnz, const int32_t* __restrict__ perm, const int32_t* __restrict__ row_of,
                           const double* __restrict__ vals, int32_t* __restrict__ t_colidx,
                           double* __restrict__ t_vals) {
    for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < nnz; p += (int64_t)gridDim.x * blockDim.x) {
        int32_t k = perm[p];
        t_colidx[p] = row_of[k];
        t_vals[p] = vals[k];
    }
}

int build_transpose(Ctx* ctx, int m, int n, int64_t nnz, const int32_t* rowptr, const int32_t* colidx,
                    const double* vals, int32_t* t_rowptr, int32_t* t_colidx, double* t_vals) {
    cudaStream_t s = ctx->stream;
    B2P_CUDA(ctx, cudaMemsetAsync(t_rowptr, 0, sizeof(int32_t) * (n + 1), s));
    if (nnz == 0) return B2P_OK;
    DBuf<int32_t>&row_of = ctx->tr_row, &keys_out = ctx->tr_keys, &perm_in = ctx->tr_in, &perm_out = ctx->tr_out;
    B2P_CUDA(ctx, row_of.reserve(nnz));
    B2P_CUDA(ctx, keys_out.reserve(nnz));
    B2P_CUDA(ctx, perm_in.reserve(nnz));
    B2P_CUDA(ctx, perm_out.reserve(nnz));
    unsigned g = grid_for(std::max<int64_t>(m, 1), 256, ctx->sm_count);
    k_row_of<<<g, 256, 0, s>>>(m, rowptr, row_of.p);
    unsigned gz = grid_for(nnz, 256, ctx->sm_count);
    k_iota<<<gz, 256, 0, s>>>(nnz, perm_in.p);
    k_count<<<gz, 256, 0, s>>>(nnz, colidx, t_rowptr + 1);
    B2P_LAUNCH(ctx);
    int end_bit = 1;
    while (end_bit < 31 && (1LL << end_bit) <= n) ++end_bit;
    // Stable LSD radix sort by column: entries of one column keep their row-major
    // order, so row indices ascend inside every column of the transpose.
    size_t tmp_sort = 0, tmp_scan = 0;
    B2P_CUDA(ctx, cub::DeviceRadixSort::SortPairs(nullptr, tmp_sort, colidx, keys_out.p, perm_in.p, perm_out.p,
                                                  (int)nnz, 0, end_bit, s));
    B2P_CUDA(ctx, cub::DeviceScan::InclusiveSum(nullptr, tmp_scan, t_rowptr + 1, t_rowptr + 1, n, s));
    B2P_CUDA(ctx, ctx->cub_tmp.reserve(std::max(tmp_sort, tmp_scan)));
    size_t tb = ctx->cub_tmp.bytes();
    B2P_CUDA(ctx, cub::DeviceRadixSort::SortPairs(ctx->cub_tmp.p, tb, colidx, keys_out.p, perm_in.p, perm_out.p,
                                                  (int)nnz, 0, end_bit, s));
    tb = ctx->cub_tmp.bytes();
    B2P_CUDA(ctx, cub::DeviceScan::InclusiveSum(ctx->cub_tmp.p, tb, t_rowptr + 1, t_rowptr + 1, n, s));
    k_gather_t<<<gz, 256, 0, s>>>(nnz, perm_out.p, row_of.p, vals, t_colidx, t_vals);
    B2P_LAUNCH(ctx);
    ctx->launches += 4;
    // a large matrix's temporaries are freed on return; make sure the stream is done with them
    B2P_CUDA(ctx, cudaStreamSynchronize(s));
    if (nnz > kKeepTranspose)
        for (auto* d : {&row_of, &keys_out, &perm_in, &perm_out}) d->release();
    return B2P_OK;
}

// ---------------------------------------------------------------- validation
// CSRMatrix::is_valid (src/sparse_matrix.cpp:187-207): indices in range and strictly ascending.
__global__ void k_validate_csr(int m, int n, const int32_t* __restrict__ rowptr, const int32_t* __restrict__ colidx,
                               int32_t* __restrict__ bad) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < m; i += gridDim.x * blockDim.x) {
        int prev = -1;
        for (int k = rowptr[i]; k < rowptr[i + 1]; ++k) {
            int c = colidx[k];
            if (c < 0 || c >= n || c <= prev) { atomicExch(bad, i + 1); break; }
            prev = c;
        }
    }
}

static int host_rowptr_ok(int m, int64_t nnz, const int32_t* rowptr) {
    if (rowptr[0] != 0 || (int64_t)rowptr[m] != nnz) return 0;
    for (int i = 0; i < m; ++i)
        if (rowptr[i + 1] < rowptr[i]) return 0;
    return 1;
}

// ---------------------------------------------------------------- GpuBackend primitives
__global__ void k_spmv_f64(int m, const int32_t* __restrict__ rowptr, const int32_t* __restrict__ colidx,
                           const double* __restrict__ vals, const double* __restrict__ x, double* __restrict__ y) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < m; i += gridDim.x * blockDim.x) {
        double sum = 0.0;
        for (int k = rowptr[i]; k < rowptr[i + 1]; ++k) sum += vals[k] * x[colidx[k]];
        y[i] = sum;
    }
}

// y = A x of an unchecked matrix: entries whose column is out of range or not above the one before
// are not read through and mark *bad (as k_validate_csr does).
__global__ void k_spmv_checked(int m, int n, const int32_t* __restrict__ rowptr, const int32_t* __restrict__ colidx,
                               const double* __restrict__ vals, const double* __restrict__ x, double* __restrict__ y,
                               int32_t* __restrict__ bad) {
    constexpr int B = 8;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < m; i += gridDim.x * blockDim.x) {
        double sum = 0.0;
        int prev = -1;
        const int e1 = rowptr[i + 1];
        for (int k = rowptr[i]; k < e1; k += B) {
            int c[B];
            double v[B], g[B];
#pragma unroll
            for (int u = 0; u < B; ++u) {
                c[u] = k + u < e1 ? colidx[k + u] : -1;
                v[u] = k + u < e1 ? vals[k + u] : 0.0;
            }
#pragma unroll
            for (int u = 0; u < B; ++u) {
                const bool ok = c[u] >= 0 && c[u] < n;
                g[u] = ok ? x[c[u]] : 0.0;
                if (k + u < e1) {
                    if (!ok || c[u] <= prev) atomicExch(bad, i + 1);
                    prev = c[u];
                }
            }
#pragma unroll
            for (int u = 0; u < B; ++u)
                if (k + u < e1) sum += v[u] * g[u];
        }
        y[i] = sum;
    }
}

// w = A^T y of a small unchecked matrix in one CTA, without a transpose: the products to shared
// memory, then one warp adds them row after row, as the reference scatter does (the columns of a
// row are distinct, so its entries go side by side; a row that is not is refused anyway).
__global__ void __launch_bounds__(1024, 1) k_spmv_t_small(int m, int n, const int32_t* __restrict__ rowptr,
                                                          const int32_t* __restrict__ colidx,
                                                          const double* __restrict__ vals, const double* __restrict__ y,
                                                          double* __restrict__ w, int32_t* __restrict__ bad,
                                                          int rows_off) {
    extern __shared__ double sh[];
    const int nnz = rowptr[m], lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double *ws = sh, *prod = ws + n;
    int16_t* col = reinterpret_cast<int16_t*>(prod + nnz);  // -1: not read through
    for (int j = threadIdx.x; j < n; j += blockDim.x) ws[j] = 0.0;
    for (int i = threadIdx.x; i <= m; i += blockDim.x) reinterpret_cast<int*>(sh + rows_off)[i] = rowptr[i];
    for (int i = warp; i < m; i += blockDim.x >> 5) {
        const int e0 = rowptr[i], e1 = rowptr[i + 1];
        const double yi = y[i];
        for (int e = e0 + lane; e < e1; e += 32) {
            const int c = colidx[e], before = e > e0 ? colidx[e - 1] : -1;
            const bool ok = c >= 0 && c < n;
            if (!ok || c <= before) atomicExch(bad, i + 1);
            col[e] = ok ? (int16_t)c : (int16_t)-1;
            prod[e] = vals[e] * yi;
        }
    }
    __syncthreads();
    if (warp == 0) {
        int* rows = reinterpret_cast<int*>(sh + rows_off);
        int e = lane < rows[1] ? lane : -1;  // this lane's entry of the next step, read ahead
        int c = e >= 0 ? col[e] : -1;
        double p = e >= 0 ? prod[e] : 0.0;
        for (int i = 0, b = 0; i < m;) {
            const int c0 = c;
            const double p0 = p;
            b += 32;
            if (b >= rows[i + 1]) b = rows[++i];
            e = i < m && b + lane < rows[i + 1] ? b + lane : -1;
            c = e >= 0 ? col[e] : -1;
            p = e >= 0 ? prod[e] : 0.0;
            if (c0 >= 0) ws[c0] += p0;
            __syncwarp();
        }
    }
    __syncthreads();
    for (int j = threadIdx.x; j < n; j += blockDim.x) w[j] = ws[j];
}

__global__ void k_vec(int op, size_t n, double alpha, const double* __restrict__ a, const double* __restrict__ b,
                      double* __restrict__ out) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        double r;
        switch (op) {
            case B2P_VEC_ADD: r = a[i] + b[i]; break;
            case B2P_VEC_SUB: r = a[i] - b[i]; break;
            case B2P_VEC_SCALE: r = alpha * a[i]; break;
            default: r = alpha * a[i] + b[i]; break;
        }
        out[i] = r;
    }
}

// Deterministic two-pass FP64 reduction: fixed-size grid, per-block partials in a
// fixed order, then one block sums the partials in index order.
constexpr int kRedBlocks = 256;
constexpr int kRedThreads = 256;

__global__ void k_dot_partial(size_t n, const double* __restrict__ a, const double* __restrict__ b,
                              double* __restrict__ partial) {
    __shared__ double sh[kRedThreads / 32];
    double s = 0.0;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        s += a[i] * (b ? b[i] : a[i]);
    s = warp_sum(s);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < kRedThreads / 32; ++w) t += sh[w];
        partial[blockIdx.x] = t;
    }
}

__global__ void k_sum_partials(int count, const double* __restrict__ partial, double* __restrict__ out) {
    __shared__ double sh[kRedThreads / 32];
    double s = 0.0;
    for (int i = threadIdx.x; i < count; i += blockDim.x) s += partial[i];
    s = warp_sum(s);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < kRedThreads / 32; ++w) t += sh[w];
        out[0] = t;
    }
}

// Events around the phases of a call, recorded only where the caller asked for its times; the
// context keeps them.
struct PhaseTimer {
    Ctx* ctx;
    bool ok;
    PhaseTimer(Ctx* c, const b2p_timing_t* t) : ctx(c), ok(t != nullptr) {
        for (auto& x : c->tev)
            if (ok && !x && cudaEventCreate(&x) != cudaSuccess) ok = false;
    }
    void mark(int phase) {
        if (ok) cudaEventRecord(ctx->tev[phase], ctx->stream);
    }
    void fill(b2p_timing_t* t, double host_t0) {
        if (!t || !ok) return;
        float a = 0, b = 0, c = 0;
        cudaEventElapsedTime(&a, ctx->tev[0], ctx->tev[1]);
        cudaEventElapsedTime(&b, ctx->tev[1], ctx->tev[2]);
        cudaEventElapsedTime(&c, ctx->tev[2], ctx->tev[3]);
        t->h2d_time_ms = a;
        t->kernel_time_ms = b;
        t->d2h_time_ms = c;
        double total = now_ms() - host_t0;
        t->sync_time_ms = std::max(0.0, total - (a + b + c));
        t->total_gpu_time_ms = total;
    }
};

// The transfers of one call.  A call of up to kPackBytes packs its inputs into one buffer and gets
// its outputs back through it: one copy each way instead of one per argument (each costs
// several microseconds before its first byte).  The buffer is pageable: pinning it took 3 ms
// in a context's first call and saved less than a microsecond in the others.  A larger call
// copies argument by argument, as they are.
struct CallIO {
    static constexpr size_t kPackBytes = 1 << 20;
    Ctx* ctx;
    bool packed = false;
    size_t used = 0, in_bytes = 0;
    struct Out {
        void* host;
        const void* dev;
        size_t at, bytes;
    };
    std::vector<Out> outs;

    static size_t round(size_t b) { return (b + 15) & ~(size_t)15; }
    // total: bytes of all arguments, each rounded up
    int begin(Ctx* c, size_t total) {
        ctx = c;
        packed = total <= kPackBytes;
        if (packed) {
            B2P_CUDA(ctx, ctx->s_pack.reserve(total));
            if (ctx->h_pack.size() < total) ctx->h_pack.resize(total);
        }
        return B2P_OK;
    }
    template <typename T>
    int in(DBuf<T>& buf, const T* src, size_t n, T** dev) {
        if (packed) {
            std::memcpy(ctx->h_pack.data() + used, src, n * sizeof(T));
            *dev = reinterpret_cast<T*>(ctx->s_pack.p + used);
            used += round(n * sizeof(T));
            return B2P_OK;
        }
        B2P_CUDA(ctx, buf.reserve(n));
        *dev = buf.p;
        if (n) B2P_CUDA(ctx, cudaMemcpyAsync(buf.p, src, n * sizeof(T), cudaMemcpyHostToDevice, ctx->stream));
        return B2P_OK;
    }
    int send() {  // after the last input
        in_bytes = used;
        if (packed && used)
            B2P_CUDA(ctx, cudaMemcpyAsync(ctx->s_pack.p, ctx->h_pack.data(), used, cudaMemcpyHostToDevice, ctx->stream));
        return B2P_OK;
    }
    template <typename T>
    int out(DBuf<T>& buf, T* dst, size_t n, T** dev) {
        if (packed) {
            *dev = reinterpret_cast<T*>(ctx->s_pack.p + used);
            outs.push_back({dst, *dev, used, n * sizeof(T)});
            used += round(n * sizeof(T));
            return B2P_OK;
        }
        B2P_CUDA(ctx, buf.reserve(n));
        *dev = buf.p;
        outs.push_back({dst, buf.p, 0, n * sizeof(T)});
        return B2P_OK;
    }
    int receive() {  // queues the copies back
        if (packed) {
            B2P_CUDA(ctx, cudaMemcpyAsync(ctx->h_pack.data() + in_bytes, ctx->s_pack.p + in_bytes, used - in_bytes,
                                          cudaMemcpyDeviceToHost, ctx->stream));
            return B2P_OK;
        }
        for (const Out& o : outs)
            B2P_CUDA(ctx, cudaMemcpyAsync(o.host, o.dev, o.bytes, cudaMemcpyDeviceToHost, ctx->stream));
        return B2P_OK;
    }
    // waits and hands the outputs over; `bad` (the last output) nonzero: only that one
    int finish(const int32_t* bad = nullptr) {
        B2P_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
        if (packed && bad) {
            const Out& o = outs.back();
            std::memcpy(o.host, ctx->h_pack.data() + o.at, o.bytes);
            if (*bad) return B2P_OK;
        }
        if (packed)
            for (const Out& o : outs) std::memcpy(o.host, ctx->h_pack.data() + o.at, o.bytes);
        return B2P_OK;
    }
};
#define B2P_DO(call)                 \
    do {                             \
        int _st = (call);            \
        if (_st != B2P_OK) return _st; \
    } while (0)

}  // namespace b2p

using namespace b2p;

static Ctx* as_ctx(void* p) { return static_cast<Ctx*>(p); }

extern "C" {

void b2p_params_default(b2p_params* p) {
    if (!p) return;
    std::memset(p, 0, sizeof(*p));
    p->engine = B2P_ENGINE_REFERENCE;
    p->precision = B2P_FP64;
    p->max_iterations = 50000;
    p->feasibility_tolerance = 1e-7;
    p->primal_step_size = 0.01;
    p->dual_step_size = 0.01;
    p->adaptive_step_size = 1;
    p->check_frequency = 100;
    p->eps_rel_kkt = 1e-6;
    p->check_every = 64;
    p->ruiz_iterations = 10;
    p->reflection = 1.0;
    p->restart_sufficient = 0.2;
    p->restart_necessary = 0.8;
    p->restart_artificial = 0.36;
    p->primal_weight = 0.0;
    p->step_safety = 0.998;
    p->refinement_rounds = -1;
    p->time_limit_s = 0.0;
    p->lanes_per_row = 0;
    p->eps_objective = 0.0;
    p->eps_infeasible = 1e-8;
}

int b2p_device_info(int device, b2p_device_info_t* out) {
    if (!out) return B2P_INVALID_ARGUMENT;
    std::memset(out, 0, sizeof(*out));
    int count = 0;
    cudaError_t e = cudaGetDeviceCount(&count);
    if (e != cudaSuccess || count <= device || device < 0) {
        std::snprintf(out->device_name, sizeof(out->device_name), "None");
        std::snprintf(out->status_message, sizeof(out->status_message), "no CUDA device %d: %s", device,
                      e != cudaSuccess ? cudaGetErrorString(e) : "index out of range");
        return B2P_GPU_UNAVAILABLE;
    }
    cudaDeviceProp prop;
    if (cudaGetDeviceProperties(&prop, device) != cudaSuccess) return B2P_GPU_UNAVAILABLE;
    std::snprintf(out->device_name, sizeof(out->device_name), "%s", prop.name);
    out->total_memory_bytes = prop.totalGlobalMem;
    out->compute_capability_major = prop.major;
    out->compute_capability_minor = prop.minor;
    out->multiprocessor_count = prop.multiProcessorCount;
    out->l2_cache_bytes = prop.l2CacheSize;
    int cur = 0;
    cudaGetDevice(&cur);
    cudaSetDevice(device);
    size_t fr = 0, tot = 0;
    if (cudaMemGetInfo(&fr, &tot) == cudaSuccess) out->free_memory_bytes = fr;
    cudaSetDevice(cur);
    // The kernels are built for sm_100a only.
    out->is_available = (prop.major == 10 && prop.minor == 0) ? 1 : 0;
    std::snprintf(out->status_message, sizeof(out->status_message), "%s (sm_%d%d, %d SMs, %.1f GiB)%s", prop.name,
                  prop.major, prop.minor, prop.multiProcessorCount, prop.totalGlobalMem / 1073741824.0,
                  out->is_available ? "" : ": this library is built for sm_100a only");
    return out->is_available ? B2P_OK : B2P_GPU_UNAVAILABLE;
}

int b2p_ctx_create(int device, void** ctx_out) {
    if (!ctx_out) return B2P_INVALID_ARGUMENT;
    *ctx_out = nullptr;
    b2p_device_info_t info;
    int st = b2p_device_info(device, &info);
    if (st != B2P_OK) return st;
    Ctx* ctx = new (std::nothrow) Ctx();
    if (!ctx) return B2P_OUT_OF_MEMORY;
    ctx->device = device;
    ctx->sm_count = info.multiprocessor_count;
    ctx->l2_bytes = info.l2_cache_bytes;
    if (cudaSetDevice(device) != cudaSuccess || cudaStreamCreateWithFlags(&ctx->own_stream, cudaStreamNonBlocking) != cudaSuccess ||
        cudaEventCreate(&ctx->ev0) != cudaSuccess || cudaEventCreate(&ctx->ev1) != cudaSuccess) {
        delete ctx;
        return B2P_GPU_UNAVAILABLE;
    }
    ctx->stream = ctx->own_stream;
    *ctx_out = ctx;
    return B2P_OK;
}

int b2p_ctx_set_stream(void* p, void* stream) {
    Ctx* ctx = as_ctx(p);
    if (!ctx) return B2P_GPU_UNINITIALIZED;
    cudaSetDevice(ctx->device);
    B2P_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    ctx->stream = stream ? static_cast<cudaStream_t>(stream) : ctx->own_stream;
    return B2P_OK;
}

int b2p_kernel_timing(void* p, const b2p_params* params, int reps, double* primal_ms, double* dual_ms,
                      double* primal_bytes, double* dual_bytes) {
    Ctx* ctx = as_ctx(p);
    if (!ctx) return B2P_GPU_UNINITIALIZED;
    if (!ctx->has_lp || !ctx->hw) {
        ctx->err = "b2p_kernel_timing: solve an uploaded LP with the Halpern engine first";
        return B2P_NO_LP;
    }
    if (!params || reps <= 0) return B2P_INVALID_ARGUMENT;
    cudaSetDevice(ctx->device);
    return halpern_kernel_timing(ctx, params, reps, primal_ms, dual_ms, primal_bytes, dual_bytes);
}

int b2p_ctx_destroy(void* p) {
    Ctx* ctx = as_ctx(p);
    if (!ctx) return B2P_INVALID_ARGUMENT;
    cudaSetDevice(ctx->device);
    cudaStreamSynchronize(ctx->stream);
    ref_free(ctx);
    halpern_free(ctx);
    batch_free(ctx);
    mlp_free(ctx);
    ctx->lp.~DevLP();
    new (&ctx->lp) DevLP();
    for (auto& x : ctx->tev)
        if (x) cudaEventDestroy(x);
    if (ctx->ev0) cudaEventDestroy(ctx->ev0);
    if (ctx->ev1) cudaEventDestroy(ctx->ev1);
    if (ctx->own_stream) cudaStreamDestroy(ctx->own_stream);
    delete ctx;
    return B2P_OK;
}

const char* b2p_last_error(void* p) {
    Ctx* ctx = as_ctx(p);
    if (!ctx) return "null context";
    return ctx->err.c_str();
}

// ---- GpuBackend::spmv (gpu_backend.cpp:34-86): INVALID_ARGUMENT on an empty matrix or missing x.
int b2p_spmv(void* p, int m, int n, const int32_t* rowptr, const int32_t* colidx, const double* vals,
             const double* x, double* y, b2p_timing_t* timing) {
    Ctx* ctx = as_ctx(p);
    if (!ctx) return B2P_GPU_UNINITIALIZED;
    if (m <= 0 || n <= 0 || !rowptr || !x || !y) return B2P_INVALID_ARGUMENT;
    int64_t nnz = rowptr[m];
    if (nnz > 0 && (!colidx || !vals)) return B2P_INVALID_ARGUMENT;
    if (!host_rowptr_ok(m, nnz, rowptr)) return B2P_INVALID_ARGUMENT;
    cudaSetDevice(ctx->device);
    double t0 = now_ms();
    PhaseTimer pt(ctx, timing);
    cudaStream_t s = ctx->stream;
    int32_t *rp, *ci, *flag, bad = 0;
    double *va, *xd, *yd;
    CallIO io;
    B2P_DO(io.begin(ctx, CallIO::round(4 * ((size_t)m + 1)) + CallIO::round(4 * nnz) + CallIO::round(8 * nnz) + 8 * ((size_t)n + m) + 64));
    pt.mark(0);
    B2P_DO(io.in(ctx->s_rowptr, rowptr, (size_t)m + 1, &rp));
    B2P_DO(io.in(ctx->s_colidx, colidx, nnz, &ci));
    B2P_DO(io.in(ctx->s_vals, vals, nnz, &va));
    B2P_DO(io.in(ctx->s_x, x, n, &xd));
    B2P_DO(io.send());
    B2P_DO(io.out(ctx->s_y, y, m, &yd));
    B2P_DO(io.out(ctx->s_flag, &bad, 1, &flag));
    B2P_CUDA(ctx, cudaMemsetAsync(flag, 0, sizeof(int32_t), s));
    pt.mark(1);
    k_spmv_checked<<<grid_for(m, 128, ctx->sm_count), 128, 0, s>>>(m, n, rp, ci, va, xd, yd, flag);
    B2P_LAUNCH(ctx);
    ctx->launches += 1;
    pt.mark(2);
    B2P_DO(io.receive());
    pt.mark(3);
    B2P_DO(io.finish());
    pt.fill(timing, t0);
    if (bad) {
        ctx->err = "CSR column indices out of range or not strictly ascending in row " + std::to_string(bad - 1);
        return B2P_INVALID_ARGUMENT;
    }
    return B2P_OK;
}

// A^T y with the transpose built on the device; the sum over each column runs in
// ascending row order, as the reference scatter (src/sparse_matrix.cpp:175-185) does.
int b2p_spmv_t(void* p, int m, int n, const int32_t* rowptr, const int32_t* colidx, const double* vals,
               const double* yv, double* w, b2p_timing_t* timing) {
    Ctx* ctx = as_ctx(p);
    if (!ctx) return B2P_GPU_UNINITIALIZED;
    if (m <= 0 || n <= 0 || !rowptr || !yv || !w) return B2P_INVALID_ARGUMENT;
    int64_t nnz = rowptr[m];
    if (nnz > 0 && (!colidx || !vals)) return B2P_INVALID_ARGUMENT;
    if (!host_rowptr_ok(m, nnz, rowptr)) return B2P_INVALID_ARGUMENT;
    cudaSetDevice(ctx->device);
    double t0 = now_ms();
    PhaseTimer pt(ctx, timing);
    cudaStream_t s = ctx->stream;
    int32_t *rp, *ci, *flag, bad = 0;
    double *va, *yd, *wd;
    CallIO io;
    B2P_DO(io.begin(ctx, CallIO::round(4 * ((size_t)m + 1)) + CallIO::round(4 * nnz) + CallIO::round(8 * nnz) + 8 * ((size_t)n + m) + 64));
    pt.mark(0);
    B2P_DO(io.in(ctx->s_rowptr, rowptr, (size_t)m + 1, &rp));
    B2P_DO(io.in(ctx->s_colidx, colidx, nnz, &ci));
    B2P_DO(io.in(ctx->s_vals, vals, nnz, &va));
    B2P_DO(io.in(ctx->s_x, yv, m, &yd));
    B2P_DO(io.send());
    B2P_DO(io.out(ctx->s_y, w, n, &wd));
    B2P_DO(io.out(ctx->s_flag, &bad, 1, &flag));
    B2P_CUDA(ctx, cudaMemsetAsync(flag, 0, sizeof(int32_t), s));
    pt.mark(1);
    auto invalid = [&]() {
        ctx->err = "CSR column indices out of range or not strictly ascending in row " + std::to_string(bad - 1);
        return B2P_INVALID_ARGUMENT;
    };
    // small: its products and sums fit one CTA, whose one adding warp takes 0.1 us for a row of up to 32
    // entries (the kernel by device events: 38 us at 300 rows of 17 entries, 109 at 1,000 of 12 or of 5);
    // the sort, scan and waits of the transpose took 150 us whatever the size
    if (io.packed && nnz <= 12288 && n <= 8192 && m <= 1024) {
        const int rows_off = n + (int)nnz + ((int)nnz + 3) / 4;  // in doubles: sums, products, columns, then row pointers
        const size_t small = 8 * (size_t)rows_off + 4 * ((size_t)m + 1);
        B2P_CUDA(ctx, open_smem(ctx, k_spmv_t_small));
        k_spmv_t_small<<<1, 1024, small, s>>>(m, n, rp, ci, va, yd, wd, flag, rows_off);
        B2P_LAUNCH(ctx);
        ctx->launches += 1;
    } else {
        k_validate_csr<<<grid_for(m, 256, ctx->sm_count), 256, 0, s>>>(m, n, rp, ci, flag);
        B2P_CUDA(ctx, cudaMemcpyAsync(&bad, flag, sizeof(int32_t), cudaMemcpyDeviceToHost, s));
        B2P_CUDA(ctx, cudaStreamSynchronize(s));
        if (bad) return invalid();
        B2P_CUDA(ctx, ctx->s_t_rowptr.reserve((size_t)n + 1));
        B2P_CUDA(ctx, ctx->s_t_colidx.reserve(nnz));
        B2P_CUDA(ctx, ctx->s_t_vals.reserve(nnz));
        B2P_DO(build_transpose(ctx, m, n, nnz, rp, ci, va, ctx->s_t_rowptr.p, ctx->s_t_colidx.p, ctx->s_t_vals.p));
        k_spmv_f64<<<grid_for(n, 256, ctx->sm_count), 256, 0, s>>>(n, ctx->s_t_rowptr.p, ctx->s_t_colidx.p, ctx->s_t_vals.p,
                                                                   yd, wd);
        B2P_LAUNCH(ctx);
        ctx->launches += 2;
    }
    pt.mark(2);
    B2P_DO(io.receive());
    pt.mark(3);
    B2P_DO(io.finish(&bad));
    pt.fill(timing, t0);
    return bad ? invalid() : B2P_OK;
}

int b2p_vector_op(void* p, int op, size_t n, double alpha, const double* a, const double* bv, double* out,
                  b2p_timing_t* timing) {
    Ctx* ctx = as_ctx(p);
    if (!ctx) return B2P_GPU_UNINITIALIZED;
    if (op < 0 || op > 3 || !a || !out) return B2P_INVALID_ARGUMENT;
    bool needs_b = (op != B2P_VEC_SCALE);
    if (needs_b && !bv) return B2P_INVALID_ARGUMENT;
    if (n == 0) return B2P_OK;
    cudaSetDevice(ctx->device);
    double t0 = now_ms();
    PhaseTimer pt(ctx, timing);
    double *ad, *bd = nullptr, *od;
    CallIO io;
    B2P_DO(io.begin(ctx, 24 * n + 64));
    pt.mark(0);
    B2P_DO(io.in(ctx->s_x, a, n, &ad));
    if (needs_b) B2P_DO(io.in(ctx->s_y, bv, n, &bd));
    B2P_DO(io.send());
    B2P_DO(io.out(ctx->s_z, out, n, &od));
    pt.mark(1);
    k_vec<<<grid_for((int64_t)n, 256, ctx->sm_count), 256, 0, ctx->stream>>>(op, n, alpha, ad, bd, od);
    B2P_LAUNCH(ctx);
    ctx->launches += 1;
    pt.mark(2);
    B2P_DO(io.receive());
    pt.mark(3);
    B2P_DO(io.finish());
    pt.fill(timing, t0);
    return B2P_OK;
}

static int dot_impl(Ctx* ctx, size_t n, const double* a, const double* bv, double* out, b2p_timing_t* timing,
                    bool sqrt_out) {
    if (!ctx) return B2P_GPU_UNINITIALIZED;
    if (!a || !out) return B2P_INVALID_ARGUMENT;
    if (n == 0) {
        *out = 0.0;
        return B2P_OK;
    }
    cudaSetDevice(ctx->device);
    double t0 = now_ms();
    PhaseTimer pt(ctx, timing);
    cudaStream_t s = ctx->stream;
    double *ad, *bd = nullptr, *rd, r = 0.0;
    DBuf<double>& sums = ctx->s_t_vals;  // the blocks' partial sums
    CallIO io;
    B2P_DO(io.begin(ctx, 16 * n + 64));
    B2P_CUDA(ctx, sums.reserve(kRedBlocks));
    pt.mark(0);
    B2P_DO(io.in(ctx->s_x, a, n, &ad));
    if (bv) B2P_DO(io.in(ctx->s_y, bv, n, &bd));
    B2P_DO(io.send());
    B2P_DO(io.out(ctx->s_z, &r, 1, &rd));
    pt.mark(1);
    k_dot_partial<<<kRedBlocks, kRedThreads, 0, s>>>(n, ad, bd, sums.p);
    k_sum_partials<<<1, kRedThreads, 0, s>>>(kRedBlocks, sums.p, rd);
    B2P_LAUNCH(ctx);
    ctx->launches += 2;
    pt.mark(2);
    B2P_DO(io.receive());
    pt.mark(3);
    B2P_DO(io.finish());
    pt.fill(timing, t0);
    *out = sqrt_out ? std::sqrt(r) : r;
    return B2P_OK;
}

int b2p_dot(void* p, size_t n, const double* a, const double* b, double* out, b2p_timing_t* timing) {
    if (!b) return B2P_INVALID_ARGUMENT;
    return dot_impl(as_ctx(p), n, a, b, out, timing, false);
}

int b2p_norm2(void* p, size_t n, const double* a, double* out, b2p_timing_t* timing) {
    return dot_impl(as_ctx(p), n, a, nullptr, out, timing, true);
}

// ---- single LP upload
int b2p_upload_lp(void* p, int m, int n, int64_t nnz, const int32_t* rowptr, const int32_t* colidx,
                  const double* vals, const double* b, const double* c, const double* lb, const double* ub,
                  const uint8_t* is_eq) {
    Ctx* ctx = as_ctx(p);
    if (!ctx) return B2P_GPU_UNINITIALIZED;
    if (m <= 0 || n <= 0 || nnz < 0 || nnz > INT32_MAX || !rowptr || !b || !c || !lb || !ub || !is_eq) {
        ctx->err = "b2p_upload_lp: empty LP or null argument";
        return B2P_INVALID_ARGUMENT;
    }
    if (nnz > 0 && (!colidx || !vals)) return B2P_INVALID_ARGUMENT;
    if (!host_rowptr_ok(m, nnz, rowptr)) {
        ctx->err = "b2p_upload_lp: row pointer array is not a valid CSR offset array";
        return B2P_INVALID_ARGUMENT;
    }
    for (int j = 0; j < n; ++j) {
        if (std::isnan(lb[j]) || std::isnan(ub[j]) || std::isnan(c[j])) {
            ctx->err = "b2p_upload_lp: NaN in c / lb / ub";
            return B2P_INVALID_ARGUMENT;
        }
    }
    cudaSetDevice(ctx->device);
    cudaStream_t s = ctx->stream;
    ctx->has_lp = false;
    DevLP& L = ctx->lp;
    L.m = m;
    L.n = n;
    L.nnz = nnz;
    B2P_CUDA(ctx, L.rowptr.reserve(m + 1));
    B2P_CUDA(ctx, L.colidx.reserve(nnz));
    B2P_CUDA(ctx, L.vals.reserve(nnz));
    B2P_CUDA(ctx, L.t_rowptr.reserve(n + 1));
    B2P_CUDA(ctx, L.t_colidx.reserve(nnz));
    B2P_CUDA(ctx, L.t_vals.reserve(nnz));
    B2P_CUDA(ctx, L.b.reserve(m));
    B2P_CUDA(ctx, L.c.reserve(n));
    B2P_CUDA(ctx, L.lb.reserve(n));
    B2P_CUDA(ctx, L.ub.reserve(n));
    B2P_CUDA(ctx, L.is_eq.reserve(m));
    B2P_CUDA(ctx, ctx->s_flag.reserve(1));
    B2P_CUDA(ctx, cudaMemcpyAsync(L.rowptr.p, rowptr, sizeof(int32_t) * (m + 1), cudaMemcpyHostToDevice, s));
    if (nnz) {
        B2P_CUDA(ctx, cudaMemcpyAsync(L.colidx.p, colidx, sizeof(int32_t) * nnz, cudaMemcpyHostToDevice, s));
        B2P_CUDA(ctx, cudaMemcpyAsync(L.vals.p, vals, sizeof(double) * nnz, cudaMemcpyHostToDevice, s));
    }
    B2P_CUDA(ctx, cudaMemcpyAsync(L.b.p, b, sizeof(double) * m, cudaMemcpyHostToDevice, s));
    B2P_CUDA(ctx, cudaMemcpyAsync(L.c.p, c, sizeof(double) * n, cudaMemcpyHostToDevice, s));
    B2P_CUDA(ctx, cudaMemcpyAsync(L.lb.p, lb, sizeof(double) * n, cudaMemcpyHostToDevice, s));
    B2P_CUDA(ctx, cudaMemcpyAsync(L.ub.p, ub, sizeof(double) * n, cudaMemcpyHostToDevice, s));
    B2P_CUDA(ctx, cudaMemcpyAsync(L.is_eq.p, is_eq, m, cudaMemcpyHostToDevice, s));
    B2P_CUDA(ctx, cudaMemsetAsync(ctx->s_flag.p, 0, sizeof(int32_t), s));
    k_validate_csr<<<grid_for(m, 256, ctx->sm_count), 256, 0, s>>>(m, n, L.rowptr.p, L.colidx.p, ctx->s_flag.p);
    B2P_LAUNCH(ctx);
    ctx->launches += 1;
    int32_t bad = 0;
    B2P_CUDA(ctx, cudaMemcpyAsync(&bad, ctx->s_flag.p, sizeof(int32_t), cudaMemcpyDeviceToHost, s));
    B2P_CUDA(ctx, cudaStreamSynchronize(s));
    if (bad) {
        ctx->err = "b2p_upload_lp: column indices out of range or not strictly ascending in row " + std::to_string(bad - 1);
        return B2P_INVALID_ARGUMENT;
    }
    int st = build_transpose(ctx, m, n, nnz, L.rowptr.p, L.colidx.p, L.vals.p, L.t_rowptr.p, L.t_colidx.p, L.t_vals.p);
    if (st) return st;
    double bn = 0, cn = 0;
    for (int i = 0; i < m; ++i) bn += b[i] * b[i];
    for (int j = 0; j < n; ++j) cn += c[j] * c[j];
    L.bnorm = std::sqrt(bn);
    L.cnorm = std::sqrt(cn);
    L.mean_row_len = (double)nnz / m;
    L.mean_col_len = (double)nnz / n;
    int mr = 0;
    for (int i = 0; i < m; ++i) mr = std::max(mr, rowptr[i + 1] - rowptr[i]);
    L.max_row_len = mr;
    ctx->lp_gen += 1;
    ctx->has_lp = true;
    return B2P_OK;
}

int b2p_solve(void* p, const b2p_params* params, const double* x0, const double* y0, b2p_result* result,
              double* x_out, double* y_out) {
    Ctx* ctx = as_ctx(p);
    if (!ctx) return B2P_GPU_UNINITIALIZED;
    if (!result) return B2P_INVALID_ARGUMENT;
    if (!ctx->has_lp) {
        ctx->err = "b2p_solve: no LP uploaded";
        return B2P_NO_LP;
    }
    b2p_params def;
    b2p_params_default(&def);
    const b2p_params* pp = params ? params : &def;
    std::memset(result, 0, sizeof(*result));
    if (pp->max_iterations < 0 || pp->check_frequency <= 0 || pp->check_every <= 0) {
        ctx->err = "b2p_solve: max_iterations < 0 or non-positive check cadence";
        return B2P_INVALID_ARGUMENT;
    }
    cudaSetDevice(ctx->device);
    int64_t l0 = ctx->launches;
    double t0 = now_ms();
    int st;
    if (pp->engine == B2P_ENGINE_REFERENCE)
        st = ref_engine_solve(ctx, pp, result, x_out, y_out);
    else if (pp->engine == B2P_ENGINE_HALPERN)
        st = halpern_engine_solve(ctx, pp, x0, y0, result, x_out, y_out);
    else {
        ctx->err = "b2p_solve: unknown engine";
        return B2P_INVALID_ARGUMENT;
    }
    result->solve_time_ms = now_ms() - t0;
    result->kernel_launches = ctx->launches - l0;
    return st;
}

}  // extern "C"
