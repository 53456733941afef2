// Context, device discovery, error text and the MatVec-operator entry points of the C ABI.
#include <cstring>
#include <iterator>
#include <map>
#include <mutex>
#include <string>

#include "common.cuh"
#include <algorithm>

#include "gemm_quant.cuh"
#include "gemv.cuh"
#include "prompt.cuh"
#include "qgemv.cuh"

namespace juno {

static thread_local char g_err[512] = "";

void set_error(const char *fmt, ...) {
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_err, sizeof(g_err), fmt, ap);
    va_end(ap);
}
const char *get_error() { return g_err; }

int ctx_check(juno_ctx *c) {
    if (!c) {
        set_error("context is null");
        return JUNO_ERR_INVALID_ARG;
    }
    if (c->magic != kMagicCtx) {
        set_error("context is closed");
        return JUNO_ERR_CLOSED;
    }
    return JUNO_OK;
}

int ensure_device(void **ptr, size_t *cur, size_t want) {
    if (*cur >= want && *ptr) return JUNO_OK;
    void *np = nullptr;
    cudaError_t e = cudaMalloc(&np, want);
    if (e != cudaSuccess) {
        cudaGetLastError();
        set_error("cudaMalloc of %zu bytes failed: %s", want, cudaGetErrorString(e));
        return JUNO_ERR_OOM;
    }
    if (*ptr) {
        cudaDeviceSynchronize();
        cudaFree(*ptr);
    }
    *ptr = np;
    *cur = want;
    return JUNO_OK;
}

int ensure_pinned(juno_ctx *c, size_t want) {
    if (c->pinned_bytes >= want && c->pinned) return JUNO_OK;
    if (c->pinned) cudaFreeHost(c->pinned);
    c->pinned = nullptr;
    c->pinned_bytes = 0;
    cudaError_t e = cudaMallocHost(&c->pinned, want);
    if (e != cudaSuccess) {
        cudaGetLastError();
        set_error("cudaMallocHost of %zu bytes failed: %s", want, cudaGetErrorString(e));
        return JUNO_ERR_OOM;
    }
    c->pinned_bytes = want;
    return JUNO_OK;
}

int wait_status(juno_ctx *c, WaitWord which) {
    const unsigned code = __atomic_exchange_n(c->gemv_scratch.qerr_host + which, 0u, __ATOMIC_ACQ_REL);
    if (!code) return JUNO_OK;
    if ((code & 0xffu) == kErrStackWait)
        set_error("a matrix product gave up waiting inside a kernel (stage %u of block %u)", (code >> 8) & 0xffu, code >> 16);
    else if ((code & 0xffu) >= 3u)
        set_error("tensor-parallel rank %u did not deliver its %s within a second (this rank gave up waiting)", (code >> 8) & 0xffu,
                  (code & 0xffu) == 3u ? "partial products" : "greedy pick");
    else
        set_error("a GEMV warp gave up waiting for a weight tile (warp %u of block %u)", (code >> 8) & 0xffu, code >> 16);
    return JUNO_ERR_TIMEOUT;
}

// Page-locked blocks for results that a host reads.  One pool for the process, because a result may outlive the context that wrote
// it.  A block is at most an eighth longer than asked for (short ones: a multiple of 256 KB), all of them together have at most
// kHostPoolBytes; those that nobody holds are given back when a context closes, and as many of them as it takes when another size needs
// the room.
constexpr size_t kHostPoolBytes = (size_t)96 << 20, kHostBlockMin = (size_t)256 << 10;
struct HostPool {
    std::mutex mu;
    std::map<void *, size_t> held;
    std::multimap<size_t, void *> idle;
    size_t held_bytes = 0, idle_bytes = 0;
    static size_t block_size(size_t bytes) {
        size_t unit = kHostBlockMin;
        while (unit * 16 <= bytes) unit *= 2;
        return (bytes + unit - 1) / unit * unit;
    }
    void hold(void *p, size_t size) {
        held[p] = size;
        held_bytes += size;
    }
    // Gives idle blocks back, the longest first, until at most `most` bytes of them are left.
    void release_idle(size_t most) {
        while (idle_bytes > most) {
            const auto it = std::prev(idle.end());
            cudaFreeHost(it->second);
            idle_bytes -= it->first;
            idle.erase(it);
        }
    }
};
static HostPool &host_pool() {
    static HostPool *p = new HostPool();  // never destroyed: results may be dropped while the process exits
    return *p;
}

}  // namespace juno

using namespace juno;

extern "C" {

int juno_host_alloc(juno_ctx *c, int64_t bytes, void **out) {
    JUNO_TRY(ctx_check(c));
    JUNO_REQUIRE(out && bytes > 0, "bad host allocation (%lld bytes)", (long long)bytes);
    const size_t size = HostPool::block_size((size_t)std::min<int64_t>(bytes, kHostPoolBytes + 1));
    HostPool &h = host_pool();
    std::lock_guard<std::mutex> lk(h.mu);
    const auto it = h.idle.lower_bound(size);
    if (it != h.idle.end() && it->first <= size + size / 4) {
        *out = it->second;
        h.hold(it->second, it->first);
        h.idle_bytes -= it->first;
        h.idle.erase(it);
        return JUNO_OK;
    }
    void *p = nullptr;
    bool ok = h.held_bytes + size <= kHostPoolBytes;  // otherwise giving back would not help
    if (ok) {
        DeviceGuard g(c->device);
        h.release_idle(kHostPoolBytes - h.held_bytes - size);
        ok = cudaHostAlloc(&p, size, cudaHostAllocPortable) == cudaSuccess;
        if (!ok) cudaGetLastError();
    }
    if (!ok) {
        set_error("no page-locked block of %lld bytes is free", (long long)bytes);
        return JUNO_ERR_OOM;
    }
    h.hold(p, size);
    *out = p;
    return JUNO_OK;
}

int juno_host_free(void *block) {
    HostPool &h = host_pool();
    std::lock_guard<std::mutex> lk(h.mu);
    const auto it = h.held.find(block);
    JUNO_REQUIRE(it != h.held.end(), "not a block of juno_host_alloc");
    h.idle.emplace(it->second, block);
    h.idle_bytes += it->second;
    h.held_bytes -= it->second;
    h.held.erase(it);
    return JUNO_OK;
}

const char *juno_last_error(void) { return get_error(); }

int juno_device_count(int32_t *count) {
    if (!count) return JUNO_ERR_INVALID_ARG;
    int n = 0;
    cudaError_t e = cudaGetDeviceCount(&n);
    if (e != cudaSuccess) {  // no driver / no device: fail soft like CudaAvailability
        cudaGetLastError();
        n = 0;
    }
    *count = n;
    return JUNO_OK;
}

int juno_device_name(int32_t device, char *buf, int32_t buf_len) {
    JUNO_REQUIRE(buf && buf_len > 0, "name buffer missing");
    cudaDeviceProp prop;
    JUNO_CUDA_TRY(cudaGetDeviceProperties(&prop, device));
    snprintf(buf, (size_t)buf_len, "%s", prop.name);
    return JUNO_OK;
}

int juno_device_total_mem(int32_t device, int64_t *bytes) {
    JUNO_REQUIRE(bytes, "bytes is null");
    cudaDeviceProp prop;
    JUNO_CUDA_TRY(cudaGetDeviceProperties(&prop, device));
    *bytes = (int64_t)prop.totalGlobalMem;
    return JUNO_OK;
}

int juno_ctx_create(int32_t device, juno_ctx **out) {
    JUNO_REQUIRE(out, "out is null");
    int n = 0;
    if (cudaGetDeviceCount(&n) != cudaSuccess || n == 0) {
        cudaGetLastError();
        set_error("no CUDA device available (this backend has no CPU fallback)");
        return JUNO_ERR_CUDA;
    }
    JUNO_REQUIRE(device >= 0 && device < n, "device %d out of range [0,%d)", device, n);
    cudaDeviceProp prop;
    JUNO_CUDA_TRY(cudaGetDeviceProperties(&prop, device));
    if (prop.major != 10) {
        set_error("device %d is sm_%d%d; this library contains sm_100a code only", device, prop.major, prop.minor);
        return JUNO_ERR_UNSUPPORTED;
    }
    DeviceGuard g(device);
    juno_ctx *c = new juno_ctx();
    c->magic = kMagicCtx;
    c->device = device;
    c->sm_count = prop.multiProcessorCount;
    c->smem_optin = prop.sharedMemPerBlockOptin;
    cudaError_t e = cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking);
    if (e != cudaSuccess) {
        set_error("cudaStreamCreateWithFlags failed: rc=%d (%s)", (int)e, cudaGetErrorString(e));
        delete c;
        return JUNO_ERR_CUDA;
    }
    // one word in mapped host memory: a kernel that gave up a wait leaves its code there, the host reads it for free
    if (e == cudaSuccess) e = cudaHostAlloc((void **)&c->gemv_scratch.qerr_host, 64, cudaHostAllocMapped);
    if (e == cudaSuccess) {
        memset(c->gemv_scratch.qerr_host, 0, 64);
        e = cudaHostGetDevicePointer((void **)&c->gemv_scratch.qerr, c->gemv_scratch.qerr_host, 0);
    }
    if (e != cudaSuccess) {
        set_error("context set-up failed: rc=%d (%s)", (int)e, cudaGetErrorString(e));
        delete c;
        return e == cudaErrorMemoryAllocation ? JUNO_ERR_OOM : JUNO_ERR_CUDA;
    }
    *out = c;
    return JUNO_OK;
}

int juno_ctx_destroy(juno_ctx *c) {
    JUNO_TRY(ctx_check(c));
    std::lock_guard<std::recursive_mutex> lk(c->mu);
    DeviceGuard g(c->device);
    cudaStreamSynchronize(c->stream);
    if (c->gemv_scratch.ximg) cudaFree(c->gemv_scratch.ximg);
    if (c->gemv_scratch.xscale) cudaFree(c->gemv_scratch.xscale);
    if (c->gemv_scratch.qerr_host) cudaFreeHost(c->gemv_scratch.qerr_host);
    if (c->stage_x) cudaFree(c->stage_x);
    if (c->stage_y) cudaFree(c->stage_y);
    if (c->pinned) cudaFreeHost(c->pinned);
    cudaStreamDestroy(c->stream);
    {
        HostPool &h = host_pool();
        std::lock_guard<std::mutex> hk(h.mu);
        h.release_idle(0);
    }
    c->magic = kMagicDead;  // record kept: a second destroy reports CLOSED
    return JUNO_OK;
}

int juno_ctx_device(juno_ctx *c, int32_t *device) {
    JUNO_TRY(ctx_check(c));
    JUNO_REQUIRE(device, "device is null");
    *device = c->device;
    return JUNO_OK;
}

int juno_ctx_synchronize(juno_ctx *c) {
    JUNO_TRY(ctx_check(c));
    DeviceGuard g(c->device);
    JUNO_CUDA_TRY(cudaStreamSynchronize(c->stream));
    return wait_status(c, WAIT_ENQUEUED);
}

int juno_ctx_stream(juno_ctx *c, void **stream) {
    JUNO_TRY(ctx_check(c));
    JUNO_REQUIRE(stream, "stream is null");
    *stream = (void *)c->stream;
    return JUNO_OK;
}

int juno_ctx_profile(juno_ctx *c, int32_t enable) {
    JUNO_TRY(ctx_check(c));
    std::lock_guard<std::recursive_mutex> lk(c->mu);
    c->profiling = enable != 0;
    return JUNO_OK;
}

int juno_ctx_profile_read(juno_ctx *c, juno_profile_entry *out, int32_t n_entries, int32_t reset) {
    JUNO_TRY(ctx_check(c));
    JUNO_REQUIRE(out && n_entries >= 1, "bad output array");
    std::lock_guard<std::recursive_mutex> lk(c->mu);
    DeviceGuard g(c->device);
    JUNO_CUDA_TRY(cudaStreamSynchronize(c->stream));
    for (auto &sp : c->prof_spans) {
        float ms = 0.f;
        if (cudaEventElapsedTime(&ms, sp.e0, sp.e1) == cudaSuccess) {
            c->prof_ms[sp.cat] += ms;
            c->prof_bytes[sp.cat] += sp.bytes;
            c->prof_launches[sp.cat]++;
        }
        cudaEventDestroy(sp.e0);
        cudaEventDestroy(sp.e1);
    }
    cudaGetLastError();
    c->prof_spans.clear();
    for (int i = 0; i < n_entries && i < PROF_COUNT; i++) {
        out[i].launches = c->prof_launches[i];
        out[i].ms = c->prof_ms[i];
        out[i].algo_bytes = c->prof_bytes[i];
    }
    if (reset)
        for (int i = 0; i < PROF_COUNT; i++) {
            c->prof_launches[i] = 0;
            c->prof_ms[i] = c->prof_bytes[i] = 0;
        }
    return JUNO_OK;
}

int juno_ctx_counters(juno_ctx *c, juno_counters *out, int32_t reset) {
    JUNO_TRY(ctx_check(c));
    if (out) {
        out->kernel_launches = c->kernel_launches.load();
        out->gemv_calls = c->gemv_calls.load();
        out->forward_calls = c->forward_calls.load();
        out->h2d_bytes = c->h2d_bytes.load();
        out->d2h_bytes = c->d2h_bytes.load();
    }
    if (reset) {
        c->kernel_launches = 0;
        c->gemv_calls = 0;
        c->forward_calls = 0;
        c->h2d_bytes = 0;
        c->d2h_bytes = 0;
    }
    return JUNO_OK;
}

// ── MatVec operator ────────────────────────────────────────────────────────────
int juno_qmat_upload(juno_ctx *c, const void *blocks, int32_t type, int64_t rows, int64_t cols, juno_qmat **out) {
    JUNO_TRY(ctx_check(c));
    JUNO_REQUIRE(blocks && out, "null argument");
    std::lock_guard<std::recursive_mutex> lk(c->mu);
    DeviceGuard g(c->device);
    return qmat_create(c, blocks, type, rows, cols, 0, rows, 0, 0, out);
}

int juno_qmat_free(juno_qmat *m) {
    if (!m) {
        set_error("matrix is null");
        return JUNO_ERR_INVALID_ARG;
    }
    if (m->magic != kMagicQmat) {
        set_error("matrix handle is closed");
        return JUNO_ERR_CLOSED;
    }
    std::lock_guard<std::recursive_mutex> lk(m->ctx->mu);
    return qmat_destroy(m);
}

static int qmat_check(juno_qmat *m) {
    if (!m) {
        set_error("matrix is null");
        return JUNO_ERR_INVALID_ARG;
    }
    if (m->magic != kMagicQmat) {
        set_error("matrix handle is closed");
        return JUNO_ERR_CLOSED;
    }
    return JUNO_OK;
}

int juno_qmat_shape(juno_qmat *m, int64_t *rows, int64_t *cols, int32_t *type) {
    JUNO_TRY(qmat_check(m));
    if (rows) *rows = m->rows;
    if (cols) *cols = m->cols;
    if (type) *type = m->type;
    return JUNO_OK;
}

static int gemv_on_stream(juno_ctx *c, juno_qmat *m, const float *x, int batch, float *y, cudaStream_t st) {
    if (!m->tiled) return launch_gemv_raw(c, m, x, batch, y, st);
    const bool batched = batch >= gemm_min_batch();
    if (!batched) {
        QGemvArgs q;
        q.nseg = 1;
        q.seg[0].w = m->dev;
        q.seg[0].out = y;
        q.seg[0].rows = (int)m->rows;
        q.seg[0].row_tiles = (int)m->row_tiles;
        q.seg[0].type = m->type;
        q.K = (int)m->cols;
        q.batch = batch;
        q.ld_out = (int)m->rows;
        q.x = x;
        q.ldx = (int)m->cols;
        return launch_qgemv(c, q, st);
    }
    const size_t need = (size_t)m->cols * 2 * std::min(batch, kGemmMaxBatch);
    void *pi = c->gemv_scratch.ximg;
    JUNO_TRY(ensure_device(&pi, &c->gemv_scratch.ximg_bytes, need));
    c->gemv_scratch.ximg = (uint8_t *)pi;
    if (!c->gemv_scratch.xscale) {
        cudaError_t e = cudaMalloc((void **)&c->gemv_scratch.xscale, kGemmMaxBatch * sizeof(float));
        if (e != cudaSuccess) {
            cudaGetLastError();
            set_error("cudaMalloc of %zu bytes failed: %s", kGemmMaxBatch * sizeof(float), cudaGetErrorString(e));
            return JUNO_ERR_OOM;
        }
    }
    // one pass over the weights per group of up to kGemmMaxBatch rows
    for (int b0 = 0; b0 < batch; b0 += kGemmMaxBatch) {
        StageRowsArgs s;
        s.x = x + (size_t)b0 * m->cols;
        s.n = std::min(kGemmMaxBatch, batch - b0);
        s.K = (int)m->cols;
        s.out = c->gemv_scratch.ximg;
        s.scale = c->gemv_scratch.xscale;
        s.quant_order = true;
        JUNO_TRY(launch_stage_rows(c, s, st));
        GemmQuantArgs a;
        a.seg[0].w = m->dev;
        a.seg[0].out = y + (size_t)b0 * m->rows;
        a.seg[0].rows = (int)m->rows;
        a.seg[0].row_tiles = (int)m->row_tiles;
        a.seg[0].type = m->type;
        a.seg[0].row_pow = m->row_pow;
        a.K = s.K;
        a.n = s.n;
        a.x = s.out;
        a.scale = s.scale;
        a.ld_out = (int)m->rows;
        JUNO_TRY(launch_gemm_quant(c, a, st));
    }
    return JUNO_OK;
}

int juno_gemv_device(juno_ctx *c, juno_qmat *m, const float *x_dev, int32_t batch, float *y_dev, void *stream) {
    JUNO_TRY(ctx_check(c));
    JUNO_TRY(qmat_check(m));
    JUNO_REQUIRE(m->ctx == c, "matrix belongs to another context");
    JUNO_REQUIRE(x_dev && y_dev && batch >= 1, "bad gemv arguments (batch=%d)", batch);
    std::lock_guard<std::recursive_mutex> lk(c->mu);
    DeviceGuard g(c->device);
    c->gemv_calls++;
    unsigned *const blocking = c->gemv_scratch.qerr;
    c->gemv_scratch.qerr = blocking + WAIT_ENQUEUED;
    const int rc = gemv_on_stream(c, m, x_dev, batch, y_dev, stream ? (cudaStream_t)stream : c->stream);
    c->gemv_scratch.qerr = blocking;
    return rc;
}

int juno_gemv(juno_ctx *c, juno_qmat *m, const float *x_host, int32_t batch, float *y_host) {
    JUNO_TRY(ctx_check(c));
    JUNO_TRY(qmat_check(m));
    JUNO_REQUIRE(m->ctx == c, "matrix belongs to another context");
    JUNO_REQUIRE(x_host && y_host, "null vector");
    JUNO_REQUIRE(batch >= 1 && batch <= 4096, "batch %d out of range", batch);
    std::lock_guard<std::recursive_mutex> lk(c->mu);
    DeviceGuard g(c->device);
    const size_t xb = (size_t)batch * m->cols * sizeof(float), yb = (size_t)batch * m->rows * sizeof(float);
    void *px = c->stage_x, *py = c->stage_y;
    JUNO_TRY(ensure_device(&px, &c->stage_x_bytes, xb));
    c->stage_x = (float *)px;
    JUNO_TRY(ensure_device(&py, &c->stage_y_bytes, yb));
    c->stage_y = (float *)py;
    JUNO_CUDA_TRY(cudaMemcpyAsync(c->stage_x, x_host, xb, cudaMemcpyHostToDevice, c->stream));
    c->gemv_calls++;
    JUNO_TRY(gemv_on_stream(c, m, c->stage_x, batch, c->stage_y, c->stream));
    JUNO_CUDA_TRY(cudaMemcpyAsync(y_host, c->stage_y, yb, cudaMemcpyDeviceToHost, c->stream));
    JUNO_CUDA_TRY(cudaStreamSynchronize(c->stream));
    JUNO_TRY(wait_status(c, WAIT_BLOCKING));
    c->h2d_bytes += (int64_t)xb;
    c->d2h_bytes += (int64_t)yb;
    return JUNO_OK;
}

int juno_dequantize(juno_ctx *c, juno_qmat *m, int64_t row_start, int64_t n_rows, float *out_host) {
    JUNO_TRY(ctx_check(c));
    JUNO_TRY(qmat_check(m));
    JUNO_REQUIRE(out_host, "out is null");
    JUNO_REQUIRE(row_start >= 0 && n_rows >= 0 && row_start + n_rows <= m->rows, "row range [%lld,+%lld) outside %lld rows",
                 (long long)row_start, (long long)n_rows, (long long)m->rows);
    if (n_rows == 0) return JUNO_OK;
    std::lock_guard<std::recursive_mutex> lk(c->mu);
    DeviceGuard g(c->device);
    const size_t bytes = (size_t)n_rows * m->cols * sizeof(float);
    void *py = c->stage_y;
    JUNO_TRY(ensure_device(&py, &c->stage_y_bytes, bytes));
    c->stage_y = (float *)py;
    JUNO_TRY(launch_dequant(c, m, row_start, n_rows, c->stage_y, c->stream));
    JUNO_CUDA_TRY(cudaMemcpyAsync(out_host, c->stage_y, bytes, cudaMemcpyDeviceToHost, c->stream));
    JUNO_CUDA_TRY(cudaStreamSynchronize(c->stream));
    c->d2h_bytes += (int64_t)bytes;
    return JUNO_OK;
}

int juno_sgemv_f32(juno_ctx *c, const float *a_host, const float *x_host, int64_t rows, int64_t cols, float *y_host) {
    JUNO_TRY(ctx_check(c));
    JUNO_REQUIRE(a_host && x_host && y_host, "null argument");
    JUNO_REQUIRE(rows >= 1 && cols >= 1, "rows*cols must be positive (rows=%lld cols=%lld)", (long long)rows,
                 (long long)cols);
    juno_qmat *m = nullptr;
    JUNO_TRY(juno_qmat_upload(c, a_host, JUNO_TYPE_F32, rows, cols, &m));
    int rc = juno_gemv(c, m, x_host, 1, y_host);
    juno_qmat_free(m);
    delete m;
    return rc;
}

}  // extern "C"
