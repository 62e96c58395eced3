// Context, memory, transfer and timing entry points of the C ABI.
#include <stdarg.h>
#include <string.h>

#include <stdlib.h>

#include <map>
#include <mutex>
#include <new>
#include <unordered_map>
#include <vector>

#include "common.cuh"
#include "launch.cuh"

static thread_local char g_error[512] = "";

int32_t katsu_set_error(int32_t code, const char *fmt, ...) {
    va_list args;
    va_start(args, fmt);
    vsnprintf(g_error, sizeof(g_error), fmt, args);
    va_end(args);
    return code;
}

extern "C" const char *katsu_cuda_last_error_string(void) { return g_error; }

int32_t katsu_bind(katsu_cuda_ctx *ctx) {
    if (ctx == nullptr) return katsu_set_error(KATSU_ERR_INVALID_ARG, "null context");
    KATSU_CUDA_TRY(cudaSetDevice(ctx->device));
    return KATSU_OK;
}

int32_t katsu_prepare_kernel(katsu_cuda_ctx *ctx, const void *kernel, size_t smem) {
    // contexts of several threads may launch the same kernel for the first time
    static std::mutex lock;
    static std::unordered_map<const void *, size_t> *prepared = new std::unordered_map<const void *, size_t>[64];
    const std::lock_guard<std::mutex> hold(lock);
    std::unordered_map<const void *, size_t> &of_device = prepared[ctx->device & 63];
    const auto it = of_device.find(kernel);
    if (it != of_device.end() && it->second >= smem) return KATSU_OK;
    if (smem) KATSU_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    KATSU_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared));
    try {
        of_device[kernel] = smem;
    } catch (...) {  // no host memory for the entry: set again by the next launch
    }
    return KATSU_OK;
}

// ---- freed blocks ----------------------------------------------------------------------------------------------
// A training step frees and allocates the same few buffers of up to hundreds of megabytes.  The pool serves that from
// cached memory only while it finds a fitting piece; when steps of different sizes alternate it maps and unmaps physical
// memory inside a step (the small CNN's step took 3 to 40 ms that way, 2 ms of it kernels).  So a freed block stays
// whole and goes to the next request of nearly its size.  All use of a context's blocks is on its one stream, so reuse
// needs no event, and one host thread drives a context.  At most an eighth of the device's memory is held; an allocation
// (the scratch block's too) that fails gives everything held back and tries again; shutdown gives everything back.
struct KatsuBlock {
    size_t bytes;
    bool held;  // freed by the caller and not handed out again
};

struct KatsuBlockCache {
    std::unordered_map<void *, KatsuBlock> blocks;  // every block this context has handed out or holds
    std::multimap<size_t, void *> held;
    size_t held_bytes = 0, most_bytes = 0;
    std::vector<void *> retired;  // earlier scratch blocks that captured graphs refer to
};

static size_t block_bytes(size_t bytes) {
    const size_t grain = bytes < (size_t(1) << 20) ? 512 : size_t(2) << 20;
    return (bytes + grain - 1) / grain * grain;
}

bool katsu_capturing(const katsu_cuda_ctx *ctx) {
    cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
    return cudaStreamIsCapturing(ctx->stream, &status) == cudaSuccess && status != cudaStreamCaptureStatusNone;
}

static void give_back_blocks(katsu_cuda_ctx *ctx) {
    KatsuBlockCache &cache = *ctx->blocks;
    for (auto &entry : cache.held) {
        cache.blocks.erase(entry.second);
        cudaFreeAsync(entry.second, ctx->stream);
    }
    cache.held.clear();
    cache.held_bytes = 0;
}

// While the stream is being captured the cache stays out of it: what a capture allocates belongs to its graph.
static int32_t take_block(katsu_cuda_ctx *ctx, size_t bytes, void **out) {
    if (katsu_capturing(ctx)) return katsu_pool_alloc(ctx, bytes, out);
    KatsuBlockCache &cache = *ctx->blocks;
    const size_t want = block_bytes(bytes);
    auto it = cache.held.lower_bound(want);
    if (it != cache.held.end() && it->first <= want + want / 8) {
        *out = it->second;
        cache.held_bytes -= it->first;
        cache.held.erase(it);
        cache.blocks.find(*out)->second.held = false;
        return KATSU_OK;
    }
    KATSU_TRY(katsu_pool_alloc(ctx, want, out));
    try {
        cache.blocks[*out] = KatsuBlock{want, false};
    } catch (...) {  // no host memory for the entry: the block goes straight back to the pool when it is freed
    }
    return KATSU_OK;
}

// *kept = false when the block has to go to the driver (another context of the device handed it out, a capture runs, or
// the cache is full).  A block that the caller has freed already is refused, as the driver refuses it.
static int32_t keep_block(katsu_cuda_ctx *ctx, void *ptr, bool *kept) {
    *kept = false;
    KatsuBlockCache &cache = *ctx->blocks;
    auto it = cache.blocks.find(ptr);
    if (it == cache.blocks.end()) return KATSU_OK;
    if (it->second.held) return katsu_set_error(KATSU_ERR_CUDA, "block %p is freed twice", ptr);
    if (katsu_capturing(ctx)) return KATSU_OK;
    const size_t bytes = it->second.bytes;
    try {
        if (cache.held_bytes + bytes <= cache.most_bytes) {
            cache.held.emplace(bytes, ptr);
            cache.held_bytes += bytes;
            it->second.held = *kept = true;
            return KATSU_OK;
        }
    } catch (...) {
    }
    cache.blocks.erase(it);
    return KATSU_OK;
}

static cudaError_t pool_malloc(katsu_cuda_ctx *ctx, size_t bytes, void **out) {
    return ctx->pool != nullptr ? cudaMallocFromPoolAsync(out, bytes, (cudaMemPool_t)ctx->pool, ctx->stream)
                                : cudaMallocAsync(out, bytes, ctx->stream);
}

int32_t katsu_pool_alloc(katsu_cuda_ctx *ctx, size_t bytes, void **out) {
    cudaError_t err = pool_malloc(ctx, bytes, out);
    if (err != cudaSuccess && !ctx->blocks->held.empty() && !katsu_capturing(ctx)) {
        cudaGetLastError();
        give_back_blocks(ctx);
        cudaStreamSynchronize(ctx->stream);
        err = pool_malloc(ctx, bytes, out);
    }
    if (err != cudaSuccess) {
        cudaGetLastError();
        *out = nullptr;
        return katsu_set_error(KATSU_ERR_ALLOC, "stream-ordered allocation of %zu bytes: %s", bytes,
                               cudaGetErrorString(err));
    }
    return KATSU_OK;
}

// A graph's kernels and tensor maps hold the address of the scratch block that they were captured with, for as long as the
// caller keeps the graph.  So a block that a capture has used is never given back before shutdown, and a block that a capture
// asks for is allocated beside it: allocated on the capturing stream it would belong to the graph, and be there only while
// the graph runs.  One block is kept back for every growth behind a capture.
int32_t katsu_scratch(katsu_cuda_ctx *ctx, size_t floats, float **out) {
    const bool capturing = katsu_capturing(ctx);
    if (floats > ctx->scratch_floats) {
        const size_t want = floats < (size_t(1) << 20) ? (size_t(1) << 20) : floats;
        void *p = nullptr;
        if (capturing || ctx->scratch_captured) {
            try {
                ctx->blocks->retired.reserve(ctx->blocks->retired.size() + 1);
            } catch (...) {
                return katsu_set_error(KATSU_ERR_ALLOC, "out of host memory");
            }
        }
        if (capturing) {
            cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
            KATSU_CUDA_TRY(cudaThreadExchangeStreamCaptureMode(&mode));
            const cudaError_t err = cudaMalloc(&p, want * sizeof(float));
            cudaThreadExchangeStreamCaptureMode(&mode);
            if (err != cudaSuccess) {
                cudaGetLastError();
                return katsu_set_error(KATSU_ERR_ALLOC, "scratch of %zu bytes: %s", want * sizeof(float), cudaGetErrorString(err));
            }
        }
        // Stream-ordered: launches already queued keep the old block until they have run, and the
        // new one comes from the context's pool, so growing the scratch does not stall the device.
        if (ctx->scratch && (capturing || ctx->scratch_captured)) ctx->blocks->retired.push_back(ctx->scratch);
        else if (ctx->scratch) KATSU_CUDA_TRY(cudaFreeAsync(ctx->scratch, ctx->stream));
        ctx->scratch = nullptr;
        ctx->scratch_floats = 0;
        ctx->scratch_captured = false;
        if (!capturing) KATSU_TRY(katsu_pool_alloc(ctx, want * sizeof(float), &p));
        ctx->scratch = (float *)p;
        ctx->scratch_floats = want;
    }
    if (capturing) ctx->scratch_captured = true;
    *out = ctx->scratch;
    return KATSU_OK;
}

// Reads the status word of the bounded device-side waits after the host has waited for the stream
// (or for an event behind the kernels in question).  A non-zero word means some wait gave up: the
// results behind it are undefined, so every synchronising entry point reports it, and the word is
// cleared so that the context's next launches run normally again.
static int32_t katsu_report_status(katsu_cuda_ctx *ctx, int status) {
    if (status == 0) return KATSU_OK;
    cudaMemsetAsync(ctx->status, 0, sizeof(int), ctx->stream);
    cudaStreamSynchronize(ctx->stream);
    return katsu_set_error(KATSU_ERR_TIMEOUT, "a device-side wait gave up (status word %d)", status);
}

// Waits for the context's stream; the status word travels behind the queued work into a page-locked
// mirror, so the check costs no second synchronisation.
int32_t katsu_sync_and_check(katsu_cuda_ctx *ctx) {
    KATSU_CUDA_TRY(cudaMemcpyAsync(ctx->status_host, ctx->status, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
    KATSU_CUDA_TRY(cudaStreamSynchronize(ctx->stream));
    return katsu_report_status(ctx, *ctx->status_host);
}

extern "C" int32_t katsu_cuda_device_count(int32_t *out_count) {
    KATSU_REQUIRE(out_count != nullptr, "out_count is null");
    int n = 0;
    cudaError_t err = cudaGetDeviceCount(&n);
    if (err != cudaSuccess) {
        *out_count = 0;
        return katsu_set_error(KATSU_ERR_NO_DEVICE, "cudaGetDeviceCount: %s", cudaGetErrorString(err));
    }
    *out_count = n;
    return KATSU_OK;
}

extern "C" int32_t katsu_cuda_init(int32_t device, katsu_cuda_ctx **out_ctx) {
    KATSU_REQUIRE(out_ctx != nullptr, "out_ctx is null");
    *out_ctx = nullptr;
    int n = 0;
    cudaError_t err = cudaGetDeviceCount(&n);
    if (err != cudaSuccess || n == 0)
        return katsu_set_error(KATSU_ERR_NO_DEVICE, "no CUDA device: %s", cudaGetErrorString(err));
    if (device < 0 || device >= n)
        return katsu_set_error(KATSU_ERR_NO_DEVICE, "device ordinal %d out of range (0..%d)", device, n - 1);
    KATSU_CUDA_TRY(cudaSetDevice(device));
    cudaDeviceProp prop;
    KATSU_CUDA_TRY(cudaGetDeviceProperties(&prop, device));
    if (prop.major != 10)
        return katsu_set_error(KATSU_ERR_NO_DEVICE,
                               "device %d is sm_%d%d; this library only carries sm_100a code", device,
                               prop.major, prop.minor);
    katsu_cuda_ctx *ctx = new (std::nothrow) katsu_cuda_ctx();
    if (ctx == nullptr) return katsu_set_error(KATSU_ERR_ALLOC, "out of host memory");
    memset(ctx, 0, sizeof(*ctx));
    ctx->device = device;
    ctx->num_sms = prop.multiProcessorCount;
    ctx->precision = KATSU_MODE_3XTF32;
    ctx->blocks = new (std::nothrow) KatsuBlockCache();
    if (ctx->blocks == nullptr) {
        delete ctx;
        return katsu_set_error(KATSU_ERR_ALLOC, "out of host memory");
    }
    ctx->blocks->most_bytes = prop.totalGlobalMem / 8;
    // katsu_cuda_alloc / katsu_cuda_free and the kernels' scratch are stream-ordered allocations
    // from a pool private to this context that keeps freed blocks cached: an autograd step
    // allocates and frees the same few hundred MB of adjoint buffers every time, and cudaMalloc /
    // cudaFree each cost a device-wide synchronisation (measured: 34 ms -> a few ms per step of
    // the small CNN).  The pool is the context's own, so the host program's other users of the
    // device's default pool keep their release behaviour; it is destroyed at shutdown.
    {
        cudaMemPoolProps props;
        memset(&props, 0, sizeof(props));
        props.allocType = cudaMemAllocationTypePinned;
        props.handleTypes = cudaMemHandleTypeNone;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = device;
        cudaMemPool_t pool = nullptr;
        if (cudaMemPoolCreate(&pool, &props) == cudaSuccess) {
            unsigned long long keep = ~0ull;
            cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
            ctx->pool = pool;
        }
        cudaGetLastError();  // without a private pool the allocations fall back to cudaMallocAsync's default pool
    }
    err = cudaStreamCreateWithFlags(&ctx->stream, cudaStreamNonBlocking);
    if (err == cudaSuccess) err = cudaMalloc(&ctx->status, sizeof(int));
    if (err == cudaSuccess) err = cudaHostAlloc((void **)&ctx->status_host, sizeof(int), cudaHostAllocDefault);
    if (err == cudaSuccess) err = cudaMemsetAsync(ctx->status, 0, sizeof(int), ctx->stream);
    if (err == cudaSuccess) err = cudaMalloc(&ctx->f16_state, 1024);
    if (err == cudaSuccess) err = cudaMemsetAsync(ctx->f16_state, 0, 1024, ctx->stream);
    if (err != cudaSuccess) {
        if (ctx->status_host) cudaFreeHost(ctx->status_host);
        if (ctx->status) cudaFree(ctx->status);
        if (ctx->f16_state) cudaFree(ctx->f16_state);
        if (ctx->stream) cudaStreamDestroy(ctx->stream);
        if (ctx->pool) cudaMemPoolDestroy((cudaMemPool_t)ctx->pool);
        cudaGetLastError();
        delete ctx->blocks;
        delete ctx;
        return katsu_set_error(KATSU_ERR_CUDA, "context setup: %s", cudaGetErrorString(err));
    }
    *ctx->status_host = 0;
    *out_ctx = ctx;
    return KATSU_OK;
}

int32_t katsu_comm_destroy_impl(katsu_cuda_ctx *ctx);

extern "C" int32_t katsu_cuda_shutdown(katsu_cuda_ctx *ctx) {
    KATSU_TRY(katsu_bind(ctx));
    cudaStreamSynchronize(ctx->stream);
    if (ctx->comm) katsu_comm_destroy_impl(ctx);
    give_back_blocks(ctx);
    cudaStreamSynchronize(ctx->stream);
    if (ctx->scratch) cudaFree(ctx->scratch);
    for (void *block : ctx->blocks->retired) cudaFree(block);
    if (ctx->flush) cudaFree(ctx->flush);
    if (ctx->status) cudaFree(ctx->status);
    if (ctx->f16_state) cudaFree(ctx->f16_state);
    if (ctx->status_host) cudaFreeHost(ctx->status_host);
    cudaStreamDestroy(ctx->stream);
    // blocks still held by the caller stay valid: the driver releases the pool with its last allocation
    if (ctx->pool) cudaMemPoolDestroy((cudaMemPool_t)ctx->pool);
    cudaGetLastError();
    delete ctx->blocks;
    delete ctx;
    return KATSU_OK;
}

extern "C" int32_t katsu_cuda_set_precision(katsu_cuda_ctx *ctx, int32_t mode) {
    KATSU_REQUIRE(ctx != nullptr, "null context");
    KATSU_REQUIRE(mode == KATSU_MODE_3XTF32 || mode == KATSU_MODE_TF32 || mode == KATSU_MODE_FP32,
                  "unknown precision mode");
    ctx->precision = mode;
    return KATSU_OK;
}

extern "C" int32_t katsu_cuda_get_precision(katsu_cuda_ctx *ctx, int32_t *out_mode) {
    KATSU_REQUIRE(ctx != nullptr && out_mode != nullptr, "null argument");
    *out_mode = ctx->precision;
    return KATSU_OK;
}

extern "C" int32_t katsu_cuda_launch_count(katsu_cuda_ctx *ctx, uint64_t *out_count) {
    KATSU_REQUIRE(ctx != nullptr && out_count != nullptr, "null argument");
    *out_count = ctx->launches;
    return KATSU_OK;
}

extern "C" int32_t katsu_cuda_stream(katsu_cuda_ctx *ctx, void **out_stream) {
    KATSU_REQUIRE(ctx != nullptr && out_stream != nullptr, "null argument");
    *out_stream = (void *)ctx->stream;
    return KATSU_OK;
}

// ---- memory ----------------------------------------------------------------
extern "C" int32_t katsu_cuda_alloc_uninit(katsu_cuda_ctx *ctx, size_t count, float **out_ptr) {
    KATSU_REQUIRE(out_ptr != nullptr, "out_ptr is null");
    *out_ptr = nullptr;
    KATSU_TRY(katsu_bind(ctx));
    if (count == 0) return KATSU_OK;
    if (count > SIZE_MAX / sizeof(float) / 2)
        return katsu_set_error(KATSU_ERR_ALLOC, "allocation of %zu floats overflows", count);
    void *p = nullptr;
    KATSU_TRY(take_block(ctx, count * sizeof(float), &p));
    *out_ptr = (float *)p;
    return KATSU_OK;
}

extern "C" int32_t katsu_cuda_alloc(katsu_cuda_ctx *ctx, size_t count, float **out_ptr) {
    KATSU_TRY(katsu_cuda_alloc_uninit(ctx, count, out_ptr));
    if (count == 0) return KATSU_OK;
    cudaError_t err = cudaMemsetAsync(*out_ptr, 0, count * sizeof(float), ctx->stream);
    if (err != cudaSuccess) {
        katsu_cuda_free(ctx, *out_ptr);
        *out_ptr = nullptr;
        return katsu_set_error(KATSU_ERR_CUDA, "cudaMemsetAsync: %s", cudaGetErrorString(err));
    }
    return KATSU_OK;
}

extern "C" int32_t katsu_cuda_free(katsu_cuda_ctx *ctx, float *ptr) {
    KATSU_TRY(katsu_bind(ctx));
    if (ptr == nullptr) return KATSU_OK;
    // Stream-ordered: work already queued on this context's stream may still use the block;
    // work queued on another context must have been synchronised by the caller.
    bool kept = false;
    KATSU_TRY(keep_block(ctx, ptr, &kept));
    if (!kept) KATSU_CUDA_TRY(cudaFreeAsync(ptr, ctx->stream));
    return KATSU_OK;
}

extern "C" int32_t katsu_cuda_zero(katsu_cuda_ctx *ctx, float *dst, size_t count) {
    KATSU_TRY(katsu_bind(ctx));
    if (count == 0) return KATSU_OK;
    KATSU_REQUIRE(dst != nullptr, "dst is null");
    KATSU_CUDA_TRY(cudaMemsetAsync(dst, 0, count * sizeof(float), ctx->stream));
    return KATSU_OK;
}

extern "C" int32_t katsu_cuda_h2d(katsu_cuda_ctx *ctx, float *dst_device, const float *src_host, size_t count) {
    KATSU_TRY(katsu_bind(ctx));
    if (count == 0) return KATSU_OK;
    KATSU_REQUIRE(dst_device != nullptr && src_host != nullptr, "null buffer");
    KATSU_CUDA_TRY(cudaMemcpyAsync(dst_device, src_host, count * sizeof(float), cudaMemcpyHostToDevice,
                                   ctx->stream));
    return KATSU_OK;
}

extern "C" int32_t katsu_cuda_d2h(katsu_cuda_ctx *ctx, float *dst_host, const float *src_device, size_t count) {
    KATSU_TRY(katsu_bind(ctx));
    if (count != 0) {
        KATSU_REQUIRE(dst_host != nullptr && src_device != nullptr, "null buffer");
        KATSU_CUDA_TRY(cudaMemcpyAsync(dst_host, src_device, count * sizeof(float), cudaMemcpyDeviceToHost,
                                       ctx->stream));
    }
    // the data is only as good as the kernels that produced it: a wait that gave up is reported here too
    return katsu_sync_and_check(ctx);
}

extern "C" int32_t katsu_cuda_d2h_async(katsu_cuda_ctx *ctx, float *dst_host, const float *src_device, size_t count) {
    KATSU_TRY(katsu_bind(ctx));
    if (count == 0) return KATSU_OK;
    KATSU_REQUIRE(dst_host != nullptr && src_device != nullptr, "null buffer");
    KATSU_CUDA_TRY(cudaMemcpyAsync(dst_host, src_device, count * sizeof(float), cudaMemcpyDeviceToHost, ctx->stream));
    return KATSU_OK;
}

extern "C" int32_t katsu_cuda_d2d(katsu_cuda_ctx *ctx, float *dst_device, const float *src_device, size_t count) {
    KATSU_TRY(katsu_bind(ctx));
    if (count == 0) return KATSU_OK;
    KATSU_REQUIRE(dst_device != nullptr && src_device != nullptr, "null buffer");
    KATSU_CUDA_TRY(cudaMemcpyAsync(dst_device, src_device, count * sizeof(float), cudaMemcpyDeviceToDevice,
                                   ctx->stream));
    return KATSU_OK;
}

extern "C" int32_t katsu_cuda_host_alloc(katsu_cuda_ctx *ctx, size_t count, float **out_ptr) {
    KATSU_REQUIRE(out_ptr != nullptr, "out_ptr is null");
    *out_ptr = nullptr;
    KATSU_TRY(katsu_bind(ctx));
    if (count == 0) return KATSU_OK;
    void *p = nullptr;
    cudaError_t err = cudaHostAlloc(&p, count * sizeof(float), cudaHostAllocDefault);
    if (err != cudaSuccess) {
        cudaGetLastError();
        return katsu_set_error(KATSU_ERR_ALLOC, "cudaHostAlloc(%zu bytes): %s", count * sizeof(float),
                               cudaGetErrorString(err));
    }
    *out_ptr = (float *)p;
    return KATSU_OK;
}

extern "C" int32_t katsu_cuda_host_free(katsu_cuda_ctx *ctx, float *ptr) {
    KATSU_TRY(katsu_bind(ctx));
    if (ptr == nullptr) return KATSU_OK;
    KATSU_CUDA_TRY(cudaFreeHost(ptr));
    return KATSU_OK;
}

extern "C" int32_t katsu_cuda_sync(katsu_cuda_ctx *ctx) {
    KATSU_TRY(katsu_bind(ctx));
    return katsu_sync_and_check(ctx);
}

// ---- timing ----------------------------------------------------------------
extern "C" int32_t katsu_cuda_event_create(katsu_cuda_ctx *ctx, katsu_cuda_event **out_event) {
    KATSU_REQUIRE(out_event != nullptr, "out_event is null");
    KATSU_TRY(katsu_bind(ctx));
    katsu_cuda_event *e = new (std::nothrow) katsu_cuda_event();
    if (e == nullptr) return katsu_set_error(KATSU_ERR_ALLOC, "out of host memory");
    cudaError_t err = cudaEventCreate(&e->ev);
    if (err != cudaSuccess) {
        delete e;
        return katsu_set_error(KATSU_ERR_CUDA, "cudaEventCreate: %s", cudaGetErrorString(err));
    }
    *out_event = e;
    return KATSU_OK;
}

extern "C" int32_t katsu_cuda_event_record(katsu_cuda_ctx *ctx, katsu_cuda_event *event) {
    KATSU_REQUIRE(event != nullptr, "event is null");
    KATSU_TRY(katsu_bind(ctx));
    KATSU_CUDA_TRY(cudaEventRecord(event->ev, ctx->stream));
    return KATSU_OK;
}

extern "C" int32_t katsu_cuda_wait_event(katsu_cuda_ctx *ctx, katsu_cuda_event *event) {
    KATSU_REQUIRE(event != nullptr, "event is null");
    KATSU_TRY(katsu_bind(ctx));
    KATSU_CUDA_TRY(cudaStreamWaitEvent(ctx->stream, event->ev, 0));
    return KATSU_OK;
}

extern "C" int32_t katsu_cuda_event_elapsed_ms(katsu_cuda_ctx *ctx, katsu_cuda_event *start,
                                               katsu_cuda_event *stop, float *out_ms) {
    KATSU_REQUIRE(start != nullptr && stop != nullptr && out_ms != nullptr, "null argument");
    KATSU_TRY(katsu_bind(ctx));
    KATSU_CUDA_TRY(cudaEventSynchronize(stop->ev));
    KATSU_CUDA_TRY(cudaEventElapsedTime(out_ms, start->ev, stop->ev));
    // The kernels in front of `stop` have run: a time measured over a wait that gave up is not a
    // measurement.  The word is read directly (work queued behind `stop` may still be running).
    int status = 0;
    KATSU_CUDA_TRY(cudaMemcpy(&status, ctx->status, sizeof(int), cudaMemcpyDeviceToHost));
    return katsu_report_status(ctx, status);
}

extern "C" int32_t katsu_cuda_event_destroy(katsu_cuda_ctx *ctx, katsu_cuda_event *event) {
    KATSU_TRY(katsu_bind(ctx));
    if (event == nullptr) return KATSU_OK;
    cudaEventDestroy(event->ev);
    delete event;
    return KATSU_OK;
}

extern "C" int32_t katsu_cuda_flush_l2(katsu_cuda_ctx *ctx) {
    KATSU_TRY(katsu_bind(ctx));
    const size_t floats = size_t(64) << 20;  // 256 MiB, twice the 126 MB L2
    if (ctx->flush == nullptr) {
        KATSU_CUDA_TRY(cudaMalloc(&ctx->flush, floats * sizeof(float)));
        ctx->flush_floats = floats;
    }
    KATSU_CUDA_TRY(cudaMemsetAsync(ctx->flush, 0, ctx->flush_floats * sizeof(float), ctx->stream));
    return KATSU_OK;
}
