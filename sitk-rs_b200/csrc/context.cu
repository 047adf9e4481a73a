// Context, error model and image upload/to_host.
//
// Mirrors the reference's device runtime contract: one backend per device with one
// stream (cuda/backend.rs:30-160), DeviceImage upload of any scalar pixel type to a
// device f32 volume cast as (float)(double)x (cuda/image.rs:98-106, :182-261), and
// to_host (cuda/image.rs:269-280). Complex and vector pixels are refused by name.

#include <cuda_runtime.h>
#include <cudaTypedefs.h>
#include <algorithm>
#include <cstdio>
#include <cstring>
#include <map>
#include <mutex>
#include <new>

#include "internal.h"

namespace mi {

mi_status set_error(mi_context* ctx, mi_status s, const std::string& msg) {
    if (ctx) ctx->last_error = msg;
    return s;
}

mi_status cuda_status(mi_context* ctx, cudaError_t e, const char* where) {
    mi_status s = MI_ERR_CUDA;
    if (e == cudaErrorMemoryAllocation) s = MI_ERR_OUT_OF_MEMORY;
    if (e == cudaErrorNoDevice || e == cudaErrorInsufficientDriver) s = MI_ERR_NO_DEVICE;
    std::string msg = std::string(where) + ": " + cudaGetErrorString(e);
    return set_error(ctx, s, msg);
}

// A kernel's dynamic shared-memory limit is a property of the function on the
// current device, shared by every metric in the process: it is only ever raised,
// so a metric created later with a smaller need does not shrink it under an
// earlier one.
mi_status raise_smem_limit(mi_context* ctx, const void* fn, size_t bytes) {
    static std::mutex mu;
    static std::map<std::pair<int, const void*>, size_t> lim;
    std::lock_guard<std::mutex> g(mu);
    size_t& cur = lim[{ctx->device, fn}];
    if (bytes <= cur) return MI_OK;
    const cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e != cudaSuccess) return cuda_status(ctx, e, "cudaFuncSetAttribute");
    cur = bytes;
    return MI_OK;
}

// The tensor-map encoder of the driver (cuTensorMapEncodeTiled), found once.
PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
    static const PFN_cuTensorMapEncodeTiled_v12000 fn = [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess) {
            cudaGetLastError();
            return (PFN_cuTensorMapEncodeTiled_v12000) nullptr;
        }
        return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    }();
    return fn;
}

// What an object gives back is kept for the next one. On the B200 a cudaMalloc / cudaFree
// pair takes 0.65–0.75 ms at any size up to 128 MB, a 128-byte cudaHostAlloc / cudaFreeHost
// pair 2.2 ms and a layered array 0.45 ms; the pool hands a block out and back in 4 µs.
// A metric holds about twenty blocks, so its set-up was mostly these calls.
//   device memory  a stream-ordered pool of the context for blocks below LARGE; above it spare
//                  blocks of the pool, at most SPARE_BLOCKS of LARGE_BYTES together, taken by
//                  the nearest size (the pool maps freed pages anew where a block of another
//                  size takes their place: 0.2–5 ms for 64–128 MB). Images of any size have
//                  cudaMalloc'd blocks, kept in the same way: their address may be given out,
//                  and memory of a pool is neither shared with other processes nor mapped by
//                  other devices (for all large blocks they made a process's first batch of
//                  24 pairs 42–48 ms; 30 with this, 24 with the pool alone)
//   pinned blocks  slabs of 64 small ones, kept until the context goes; of the larger ones up
//                  to PINNED_SPARES of each size of at most PINNED_KEEP bytes
//   arrays         at most SPARE_ARRAYS of SPARE_ARRAY_BYTES together, taken by exact shape
// A block is reused in the order of the context's one stream, so nothing waits. What every
// context of the device keeps (but for the slabs) goes back when a device allocation of any of
// them does not fit beside it; a context's own, when it is trimmed (for the allocators of
// others: mi_context_trim), and with the context.
constexpr unsigned long long POOL_KEEP = 256ull << 20;  // what the pool keeps of freed pages
constexpr size_t LARGE = (size_t)1 << 20, LARGE_BYTES = (size_t)4 << 30, SPARE_BLOCKS = 256;
constexpr size_t IMAGE_GRAIN = (size_t)1 << 16, SMALL_IMAGE = (size_t)16 << 20;  // the grain below LARGE
constexpr size_t SPARE_ARRAYS = 64, SPARE_ARRAY_BYTES = (size_t)1 << 30;
constexpr size_t SLAB_BLOCKS = 64, PINNED_SPARES = 4, PINNED_KEEP = (size_t)16 << 20;

namespace {

cudaError_t create_pool(mi_context* c) {
    cudaMemPoolProps props = {};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = c->device;
    cudaError_t e = cudaMemPoolCreate(&c->pool, &props);
    unsigned long long keep = POOL_KEEP;
    if (e == cudaSuccess) e = cudaMemPoolSetAttribute(c->pool, cudaMemPoolAttrReleaseThreshold, &keep);
    return e;
}

// The spare arrays beyond `count` of `bytes` together go, oldest first (spare_mutex held).
void drop_arrays(mi_context* ctx, size_t count, size_t bytes) {
    while (!ctx->spare_arrays.empty() && (ctx->spare_arrays.size() > count || ctx->spare_array_bytes > bytes)) {
        ctx->spare_array_bytes -= ctx->spare_arrays.front().bytes();
        cudaFreeArray(ctx->spare_arrays.front().array);
        ctx->spare_arrays.pop_front();
    }
}

// The spare blocks beyond `count` of `bytes` together go, oldest first (spare_mutex held).
void drop_blocks(mi_context* ctx, size_t count, size_t bytes) {
    while (!ctx->spare_blocks.empty() && (ctx->spare_blocks.size() > count || ctx->spare_block_bytes > bytes)) {
        const auto oldest = ctx->spare_blocks.begin();
        ctx->spare_block_bytes -= oldest->bytes;
        ctx->large_blocks.erase(oldest->p);
        if (oldest->image)
            cudaFree(oldest->p);
        else
            cudaFreeAsync(oldest->p, ctx->stream);
        ctx->spare_blocks.erase(oldest);
    }
}

// The contexts there are (never destroyed: a context may go at the process's end).
std::mutex& g_contexts_mutex = *new std::mutex;
std::vector<mi_context*>& g_contexts = *new std::vector<mi_context*>;

// Waits for the work of every stream, as cudaFree of a cudaMalloc'd block does: here a word
// kept for it. That is allowed while another thread captures a graph on another stream, when
// cudaDeviceSynchronize fails and invalidates the capture (a batch in another thread lost
// its registration so). False when there is no word to be had (spare_mutex held).
bool wait_for_device(mi_context* ctx) {
    if (!ctx->word && cudaMalloc(&ctx->word, 1) != cudaSuccess) {
        cudaGetLastError();
        ctx->word = nullptr;
        return false;
    }
    cudaFree(ctx->word);
    if (cudaMalloc(&ctx->word, 1) != cudaSuccess) {
        cudaGetLastError();
        ctx->word = nullptr;
    }
    return true;
}

// Everything a context keeps goes back, once no work uses it (spare_mutex held).
void drop_kept(mi_context* ctx) {
    for (const SpareBlock& b : ctx->spare_blocks) {
        ctx->large_blocks.erase(b.p);
        cudaFree(b.p);
    }
    ctx->spare_blocks.clear();
    ctx->spare_block_bytes = 0;
    drop_arrays(ctx, 0, 0);
    for (auto& c : ctx->pinned_large) {
        for (unsigned char* p : c.second) cudaFreeHost(p);
        c.second.clear();
    }
    cudaMemPoolTrimTo(ctx->pool, 0);
}

// The same of every context of the device, for an allocation of `ctx` that did not fit beside it.
void give_back(mi_context* ctx) {
    cudaGetLastError();
    std::lock_guard<std::mutex> g(g_contexts_mutex);
    // (only here does a thread hold more than one of these)
    std::vector<std::unique_lock<std::mutex>> held;
    for (mi_context* c : g_contexts)
        if (c->device == ctx->device) held.emplace_back(c->spare_mutex);
    if (!wait_for_device(ctx)) return;
    for (mi_context* c : g_contexts)
        if (c->device == ctx->device) drop_kept(c);
}

cudaError_t pool_alloc(mi_context* ctx, void** p, size_t bytes) {
    cudaError_t e = cudaMallocFromPoolAsync(p, bytes, ctx->pool, ctx->stream);
    if (e == cudaErrorMemoryAllocation) {
        give_back(ctx);
        e = cudaMallocFromPoolAsync(p, bytes, ctx->pool, ctx->stream);
    }
    if (e != cudaSuccess) *p = nullptr;
    return e;
}

// A block that is kept, or a spare one of up to a quarter more, twice as much for an image
// below SMALL_IMAGE (whose cudaMalloc takes longer than all the rest of making it).
cudaError_t block_alloc(mi_context* ctx, void** p, size_t bytes, bool image) {
    const size_t most = image && bytes < SMALL_IMAGE ? 2 * bytes : bytes + bytes / 4;
    {
        std::lock_guard<std::mutex> g(ctx->spare_mutex);
        auto best = ctx->spare_blocks.end();
        for (auto it = ctx->spare_blocks.begin(); it != ctx->spare_blocks.end(); ++it)
            if (it->image == image && it->bytes >= bytes && it->bytes <= most &&
                (best == ctx->spare_blocks.end() || it->bytes < best->bytes))
                best = it;
        if (best != ctx->spare_blocks.end()) {
            *p = best->p;
            ctx->spare_block_bytes -= best->bytes;
            ctx->spare_blocks.erase(best);
            return cudaSuccess;
        }
    }
    cudaError_t e;
    if (image) {
        e = cudaMalloc(p, bytes);
        if (e == cudaErrorMemoryAllocation) {
            give_back(ctx);
            e = cudaMalloc(p, bytes);
        }
    } else {
        e = pool_alloc(ctx, p, bytes);
    }
    if (e != cudaSuccess) {
        *p = nullptr;
        return e;
    }
    std::lock_guard<std::mutex> g(ctx->spare_mutex);
    ctx->large_blocks[*p] = SpareBlock{*p, bytes, image};
    return e;
}

}  // namespace

cudaError_t dev_alloc_bytes(mi_context* ctx, void** p, size_t bytes) {
    if (bytes < LARGE) return pool_alloc(ctx, p, bytes ? bytes : 1);
    return block_alloc(ctx, p, (bytes + LARGE - 1) & ~(LARGE - 1), false);
}

cudaError_t image_alloc(mi_context* ctx, float** p, int64_t voxels) {
    const size_t bytes = (size_t)voxels * sizeof(float), grain = bytes < LARGE ? IMAGE_GRAIN : LARGE;
    void* v = nullptr;
    const cudaError_t e = block_alloc(ctx, &v, (bytes + grain - 1) & ~(grain - 1), true);
    *p = static_cast<float*>(v);
    return e;
}

void dev_free(mi_context* ctx, void* p) {
    if (!p) return;
    std::lock_guard<std::mutex> g(ctx->spare_mutex);
    const auto large = ctx->large_blocks.find(p);
    if (large == ctx->large_blocks.end()) {
        cudaFreeAsync(p, ctx->stream);
        return;
    }
    ctx->spare_blocks.push_back(large->second);
    ctx->spare_block_bytes += large->second.bytes;
    drop_blocks(ctx, SPARE_BLOCKS, LARGE_BYTES);
}

void wait_for_all_streams(mi_context* ctx) {
    for (int turn = 0; turn < 2; ++turn) {
        {
            std::lock_guard<std::mutex> g(ctx->spare_mutex);
            if (wait_for_device(ctx)) return;
        }
        give_back(ctx);
    }
    cudaDeviceSynchronize();
}

void context_release(mi_context* ctx) {
    if (ctx->holders.fetch_sub(1, std::memory_order_acq_rel) != 1) return;
    {
        std::lock_guard<std::mutex> g(g_contexts_mutex);
        g_contexts.erase(std::remove(g_contexts.begin(), g_contexts.end(), ctx), g_contexts.end());
    }
    cudaSetDevice(ctx->device);
    cudaStreamSynchronize(ctx->stream);
    cudaStreamDestroy(ctx->stream);
    drop_kept(ctx);
    for (unsigned char* slab : ctx->pinned_slabs) cudaFreeHost(slab);
    cudaFree(ctx->word);
    cudaMemPoolDestroy(ctx->pool);
    delete ctx;
}

// Larger blocks come in powers of two.
static size_t pinned_class(size_t bytes) {
    size_t c = 4096;
    while (c < bytes) c <<= 1;
    return c;
}

cudaError_t pinned_alloc(mi_context* ctx, void** host, void** dev, size_t bytes) {
    std::lock_guard<std::mutex> g(ctx->spare_mutex);
    std::vector<unsigned char*>& spare = bytes <= PINNED_BLOCK ? ctx->pinned_spare : ctx->pinned_large[pinned_class(bytes)];
    if (spare.empty()) {
        const size_t block = bytes <= PINNED_BLOCK ? PINNED_BLOCK : pinned_class(bytes);
        const size_t blocks = bytes <= PINNED_BLOCK ? SLAB_BLOCKS : 1;
        void* slab = nullptr;
        const cudaError_t e = cudaHostAlloc(&slab, blocks * block, cudaHostAllocMapped);
        if (e != cudaSuccess) return e;
        if (bytes <= PINNED_BLOCK) ctx->pinned_slabs.push_back(static_cast<unsigned char*>(slab));
        for (size_t i = blocks; i-- > 0;) spare.push_back(static_cast<unsigned char*>(slab) + i * block);
    }
    unsigned char* h = spare.back();
    if (dev) {
        const cudaError_t e = cudaHostGetDevicePointer(dev, h, 0);
        if (e != cudaSuccess) return e;
    }
    spare.pop_back();
    *host = h;
    return cudaSuccess;
}

void pinned_free(mi_context* ctx, void* host, size_t bytes) {
    if (!host) return;
    std::lock_guard<std::mutex> g(ctx->spare_mutex);
    if (bytes <= PINNED_BLOCK) {
        ctx->pinned_spare.push_back(static_cast<unsigned char*>(host));
        return;
    }
    std::vector<unsigned char*>& spare = ctx->pinned_large[pinned_class(bytes)];
    if (pinned_class(bytes) <= PINNED_KEEP && spare.size() < PINNED_SPARES)
        spare.push_back(static_cast<unsigned char*>(host));
    else
        cudaFreeHost(host);
}

cudaError_t array_alloc(mi_context* ctx, cudaArray_t* out, const cudaExtent& ext, size_t element, bool layered) {
    {
        std::lock_guard<std::mutex> g(ctx->spare_mutex);
        for (auto it = ctx->spare_arrays.begin(); it != ctx->spare_arrays.end(); ++it)
            if (it->extent[0] == ext.width && it->extent[1] == ext.height && it->extent[2] == ext.depth &&
                it->element == element && it->layered == layered) {
                *out = it->array;
                ctx->spare_array_bytes -= it->bytes();
                ctx->spare_arrays.erase(it);
                return cudaSuccess;
            }
    }
    const cudaChannelFormatDesc fmt =
        element == 2 ? cudaCreateChannelDesc<unsigned short>() : cudaCreateChannelDesc<float>();
    cudaError_t e = cudaMalloc3DArray(out, &fmt, ext, layered ? cudaArrayLayered : 0);
    if (e == cudaErrorMemoryAllocation) {
        give_back(ctx);
        e = cudaMalloc3DArray(out, &fmt, ext, layered ? cudaArrayLayered : 0);
    }
    return e;
}

void array_free(mi_context* ctx, cudaArray_t array, const cudaExtent& ext, size_t element, bool layered) {
    if (!array) return;
    std::lock_guard<std::mutex> g(ctx->spare_mutex);
    ctx->spare_arrays.push_back(SpareArray{array, {ext.width, ext.height, ext.depth}, element, layered});
    ctx->spare_array_bytes += ctx->spare_arrays.back().bytes();
    drop_arrays(ctx, SPARE_ARRAYS, SPARE_ARRAY_BYTES);
}

}  // namespace mi

namespace {

template <typename T>
__global__ void k_cast_to_f32(const T* __restrict__ src, float* __restrict__ dst, int64_t n) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (; i < n; i += stride) dst[i] = (float)(double)src[i];
}

size_t dtype_size(int dt) {
    switch (dt) {
        case MI_U8: case MI_I8: return 1;
        case MI_U16: case MI_I16: return 2;
        case MI_U32: case MI_I32: case MI_F32: return 4;
        case MI_U64: case MI_I64: case MI_F64: return 8;
        default: return 0;
    }
}

bool geometry_ok(const mi_geometry* g) {
    if (!g) return false;
    for (int d = 0; d < 3; ++d)
        if (g->size[d] <= 0) return false;
    return true;
}

template <typename T>
void launch_cast(const void* src, float* dst, int64_t n, int sms, cudaStream_t st) {
    int block = 256;
    int64_t want = (n + block - 1) / block;
    int grid = (int)(want < (int64_t)sms * 8 ? want : (int64_t)sms * 8);
    if (grid < 1) grid = 1;
    k_cast_to_f32<T><<<grid, block, 0, st>>>((const T*)src, dst, n);
}

}  // namespace

extern "C" {

const char* mi_status_string(mi_status s) {
    switch (s) {
        case MI_OK: return "ok";
        case MI_ERR_INVALID_ARGUMENT: return "invalid argument";
        case MI_ERR_NO_DEVICE: return "no CUDA device";
        case MI_ERR_CUDA: return "CUDA runtime error";
        case MI_ERR_OUT_OF_MEMORY: return "out of device memory";
        case MI_ERR_UNSUPPORTED_PIXEL_TYPE: return "unsupported pixel type (complex or vector)";
        case MI_ERR_SINGULAR_DIRECTION: return "moving image's direction matrix is singular";
        case MI_ERR_TOO_FEW_HISTOGRAM_BINS: return "too few histogram bins (need at least 5)";
        case MI_ERR_CONSTANT_FIXED: return "constant intensity: fixed";
        case MI_ERR_CONSTANT_MOVING: return "constant intensity: moving";
        case MI_ERR_SAMPLE_INDEX_OUT_OF_GRID: return "sample index outside the fixed grid";
        case MI_ERR_MASK_SIZE_MISMATCH: return "mask size does not match its image";
        case MI_ERR_NON_AFFINE_TRANSFORM: return "transform's Jacobian is not affine in the point";
        case MI_ERR_POINT_MAP_STAGE_COUNT: return "too many point-map stages";
        case MI_ERR_TOO_MANY_HISTOGRAM_BINS: return "too many histogram bins for the device histogram";
        case MI_ERR_TIMEOUT: return "a bounded device wait gave up";
        case MI_ERR_NOT_CONVERGED: return "not converged";
    }
    return "unknown status";
}

mi_status mi_context_create(int device, mi_context** out) {
    if (!out) return MI_ERR_INVALID_ARGUMENT;
    *out = nullptr;
    int count = 0;
    cudaError_t e = cudaGetDeviceCount(&count);
    if (e != cudaSuccess || count == 0) return MI_ERR_NO_DEVICE;
    if (device < 0 || device >= count) return MI_ERR_INVALID_ARGUMENT;
    mi_context* c = new (std::nothrow) mi_context();
    if (!c) return MI_ERR_OUT_OF_MEMORY;
    c->device = device;
    e = cudaSetDevice(device);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&c->num_sms, cudaDevAttrMultiProcessorCount, device);
    int l2 = 0;
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&l2, cudaDevAttrL2CacheSize, device);
    c->l2_bytes = (size_t)l2;
    if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = mi::create_pool(c);
    if (e == cudaSuccess) e = cudaMalloc(&c->word, 1);
    if (e != cudaSuccess) {
        if (c->pool) cudaMemPoolDestroy(c->pool);
        if (c->stream) cudaStreamDestroy(c->stream);
        delete c;
        return e == cudaErrorNoDevice ? MI_ERR_NO_DEVICE : MI_ERR_CUDA;
    }
    {
        std::lock_guard<std::mutex> g(mi::g_contexts_mutex);
        mi::g_contexts.push_back(c);
    }
    *out = c;
    return MI_OK;
}

mi_status mi_context_trim(mi_context* ctx) {
    if (!ctx) return MI_ERR_INVALID_ARGUMENT;
    MI_CHECK_CUDA(ctx, cudaSetDevice(ctx->device));
    MI_CHECK_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    std::lock_guard<std::mutex> g(ctx->spare_mutex);
    mi::drop_kept(ctx);
    return MI_OK;
}

mi_status mi_context_destroy(mi_context* ctx) {
    if (!ctx) return MI_ERR_INVALID_ARGUMENT;
    cudaSetDevice(ctx->device);
    cudaStreamSynchronize(ctx->stream);
    {
        std::lock_guard<std::mutex> g(ctx->spare_mutex);
        mi::drop_kept(ctx);
    }
    mi::context_release(ctx);
    return MI_OK;
}

mi_status mi_context_sync(mi_context* ctx) {
    if (!ctx) return MI_ERR_INVALID_ARGUMENT;
    MI_CHECK_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    return MI_OK;
}

const char* mi_last_error(const mi_context* ctx) {
    return ctx ? ctx->last_error.c_str() : "null context";
}

void* mi_context_stream(mi_context* ctx) { return ctx ? (void*)ctx->stream : nullptr; }

mi_status mi_image_upload(mi_context* ctx, const void* host, mi_dtype dtype,
                          const mi_geometry* geometry, mi_image** out) {
    if (!ctx || !host || !out) return MI_ERR_INVALID_ARGUMENT;
    *out = nullptr;
    if (dtype == MI_COMPLEX_F32 || dtype == MI_VECTOR_F32)
        return mi::set_error(ctx, MI_ERR_UNSUPPORTED_PIXEL_TYPE,
                             "DeviceImage holds scalar voxels only; complex and vector pixels are refused");
    size_t es = dtype_size(dtype);
    if (es == 0) return mi::set_error(ctx, MI_ERR_INVALID_ARGUMENT, "unknown pixel type");
    if (!geometry_ok(geometry)) return mi::set_error(ctx, MI_ERR_INVALID_ARGUMENT, "bad geometry");
    MI_CHECK_CUDA(ctx, cudaSetDevice(ctx->device));
    int64_t n = geometry->size[0] * geometry->size[1] * geometry->size[2];
    float* d = nullptr;
    MI_CHECK_CUDA(ctx, mi::image_alloc(ctx, &d, n));
    cudaError_t e = cudaSuccess;
    if (dtype == MI_F32) {
        e = cudaMemcpyAsync(d, host, (size_t)n * 4, cudaMemcpyHostToDevice, ctx->stream);
    } else {
        void* tmp = nullptr;
        e = mi::dev_alloc(ctx, &tmp, (size_t)n * es);
        if (e == cudaSuccess) e = cudaMemcpyAsync(tmp, host, (size_t)n * es, cudaMemcpyHostToDevice, ctx->stream);
        if (e == cudaSuccess) {
            switch (dtype) {
                case MI_U8: launch_cast<uint8_t>(tmp, d, n, ctx->num_sms, ctx->stream); break;
                case MI_I8: launch_cast<int8_t>(tmp, d, n, ctx->num_sms, ctx->stream); break;
                case MI_U16: launch_cast<uint16_t>(tmp, d, n, ctx->num_sms, ctx->stream); break;
                case MI_I16: launch_cast<int16_t>(tmp, d, n, ctx->num_sms, ctx->stream); break;
                case MI_U32: launch_cast<uint32_t>(tmp, d, n, ctx->num_sms, ctx->stream); break;
                case MI_I32: launch_cast<int32_t>(tmp, d, n, ctx->num_sms, ctx->stream); break;
                case MI_U64: launch_cast<unsigned long long>(tmp, d, n, ctx->num_sms, ctx->stream); break;
                case MI_I64: launch_cast<long long>(tmp, d, n, ctx->num_sms, ctx->stream); break;
                case MI_F64: launch_cast<double>(tmp, d, n, ctx->num_sms, ctx->stream); break;
                default: break;
            }
            e = cudaGetLastError();
        }
        if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
        mi::dev_free(ctx, tmp);
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    if (e != cudaSuccess) {
        mi::dev_free(ctx, d);
        return mi::cuda_status(ctx, e, "mi_image_upload");
    }
    mi_image* img = new (std::nothrow) mi_image();
    if (!img) {
        mi::dev_free(ctx, d);
        return MI_ERR_OUT_OF_MEMORY;
    }
    img->ctx = ctx;
    img->geo = *geometry;
    img->data = d;
    img->n = n;
    *out = img;
    return MI_OK;
}

mi_status mi_image_from_device(mi_context* ctx, const float* device_ptr, const mi_geometry* geometry,
                               mi_image** out) {
    if (!ctx || !device_ptr || !out) return MI_ERR_INVALID_ARGUMENT;
    *out = nullptr;
    if (!geometry_ok(geometry)) return mi::set_error(ctx, MI_ERR_INVALID_ARGUMENT, "bad geometry");
    MI_CHECK_CUDA(ctx, cudaSetDevice(ctx->device));
    int64_t n = geometry->size[0] * geometry->size[1] * geometry->size[2];
    float* d = nullptr;
    MI_CHECK_CUDA(ctx, mi::image_alloc(ctx, &d, n));
    cudaError_t e = cudaMemcpyAsync(d, device_ptr, (size_t)n * 4, cudaMemcpyDeviceToDevice, ctx->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    if (e != cudaSuccess) {
        mi::dev_free(ctx, d);
        return mi::cuda_status(ctx, e, "mi_image_from_device");
    }
    mi_image* img = new (std::nothrow) mi_image();
    if (!img) {
        mi::dev_free(ctx, d);
        return MI_ERR_OUT_OF_MEMORY;
    }
    img->ctx = ctx;
    img->geo = *geometry;
    img->data = d;
    img->n = n;
    *out = img;
    return MI_OK;
}

mi_status mi_image_to_host(const mi_image* img, float* dst, size_t n_elements) {
    if (!img || !dst) return MI_ERR_INVALID_ARGUMENT;
    if ((int64_t)n_elements < img->n)
        return mi::set_error(img->ctx, MI_ERR_INVALID_ARGUMENT, "destination smaller than the image");
    MI_CHECK_CUDA(img->ctx, cudaSetDevice(img->ctx->device));
    MI_CHECK_CUDA(img->ctx, cudaMemcpyAsync(dst, img->data, (size_t)img->n * 4, cudaMemcpyDeviceToHost,
                                            img->ctx->stream));
    MI_CHECK_CUDA(img->ctx, cudaStreamSynchronize(img->ctx->stream));
    return MI_OK;
}

mi_status mi_image_geometry(const mi_image* img, mi_geometry* out) {
    if (!img || !out) return MI_ERR_INVALID_ARGUMENT;
    *out = img->geo;
    return MI_OK;
}

const float* mi_image_device_ptr(const mi_image* img) {
    if (!img) return nullptr;
    img->lent = true;
    return img->data;
}

mi_status mi_image_free(mi_image* img) {
    if (!img) return MI_ERR_INVALID_ARGUMENT;
    cudaSetDevice(img->ctx->device);
    // Voxels that were lent out (mi_image_device_ptr) may still be read by work of any stream;
    // the library's own calls are done with them, or come before the block's next use.
    if (img->lent) mi::wait_for_all_streams(img->ctx);
    mi::dev_free(img->ctx, img->data);
    delete img;
    return MI_OK;
}

}  // extern "C"
