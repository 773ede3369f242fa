// ReduceTexture (glslppm.cpp:170-209) as a stage-level entry point.
//
// The reference reduces an R x R RGBA32F texture to one texel by drawing quads of R/2, R/4, ... 1
// pixels into a ping-pong texture; each output texel applies min.fs / max.fs / sum.fs to the four
// texels (i,j), (i+n,j), (i,j+n), (i+n,j+n) of the previous level, and the host reads texel (0,0).
// The folds of consecutive levels of one output texel read inputs that no other output reads, so a
// launch does up to four levels (no texel written between) until at most 128 x 128 texels are left,
// which one block folds to the end.  The sums are evaluated as ((v0 + v1) + v2) + v3
// with non-fused adds in the reference's order, so all three results are bit-identical to its fold.
//
// 1024 x 1024 (16 MiB): two launches instead of ten, and a scratch kept between calls: 249 -> 36 us a
// call, most of it launches, the copy of the result and the wait.
#include <cstdint>
#include <mutex>

#include <cuda.h>  // driver types only (CUcontext, CUresult); nothing is linked
#include <cuda_runtime.h>

#include "../host/scene_internal.h"
#include "device_common.cuh"

namespace sppm_dev {

template <int OP>
__device__ __forceinline__ float4 fold4(const float4& v0, const float4& v1, const float4& v2, const float4& v3) {
    auto f = [](float a, float b, float c, float d) {
        if (OP == SPPM_REDUCE_MIN) return fminf(fminf(a, b), fminf(c, d));
        if (OP == SPPM_REDUCE_MAX) return fmaxf(fmaxf(a, b), fmaxf(c, d));
        return __fadd_rn(__fadd_rn(__fadd_rn(a, b), c), d);
    };
    return make_float4(f(v0.x, v1.x, v2.x, v3.x), f(v0.y, v1.y, v2.y, v3.y), f(v0.z, v1.z, v2.z, v3.z),
                       f(v0.w, v1.w, v2.w, v3.w));
}

// texel (i, j) after folding the 2^K n x 2^K n texels of src to n x n, level by level
template <int OP, int K>
__device__ __forceinline__ float4 fold_levels(const float4* __restrict__ src, size_t stride, uint32_t i, uint32_t j,
                                              uint32_t n) {
    if constexpr (K == 0) {
        return src[j * stride + i];
    } else {
        return fold4<OP>(fold_levels<OP, K - 1>(src, stride, i, j, 2 * n),
                         fold_levels<OP, K - 1>(src, stride, i + n, j, 2 * n),
                         fold_levels<OP, K - 1>(src, stride, i, j + n, 2 * n),
                         fold_levels<OP, K - 1>(src, stride, i + n, j + n, 2 * n));
    }
}

// K levels: dst [n][n] of row length dst_stride.  In place (dst == src, equal strides) a thread reads
// its own output texel and texels outside the output square, which no thread writes.
template <int OP, int K>
__global__ void __launch_bounds__(128) k_reduce_levels(const float4* src, uint32_t src_stride, float4* dst,
                                                     uint32_t dst_stride, uint32_t n) {
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n * n) return;
    const uint32_t i = t % n, j = t / n;
    dst[(size_t)j * dst_stride + i] = fold_levels<OP, K>(src, src_stride, i, j, n);
}

// Four levels, 256 input texels an output: a block folds 32 outputs, each of its 16 warps two levels of
// one sixteenth of their inputs (16 loads a thread, all of a 1024 x 1024 texture in flight at once), and
// the last two levels through shared memory.  In place as above: a block reads its own output texels
// before the barrier and writes them after it.  64 texels a thread, three levels without shared
// memory, took 12.4 us for 1024 x 1024 (16 MiB) and left four times the texels for the one block of the
// tail, 6.0 us; this 6.7 and 4.2.
template <int OP>
__global__ void __launch_bounds__(512) k_reduce_levels4(const float4* src, uint32_t src_stride, float4* dst,
                                                      uint32_t dst_stride, uint32_t n) {
    __shared__ float4 s[16][32];
    const uint32_t lane = threadIdx.x & 31u, q1 = threadIdx.x >> 7, q2 = (threadIdx.x >> 5) & 3u;
    const uint32_t t = blockIdx.x * 32 + lane, i = t % n, j = t / n;
    if (t < n * n)
        s[threadIdx.x >> 5][lane] =
            fold_levels<OP, 2>(src, src_stride, i + (q1 & 1u) * n + (q2 & 1u) * 2 * n,
                               j + (q1 >> 1) * n + (q2 >> 1) * 2 * n, 4 * n);
    __syncthreads();
    if (t < n * n && q2 == 0)
        s[threadIdx.x >> 5][lane] = fold4<OP>(s[4 * q1][lane], s[4 * q1 + 1][lane], s[4 * q1 + 2][lane], s[4 * q1 + 3][lane]);
    __syncthreads();
    if (t < n * n && threadIdx.x < 32)
        dst[(size_t)j * dst_stride + i] = fold4<OP>(s[0][lane], s[4][lane], s[8][lane], s[12][lane]);
}

// the last levels in one block: n x n texels (n <= kReduceTail) to one.  A thread folds up to two
// levels from memory, the rest go through shared memory.
constexpr uint32_t kReduceTail = 128;
template <int OP>
__global__ void __launch_bounds__(1024) k_reduce_tail(const float4* src, uint32_t stride, uint32_t n, float4* out) {
    __shared__ float4 s[32 * 32];
    const uint32_t m = n <= 32 ? n : 32;  // side after the fold from memory
    const uint32_t t = threadIdx.x;
    if (t < m * m) {
        const uint32_t i = t % m, j = t / m;
        s[t] = n <= 32 ? fold_levels<OP, 0>(src, stride, i, j, m)
                       : (n == 64 ? fold_levels<OP, 1>(src, stride, i, j, m) : fold_levels<OP, 2>(src, stride, i, j, m));
    }
    // rows keep their length m: as in place above, no thread reads what another writes
    for (uint32_t h = m / 2; h >= 1; h /= 2) {
        __syncthreads();
        if (t < h * h) {
            const uint32_t i = t % h, j = t / h;
            s[j * m + i] = fold_levels<OP, 1>(s, m, i, j, h);
        }
    }
    if (t == 0) *out = s[0];
}

template <int OP>
static void reduce_op(const float4* src, uint32_t n, float4* scratch, cudaStream_t s) {
    uint32_t stride = n;
    while (n > kReduceTail) {
        const uint32_t k = n >= 8 * kReduceTail ? 4 : (n == 4 * kReduceTail ? 2 : 1), m = n >> k;
        const uint32_t out_stride = src == scratch ? stride : m, blocks = (m * m + 127) / 128;
        if (k == 4) k_reduce_levels4<OP><<<(m * m + 31) / 32, 512, 0, s>>>(src, stride, scratch, out_stride, m);
        else if (k == 2) k_reduce_levels<OP, 2><<<blocks, 128, 0, s>>>(src, stride, scratch, out_stride, m);
        else k_reduce_levels<OP, 1><<<blocks, 128, 0, s>>>(src, stride, scratch, out_stride, m);
        src = scratch;
        stride = out_stride;
        n = m;
    }
    k_reduce_tail<OP><<<1, 1024, 0, s>>>(src, stride, n, scratch);
}

// texels of scratch: the first launch's output, at least the result's
size_t reduce_scratch_texels(uint32_t resolution) {
    if (resolution <= kReduceTail) return 1;
    const size_t m = resolution >= 8 * kReduceTail ? resolution / 16 : kReduceTail;
    return m * m;
}

// all levels of one reduction; the result is scratch[0] when the last launch completes
void launch_reduce_texture(const float4* tex, uint32_t resolution, uint32_t op, float4* scratch, cudaStream_t s) {
    if (op == SPPM_REDUCE_MIN) reduce_op<SPPM_REDUCE_MIN>(tex, resolution, scratch, s);
    else if (op == SPPM_REDUCE_MAX) reduce_op<SPPM_REDUCE_MAX>(tex, resolution, scratch, s);
    else reduce_op<SPPM_REDUCE_SUM>(tex, resolution, scratch, s);
}

}  // namespace sppm_dev

using sppm::fail;

// ---- variant without device allocation ---------------------------------------------------------
// Its scratch is this file-scope device array, the first launch's output at any size up to the largest:
// 128 x 128 float4 = 256 KiB, held by every GPU that loads the library until the process exits.  Host
// code must not pass `g_reduce_scratch` itself to a kernel (on the host it names a host-side shadow, not
// device memory): the device address is looked up with cudaGetSymbolAddress once per device and context,
// with that device current, and cached.
static __device__ __align__(256) float4 g_reduce_scratch[sppm_dev::kReduceTail * sppm_dev::kReduceTail];
static_assert(SPPM_REDUCE_NOALLOC_MAX_RESOLUTION <= 16 * sppm_dev::kReduceTail, "the scratch holds the first launch's output");

namespace {
// The device address of g_reduce_scratch belongs to the CUDA context that loaded the library's
// device code: a device reset (cudaDeviceReset) destroys that context and the next runtime call
// creates a new one, in which the array may sit elsewhere.  The cache is therefore keyed on the
// context's unique id (cuCtxGetId, never reused within a process), read through driver entry
// points that the runtime hands out, so the library needs no link against the driver library.
typedef CUresult (*PFN_ctx_get_current)(CUcontext*);
typedef CUresult (*PFN_ctx_get_id)(CUcontext, unsigned long long*);

struct ScratchEntry {
    unsigned long long ctx_id;
    float4* ptr;
};
std::mutex g_scratch_mutex;
ScratchEntry g_scratch_cache[64];  // per device ordinal: the context it was looked up in, address
PFN_ctx_get_current g_ctx_get_current = nullptr;
PFN_ctx_get_id g_ctx_get_id = nullptr;

// id of the current context, 0 when none is current (after a reset, before the next runtime call)
int current_context_id(unsigned long long* id) {
    *id = 0;
    if (!g_ctx_get_current || !g_ctx_get_id) {
        void* f1 = nullptr;
        void* f2 = nullptr;
        cudaDriverEntryPointQueryResult q1 = cudaDriverEntryPointSymbolNotFound, q2 = cudaDriverEntryPointSymbolNotFound;
        cudaError_t e = cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &f1, 12000, cudaEnableDefault, &q1);
        if (e == cudaSuccess) e = cudaGetDriverEntryPointByVersion("cuCtxGetId", &f2, 12000, cudaEnableDefault, &q2);
        if (e != cudaSuccess || q1 != cudaDriverEntryPointSuccess || q2 != cudaDriverEntryPointSuccess || !f1 || !f2)
            return fail(SPPM_ERR_CUDA, "driver entry points cuCtxGetCurrent/cuCtxGetId unavailable: %s",
                        cudaGetErrorString(e));
        g_ctx_get_current = reinterpret_cast<PFN_ctx_get_current>(f1);
        g_ctx_get_id = reinterpret_cast<PFN_ctx_get_id>(f2);
    }
    CUcontext ctx = nullptr;
    if (g_ctx_get_current(&ctx) != CUDA_SUCCESS) return fail(SPPM_ERR_CUDA, "cuCtxGetCurrent failed");
    if (ctx && g_ctx_get_id(ctx, id) != CUDA_SUCCESS) return fail(SPPM_ERR_CUDA, "cuCtxGetId failed");
    return SPPM_OK;
}

// Set-up of the entry point: on the first call in a device's current context (and again after a
// device reset replaced that context), the array's device address is looked up with that device
// current and cached; later calls in the same context reuse it.
int scratch_address(float4** out) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return fail(SPPM_ERR_CUDA, "cudaGetDevice failed: %s", cudaGetErrorString(e));
    if (dev < 0 || dev >= 64) return fail(SPPM_ERR_ARG, "device ordinal %d out of range", dev);
    std::lock_guard<std::mutex> lock(g_scratch_mutex);
    unsigned long long id = 0;
    int st = current_context_id(&id);
    if (st) return st;
    ScratchEntry& c = g_scratch_cache[dev];
    if (id == 0 || !c.ptr || c.ctx_id != id) {
        // also makes the device's primary context current when none is
        void* p = nullptr;
        e = cudaGetSymbolAddress(&p, g_reduce_scratch);
        if (e != cudaSuccess || !p)
            return fail(SPPM_ERR_CUDA, "cudaGetSymbolAddress(g_reduce_scratch) failed: %s", cudaGetErrorString(e));
        if (id == 0 && (st = current_context_id(&id)) != SPPM_OK) return st;
        c.ptr = static_cast<float4*>(p);
        c.ctx_id = id;
    }
    *out = c.ptr;
    return SPPM_OK;
}
// The scratch of sppm_reduce_texture: up to kKeptScratch buffers per CUDA context are kept between calls
// (an allocation that a synchronization gives back to the system costs the call 100 us and more), each
// as large as a call that took it has needed: 256 KiB, 1 MiB from a resolution of 4096, 4 at 8192, 16 at
// 16384.  A call takes one out of its context's list and puts it back once its stream has been
// synchronized, so no two calls share one; a call that finds none, kKeptScratch others being under way,
// allocates its own.  They are the context's (cudaMalloc), so they end with it; a pool's allocations would
// outlive it.  Context ids are never reused, so the list of a context that is gone is never looked up
// again; contexts beyond kKeptContexts keep nothing.
constexpr size_t kLeastScratch = sppm_dev::kReduceTail * sppm_dev::kReduceTail, kKeptScratch = 4, kKeptContexts = 64;
struct Scratch {
    float4* ptr;
    size_t texels;
};
struct ScratchList {
    unsigned long long ctx_id;
    size_t made, n;  // buffers made, and of them free
    Scratch free[kKeptScratch];
};
ScratchList g_scratch_lists[kKeptContexts];
size_t g_scratch_contexts = 0;

// the list of context `id`, null when there is no room for one (g_scratch_mutex held)
ScratchList* scratch_list(unsigned long long id) {
    for (size_t i = 0; i < g_scratch_contexts; i++)
        if (g_scratch_lists[i].ctx_id == id) return &g_scratch_lists[i];
    if (g_scratch_contexts == kKeptContexts) return nullptr;
    g_scratch_lists[g_scratch_contexts] = ScratchList{id, 0, 0, {}};
    return &g_scratch_lists[g_scratch_contexts++];
}

// a kept buffer for a call on stream s, null when the call has to allocate its own; *id: its context
Scratch take_scratch(cudaStream_t s, size_t texels, unsigned long long* id) {
    const Scratch none{nullptr, 0};
    // (a stream under capture cannot be waited for: the call fails there, as it does without this)
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(s, &capture) != cudaSuccess) {
        cudaGetLastError();
        return none;
    }
    if (capture != cudaStreamCaptureStatusNone) return none;
    std::lock_guard<std::mutex> lock(g_scratch_mutex);
    if (current_context_id(id) != SPPM_OK) return none;
    if (*id == 0) {  // a thread's first CUDA call: make its device's primary context current
        int dev = 0;
        if (cudaGetDevice(&dev) != cudaSuccess || cudaSetDevice(dev) != cudaSuccess) {
            cudaGetLastError();
            return none;
        }
        if (current_context_id(id) != SPPM_OK || *id == 0) return none;
    }
    ScratchList* list = scratch_list(*id);
    if (!list) return none;
    size_t at = 0;
    while (at < list->n && list->free[at].texels < texels) at++;
    if (at < list->n) {
        const Scratch found = list->free[at];
        list->free[at] = list->free[--list->n];
        return found;
    }
    if (list->made == kKeptScratch && !list->n) return none;
    Scratch made{nullptr, texels > kLeastScratch ? texels : kLeastScratch};
    // another thread's capture does not bear on these calls
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    cudaThreadExchangeStreamCaptureMode(&mode);
    if (list->made == kKeptScratch) {  // a larger one in the place of one that is too small
        cudaFree(list->free[--list->n].ptr);
        list->made--;
    }
    const cudaError_t e = cudaMalloc(&made.ptr, made.texels * sizeof(float4));
    cudaThreadExchangeStreamCaptureMode(&mode);
    if (e != cudaSuccess) {
        cudaGetLastError();
        return none;
    }
    list->made++;
    return made;
}

void put_scratch(unsigned long long id, Scratch scratch) {
    std::lock_guard<std::mutex> lock(g_scratch_mutex);
    ScratchList* list = scratch_list(id);
    list->free[list->n++] = scratch;
}
}  // namespace

extern "C" int sppm_reduce_texture_noalloc(const float* d_texture, uint32_t resolution, uint32_t op, float out[4],
                                           void* stream) {
    if (!d_texture || !out) return fail(SPPM_ERR_ARG, "sppm_reduce_texture_noalloc: null argument");
    if (resolution < 2 || (resolution & (resolution - 1)))
        return fail(SPPM_ERR_ARG, "sppm_reduce_texture_noalloc: resolution %u must be a power of two >= 2", resolution);
    if (resolution > SPPM_REDUCE_NOALLOC_MAX_RESOLUTION)
        return fail(SPPM_ERR_ARG,
                    "sppm_reduce_texture_noalloc: resolution %u exceeds the maximum %u of its fixed scratch "
                    "(use sppm_reduce_texture)", resolution, (unsigned)SPPM_REDUCE_NOALLOC_MAX_RESOLUTION);
    if (op > SPPM_REDUCE_SUM) return fail(SPPM_ERR_ARG, "sppm_reduce_texture_noalloc: unknown op %u", op);
    if (reinterpret_cast<uintptr_t>(d_texture) & 15) return fail(SPPM_ERR_ARG, "texture must be 16-byte aligned");
    float4* scratch = nullptr;
    int st = scratch_address(&scratch);
    if (st) return st;
    cudaStream_t s = (cudaStream_t)stream;
    // no clearing needed: every level writes each scratch texel it later reads
    sppm_dev::launch_reduce_texture(reinterpret_cast<const float4*>(d_texture), resolution, op, scratch, s);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpyAsync(out, scratch, sizeof(float4), cudaMemcpyDeviceToHost, s);
    const cudaError_t e2 = cudaStreamSynchronize(s);
    if (e != cudaSuccess || e2 != cudaSuccess)
        return fail(SPPM_ERR_CUDA, "sppm_reduce_texture_noalloc failed: %s",
                    cudaGetErrorString(e != cudaSuccess ? e : e2));
    return SPPM_OK;
}

extern "C" int sppm_reduce_texture(const float* d_texture, uint32_t resolution, uint32_t op, float out[4],
                                   void* stream) {
    if (!d_texture || !out) return fail(SPPM_ERR_ARG, "sppm_reduce_texture: null argument");
    if (resolution < 2 || (resolution & (resolution - 1)) || resolution > 16384)
        return fail(SPPM_ERR_ARG, "sppm_reduce_texture: resolution %u must be a power of two in [2, 16384]", resolution);
    if (op > SPPM_REDUCE_SUM) return fail(SPPM_ERR_ARG, "sppm_reduce_texture: unknown op %u", op);
    if (reinterpret_cast<uintptr_t>(d_texture) & 15) return fail(SPPM_ERR_ARG, "texture must be 16-byte aligned");
    cudaStream_t s = (cudaStream_t)stream;
    const size_t texels = sppm_dev::reduce_scratch_texels(resolution);
    unsigned long long id = 0;
    const Scratch kept = take_scratch(s, texels, &id);
    float4* scratch = kept.ptr;
    cudaError_t e = cudaSuccess;
    if (!scratch) e = cudaMallocAsync(&scratch, texels * sizeof(float4), s);
    if (e != cudaSuccess) return fail(SPPM_ERR_OOM, "sppm_reduce_texture: scratch allocation failed: %s", cudaGetErrorString(e));
    sppm_dev::launch_reduce_texture(reinterpret_cast<const float4*>(d_texture), resolution, op, scratch, s);
    e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpyAsync(out, scratch, sizeof(float4), cudaMemcpyDeviceToHost, s);
    if (!kept.ptr) cudaFreeAsync(scratch, s);
    const cudaError_t e2 = cudaStreamSynchronize(s);
    if (kept.ptr && e2 == cudaSuccess) put_scratch(id, kept);  // (else the stream may still work in it)
    if (e != cudaSuccess || e2 != cudaSuccess) {
        cudaGetLastError();  // reported here, not by the next call's launch
        return fail(SPPM_ERR_CUDA, "sppm_reduce_texture failed: %s", cudaGetErrorString(e != cudaSuccess ? e : e2));
    }
    return SPPM_OK;
}
