// extern "C" entry points of libvsparse_b200: argument validation and kernel dispatch.
//
// Each operator entry point checks its arguments on the host, picks the template instantiation for
// (path, element types, vector length) and enqueues the kernel(s) on the caller's stream.  Nothing here
// synchronises; the *_host convenience forms allocate and say so, and the tensor-core SpMM keeps one plan
// scratch buffer per calling stream, taken from the stream-ordered allocator the first time (and when a larger
// matrix needs a larger one).
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <algorithm>
#include <atomic>
#include <cstring>
#include <cmath>
#include <memory>
#include <mutex>
#include <thread>
#include <functional>
#include <unordered_map>
#include <utility>
#include <vector>

#include "vsparse_b200.h"
#include "common.cuh"
#include "cuda_core.cuh"
#include "attention.cuh"
#include "spmm_tc.cuh"
#include "spmm_cc_tile.cuh"
#include "spmm_tma.cuh"
#include "spmm_dense.cuh"
#include "spmm_direct.cuh"
#include "sddmm_pair.cuh"
#include "spmm_pair.cuh"
#include "densify.cuh"
#include "spmm_split.cuh"
#include "spmm_t.cuh"
#include "sddmm_tc.cuh"
#include "sddmm_tma.cuh"
#include "sddmm_dense.cuh"
#include "sddmm_direct.cuh"
#include "tc_selftest.cuh"

#define VS_EXPORT extern "C" __attribute__((visibility("default")))
#define VS_CUDA_TRY(expr)                      \
    do {                                       \
        cudaError_t e__ = (expr);              \
        if (e__ != cudaSuccess) return (int)e__; \
    } while (0)

namespace {

using namespace vs;

// Per-device status word, OR-ed into by kernels whose bounded waits ran out.
__device__ uint32_t g_device_status = 0;

constexpr int kMaxDevices = 64;
struct Scratch {
    std::mutex use;         // held by a call from the look at `ptr` to its last launch
    bool retired = false;   // no longer in the table
    void *ptr = nullptr;
    size_t bytes = 0;
    // the capture that last asked for scratch on this stream, and what it was given (memory of the graph, see graph_scratch)
    unsigned long long capture = 0;
    void *capture_ptr = nullptr;
    size_t capture_bytes = 0;
};
struct DeviceInfo {
    bool ready = false;
    int sm_count = 0;
    uint32_t *status = nullptr;
    // Plan scratch of the densifying SpMM, one buffer per stream that has called it: calls on one stream run
    // in order, so they can share a buffer; calls on different streams cannot.  cudaStreamPerThread is one handle
    // value that names a different stream in every host thread, so there the calling thread is part of the key.
    struct Key {
        cudaStream_t stream;
        std::thread::id thread;
        bool operator==(const Key &o) const { return stream == o.stream && thread == o.thread; }
    };
    struct KeyHash {
        size_t operator()(const Key &k) const {
            return std::hash<const void *>()(static_cast<const void *>(k.stream)) ^ (std::hash<std::thread::id>()(k.thread) * 0x9e3779b97f4a7c15ull);
        }
    };
    std::unordered_map<Key, std::shared_ptr<Scratch>, KeyHash> scratch;
    static Key key_of(cudaStream_t s) { return Key{s, s == cudaStreamPerThread ? std::this_thread::get_id() : std::thread::id()}; }
};
DeviceInfo g_devices[kMaxDevices];
std::mutex g_devices_mutex;

// Whether the calling thread has a current context (cuCtxGetCurrent, fetched from the driver at first use).
bool context_is_current() {
    typedef CUresult (*GetCurrentFn)(CUcontext *);
    static const GetCurrentFn fn = []() -> GetCurrentFn {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &p, cudaEnableDefault, &q) != cudaSuccess) return nullptr;
        return q == cudaDriverEntryPointSuccess ? reinterpret_cast<GetCurrentFn>(p) : nullptr;
    }();
    CUcontext current = nullptr;
    return fn && fn(&current) == CUDA_SUCCESS && current;
}

int device_info(DeviceInfo **out) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return (int)e;
    if (dev < 0 || dev >= kMaxDevices) return VS_ERR_ARG;
    // A thread that has made no runtime call yet (autograd's backward thread, say) has no current context, and the
    // driver's cuTensorMapEncodeTiled refuses to work without one: its first call would take the kernels that need no
    // tensor maps.  Setting the device binds the device's primary context; a context that the caller has made current stays.
    if (!context_is_current()) {
        e = cudaSetDevice(dev);
        if (e != cudaSuccess) return (int)e;
    }
    std::lock_guard<std::mutex> lock(g_devices_mutex);
    DeviceInfo &d = g_devices[dev];
    if (!d.ready) {
        e = cudaDeviceGetAttribute(&d.sm_count, cudaDevAttrMultiProcessorCount, dev);
        if (e != cudaSuccess) return (int)e;
        e = cudaGetSymbolAddress(reinterpret_cast<void **>(&d.status), g_device_status);
        if (e != cudaSuccess) return (int)e;
        d.ready = true;
    }
    *out = &d;
    return VS_OK;
}

// Set for the duration of an entry point that promises not to allocate: the tensor-core formulations that need
// plan scratch are skipped on this thread, the kernels that need none take the call.
thread_local bool t_no_scratch = false;
struct NoScratchScope {
    bool saved;
    explicit NoScratchScope(bool on = true) : saved(t_no_scratch) { t_no_scratch |= on; }
    ~NoScratchScope() { t_no_scratch = saved; }
};

// A workspace handed over by the caller (vs_set_workspace) for the calls of this host thread.
thread_local bool t_ws_set = false;
thread_local void *t_ws_ptr = nullptr;
thread_local int64_t t_ws_bytes = 0;

// What the calls of this host thread are parts of (vs_set_part_of; 0: nothing): choices that decide in which order sums are formed are made as
// for the whole call.
thread_local int t_whole_columns = 0, t_whole_batch = 0;

// Scratch for captured work belongs to the graph: a buffer that the library keeps for a stream is replaced by a later, larger
// call and used by other calls beside a replay.  The graph and whatever is instantiated from it hold a reference (a CUDA user
// object); when the last one goes, the buffer comes back to this list and serves another capture, or is freed: by
// vs_release_scratch, or here when the list holds more than kMaxReturnedBytes.
struct GraphScratch {
    int device;
    void *ptr;
    size_t bytes;
};
constexpr size_t kMaxReturnedBytes = 256u << 20;
struct ReturnedScratch {
    std::mutex lock;   // nothing else is locked and no CUDA call made under it: the driver calls returned() from a thread of its own
    std::vector<GraphScratch *> list;
};
ReturnedScratch &returned_scratch() {
    static ReturnedScratch *r = new ReturnedScratch;   // never destroyed: graphs may outlive the library's static objects
    return *r;
}
void CUDART_CB graph_scratch_returned(void *buffer) {
    ReturnedScratch &r = returned_scratch();
    std::lock_guard<std::mutex> guard(r.lock);
    r.list.push_back(static_cast<GraphScratch *>(buffer));
}
// Allocating and freeing beside a capture, which forbids them unless the thread says that it knows what it does.
struct RelaxedCapture {
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    RelaxedCapture() { (void)cudaThreadExchangeStreamCaptureMode(&mode); }
    ~RelaxedCapture() { (void)cudaThreadExchangeStreamCaptureMode(&mode); }
};
// Frees returned buffers of `device` until those left hold at most `keep` bytes.
void free_returned_scratch(int device, size_t keep) {
    std::vector<GraphScratch *> gone;
    {
        ReturnedScratch &r = returned_scratch();
        std::lock_guard<std::mutex> guard(r.lock);
        size_t held = 0;
        for (size_t i = 0; i < r.list.size();) {
            if (r.list[i]->device == device && (held += r.list[i]->bytes) > keep) {
                gone.push_back(r.list[i]);
                r.list.erase(r.list.begin() + i);
            } else {
                ++i;
            }
        }
    }
    RelaxedCapture relaxed;
    for (GraphScratch *g : gone) {
        (void)cudaFree(g->ptr);
        delete g;
    }
}
int graph_scratch(cudaGraph_t graph, size_t bytes, void **out) {
    int device = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess) return (int)e;
    RelaxedCapture relaxed;
    GraphScratch *buffer = nullptr;
    {
        ReturnedScratch &r = returned_scratch();
        std::lock_guard<std::mutex> guard(r.lock);
        auto best = r.list.end();   // the smallest that is large enough
        for (auto it = r.list.begin(); it != r.list.end(); ++it)
            if ((*it)->device == device && (*it)->bytes >= bytes && (best == r.list.end() || (*it)->bytes < (*best)->bytes)) best = it;
        if (best != r.list.end()) {
            buffer = *best;
            r.list.erase(best);
        }
    }
    if (!buffer) {
        free_returned_scratch(device, kMaxReturnedBytes);
        void *ptr = nullptr;
        e = cudaMalloc(&ptr, bytes);
        if (e != cudaSuccess) {
            (void)cudaGetLastError();
            return (int)e;
        }
        buffer = new GraphScratch{device, ptr, bytes};
    }
    cudaUserObject_t owner = nullptr;
    e = cudaUserObjectCreate(&owner, buffer, graph_scratch_returned, 1, cudaUserObjectNoDestructorSync);
    if (e != cudaSuccess) {
        (void)cudaGetLastError();
        graph_scratch_returned(buffer);
        return (int)e;
    }
    *out = buffer->ptr;
    e = cudaGraphRetainUserObject(graph, owner, 1, cudaGraphUserObjectMove);
    if (e != cudaSuccess) {
        (void)cudaGetLastError();
        (void)cudaUserObjectRelease(owner, 1);   // the buffer goes back to the list
        return (int)e;
    }
    return VS_OK;
}

// The graph that `s` is being captured into and the capture's number, unique in the process; null without a capture.
cudaGraph_t capture_graph(cudaStream_t s, unsigned long long *id) {
    cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
    cudaGraph_t graph = nullptr;
    if (cudaStreamGetCaptureInfo(s, &st, id, &graph) != cudaSuccess) {
        (void)cudaGetLastError();
        return nullptr;
    }
    return st == cudaStreamCaptureStatusActive ? graph : nullptr;
}

// The plan scratch of one call.  The call's kernels share it, so nothing else may be enqueued on the stream between them that
// uses it too: the object holds the stream's buffer against other host threads until it goes out of scope behind the last
// launch.
class PlanScratch {
public:
    // At least `bytes` for work enqueued on `stream`.  Grows by stream-ordered allocation (the old buffer is released behind the
    // work already enqueued) and lives until vs_release_scratch or the end of the process.  While the stream is being captured
    // the buffer is the graph's; the calls that one capture makes on one stream follow one another in the graph too, so they share one.
    int take(DeviceInfo *d, cudaStream_t stream, size_t bytes, void **out) {
        if (t_ws_set) {   // the caller's buffer or nothing: never allocate behind a caller that manages memory itself
            if ((int64_t)bytes > t_ws_bytes) return VS_ERR_SHAPE;
            *out = t_ws_ptr;
            return VS_OK;
        }
        do {
            lock_ = {};
            {
                std::lock_guard<std::mutex> table(g_devices_mutex);
                std::shared_ptr<Scratch> &entry = d->scratch[DeviceInfo::key_of(stream)];
                if (!entry) entry = std::make_shared<Scratch>();
                held_ = entry;
            }
            lock_ = std::unique_lock<std::mutex>(held_->use);
        } while (held_->retired);   // released while this thread waited for it
        unsigned long long capture = 0;
        if (cudaGraph_t graph = capture_graph(stream, &capture)) {
            if (held_->capture != capture || held_->capture_bytes < bytes) {
                const size_t want = held_->capture == capture ? std::max(bytes, 2 * held_->capture_bytes) : bytes;
                const int rc = graph_scratch(graph, want, &held_->capture_ptr);
                held_->capture = rc == VS_OK ? capture : 0;
                held_->capture_bytes = want;
                if (rc != VS_OK) return rc;
            }
            *out = held_->capture_ptr;
            return VS_OK;
        }
        if (held_->bytes < bytes) {
            size_t want = 1u << 20;
            while (want < bytes) want <<= 1;
            if (bytes > 1u << 20) want = (bytes + want / 16 - 1) / (want / 16) * (want / 16);   // an eighth too much at most
            void *fresh = nullptr;
            cudaError_t e = cudaMallocAsync(&fresh, want, stream);
            if (e != cudaSuccess) {
                (void)cudaGetLastError();
                return (int)e;
            }
            if (held_->ptr) (void)cudaFreeAsync(held_->ptr, stream);
            held_->ptr = fresh;
            held_->bytes = want;
        }
        *out = held_->ptr;
        return VS_OK;
    }

private:
    std::shared_ptr<Scratch> held_;   // outlives the lock on it
    std::unique_lock<std::mutex> lock_;
};

inline bool aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }
inline bool valid_v(int v) { return v == 1 || v == 2 || v == 4 || v == 8; }
inline int elem_size(int dtype) { return dtype == VS_F16 ? 2 : 4; }
inline bool stride_ok(int64_t stride, int dtype) { return stride >= 0 && (stride * elem_size(dtype)) % 16 == 0; }

template <typename K> int set_smem(K kernel, int bytes) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    return e == cudaSuccess ? VS_OK : (int)e;
}
// The same for a kernel whose shared memory never changes: asked once per device (`done`, one bit per device, belongs
// to one kernel), not once per call, where it costs about as much as a tensor map.
typedef std::atomic<uint64_t> DeviceBits;
static_assert(kMaxDevices <= 64, "one bit per device");
template <typename K> int set_smem_once(K kernel, int bytes, DeviceBits &done) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return set_smem(kernel, bytes);
    const uint64_t bit = 1ull << dev;
    if (done.load(std::memory_order_acquire) & bit) return VS_OK;
    const int rc = set_smem(kernel, bytes);
    if (rc == VS_OK) done.fetch_or(bit, std::memory_order_release);
    return rc;
}

// Launches `kernel` so that it may start while the kernel ahead of it in the stream is still running (programmatic
// dependent launch); such a kernel calls pdl_wait() before it reads anything written earlier in the stream.
// VSPARSE_B200_PDL=0 launches the ordinary way.
template <typename... Exp, typename... Act>
cudaError_t launch_overlapped(void (*kernel)(Exp...), unsigned grid, unsigned block, size_t smem, cudaStream_t s, Act &&...args) {
    static const bool overlap = []() {
        const char *e = std::getenv("VSPARSE_B200_PDL");
        return !(e && !std::strcmp(e, "0"));
    }();
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = overlap ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, std::forward<Act>(args)...);
}

// Launches clusters of `size` CTAs, `grid` CTAs in all, as a programmatic dependent.
template <typename... Exp, typename... Act>
cudaError_t launch_clusters(void (*kernel)(Exp...), unsigned grid, unsigned size, unsigned block, size_t smem, cudaStream_t s, Act &&...args) {
    static const bool overlap = []() {
        const char *e = std::getenv("VSPARSE_B200_PDL");
        return !(e && !std::strcmp(e, "0"));
    }();
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = size;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = overlap ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, kernel, std::forward<Act>(args)...);
}

// Launches `pairs` clusters of two CTAs (tcgen05 cta_group::2 kernels), optionally as a programmatic dependent.
template <typename... Exp, typename... Act>
cudaError_t launch_pairs(void (*kernel)(Exp...), unsigned pairs, unsigned block, size_t smem, cudaStream_t s, bool overlapped,
                         Act &&...args) {
    static const bool overlap = []() {
        const char *e = std::getenv("VSPARSE_B200_PDL");
        return !(e && !std::strcmp(e, "0"));
    }();
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * pairs);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = (overlapped && overlap) ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, kernel, std::forward<Act>(args)...);
}

// Diagnostic: CUDA events around the multiplying kernels of the dense tensor-core paths (vs_kernel_timing).  Off by
// default; while on, every such kernel is bracketed by two events on its stream, which also keeps it from
// overlapping the kernels before and behind it (it is timed alone, as a profiler's launch list shows it).
struct KernelTiming {
    std::mutex lock;
    bool on = false;
    std::vector<std::pair<cudaEvent_t, cudaEvent_t>> pairs;
};
KernelTiming &kernel_timing() {
    static KernelTiming t;
    return t;
}
struct TimedLaunch {   // records the opening event on construction, the closing one on destruction
    cudaStream_t s;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    explicit TimedLaunch(cudaStream_t stream) : s(stream) {
        KernelTiming &t = kernel_timing();
        std::lock_guard<std::mutex> g(t.lock);
        if (!t.on) return;
        if (cudaEventCreate(&e0) != cudaSuccess || cudaEventCreate(&e1) != cudaSuccess) { e0 = e1 = nullptr; (void)cudaGetLastError(); return; }
        cudaEventRecord(e0, s);
    }
    ~TimedLaunch() {
        if (!e0) return;
        cudaEventRecord(e1, s);
        KernelTiming &t = kernel_timing();
        std::lock_guard<std::mutex> g(t.lock);
        t.pairs.emplace_back(e0, e1);
    }
};

// cuTensorMapEncodeTiled, fetched from the driver at first use (the library does not link libcuda).
typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn encode_tiled_fn() {
    static EncodeTiledFn fn = []() -> EncodeTiledFn {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess) return nullptr;
        return q == cudaDriverEntryPointSuccess ? reinterpret_cast<EncodeTiledFn>(p) : nullptr;
    }();
    return fn;
}

// Tensor map of a row-major fp16 matrix [rows x cols] for row gathers: box = 64 columns x 1 row, 128-byte
// swizzle, zero fill outside the matrix.
int make_gather_map(CUtensorMap *map, const void *ptr, uint64_t rows, uint64_t cols) {
    EncodeTiledFn fn = encode_tiled_fn();
    if (!fn) return VS_ERR_DEVICE;
    const cuuint64_t dims[2] = {cols, rows};
    const cuuint64_t strides[1] = {cols * 2};
    const cuuint32_t box[2] = {64, 1};
    const cuuint32_t estr[2] = {1, 1};
    CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void *>(ptr), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? VS_OK : VS_ERR_ARG;
}

// Tensor map of a batch of row-major matrices, dimensions {cols, rows, batch}, for tile loads / stores of
// box_cols x box_rows elements, swizzled over the bytes of a box row (128 or 64); loads read zeros outside the
// matrix, stores are clipped there.
int make_tile_map(CUtensorMap *map, const void *ptr, bool f32, uint64_t rows, uint64_t cols, uint64_t batch,
                  uint64_t batch_stride, uint32_t box_cols, uint32_t box_rows, bool swizzled = true) {
    EncodeTiledFn fn = encode_tiled_fn();
    if (!fn) return VS_ERR_DEVICE;
    const uint64_t es = f32 ? 4 : 2;
    const cuuint64_t dims[3] = {cols, rows, batch};
    const cuuint64_t strides[2] = {cols * es, (batch > 1 ? batch_stride : rows * cols) * es};
    const cuuint32_t box[3] = {box_cols, box_rows, 1};
    const cuuint32_t estr[3] = {1, 1, 1};
    const CUtensorMapSwizzle swizzle = !swizzled ? CU_TENSOR_MAP_SWIZZLE_NONE : box_cols * es == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B;
    CUresult r = fn(map, f32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<void *>(ptr), dims,
                    strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? VS_OK : VS_ERR_ARG;
}

// The dense operand of a batch seen as {64 columns, rows, cols / 64 column blocks, batch}: one copy fetches
// 64 rows of `blocks` neighbouring 64-column blocks, each block landing as its own 64 x 128-byte slab.
// cols must be a multiple of 64.
int make_blocked_map(CUtensorMap *map, const void *ptr, uint64_t rows, uint64_t cols, uint64_t batch, uint64_t batch_stride,
                     uint32_t blocks) {
    EncodeTiledFn fn = encode_tiled_fn();
    if (!fn) return VS_ERR_DEVICE;
    const cuuint64_t dims[4] = {64, rows, cols / 64, batch};
    const cuuint64_t strides[3] = {cols * 2, 128, (batch > 1 ? batch_stride : rows * cols) * 2};
    const cuuint32_t box[4] = {64, 64, blocks, 1};
    const cuuint32_t estr[4] = {1, 1, 1, 1};
    CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 4, const_cast<void *>(ptr), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? VS_OK : VS_ERR_ARG;
}

// Tiles of cols x rows fp16 (or bf16) values, `parts` of them side by side, one after another: {cols, rows, parts, tiles}, a copy takes
// all parts of `box_tiles` tiles.  128-byte swizzle (cols = 64).
int make_packed_map(CUtensorMap *map, const void *ptr, uint64_t cols, uint64_t rows, uint64_t parts, uint64_t tiles, uint32_t box_tiles) {
    EncodeTiledFn fn = encode_tiled_fn();
    if (!fn || tiles > 0x7fffffffull) return VS_ERR_DEVICE;
    const cuuint64_t dims[4] = {cols, rows, parts, tiles};
    const cuuint64_t strides[3] = {cols * 2, cols * rows * 2, cols * rows * parts * 2};
    const cuuint32_t box[4] = {(cuuint32_t)cols, (cuuint32_t)rows, (cuuint32_t)parts, box_tiles};
    const cuuint32_t estr[4] = {1, 1, 1, 1};
    CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 4, const_cast<void *>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                    CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? VS_OK : VS_ERR_ARG;
}

// ---- SpMM dispatch ----------------------------------------------------------------------------------------
// 16-byte chunks of the dense width per thread of spmm_cc_kernel: several where the width allows it and the accumulators
// stay in registers (64 at most); VSPARSE_B200_SPMM_CC_CHUNKS=1|2|4 caps them.
int spmm_cc_chunks(int VE, int E, int N) {
    const char *e = std::getenv("VSPARSE_B200_SPMM_CC_CHUNKS");
    const int cap = e ? std::atoi(e) : 4;
    return (VE <= 16 && cap >= 4 && N % (128 * E) == 0) ? 4 : (VE <= 32 && cap >= 2 && N % (64 * E) == 0) ? 2 : 1;
}
int64_t spmm_cc_tile_ctas(const SpmmParams &p) {
    return (((int64_t)p.m_vec + cctile::kWarps - 1) / cctile::kWarps) * (((int64_t)p.N + cctile::kCols - 1) / cctile::kCols) * p.batch;
}
// Whether the fp32 product goes to the kernel that stages tiles of B.  Its CTAs take an SM each: where one wave of them
// holds the product it won or drew at every V, size and sparsity measured from 128 columns up (up to 4x; with 64 columns
// and a few entries per vector-row it lost, 5.5 against 4.3 us).  With two waves it still wins where the other kernel is
// left with under eight warps per SM (1024 x 1024 x 1024 at V = 2, 50 / 90 / 98 % sparse: 60 / 23 / 12.5 against 131 / 39 / 12.5 us), and
// loses where that has more (2048 x 512 x 256 at V = 1: 31 / 12.6 / 8.5 against 29 / 11.5 / 6.4).
// VSPARSE_B200_SPMM_CC=rows|tiles|few chooses one.
bool spmm_cc_tiles_chosen(int V, const SpmmParams &p, const DeviceInfo *d) {
    if (p.K < 1 || p.K > 1 << 30) return false;   // tile coordinates and column sums in 32 bits
    const int64_t ctas = spmm_cc_tile_ctas(p);
    if (ctas > 0x7fffffffll) return false;
    const char *e = std::getenv("VSPARSE_B200_SPMM_CC");
    if (e && !std::strcmp(e, "rows")) return false;
    if (e && !std::strcmp(e, "tiles")) return true;
    const int64_t threads = (int64_t)p.m_vec * (p.N / 4) / spmm_cc_chunks(4 * V, 4, p.N) * p.batch;
    return p.K >= 128 && (ctas <= d->sm_count || (ctas <= 2 * d->sm_count && threads <= (int64_t)d->sm_count * 256));
}
// Bytes of a lane's columns in spmm_cc_few_kernel, or 0 where the others are the quicker ones: up to 20 of its warps per SM of 4-byte lanes at any V; where
// rows would go to spmm_cc_kernel (no `tiles`) up to 96 at V = 2, and at V = 1 16-byte lanes up to 28.  us, as before / 4-byte / 16-byte lanes, warps of the
// latter: fp16, V = 1, 132 rows x 4400 x 64, 55 % (66) 320 / 49 / 137, V = 2, 313 x 1019 x 48, 67 % (118) 78 / 18.5 / 51; fp32, V = 2, 110 x 4142 x 208, 59 %
// (220) 134 / 68 / 220, V = 8, 50 x 2520 x 1784, 82 % (700) 72 / 55 / 116, V = 4, 68 x 1805 x 1940, 76 % (1088) 46 / 47 / 107; V = 1, 2416 x 1272 x 216, 60 %
// (4832) 115 / 109 / 70, 575 x 139 x 1432, 78 % (6900) 12.3 / 22.6 / 13.1; V = 2, 200 x 1350 x 2100, 62 % (3400) 130 / 97 / 100, 147 x 130 x 3360, 54 %
// (3969) 20.5 / 22.5 / 17.5.  VSPARSE_B200_SPMM_CC=few chooses the 4-byte lanes.
int spmm_cc_few_bytes(int V, int chunk_elems, const SpmmParams &p, bool tiles, const DeviceInfo *d) {
    const char *e = std::getenv("VSPARSE_B200_SPMM_CC");
    if (e) return !std::strcmp(e, "few") ? 4 : 0;
    const int64_t rows = (int64_t)p.m_vec * p.batch;
    if (rows * ((p.N + 8 * chunk_elems - 1) / (8 * chunk_elems)) <= 20 * (int64_t)d->sm_count) return 4;
    const int64_t wide = rows * ((p.N + 32 * chunk_elems - 1) / (32 * chunk_elems));
    if (tiles || wide > 28 * (int64_t)d->sm_count) return 0;
    return V == 1 ? 16 : V == 2 && wide <= 24 * (int64_t)d->sm_count ? 4 : 0;
}
// Leaves *taken false where no tensor map can be made.
template <int V> int launch_spmm_cc_tile(const SpmmParams &p, DeviceInfo *d, cudaStream_t s, bool *taken) {
    using L = cctile::Layout<V>;
    const int groups = (int)(((int64_t)p.m_vec + cctile::kWarps - 1) / cctile::kWarps), slabs = (int)(((int64_t)p.N + cctile::kCols - 1) / cctile::kCols);
    CUtensorMap map;
    if (make_tile_map(&map, p.rhs, true, (uint64_t)p.K, (uint64_t)p.N, p.stride_rhs ? (uint64_t)p.batch : 1, (uint64_t)p.stride_rhs, cctile::kCols,
                      cctile::kTile, false) != VS_OK)
        return VS_OK;
    auto kernel = cctile::spmm_cc_tile_kernel<V>;
    static DeviceBits done;
    const int rc = set_smem_once(kernel, L::kSmemBytes, done);
    if (rc != VS_OK) return rc;
    *taken = true;
    kernel<<<(unsigned)groups * slabs * p.batch, cctile::kThreads, L::kSmemBytes, s>>>(p, map, groups, slabs, d->status);
    return (int)cudaGetLastError();
}
int spmm_cc_tile(int V, const SpmmParams &p, cudaStream_t s, bool *taken) {
    DeviceInfo *d = nullptr;
    const int rc = device_info(&d);
    if (rc != VS_OK) return rc;
    if (!spmm_cc_tiles_chosen(V, p, d) || spmm_cc_few_bytes(V, 4, p, true, d)) return VS_OK;
    switch (V) {
        case 1: return launch_spmm_cc_tile<1>(p, d, s, taken);
        case 2: return launch_spmm_cc_tile<2>(p, d, s, taken);
        case 4: return launch_spmm_cc_tile<4>(p, d, s, taken);
        case 8: return launch_spmm_cc_tile<8>(p, d, s, taken);
    }
    return VS_OK;
}

// Slab by slab (cuda_core.cuh) where the pieces of a row, of `want` chunks each, come in warps, and there are enough of those that the ones at work
// together share columns; half as many will do where B does not stay in L2.  us, row by row / slab by slab, 90 % sparse, thousands of warps: 4096 x 4096 x 8192
// V = 1 (64) 2628 / 2377, V = 2 (32) 1379 / 1248, V = 8 (16) 1033 / 924; 4096 x 1024 x 8192 V = 1 (64) 641 / 528, V = 4 (16) 263 / 255; 2048 x 2048 x 4096 V = 1 (16)
// 322 / 306, V = 2 (8) 169 / 180, V = 8 (4) 135 / 142; 1024 x 1024 x 8192 V = 1 (16) 167 / 157, V = 2 (8) 91 / 97; 2048 x 2048 x 8192, 67 MB of B, V = 8 (8) 297 / 268;
// 512 x 4096 x 8192 V = 2 (4) 186 / 191.  With 1024 columns nothing, or 3 % lost.
bool spmm_cc_slabs(const SpmmParams &p, int want) {
    if (p.N < kSlabColumns || p.N % (128 * want) != 0) return false;
    const int64_t warps = (int64_t)p.m_vec * (p.N / (128 * want));
    return warps >= 16384 || (warps >= 8192 && (int64_t)p.K * p.N * 4 >= 64 << 20);
}
template <typename TIn, typename TOut, int V, int kChunks> void launch_spmm_cc_as(const SpmmParams &p, dim3 grid, cudaStream_t s) {
    if constexpr (sizeof(TIn) == 4) {
        if (spmm_cc_slabs(p, kChunks)) {
            spmm_cc_kernel<TIn, TOut, V, kChunks, true><<<grid, kCcThreads, 0, s>>>(p);
            return;
        }
    }
    spmm_cc_kernel<TIn, TOut, V, kChunks><<<grid, kCcThreads, 0, s>>>(p);
}
template <typename TIn, typename TOut, int V, int kBytes> int launch_spmm_cc_few(const SpmmParams &p, cudaStream_t s) {
    const int pieces = (p.N + 32 * Piece<TIn, kBytes>::kElems - 1) / (32 * Piece<TIn, kBytes>::kElems);
    const int64_t blocks = ((int64_t)p.m_vec * pieces + kFewWarps - 1) / kFewWarps;
    if (blocks > 0x7fffffffll) return VS_ERR_SHAPE;
    spmm_cc_few_kernel<TIn, TOut, V, kBytes><<<dim3((unsigned)blocks, (unsigned)p.batch), kFewThreads, 0, s>>>(p, pieces);
    return (int)cudaGetLastError();
}
template <typename TIn, typename TOut, int V> int launch_spmm_cc(const SpmmParams &p, cudaStream_t s) {
    constexpr int E = Chunk<TIn>::kElems;
    DeviceInfo *d = nullptr;
    const int rc = device_info(&d);
    if (rc != VS_OK) return rc;
    const int few = spmm_cc_few_bytes(V, E, p, false, d);
    if (few == 4) return launch_spmm_cc_few<TIn, TOut, V, 4>(p, s);
    if constexpr (V == 1) {
        if (few == 16) return launch_spmm_cc_few<TIn, TOut, V, 16>(p, s);
    }
    const int want = spmm_cc_chunks(V * E, E, p.N);
    const int64_t items = (int64_t)p.m_vec * (p.N / E) / want;
    const int64_t blocks = (items + kCcThreads - 1) / kCcThreads;
    if (blocks > 0x7fffffffll) return VS_ERR_SHAPE;
    dim3 grid((unsigned)blocks, (unsigned)p.batch, 1);
    if constexpr (V * E <= 16) {
        if (want == 4) {
            launch_spmm_cc_as<TIn, TOut, V, 4>(p, grid, s);
            return (int)cudaGetLastError();
        }
    }
    if constexpr (V * E <= 32) {
        if (want == 2) {
            launch_spmm_cc_as<TIn, TOut, V, 2>(p, grid, s);
            return (int)cudaGetLastError();
        }
    }
    launch_spmm_cc_as<TIn, TOut, V, 1>(p, grid, s);
    return (int)cudaGetLastError();
}

int spmm_split(int V, const SpmmParams &p, cudaStream_t s, bool *taken);
template <typename TIn, typename TOut> int spmm_cc_by_v(int V, const SpmmParams &p, cudaStream_t s) {
    if constexpr (sizeof(TIn) == 4) {
        bool taken = false;
        int rc = spmm_split(V, p, s, &taken);
        if (rc != VS_OK || taken) return rc;
        rc = spmm_cc_tile(V, p, s, &taken);
        if (rc != VS_OK || taken) return rc;
    }
    switch (V) {
        case 1: return launch_spmm_cc<TIn, TOut, 1>(p, s);
        case 2: return launch_spmm_cc<TIn, TOut, 2>(p, s);
        case 4: return launch_spmm_cc<TIn, TOut, 4>(p, s);
        case 8: return launch_spmm_cc<TIn, TOut, 8>(p, s);
    }
    return VS_ERR_VEC_LENGTH;
}
template <typename TOut, int V> int launch_spmm_cc_standby(const SpmmParams &p, cudaStream_t s, DeviceInfo *d, const int32_t *plan_hdr, int plan_checks,
                                                          bool overlapped = true) {
    const int64_t blocks = ((int64_t)p.m_vec * (p.N / Chunk<__half>::kElems) * p.batch + kCcThreads - 1) / kCcThreads;
    const int64_t cap = (int64_t)d->sm_count * 8;
    const unsigned grid = (unsigned)(blocks < cap ? blocks : cap);
    if (!overlapped) {
        spmm_cc_standby_kernel<__half, TOut, V><<<grid, kCcThreads, 0, s>>>(p, plan_hdr, plan_checks, 0);
        return (int)cudaGetLastError();
    }
    return (int)launch_overlapped(spmm_cc_standby_kernel<__half, TOut, V>, grid, kCcThreads, 0, s, p, plan_hdr, plan_checks, 0);
}

// Software (cp.async) gather: works for any batch stride.
template <typename TOut, int V>
int launch_spmm_tc_cpasync(const SpmmParams &p, cudaStream_t s, DeviceInfo *d, const int32_t *plan_hdr = nullptr, int plan_checks = 0) {
    auto kernel = tcspmm::spmm_tc_kernel<TOut, V>;
    static DeviceBits smem_set;
    int rc = set_smem_once(kernel, tcspmm::kSmemBytes, smem_set);
    if (rc != VS_OK) return rc;
    const int n_tiles = (p.N + tcspmm::kTileN - 1) / tcspmm::kTileN;
    const int64_t items = (int64_t)p.batch * n_tiles * p.m_vec;
    const int64_t cap = (int64_t)tcspmm::kCtasPerSm * d->sm_count;  // persistent CTAs
    const unsigned grid = (unsigned)(items < cap ? items : cap);
    if (plan_hdr) return (int)launch_overlapped(kernel, grid, tcspmm::kThreads, tcspmm::kSmemBytes, s, p, d->status, plan_hdr, plan_checks);
    kernel<<<grid, tcspmm::kThreads, tcspmm::kSmemBytes, s>>>(p, d->status, plan_hdr, plan_checks);
    return (int)cudaGetLastError();
}

// TMA row gather: the dense operand of all batch entries must be addressable as one matrix of N-wide rows,
// i.e. the batch stride is a multiple of N (or zero / a single entry).  With `plan_hdr` the kernel returns at
// once when that plan header says that the densifying kernel has taken the call.
template <typename TOut, int V>
int launch_spmm_gather(const SpmmParams &p, cudaStream_t s, DeviceInfo *d, const int32_t *plan_hdr, int plan_checks) {
    static const bool force_cpasync = []() {
        const char *e = std::getenv("VSPARSE_B200_GATHER");
        return e && !std::strcmp(e, "cpasync");
    }();
    const bool one = p.batch == 1 || p.stride_rhs == 0;
    const int64_t rows_per_batch = one ? 0 : p.stride_rhs / p.N;
    const int64_t total_rows = (one ? 0 : (int64_t)(p.batch - 1) * rows_per_batch) + p.K;
    const bool tma_ok = !force_cpasync && p.K > 0 && (one || p.stride_rhs % p.N == 0) && total_rows < 0x7fffffffll;
    if (!tma_ok) return launch_spmm_tc_cpasync<TOut, V>(p, s, d, plan_hdr, plan_checks);
    CUtensorMap map;
    int rc = make_gather_map(&map, p.rhs, (uint64_t)total_rows, (uint64_t)p.N);
    if (rc != VS_OK) return launch_spmm_tc_cpasync<TOut, V>(p, s, d, plan_hdr, plan_checks);
    auto kernel = tmaspmm::spmm_tma_kernel<TOut, V>;
    static DeviceBits smem_set;
    rc = set_smem_once(kernel, tmaspmm::kSmemBytes, smem_set);
    if (rc != VS_OK) return rc;
    const int n_tiles = (p.N + tmaspmm::kTileN - 1) / tmaspmm::kTileN;
    const int64_t items = (int64_t)p.batch * n_tiles * p.m_vec;
    const int64_t cap = (int64_t)tmaspmm::kCtasPerSm * d->sm_count;  // persistent CTAs
    const unsigned grid = (unsigned)(items < cap ? items : cap);
    if (plan_hdr)
        return (int)launch_overlapped(kernel, grid, tmaspmm::kThreads, tmaspmm::kSmemBytes, s, p, map, (int)rows_per_batch,
                                      (int)total_rows, d->status, plan_hdr, plan_checks);
    kernel<<<grid, tmaspmm::kThreads, tmaspmm::kSmemBytes, s>>>(p, map, (int)rows_per_batch, (int)total_rows, d->status,
                                                                plan_hdr, plan_checks);
    return (int)cudaGetLastError();
}

// Which tensor-core SpMM runs.  The densifying kernel multiplies zero-filled 256 x 64 tiles of A, the gather
// kernels fetch one row of B per nonzero vector: the first costs the same whatever the sparsity, the second is
// proportional to the nonzeros.  The number of nonzeros is only known on the device (the reference signature
// does not pass it), so the choice is made there: the plan kernel compares the two costs (see there) and
// leaves a flag that one of the two kernels, both enqueued, finds set against it and returns at once.  The
// densifying kernel sets the plan's redo word if it produced a non-finite sum, so that the gather kernel redoes the
// call with the reference's semantics for Inf / NaN in rows of B that no nonzero names.
enum class SpmmMode { kAuto, kDense, kGather, kDirect };
SpmmMode spmm_mode() {   // read at every call, so that a test can switch kernels inside one process
    const char *e = std::getenv("VSPARSE_B200_SPMM");
    if (e && !std::strcmp(e, "dense")) return SpmmMode::kDense;
    if (e && !std::strcmp(e, "gather")) return SpmmMode::kGather;
    if (e && !std::strcmp(e, "direct")) return SpmmMode::kDirect;
    return SpmmMode::kAuto;
}
constexpr int64_t kMaxPlanBytes = 512ll << 20;

// Bytes of plan scratch the densifying SpMM needs: the header (verdict + one word per duplicate-checking CTA of
// the plan kernel), the bucket offsets, 8 bytes per possible entry.
inline int spmm_plan_checks(int m_vec) {   // duplicate-checking CTAs: a vector-row per warp, a few rows each at most
    const int want = (m_vec + densespmm::kPlanWarps - 1) / densespmm::kPlanWarps;
    return want < densespmm::kMaxCheckCtas ? want : densespmm::kMaxCheckCtas;
}
inline int64_t spmm_plan_header_bytes(int checks) { return ((int64_t)(4 + checks) * 4 + 15) & ~15ll; }
int64_t spmm_plan_bytes(int m_vec, int V, int K, int batch, int64_t stride_values, int64_t *capacity_out, int64_t *offsets_out) {
    const int k_blocks = (K + densespmm::kBlockK - 1) / densespmm::kBlockK;
    const int m_tiles = (int)(((int64_t)m_vec * V + densespmm::kTileM - 1) / densespmm::kTileM);
    const int groups = m_tiles * (densespmm::kTileM / densespmm::kGroupRows);
    const int plan_blocks = k_blocks * (densespmm::kBlockK / densespmm::kPlanCols);
    // entries are addressed like the nonzero vectors: at most one per (vector-row, column), and never more than
    // fit between two matrices of a batch
    int64_t capacity = (int64_t)m_vec * K;
    if (batch > 1 && stride_values > 0 && stride_values / V < capacity) capacity = stride_values / V;
    const int64_t offsets_bytes = (((int64_t)groups * (plan_blocks + 1) * 4) + 15) & ~15ll;
    if (capacity_out) *capacity_out = capacity;
    if (offsets_out) *offsets_out = offsets_bytes;
    return spmm_plan_header_bytes(spmm_plan_checks(m_vec)) + offsets_bytes + capacity * 8;
}
// The plan of A^T for the transposed product: n rows over m_vec * V columns, one entry per nonzero VECTOR of A.
int64_t spmm_t_plan_bytes(int n, int m_vec, int V, int batch, int64_t stride_values, int64_t *capacity_out, int64_t *offsets_out) {
    const int64_t M = (int64_t)m_vec * V;
    const int k_blocks = (int)((M + densespmm::kBlockK - 1) / densespmm::kBlockK);
    const int m_tiles = (n + densespmm::kTileM - 1) / densespmm::kTileM;
    const int groups = m_tiles * (densespmm::kTileM / densespmm::kGroupRows);
    const int plan_blocks = k_blocks * (densespmm::kBlockK / densespmm::kPlanCols);
    int64_t capacity = (int64_t)n * m_vec;   // at most one vector per (column of A, vector-row)
    if (batch > 1 && stride_values > 0 && stride_values / V < capacity) capacity = stride_values / V;
    const int64_t offsets_bytes = (((int64_t)groups * (plan_blocks + 1) * 4) + 15) & ~15ll;
    if (capacity_out) *capacity_out = capacity;
    if (offsets_out) *offsets_out = offsets_bytes;
    return spmm_plan_header_bytes(spmm_plan_checks(n)) + offsets_bytes + capacity * 8;
}
// The same for the dense SDDMM: per-row chunk offsets and 8 bytes per mask entry.
int64_t sddmm_plan_bytes(int m_vec, int n, int nnz_vec, int64_t *offsets_out) {
    const int chunks = (n + densesddmm::kChunk - 1) / densesddmm::kChunk;
    const int64_t offsets_bytes = (((int64_t)m_vec * (chunks + 1) * 4) + 15) & ~15ll;
    if (offsets_out) *offsets_out = offsets_bytes;
    return offsets_bytes + (int64_t)nnz_vec * 8;
}

// How many pairs of CTAs of `kernel` the device holds at once (one CTA per SM, two neighbouring SMs per pair).
template <typename K> int max_resident_pairs(K kernel, int block, size_t smem, DeviceInfo *d) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * (unsigned)d->sm_count);
    cfg.blockDim = dim3((unsigned)block);
    cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess) {
        (void)cudaGetLastError();
        return 0;
    }
    return n;
}

// The densified product by pairs of CTAs (spmm_pair.cuh) takes dense widths from 128 up, the single-CTA kernel (spmm_dense.cuh) the narrower ones, and 128 where
// there are more row tiles than its CTAs.  us, single CTAs / pairs, product with the matrix
// and with its transpose: 64 x (2048 x 512 x N), V = 8, 90 % sparse: N = 128 28 / 33 and 33 / 39, 192 38 / 35 and 51 / 41, 448 65 / 59 and 85 / 64;
// 4096 x 4096 x 1984, V = 2, 70 %: 261 / 149 and 281 / 161; widths that are no multiple of 64: 64 x (2048 x 512 x 200), V = 8 45.6 / 40.0, x 264 63 / 59,
// 17 x (2062 x 1310 x 560), V = 2 (laid out) 241 / 148, 4 x (3958 x 1750 x 584), V = 1 (laid out) 195 / 81.  VSPARSE_B200_SPMM_PAIR=0 keeps every width on the former, =1 on the latter.
inline bool spmm_pair_takes(int N, int V, int64_t row_items, const DeviceInfo *d, bool from_plan = false) {
    const char *e = std::getenv("VSPARSE_B200_SPMM_PAIR");
    if (N % 8 != 0 || N < 128 || (e && !std::strcmp(e, "0"))) return false;
    if (from_plan && V <= 2 && N % 64 != 0 && !e) return false;   // scattering short vectors for the rest of a wide tile costs more than the pair saves (V = 1 41 / 34 for 64 x (1024 x 256 x 256) already)
    return N > 128 || row_items <= d->sm_count || e;
}
// Columns of B per work item of the pair kernel.  An item of 128 columns costs 0.9 of one of 256 (both fill the same tile of A), so
// 256 it is, a partly empty last tile included, unless the narrower items need fewer waves of pairs.
int spmm_pair_width(int N, int64_t row_items, int pairs) {
    if (N <= 128) return 128;
    const int64_t wide = row_items * ((N + 255) / 256), narrow = row_items * ((N + 127) / 128);
    return 9 * ((narrow + pairs - 1) / pairs) < 10 * ((wide + pairs - 1) / pairs) ? 128 : 256;
}
// How many pairs of `kernel` this device holds; -1 where it cannot run it.
template <typename K> int pair_capacity(K kernel, int threads, int (&resident)[kMaxDevices], DeviceInfo *d) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return -1;
    if (resident[dev] == 0) {   // not asked yet
        const int n = set_smem(kernel, pairspmm::kSmemBytes) == VS_OK ? max_resident_pairs(kernel, threads, pairspmm::kSmemBytes, d) : 0;
        resident[dev] = n > 0 ? n : -1;
    }
    return resident[dev];
}
// Enqueues the pair kernel for a call whose plan kernel has been enqueued; false if this device cannot hold it.
template <typename TOut, int V, bool kTransposed>
bool launch_spmm_pair(const SpmmParams &q, cudaStream_t s, DeviceInfo *d, const CUtensorMap &map, const CUtensorMap &map_out,
                      const CUtensorMap &map_b2, const int32_t *blk_offsets, const uint2 *blk_entries, int m_tiles, int k_blocks,
                      int32_t *flag, int checks, int32_t *redo, int *rc_out) {
    static int resident[kMaxDevices];
    auto kernel = pairspmm::spmm_pair_kernel<TOut, V, kTransposed>;
    const int capacity = pair_capacity(kernel, pairspmm::kThreads, resident, d);
    if (capacity < 0) return false;
    const int tn = spmm_pair_width(q.N, (int64_t)q.batch * m_tiles, capacity);
    const int n_tiles = (q.N + tn - 1) / tn;
    const int64_t items = (int64_t)q.batch * n_tiles * m_tiles;
    const unsigned pairs = (unsigned)(items < capacity ? items : capacity);
    TimedLaunch timed(s);
    *rc_out = (int)launch_pairs(kernel, pairs, pairspmm::kThreads, (size_t)pairspmm::kSmemBytes, s, true, q, map, 1, 0, map, map_out, map_b2, tn,
                                blk_offsets, blk_entries, m_tiles, n_tiles, k_blocks, d->status, flag, checks, redo);
    return true;
}

// Costs of the two formulations in SM-cycles per 128 columns of B, as the plan kernel compares them (see there).
struct SpmmCosts {
    float dense_per_stage, dense_per_entry, gather_per_row, gather_per_entry;
};
constexpr SpmmCosts kGatherCosts = {1100.0f, 0.0f, 370.0f, 4.7f};
// The same with the CUDA-core kernel as the other formulation, fitted at V = 1 and 2 to 512 x 4096 to 4096 x 4096, 64 to 1024 dense columns, 60 to
// 99.7 % sparse.
constexpr SpmmCosts cores_costs(int V) {
    return {700.0f, V == 1 ? 1.0f : V == 2 ? 0.5f : 0.0f, V == 1 ? 25.0f : V == 2 ? 50.0f : 100.0f, V == 1 ? 5.6f : V == 2 ? 13.0f : V == 4 ? 13.0f : 20.0f};
}
// What they come to where a product leaves SMs idle: the densified one has few tiles, each walking its columns in series; the CUDA-core
// kernel few rows, with 0.3 us for an entry behind the other.  Without this 4096 x 4096 x 256 at V = 2 and 99 % sparse took 34 us on tiles that the
// CUDA-core kernel needs 10 for; at 95 % the tiles' 41 against 36.
SpmmCosts cores_costs_of(const SpmmParams &p, int V, int64_t items, int units, const DeviceInfo *d) {
    SpmmCosts c = cores_costs(V);
    const float idle = std::max(1.0f, (float)units / (float)std::max<int64_t>(items, 1));
    c.dense_per_stage *= idle;
    c.dense_per_entry *= idle;
    c.gather_per_entry = std::max(c.gather_per_entry, 0.3f * 1900.0f * (float)d->sm_count * 128.0f / (float)p.N / (float)p.m_vec / (float)p.batch);
    return c;
}

// What takes a call that the densified product does not: the gather kernels (wmmaSpmm) or the CUDA-core kernel (cudaSpmm
// with fp16 results).  With a plan header: as a stand-by behind a densifying kernel.
template <typename TOut, int V, bool kCores>
int launch_spmm_other(const SpmmParams &p, cudaStream_t s, DeviceInfo *d, const int32_t *plan_hdr, int plan_checks) {
    if constexpr (kCores) {
        return plan_hdr ? launch_spmm_cc_standby<TOut, V>(p, s, d, plan_hdr, plan_checks) : launch_spmm_cc<__half, TOut, V>(p, s);
    } else {
        return launch_spmm_gather<TOut, V>(p, s, d, plan_hdr, plan_checks);
    }
}

// The sizes of the whole call that `p` is a part of (vs_set_part_of); its own where it is a part of none.
SpmmParams whole_call(const SpmmParams &p) {
    SpmmParams whole = p;
    whole.N = std::max(p.N, t_whole_columns);
    whole.batch = std::max(p.batch, t_whole_batch);
    return whole;
}
// CTAs that share a tile of the one-kernel form: as many as the tiles leave room for, two from seven chunks of 128 columns on, up to eight with three or more
// each.  us, 1 / 2 / 4 / 8: 80 x 4023 x 320, V = 8, 52 % 37 / 23 / 15.5 / 13.8;
// 1588 x 2035 x 104, V = 4, 57 % 36 / 27 / 21; 172 x 2995 x 64, V = 2, 52 % 64 / 39 / 26 / 19; 158 x 1018 x 128, V = 2, 93 % 12.6 / 10.5; but six chunks,
// 15 x (232 x 986 x 64) and alike, V = 8, 91 %: 8.3 to 9.0 / 8.7 to 10.1.  VSPARSE_B200_SPMM_SPLIT sets the most.
int spmm_direct_split(const SpmmParams &p, int V, const DeviceInfo *d) {
    const int chunks = (p.K + directspmm::kChunkK - 1) / directspmm::kChunkK;
    if (chunks < 7) return 1;
    const char *e = std::getenv("VSPARSE_B200_SPMM_SPLIT");
    const int most = e ? std::atoi(e) : directspmm::kMaxSplit;
    const int64_t tiles = ((int64_t)p.m_vec * V + directspmm::kTileM - 1) / directspmm::kTileM * ((p.N + directspmm::kTileN - 1) / directspmm::kTileN) * p.batch;
    int split = 1;
    while (2 * split <= std::min(most, directspmm::kMaxSplit) && 2 * split * tiles <= 2 * d->sm_count && std::max(7, 6 * split) <= chunks) split *= 2;
    return split;
}
// Small products in one kernel (spmm_direct.cuh), `split` CTAs to a tile; false if this call or this device cannot take it.  When the densified
// product is the cheaper one whatever the number of nonzeros, nothing else is enqueued; otherwise the kernel leaves its
// verdict where the gather kernel behind it looks for the plan kernel's.
template <typename TOut, int V, bool kCores> bool launch_spmm_direct(const SpmmParams &p, cudaStream_t s, DeviceInfo *d, SpmmCosts cost,
                                                                     bool forced, int split, int *rc_out) {
    const int m_tiles = (int)(((int64_t)p.m_vec * V + directspmm::kTileM - 1) / directspmm::kTileM);
    const int n_tiles = (p.N + directspmm::kTileN - 1) / directspmm::kTileN;
    const int64_t tiles = (int64_t)p.batch * m_tiles * n_tiles;
    if (tiles > 0x7fffffffll || p.K <= 0 || p.N % 8 != 0) return false;
    const float stages = std::ceil((float)p.m_vec * V / densespmm::kTileM) * std::ceil((float)p.K / densespmm::kBlockK);
    // Against the CUDA-core kernel it is the quicker form of a small product down to a few per cent of the vectors.  Up to 1024
    // columns, and at V > 2, a stand-by behind every call would cost more than it saves on the few below; with short vectors
    // and more columns the line is a density, which the device knows.  Forced / CUDA-core kernel, us, 90 / 95 / 98 % sparse: V = 1,
    // 2048 x 2048 x 256 53 / 37 / 28 against 53 / 31 / 17, 419 x 2665 x 64 49 / 35 / 29 against 80 / 43 / 25; V = 2, 209 vector-rows of that
    // with 256 dense columns 34 / 31 / 25 against 72 / 41 / 23.
    // V > 2: only past 4096 columns, where a product whose rows hold a few entries waits for 32 and more chunks, and with scratch.
    const bool by_density = kCores && !forced && (V <= 2 ? p.K > 1024 : p.K > 4096 && !t_no_scratch);
    const SpmmParams whole = split > 1 ? whole_call(p) : p;   // its parts share tiles where it does
    const bool many = (int64_t)whole.batch * m_tiles * ((whole.N + directspmm::kTileN - 1) / directspmm::kTileN) > 48;
    if (by_density) cost = {(V > 2 ? 0.018f : V == 2 ? 0.03f : many ? 0.045f : 0.035f) * (float)p.K * (float)p.m_vec / stages, 0.0f, 0.0f, 1.0f};
    bool always = forced || (kCores && !by_density) || (!kCores && cost.dense_per_entry == 0.0f && cost.dense_per_stage * stages < cost.gather_per_row * (float)p.m_vec);
    // A caller that says how many values there are is spared the kernel that would return at once (10 x (4 to 16 rows of tiles), 700 to 1600 columns: 2 to 3 of
    // 8 to 16 us).  The distance between the matrices of a batch is no such number, only a bound: too few for the tiles by that are too few, enough by that the
    // device has to say.
    if (!always && p.stride_values > 0) {
        const float nnz = (float)(p.stride_values / V);
        if (!(cost.dense_per_stage * stages + cost.dense_per_entry * nnz < cost.gather_per_row * (float)p.m_vec + cost.gather_per_entry * nnz)) {
            *rc_out = launch_spmm_other<TOut, V, kCores>(p, s, d, nullptr, 0);
            return true;
        }
        always = whole_call(p).batch == 1;
    }
    CUtensorMap map;
    static DeviceBits smem_set, smem_set_split;
    auto kernel = split > 1 ? directspmm::spmm_direct_kernel<TOut, V, true> : directspmm::spmm_direct_kernel<TOut, V, false>;
    if (tiles * split > 0x7fffffffll || make_tile_map(&map, p.rhs, false, (uint64_t)p.K, (uint64_t)p.N, (uint64_t)p.batch, (uint64_t)p.stride_rhs, 64, 64) != VS_OK ||
        set_smem_once(kernel, directspmm::kSmemBytes, split > 1 ? smem_set_split : smem_set) != VS_OK)
        return false;
    void *verdict = nullptr;
    PlanScratch scratch;
    if (!always && (t_no_scratch || scratch.take(d, s, 16, &verdict) != VS_OK)) return false;
    if (split > 1)
        *rc_out = (int)launch_clusters(kernel, (unsigned)(tiles * split), (unsigned)split, directspmm::kThreads, directspmm::kSmemBytes, s, p, map, m_tiles, n_tiles,
                                       cost.dense_per_stage * stages, cost.dense_per_entry, cost.gather_per_row, cost.gather_per_entry,
                                       static_cast<int32_t *>(verdict), d->status);
    else
        *rc_out = (int)launch_overlapped(kernel, (unsigned)tiles, directspmm::kThreads, directspmm::kSmemBytes, s, p, map, m_tiles, n_tiles,
                                         cost.dense_per_stage * stages, cost.dense_per_entry, cost.gather_per_row, cost.gather_per_entry,
                                         static_cast<int32_t *>(verdict), d->status);
    if (*rc_out == VS_OK && !always) {
        // Not overlapped: CTAs that become resident beside a grid of under one wave crowd onto the SMs it leaves free, and where the
        // CUDA-core kernel then does the work that cost it half its speed (V = 1, 4096 x 4096 x 256, 98 % sparse: 31 -> 46 us).
        if constexpr (kCores) *rc_out = launch_spmm_cc_standby<TOut, V>(p, s, d, static_cast<const int32_t *>(verdict), 0, false);
        else *rc_out = launch_spmm_other<TOut, V, kCores>(p, s, d, static_cast<const int32_t *>(verdict), 0);
    }
    return true;
}
// Which products are small: up to one wave of 128 x 64 tiles at two per SM the one-kernel form saves the ~9 us of the other
// launches (2048 x 512 x 256, V = 8: 15.4 -> 6.5 us; 512 x 2048 x 256: 22.3 -> 13.3), up to two waves while K is short.  Shorter
// vectors mean more entries per tile, which it scatters again for every 64 columns of B, so there the line lies at a smaller
// K (V = 2, 2048 x 2048 x 256, 60 and 95 % sparse: 85 -> 68 and 28 -> 30; 4096 x 4608 x 256, 85 % sparse: 74 -> 88).
// The entry point with the CUDA-core kernel behind it takes it at any K where short vectors meet a narrow B: the planned
// kernels' 256-row tiles leave most SMs idle there (V = 1, 4096 x 4096 x 64, 80 / 95 % sparse: 272 -> 114 and 94 -> 53 us; 128 x 4096 x
// 256: 136 -> 109 and 51 -> 50), at V = 2 up to 64 tiles (2048 vector-rows x 4096 x 64: 143 -> 71 and 58 -> 46; with 256 dense columns
// 82 -> 93 and 47 -> 60).
bool spmm_direct_wanted(const SpmmParams &p, int V, bool cores, int split, const DeviceInfo *d) {
    const int64_t m_tiles = ((int64_t)p.m_vec * V + directspmm::kTileM - 1) / directspmm::kTileM;
    const int64_t tiles = m_tiles * ((p.N + directspmm::kTileN - 1) / directspmm::kTileN) * p.batch;
    const int chunks = (p.K + directspmm::kChunkK - 1) / directspmm::kChunkK;
    if (cores && p.N <= 256 && ((V == 1 && tiles <= 2 * d->sm_count) || (V == 2 && tiles <= 64))) return true;
    // Few tiles share their columns among CTAs, which puts the line at so many times the K.  At V <= 2 a matrix laid out first is on the other side of it where
    // B is wide enough to pay for that.  us, one kernel / laid out, V = 2: 657 x 1460 x 1320, 78 % (12 chunks) 38 / 22, 909 x 1511 x 872, 57 % 50 / 25, 1180 x
    // 1966 x 640, 81 % (8 each) 29 / 24, 506 x 765 x 704, 71 % (6) 18.5 / 16.2, 1906 x 569 x 528, 76 % (5) 20.6 / 26.9; 1984 x 1031 x 320, 87 % (9) 24 / 28, 8 x (97 x
    // 762 x 192), 88 % (6) 17 / 22, 1762 x 1938 x 192, 87 % (4) 21.6 / 26, 1984 x 3120 x 192, 61 % (13) 120 / 110; one kernel / a plan, 172 x 2995 x 64 19 / 164, 16 x
    // (1062 x 2224 x 32) (9) 36 / 80, V = 1, 2 x (2792 x 4032 x 112) (16) 165 / 157.
    const int each = (chunks + split - 1) / split;
    const int short_vectors = p.N >= 512 && !t_no_scratch ? (tiles > 40 ? 5 : 6) : split > 1 ? 10 : 16;
    if (tiles <= 2 * d->sm_count) return each <= (V == 8 ? 64 : V == 4 ? 32 : short_vectors);
    return tiles <= 4 * d->sm_count && chunks <= (V >= 4 ? 4 : 1);
}
// Whether a call takes that form, and how many CTAs share a tile.  Shared tiles add up in another order than every other kernel of the tensor cores, so a part of a
// call (vs_set_part_of) has them where, and as, the whole does; where the whole has not, a part takes what is quickest for its own sizes.
bool spmm_direct_chosen(const SpmmParams &p, int V, bool cores, bool forced, const DeviceInfo *d, int *split) {
    const SpmmParams whole = whole_call(p);
    *split = spmm_direct_split(whole, V, d);
    const bool chosen = forced || spmm_direct_wanted(whole, V, cores, *split, d);
    if ((chosen && *split > 1) || (whole.N == p.N && whole.batch == p.batch)) return chosen;
    *split = 1;
    return forced || spmm_direct_wanted(p, V, cores, 1, d);
}

// The same product with A laid out densely in memory first (densify.cuh), at V <= 2, where filling the tiles from a plan is what the pair
// kernel spends its time on: a stage takes it 1 to 3 us at V = 1 (95 to 80 % sparse) and 0.8 to 1.2 at V = 2, with A laid out 0.5.  Laying it out
// takes 0.67 us per MB, once instead of for every 256 columns of B.  us, plan / laid out: V = 1, 4096 x 4096 x 1024, 80 / 95 %: 190 / 52 and
// 69 / 44, 8 x (1000 x 1000 x 640), 70 %: 79 / 39; V = 2, 4096 x 4096 x 1984, 70 %: 156 / 73, 4096 x 4096 x 256, 90 %: 50 / 41; but
// 64 x (1024 x 256 x 256), V = 1, 80 %: 34 / 41, 64 x (2048 x 512 x 256), V = 2, 90 %: 41 / 97.
// Enqueues everything and returns true, or leaves the call alone.  VSPARSE_B200_SPMM_A=plan|laid-out.
template <typename TOut, int V, bool kCores> bool launch_spmm_laid_out(const SpmmParams &p, cudaStream_t s, DeviceInfo *d, bool forced, int *rc_out) {
    const char *e = std::getenv("VSPARSE_B200_SPMM_A");
    if (e && !std::strcmp(e, "plan")) return false;
    static int resident[kMaxDevices];
    auto kernel = pairspmm::spmm_pair_kernel<TOut, 1, false, true>;   // V is the layout's business
    const int capacity = pair_capacity(kernel, pairspmm::kPreparedThreads, resident, d);
    const int64_t M = (int64_t)p.m_vec * V;
    const int m_tiles = (int)((M + pairspmm::kTileM - 1) / pairspmm::kTileM), row_tiles = (int)((M + 127) / 128);
    const int Kp = (p.K + 63) / 64 * 64, k_blocks = Kp / 64, batch_a = p.batch > 1 && p.stride_values ? p.batch : 1;
    const int64_t row_items = (int64_t)p.batch * m_tiles, a_bytes = (int64_t)batch_a * row_tiles * 128 * Kp * 2;
    if (capacity < 0 || !spmm_pair_takes(p.N, V, row_items, d) || a_bytes > (128ll << 20)) return false;
    // Widths that are no multiple of 64: where there is work for the tiles, six blocks of 64 columns and not, by the count or its bound,
    // under 5 % of the vectors (68 x (3960 x 66 x 1128), V = 1 218 us on
    // single CTAs, 312 laid out; 49 x (160 x 1166 x 336), V = 1, 96 % 26 and 32)
    if (!e && p.N % 64 != 0 && (k_blocks < 6 || (p.stride_values > 0 && (double)(p.stride_values / V) < 0.05 * p.m_vec * p.K))) return false;
    const int tn = spmm_pair_width(p.N, row_items, capacity), n_tiles = (p.N + tn - 1) / tn;
    const int64_t items = row_items * n_tiles;
    if (items * k_blocks > 0x7fffffffll) return false;
    if (!e) {
        const double waves = (double)((items + capacity - 1) / capacity);
        if (waves * k_blocks * (V == 1 ? 1.1 : 0.4) < 0.67e-6 * (double)a_bytes + 3.0) return false;
    }
    SpmmCosts c = kGatherCosts;
    if constexpr (kCores) c = cores_costs_of(p, V, items, d->sm_count / 2, d);
    const double stages = (double)m_tiles * k_blocks;
    const int64_t min_vectors = forced ? 0 : (int64_t)std::max(0.0, std::ceil((stages * c.dense_per_stage - (double)p.m_vec * c.gather_per_row) / (c.gather_per_entry - c.dense_per_entry)));
    const int checks = (int)std::min<int64_t>((int64_t)batch_a * p.m_vec, 8 * d->sm_count);
    const int64_t header = ((4 + checks) * 4 + 255) / 256 * 256;
    CUtensorMap map_a, map_b, map_b2, map_out;
    if (make_tile_map(&map_b, p.rhs, false, (uint64_t)p.K, (uint64_t)p.N, (uint64_t)p.batch, (uint64_t)p.stride_rhs, 64, 64) != VS_OK ||
        (p.N % 64 == 0 && make_blocked_map(&map_b2, p.rhs, (uint64_t)p.K, (uint64_t)p.N, (uint64_t)p.batch, (uint64_t)p.stride_rhs, 2) != VS_OK) ||
        make_tile_map(&map_out, p.out, sizeof(TOut) == 4, (uint64_t)M, (uint64_t)p.N, (uint64_t)p.batch, (uint64_t)p.stride_out, pairspmm::kStoreCols, 32) != VS_OK)
        return false;
    uint8_t *mem = nullptr;
    PlanScratch scratch;
    if (scratch.take(d, s, (size_t)(header + a_bytes), reinterpret_cast<void **>(&mem)) != VS_OK) return false;
    if (p.N % 64 != 0) map_b2 = map_b;
    if (make_packed_map(&map_a, mem + header, 64, 128, 1, (uint64_t)batch_a * row_tiles * k_blocks, 1) != VS_OK) return false;
    int32_t *verdict = reinterpret_cast<int32_t *>(mem);
    int rc = (int)launch_overlapped(densify::densify_kernel<V>, (unsigned)checks, densify::kPrepThreads, 0, s, p, batch_a, Kp, min_vectors,
                                    reinterpret_cast<uint16_t *>(mem + header), verdict);
    if (rc == VS_OK) {
        TimedLaunch timed(s);
        SpmmParams q = p;
        q.m_vec = (int)M;
        rc = (int)launch_pairs(kernel, (unsigned)std::min<int64_t>(items, capacity), pairspmm::kPreparedThreads, (size_t)pairspmm::kSmemBytes, s, true, q, map_a,
                               batch_a, row_tiles, map_b, map_out, map_b2, tn, (const int32_t *)nullptr, (const uint2 *)nullptr, m_tiles, n_tiles,
                               k_blocks, d->status, verdict, checks, verdict + kPlanRedo);
    }
    if (rc == VS_OK) rc = launch_spmm_other<TOut, V, kCores>(p, s, d, verdict, checks);
    *rc_out = rc;
    return true;
}

template <typename TOut, int V, bool kCores> int launch_spmm_tc(const SpmmParams &p, cudaStream_t s) {
    DeviceInfo *d;
    int rc = device_info(&d);
    if (rc != VS_OK) return rc;
    const SpmmMode mode = spmm_mode();
    constexpr SpmmCosts cost = kCores ? cores_costs(V) : kGatherCosts;
    const bool direct = mode == SpmmMode::kDirect;
    int split = 1;
    if ((direct || mode == SpmmMode::kAuto) && spmm_direct_chosen(p, V, kCores, direct, d, &split) &&
        launch_spmm_direct<TOut, V, kCores>(p, s, d, cost, direct, split, &rc))
        return rc;
    if constexpr (V <= 2) {
        if (!t_no_scratch && mode != SpmmMode::kGather && p.K > 0 && (p.batch == 1 || (p.stride_rhs * 2) % 16 == 0) &&
            (p.batch == 1 || (p.stride_out * sizeof(TOut)) % 16 == 0) && launch_spmm_laid_out<TOut, V, kCores>(p, s, d, mode == SpmmMode::kDense, &rc))
            return rc;
    }
    const int k_blocks = (p.K + densespmm::kBlockK - 1) / densespmm::kBlockK;
    const int m_tiles = (p.m_vec * V + densespmm::kTileM - 1) / densespmm::kTileM;
    const int n_tiles = (p.N + densespmm::kTileN - 1) / densespmm::kTileN;
    const int groups = m_tiles * (densespmm::kTileM / densespmm::kGroupRows);
    const int plan_blocks = k_blocks * (densespmm::kBlockK / densespmm::kPlanCols);
    const int rows_per_group = densespmm::kGroupRows / V;
    int64_t capacity = 0, offsets_bytes = 0;
    const int64_t plan_bytes = spmm_plan_bytes(p.m_vec, V, p.K, p.batch, p.stride_values, &capacity, &offsets_bytes);
    const int checks = spmm_plan_checks(p.m_vec);
    const size_t plan_words = (size_t)(2 * plan_blocks + rows_per_group + 1), check_words = (size_t)densespmm::kPlanWarps * plan_blocks;
    const size_t plan_smem = (plan_words > check_words ? plan_words : check_words) * 4;
    const bool dense_ok = !t_no_scratch && mode != SpmmMode::kGather && p.K > 0 && p.m_vec > 0 && p.N % 8 == 0 && plan_bytes <= kMaxPlanBytes &&
                          plan_smem <= 40 * 1024 && (p.batch == 1 || (p.stride_rhs * 2) % 16 == 0) &&
                          (p.batch == 1 || (p.stride_out * sizeof(TOut)) % 16 == 0) && aligned16(p.rhs) && aligned16(p.out);
    if (!dense_ok) return launch_spmm_other<TOut, V, kCores>(p, s, d, nullptr, 0);

    constexpr bool kOutF32 = sizeof(TOut) == 4;
    CUtensorMap map, map_out;
    if (make_tile_map(&map, p.rhs, false, (uint64_t)p.K, (uint64_t)p.N, (uint64_t)p.batch, (uint64_t)p.stride_rhs, 64, 64) != VS_OK ||
        make_tile_map(&map_out, p.out, kOutF32, (uint64_t)p.m_vec * V, (uint64_t)p.N, (uint64_t)p.batch,
                      (uint64_t)p.stride_out, densespmm::kStoreCols, 32) != VS_OK)
        return launch_spmm_other<TOut, V, kCores>(p, s, d, nullptr, 0);
    CUtensorMap map_b4 = map;
    const int use_b4 = (p.N % 64 == 0 && make_blocked_map(&map_b4, p.rhs, (uint64_t)p.K, (uint64_t)p.N, (uint64_t)p.batch,
                                                          (uint64_t)p.stride_rhs, densespmm::kTileN / 64) == VS_OK) ? 1 : 0;
    auto kernel = densespmm::spmm_dense_kernel<TOut, V, false>;
    static DeviceBits smem_set;
    rc = set_smem_once(kernel, densespmm::kSmemBytes, smem_set);
    if (rc != VS_OK) return rc;
    uint8_t *plan = nullptr;
    PlanScratch scratch;
    if (scratch.take(d, s, (size_t)plan_bytes, reinterpret_cast<void **>(&plan)) != VS_OK)
        return launch_spmm_other<TOut, V, kCores>(p, s, d, nullptr, 0);
    int32_t *flag = reinterpret_cast<int32_t *>(plan);
    const int64_t header_bytes = spmm_plan_header_bytes(checks);
    int32_t *blk_offsets = reinterpret_cast<int32_t *>(plan + header_bytes);
    uint2 *blk_entries = reinterpret_cast<uint2 *>(plan + header_bytes + offsets_bytes);
    const int force_dense = mode == SpmmMode::kDense ? 1 : 0;
    SpmmCosts planned = cost;
    if constexpr (kCores) {
        const bool pairs = (use_b4 || p.N % 64 != 0) && spmm_pair_takes(p.N, V, (int64_t)p.batch * m_tiles, d, true);
        const int tn = spmm_pair_width(p.N, (int64_t)p.batch * m_tiles, d->sm_count / 2);
        const int64_t widths = pairs ? (p.N + tn - 1) / tn : n_tiles;
        planned = cores_costs_of(p, V, (int64_t)p.batch * m_tiles * widths, pairs ? d->sm_count / 2 : d->sm_count, d);
    }
    // a dependent launch as well: in a stream of calls the plan kernel queues up behind the previous call's last kernel
    rc = (int)launch_overlapped(densespmm::dense_plan_kernel<false>, (unsigned)(groups + checks), densespmm::kPlanThreads, plan_smem, s,
                                p.row_offsets, p.col_indices, (const int32_t *)nullptr, 0, p.m_vec, p.K, groups, rows_per_group,
                                plan_blocks, blk_offsets, blk_entries, capacity, force_dense, planned.dense_per_stage,
                                planned.gather_per_row, planned.gather_per_entry, planned.dense_per_entry, flag);
    if (rc != VS_OK) return rc;
    const int64_t items = (int64_t)p.batch * n_tiles * m_tiles;
    const unsigned grid = (unsigned)(items < d->sm_count ? items : d->sm_count);   // one persistent CTA per SM
    rc = (int)cudaGetLastError();
    if (rc == VS_OK) {
        int rc_pair = VS_OK;
        if ((use_b4 || p.N % 64 != 0) && spmm_pair_takes(p.N, V, (int64_t)p.batch * m_tiles, d, true) &&
            launch_spmm_pair<TOut, V, false>(p, s, d, map, map_out, map_b4, blk_offsets, blk_entries, m_tiles, k_blocks, flag, checks, flag + kPlanRedo, &rc_pair))
            rc = rc_pair;
        else
            rc = (int)launch_overlapped(kernel, grid, densespmm::kThreads, densespmm::kSmemBytes, s, p, map, map_out, map_b4, use_b4,
                                        blk_offsets, blk_entries, m_tiles, n_tiles, k_blocks, d->status, flag, checks, flag + kPlanRedo,
                                        densespmm::Second<false>());
    }
    if (rc == VS_OK) rc = launch_spmm_other<TOut, V, kCores>(p, s, d, flag, checks);
    return rc;
}

template <typename TOut> int spmm_tc_by_v(int V, const SpmmParams &p, cudaStream_t s) {
    switch (V) {
        case 2: return launch_spmm_tc<TOut, 2, false>(p, s);
        case 4: return launch_spmm_tc<TOut, 4, false>(p, s);
        case 8: return launch_spmm_tc<TOut, 8, false>(p, s);
    }
    return VS_ERR_VEC_LENGTH;
}
// cudaSpmm with fp16 operands and results.  The results are rounded to fp16 (2^-11 of their size), so the fp32 sums may be taken
// in any order and on the tensor cores, whose products of fp16 values are exact and whose sums are fp32 too; what the densified
// product cannot do (repeated columns, non-finite values, few nonzeros) stays with the CUDA-core kernel.  fp32 results keep it
// throughout: there the order of the sums shows.  VSPARSE_B200_SPMM=gather forces the CUDA-core kernel.
// The workspace of vs_set_workspace is the tensor path's: a thread may make cuda* calls beside those, on streams of their own, so
// while one is set these take the forms without scratch.
int spmm_cores_by_v(int V, const SpmmParams &p, cudaStream_t s) {
    NoScratchScope scope(t_ws_set);
    switch (V) {
        case 1: return launch_spmm_tc<__half, 1, true>(p, s);
        case 2: return launch_spmm_tc<__half, 2, true>(p, s);
        case 4: return launch_spmm_tc<__half, 4, true>(p, s);
        case 8: return launch_spmm_tc<__half, 8, true>(p, s);
    }
    return VS_ERR_VEC_LENGTH;
}

// ---- fp32 SpMM from bf16 parts ------------------------------------------------------------------------------
template <int V, int kChunks> int launch_spmm_f32_standby(const SpmmParams &p, cudaStream_t s, DeviceInfo *d, const int32_t *verdict, int checks, int few) {
    const int64_t blocks = ((int64_t)p.m_vec * (p.N / (4 * kChunks)) * p.batch + kCcThreads - 1) / kCcThreads, cap = (int64_t)d->sm_count * 8;
    auto kernel = spmm_cc_slabs(p, kChunks) ? spmm_cc_standby_kernel<float, float, V, kChunks, true> : spmm_cc_standby_kernel<float, float, V, kChunks>;
    return (int)launch_overlapped(kernel, (unsigned)(blocks < cap ? blocks : cap), kCcThreads, 0, s, p, verdict, checks, few);
}
// Tiles, scratch and estimated time of the split product of p's matrix with N columns in `batch` problems.
struct SplitSizes {
    int batch_a, batch_b, Kp, Np, k_blocks, m_tiles, tn, n_tiles, row_tiles, slabs;
    int64_t row_items, a_elems, b_elems;
    double us;
};
SplitSizes split_sizes(const SpmmParams &p, int V, int N, int batch, int resident) {
    SplitSizes z;
    const int64_t M = (int64_t)p.m_vec * V;
    z.batch_a = batch > 1 && (p.stride_values || p.batch == 1) ? batch : 1;
    z.batch_b = batch > 1 && (p.stride_rhs || p.batch == 1) ? batch : 1;
    z.Kp = (p.K + 63) / 64 * 64;
    z.Np = (N + 63) / 64 * 64;
    z.k_blocks = z.Kp / 64;
    z.m_tiles = (int)((M + splitspmm::kTileM - 1) / splitspmm::kTileM);
    z.row_items = (int64_t)batch * z.m_tiles;
    const int64_t wide = (N + 255) / 256, narrow = (N + 127) / 128;
    auto waves = [&](int64_t items) { return (double)((items + resident - 1) / resident); };
    const double t_wide = 2.1 * waves(z.row_items * wide), t_narrow = 1.1 * waves(z.row_items * narrow);
    z.tn = t_narrow < t_wide ? 128 : 256;
    z.n_tiles = (int)(z.tn == 256 ? wide : narrow);
    z.row_tiles = (int)((M + 127) / 128);
    z.slabs = z.Np / 64;
    z.a_elems = (int64_t)z.batch_a * z.row_tiles * 128 * z.Kp;
    z.b_elems = (int64_t)z.batch_b * z.Kp * z.Np;
    z.us = z.k_blocks * std::min(t_wide, t_narrow) + (double)(6 * z.a_elems + 10 * z.b_elems) / 4.6e6 + 15.0;
    return z;
}
// Leaves *taken false where the call is not one for it.
template <int V> int launch_spmm_split(const SpmmParams &p, int64_t vectors, cudaStream_t s, bool forced, DeviceInfo *d, bool *taken) {
    static int resident[kMaxDevices];   // 0 = not asked yet, -1 = the kernel cannot run here
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return VS_OK;
    if (resident[dev] == 0) {
        const bool fits = set_smem(splitspmm::spmm_split_kernel<256>, splitspmm::kSmemBytes) == VS_OK && set_smem(splitspmm::spmm_split_kernel<128>, splitspmm::kSmemBytes) == VS_OK;
        const int n = fits ? max_resident_pairs(splitspmm::spmm_split_kernel<256>, splitspmm::kThreads, splitspmm::kSmemBytes, d) : 0;
        resident[dev] = n > 0 ? n : -1;
    }
    if (resident[dev] < 0) return VS_OK;
    const int64_t M = (int64_t)p.m_vec * V;
    const SpmmParams whole = whole_call(p);
    const SplitSizes z = split_sizes(p, V, p.N, p.batch, resident[dev]), zw = split_sizes(p, V, whole.N, whole.batch, resident[dev]);
    splitspmm::PrepParams q;
    q.batch_a = z.batch_a; q.batch_b = z.batch_b; q.Kp = z.Kp; q.Np = z.Np;
    const int k_blocks = z.k_blocks, m_tiles = z.m_tiles, tn = z.tn, n_tiles = z.n_tiles, row_tiles = z.row_tiles, slabs = z.slabs;
    const int64_t row_items = z.row_items, a_elems = z.a_elems, b_elems = z.b_elems;
    // us: 64 columns of an item by a pair, the preparation at 4.6 TB/s, launches (180 estimated, 165 to 180 measured at 4096 x 4096 x 1024; 36
    // and 36 at 1024 cubed; 25 and 25 at 512 cubed); against the CUDA-core kernel's time per vector and column (611 us
    // at V = 1, 305 at V = 2, 301 at V = 4, 258 at V = 8 for 4096 x 4096 x 1024, 80 % sparse), or, where it takes the call otherwise, against that of the
    // kernel that stages tiles of B (also where few vector-rows then go to spmm_cc_few_kernel, whose time is not fitted): per wave a start, the tiles, the entries of a vector-row (V = 8, 2048 x 4096 x 1024, 50 / 65 / 80 %
    // sparse: that kernel 228 / 165 / 103, this one 114 / 111 / 106; V = 1, 1024 x 1024 x 512: 54 / 41 / 29 and 38 / 37 / 36).  Below kMinDensity that kernel keeps every
    // dense width, so that column shards of usual matrices (90 %, at V = 4 80 % sparse) have the bits of the whole product; by cost the line would lie
    // at 0.047 (V = 1) and 0.097 (V = 4) for 4096 x 4096 x 8192.
    constexpr double kCoresPs = V <= 2 ? 0.18 : V == 4 ? 0.35 : 0.6, kTileEntryUs = V == 1 ? 0.043 : V == 2 ? 0.047 : V == 4 ? 0.061 : 0.102, kMinDensity = V == 1 ? 0.102 : V == 2 ? 0.11 : V == 4 ? 0.205 : 0.13;
    // Nor does it take a matrix whose rows are about as short on average as those that the CUDA-core kernel computes behind it.
    q.few = forced ? 0 : splitspmm::few_entries(p.K);
    double line = 1.1 * zw.us / (kCoresPs * 1e-6 * whole.N * whole.batch);
    if (spmm_cc_tiles_chosen(V, whole, d))
        line = p.m_vec * (1.1 * zw.us / (double)((spmm_cc_tile_ctas(whole) + d->sm_count - 1) / d->sm_count) - 6.0 - 0.002 * p.K) / kTileEntryUs;
    q.min_vectors = forced ? 0 : (int64_t)std::max({line, kMinDensity * p.m_vec * (double)p.K, 1.125 * q.few * p.m_vec});
    // A caller that does not say how many values there are: large products only, where two kernels that may return at once cost little.
    if (!forced && (vectors < q.min_vectors || whole.N < 256 || (p.stride_values == 0 && zw.us < 100.0))) return VS_OK;
    const int64_t units = (int64_t)q.batch_a * p.m_vec + b_elems / (8 * splitspmm::kPrepThreads) + 1;
    const int checks = (int)std::min<int64_t>(units, 8 * d->sm_count);
    const int64_t header = ((4 + checks) * 4 + 255) / 256 * 256, a_bytes = (a_elems * 6 + 255) / 256 * 256, bytes = header + a_bytes + b_elems * 6;
    if (std::max(bytes, (zw.a_elems + zw.b_elems) * 6) > kMaxPlanBytes || zw.row_items * zw.n_tiles * k_blocks > 0x7fffffffll) return VS_OK;
    CUtensorMap map_out;
    if (make_tile_map(&map_out, p.out, true, (uint64_t)M, (uint64_t)p.N, (uint64_t)p.batch, (uint64_t)p.stride_out, splitspmm::kStoreCols, 32, false) != VS_OK) return VS_OK;
    uint8_t *mem = nullptr;
    PlanScratch scratch;
    if (scratch.take(d, s, (size_t)bytes, reinterpret_cast<void **>(&mem)) != VS_OK) return VS_OK;
    q.verdict = reinterpret_cast<int32_t *>(mem);
    q.a = reinterpret_cast<uint16_t *>(mem + header);
    q.b = reinterpret_cast<uint16_t *>(mem + header + a_bytes);
    CUtensorMap map_a, map_b;
    if (make_packed_map(&map_a, q.a, 64, 128, 3, (uint64_t)q.batch_a * row_tiles * k_blocks, 1) != VS_OK ||
        make_packed_map(&map_b, q.b, 64, 64, 3, (uint64_t)q.batch_b * k_blocks * slabs, (uint32_t)(tn / 128)) != VS_OK)
        return VS_OK;
    *taken = true;
    int rc = (int)launch_overlapped(splitspmm::spmm_split_prepare<V>, (unsigned)checks, splitspmm::kPrepThreads, 0, s, p, q);
    if (rc != VS_OK) return rc;
    const int64_t items = row_items * n_tiles;
    {
        TimedLaunch timed(s);
        rc = (int)launch_pairs(tn == 256 ? splitspmm::spmm_split_kernel<256> : splitspmm::spmm_split_kernel<128>, (unsigned)std::min<int64_t>(items, resident[dev]), splitspmm::kThreads, (size_t)splitspmm::kSmemBytes, s, true,
                               p, V, map_a, map_b, map_out, q.batch_a, q.batch_b, m_tiles, n_tiles, k_blocks, row_tiles, slabs, d->status, q.verdict, checks, q.verdict + kPlanRedo);
    }
    if (rc != VS_OK) return rc;
    const int chunks = spmm_cc_chunks(4 * V, 4, p.N);
    if constexpr (V <= 4) {
        if (chunks == 4) return launch_spmm_f32_standby<V, 4>(p, s, d, q.verdict, checks, q.few);
    }
    if (chunks == 2) return launch_spmm_f32_standby<V, 2>(p, s, d, q.verdict, checks, q.few);
    return launch_spmm_f32_standby<V, 1>(p, s, d, q.verdict, checks, q.few);
}
// VSPARSE_B200_SPMM_F32=cores|split chooses one, for all rows; VSPARSE_B200_SPMM_CC, a choice among the CUDA-core kernels, chooses those.
int spmm_split(int V, const SpmmParams &p, cudaStream_t s, bool *taken) {
    const char *e = std::getenv("VSPARSE_B200_SPMM_F32");
    const bool forced = e && !std::strcmp(e, "split");
    if ((e && !std::strcmp(e, "cores")) || (!forced && std::getenv("VSPARSE_B200_SPMM_CC")) || t_no_scratch || t_ws_set || p.K < 1) return VS_OK;
    DeviceInfo *d = nullptr;
    const int rc = device_info(&d);
    if (rc != VS_OK) return rc;
    const int64_t vectors = p.stride_values > 0 ? p.stride_values / V : (int64_t)p.m_vec * p.K;
    switch (V) {
        case 1: return launch_spmm_split<1>(p, vectors, s, forced, d, taken);
        case 2: return launch_spmm_split<2>(p, vectors, s, forced, d, taken);
        case 4: return launch_spmm_split<4>(p, vectors, s, forced, d, taken);
        case 8: return launch_spmm_split<8>(p, vectors, s, forced, d, taken);
    }
    return VS_OK;
}

// ---- SDDMM dispatch ---------------------------------------------------------------------------------------
// CUDA-core SDDMM: a group of lanes per vector-row with the lhs rows in registers when the contraction length fits
// 32 chunks of 16 bytes (k <= 256 in fp16, 128 in fp32), a group of eight lanes per mask entry otherwise.
// VSPARSE_B200_SDDMM_CC=entry keeps the latter.
template <typename TIn, typename TOut, int V, int L> int launch_sddmm_cc_row(const SddmmParams &p, cudaStream_t s) {
    // groups of lanes that share a vector-row: until there are 16 warps per SM, with eight entries each or more
    DeviceInfo *d = nullptr;
    const int rc = device_info(&d);
    if (rc != VS_OK) return rc;
    int pieces = 1;
    while ((int64_t)p.m_vec * p.batch * pieces * L < 16ll * 32 * d->sm_count && p.nnz_vec / p.m_vec >= 16 * pieces && pieces < 64) pieces *= 2;
    const int64_t blocks = ((int64_t)p.m_vec * pieces * L + kCcThreads - 1) / kCcThreads;
    if (blocks > 0x7fffffffll) return VS_ERR_SHAPE;
    dim3 grid((unsigned)blocks, (unsigned)p.batch, 1);
    sddmm_cc_row_kernel<TIn, TOut, V, L><<<grid, kCcThreads, 0, s>>>(p, pieces);
    return (int)cudaGetLastError();
}
template <typename TIn, typename TOut, int V> int launch_sddmm_cc(const SddmmParams &p, cudaStream_t s) {
    const int chunks = p.k / Chunk<TIn>::kElems;
    const char *e = std::getenv("VSPARSE_B200_SDDMM_CC");
    if (chunks >= 1 && chunks <= 32 && p.m_vec > 0 && !(e && !std::strcmp(e, "entry"))) {
        if (chunks > 16) return launch_sddmm_cc_row<TIn, TOut, V, 32>(p, s);
        if (chunks > 8) return launch_sddmm_cc_row<TIn, TOut, V, 16>(p, s);
        return launch_sddmm_cc_row<TIn, TOut, V, 8>(p, s);
    }
    const int64_t blocks = ((int64_t)p.nnz_vec * 8 + kCcThreads - 1) / kCcThreads;
    if (blocks > 0x7fffffffll) return VS_ERR_SHAPE;
    dim3 grid((unsigned)blocks, (unsigned)p.batch, 1);
    sddmm_cc_kernel<TIn, TOut, V><<<grid, kCcThreads, 0, s>>>(p);
    return (int)cudaGetLastError();
}

template <typename TIn, typename TOut> int sddmm_cc_by_v(int V, const SddmmParams &p, cudaStream_t s) {
    switch (V) {
        case 1: return launch_sddmm_cc<TIn, TOut, 1>(p, s);
        case 2: return launch_sddmm_cc<TIn, TOut, 2>(p, s);
        case 4: return launch_sddmm_cc<TIn, TOut, 4>(p, s);
        case 8: return launch_sddmm_cc<TIn, TOut, 8>(p, s);
    }
    return VS_ERR_VEC_LENGTH;
}

// Software (cp.async) gather: works for any batch stride.
template <typename TOut, int V> int launch_sddmm_tc_cpasync(const SddmmParams &p, cudaStream_t s, DeviceInfo *d) {
    auto kernel = tcsddmm::sddmm_tc_kernel<TOut, V>;
    static DeviceBits smem_set;
    int rc = set_smem_once(kernel, tcsddmm::kSmemBytes, smem_set);
    if (rc != VS_OK) return rc;
    const int64_t items = (int64_t)p.batch * p.m_vec;
    const int64_t cap = 2ll * d->sm_count;
    const unsigned grid = (unsigned)(items < cap ? items : cap);
    kernel<<<grid, tcsddmm::kThreads, tcsddmm::kSmemBytes, s>>>(p, d->status);
    return (int)cudaGetLastError();
}

// TMA row gather: lhs and rhs of all batch entries must each be addressable as one matrix of k-wide rows, i.e.
// their batch strides are multiples of k (or zero / a single entry).
template <typename TOut, int V> int launch_sddmm_gather(const SddmmParams &p, cudaStream_t s, DeviceInfo *d) {
    static const bool force_cpasync = []() {
        const char *e = std::getenv("VSPARSE_B200_GATHER");
        return e && !std::strcmp(e, "cpasync");
    }();
    const int64_t m = (int64_t)p.m_vec * V;
    const bool one_r = p.batch == 1 || p.stride_rhs == 0, one_l = p.batch == 1 || p.stride_lhs == 0;
    const int64_t rpb_r = one_r ? 0 : p.stride_rhs / p.k, rpb_l = one_l ? 0 : p.stride_lhs / p.k;
    const int64_t rows_r = (one_r ? 0 : (int64_t)(p.batch - 1) * rpb_r) + p.n;
    const int64_t rows_l = (one_l ? 0 : (int64_t)(p.batch - 1) * rpb_l) + m;
    const bool tma_ok = !force_cpasync && p.n > 0 && (one_r || p.stride_rhs % p.k == 0) && (one_l || p.stride_lhs % p.k == 0) &&
                        rows_r < 0x7fffffffll && rows_l < 0x7fffffffll;
    if (!tma_ok) return launch_sddmm_tc_cpasync<TOut, V>(p, s, d);
    CUtensorMap map_r, map_l;
    if (make_gather_map(&map_r, p.rhs, (uint64_t)rows_r, (uint64_t)p.k) != VS_OK ||
        make_gather_map(&map_l, p.lhs, (uint64_t)rows_l, (uint64_t)p.k) != VS_OK)
        return launch_sddmm_tc_cpasync<TOut, V>(p, s, d);
    auto kernel = tmasddmm::sddmm_tma_kernel<TOut, V>;
    static DeviceBits smem_set;
    int rc = set_smem_once(kernel, tmasddmm::kSmemBytes, smem_set);
    if (rc != VS_OK) return rc;
    const int64_t items = (int64_t)p.batch * p.m_vec;
    const int64_t cap = (int64_t)tmasddmm::kCtasPerSm * d->sm_count;
    const unsigned grid = (unsigned)(items < cap ? items : cap);
    kernel<<<grid, tmasddmm::kThreads, tmasddmm::kSmemBytes, s>>>(p, map_r, map_l, (int)rpb_r, (int)rows_r, (int)rpb_l,
                                                                  (int)rows_l, d->status);
    return (int)cudaGetLastError();
}

// The dense SDDMM by pairs of CTAs (sddmm_pair.cuh) serves masks of up to pairsddmm::kMaxPlanColumns columns whose
// outputs can be written with vector stores; VSPARSE_B200_SDDMM_PAIR=0 keeps the single-CTA kernel.
inline bool sddmm_pair_enabled() {
    const char *e = std::getenv("VSPARSE_B200_SDDMM_PAIR");
    return !(e && !std::strcmp(e, "0"));
}
// Scratch of the pair kernel's plan: words, entry order, a twins flag per CTA of the plan.
constexpr int kCellPlanCtas = 1024;
inline int sddmm_cell_plan_ctas(int m_vec) { return std::min((m_vec + pairsddmm::kPlanWarps - 1) / pairsddmm::kPlanWarps, kCellPlanCtas); }
int64_t sddmm_pair_plan_bytes(int m_vec, int n, int nnz_vec, int64_t *words_out, int64_t *order_out) {
    const int64_t words_bytes = ((int64_t)m_vec * ((n + 31) / 32) * 8 + 15) & ~15ll, order_bytes = ((int64_t)nnz_vec * 4 + 15) & ~15ll;
    if (words_out) *words_out = words_bytes;
    if (order_out) *order_out = order_bytes;
    return words_bytes + order_bytes + 4 * (int64_t)std::min(m_vec, kCellPlanCtas);
}
// Plan, multiplying kernel and the fix-up for repeated columns; false if this call or this device cannot take them
// (nothing has been enqueued then).
template <typename TOut, int V> bool launch_sddmm_pair(const SddmmParams &p, cudaStream_t s, DeviceInfo *d, int *rc_out) {
    static int resident[kMaxDevices];   // 0 = not asked yet, -1 = the kernels cannot run here
    auto kernel = pairsddmm::sddmm_pair_kernel<TOut, V>;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return false;
    if (resident[dev] == 0) {
        const int n = set_smem(kernel, pairsddmm::kSmemBytes) == VS_OK ? max_resident_pairs(kernel, pairsddmm::kThreads, pairsddmm::kSmemBytes, d) : 0;
        resident[dev] = n > 0 ? n : -1;
    }
    if (resident[dev] < 0) return false;
    int64_t words_bytes = 0, order_bytes = 0;
    const int64_t plan_bytes = sddmm_pair_plan_bytes(p.m_vec, p.n, p.nnz_vec, &words_bytes, &order_bytes);
    if (p.n > pairsddmm::kMaxPlanColumns || plan_bytes > kMaxPlanBytes || !aligned16(p.out) ||
        (p.batch > 1 && (p.stride_out * sizeof(TOut)) % 16 != 0))
        return false;
    CUtensorMap map_l, map_r;
    if (make_tile_map(&map_l, p.lhs, false, (uint64_t)p.m_vec * V, (uint64_t)p.k, (uint64_t)p.batch, (uint64_t)p.stride_lhs, 64,
                      pairsddmm::kCtaRows) != VS_OK ||
        make_tile_map(&map_r, p.rhs, false, (uint64_t)p.n, (uint64_t)p.k, (uint64_t)p.batch, (uint64_t)p.stride_rhs, 64,
                      pairsddmm::kCtaRows) != VS_OK)
        return false;
    uint8_t *plan = nullptr;
    PlanScratch scratch;
    if (scratch.take(d, s, (size_t)plan_bytes, reinterpret_cast<void **>(&plan)) != VS_OK) return false;
    uint2 *words = reinterpret_cast<uint2 *>(plan);
    int32_t *order = reinterpret_cast<int32_t *>(plan + words_bytes);
    int32_t *twins = reinterpret_cast<int32_t *>(plan + words_bytes + order_bytes);
    // a CTA per vector-row where the rows are long, a warp, whose 32 entries take 0.3 us, where they are short: 53 skewed rows of 960 entries 22 us / 5.5, 252 of
    // 229 9.0 / 4.4; 256 of 51 4.5 with a warp
    const bool shared_rows = (int64_t)p.nnz_vec > 192ll * p.m_vec;
    const int plan_ctas = shared_rows ? std::min(p.m_vec, kCellPlanCtas) : sddmm_cell_plan_ctas(p.m_vec);
    int rc = (int)launch_overlapped(shared_rows ? pairsddmm::sddmm_cell_plan_kernel<pairsddmm::kPlanWarps> : pairsddmm::sddmm_cell_plan_kernel<1>, (unsigned)plan_ctas, pairsddmm::kPlanThreads,
                                    (size_t)(shared_rows ? 1 : pairsddmm::kPlanWarps) * ((p.n + 31) / 32) * 8, s, p.row_offsets, p.col_indices, p.m_vec, p.n, p.nnz_vec, words, order, twins);
    if (rc == VS_OK) {
        const int m_tiles = (p.m_vec * V + pairsddmm::kTile - 1) / pairsddmm::kTile;
        const int n_tiles = (p.n + pairsddmm::kTile - 1) / pairsddmm::kTile;
        const int64_t items = (int64_t)p.batch * n_tiles * m_tiles;
        const unsigned pairs = (unsigned)(items < resident[dev] ? items : resident[dev]);
        // rhs of a batch entry fits the resident slots (VSPARSE_B200_SDDMM_RESIDENT=0: stream both operands anyway)
        const char *res_env = std::getenv("VSPARSE_B200_SDDMM_RESIDENT");
        const int resident = (n_tiles * ((p.k + densesddmm::kBlockK - 1) / densesddmm::kBlockK) <= pairsddmm::kMaxResident && !(res_env && !std::strcmp(res_env, "0"))) ? 1 : 0;
        TimedLaunch timed(s);
        rc = (int)launch_pairs(kernel, pairs, pairsddmm::kThreads, (size_t)pairsddmm::kSmemBytes, s, true, p, map_l, map_r, (const uint2 *)words, (const int32_t *)order,
                               m_tiles, n_tiles, resident, d->status);
    }
    if (rc == VS_OK)
        rc = (int)launch_overlapped(pairsddmm::sddmm_twin_kernel<TOut, V>, (unsigned)std::min<int64_t>((p.nnz_vec + pairsddmm::kTwinThreads - 1) / pairsddmm::kTwinThreads, d->sm_count),
                                    pairsddmm::kTwinThreads, 0, s, p, (const uint2 *)words, (const int32_t *)order, (const int32_t *)twins, plan_ctas);
    *rc_out = rc;
    return true;
}

// Small problems in one kernel (sddmm_direct.cuh); false if this call or this device cannot take it.
template <typename TOut, int V> bool launch_sddmm_direct(const SddmmParams &p, cudaStream_t s, DeviceInfo *d, int *rc_out) {
    const int m_tiles = (int)(((int64_t)p.m_vec * V + directsddmm::kTileM - 1) / directsddmm::kTileM);
    // 64-column tiles while 128-column ones would leave SMs without a tile
    const int tn = (int64_t)p.batch * m_tiles * ((p.n + 127) / 128) >= d->sm_count ? 128 : 64;
    const int n_tiles = (p.n + tn - 1) / tn;
    const int64_t tiles = (int64_t)p.batch * m_tiles * n_tiles;
    if (tiles > 0x7fffffffll || p.n <= 0 || p.k <= 0 || p.k % 8 != 0) return false;
    CUtensorMap map_l, map_r;
    static DeviceBits smem_set;
    auto kernel = directsddmm::sddmm_direct_kernel<TOut, V>;
    if (make_tile_map(&map_l, p.lhs, false, (uint64_t)p.m_vec * V, (uint64_t)p.k, (uint64_t)p.batch, (uint64_t)p.stride_lhs, 64,
                      directsddmm::kTileM) != VS_OK ||
        make_tile_map(&map_r, p.rhs, false, (uint64_t)p.n, (uint64_t)p.k, (uint64_t)p.batch, (uint64_t)p.stride_rhs, 64, (uint32_t)tn) != VS_OK ||
        set_smem_once(kernel, directsddmm::kSmemBytes, smem_set) != VS_OK)
        return false;
    *rc_out = (int)launch_overlapped(kernel, (unsigned)tiles, directsddmm::kThreads, directsddmm::kSmemBytes, s, p, map_l, map_r, tn, m_tiles,
                                     n_tiles, d->status);
    return true;
}
// Time each form of a sampled product takes, us.  Direct: waves of 128 x 128 tiles at two per SM, each paying for its contraction (three times as much per
// block once both CTAs of an SM draw on L2) and for looking at every entry of its rows.  Dense: the launches, waves of 256 x 256 tiles, each the longer of its
// contraction and its sampling; the single-CTA kernel of wide masks takes 1.4 times as long.  Gather: rounds of a vector-row per CTA at two per SM, each entry
// by itself for every 64 contraction elements.  Fitted to 87 sizes (V = 2 to 8, 64 to 4096 rows, 64 to 4608 columns, k = 64 to 1984, 50 to 98 % sparse, batches of
// up to 256): 0.8 to 1.25 times the measured time in nine of ten, and the choice among the three within 1.4 % of the best in the mean.  (The costs
// before counted an entry of the gather kernel once whatever k, which sent 3480 x 4231, k = 960, V = 8, 56 % there: 232 us instead of 32; 4 x (376 x 2817),
// k = 1344, V = 4: 303 instead of 25.)
struct SddmmTimes {
    double direct, dense, gather;
};
SddmmTimes sddmm_times(const SddmmParams &p, int V, int sm_count) {
    const double sms = sm_count, k_blocks = std::ceil(p.k / 64.0), per_row = (double)p.nnz_vec / std::max(p.m_vec, 1), m = (double)p.m_vec * V;
    const double tiles = std::ceil(m / 128.0) * std::ceil(p.n / 128.0) * p.batch, items = std::max(1.0, std::ceil(m / 256.0) * std::ceil(p.n / 256.0) * p.batch);
    const double shared = std::min(1.0, std::max(0.0, tiles / sms - 1.0)), pairs = sms / 2;
    SddmmTimes t;
    t.direct = 2.0 + std::max(1.0, tiles / (2.0 * sms)) * (1.6 + (0.24 + 0.5 * shared) * k_blocks + (0.11 + 0.035 * shared) * std::min((double)p.m_vec, 128.0 / V) * per_row / 256.0);
    const double waves = items > 4.0 * pairs ? items / pairs : std::ceil(items / pairs);
    t.dense = 9.2 + waves * std::max(0.4 * k_blocks, 0.98 + 0.52e-3 * (double)p.nnz_vec * p.batch / items) * (p.n > pairsddmm::kMaxPlanColumns || !sddmm_pair_enabled() ? 1.4 : 1.0);
    t.gather = 6.5 + std::max(1.0, (double)p.m_vec * p.batch / (2.0 * sms)) * (0.168 + 4.1e-3 * per_row) * k_blocks;
    return t;
}
// Which planned form runs (VSPARSE_B200_SDDMM = "dense" | "gather", read at every call, forces one).  The number of entries is an argument here, so the choice
// is made on the host.
bool sddmm_use_dense(const SddmmParams &p, int V, int sm_count) {
    const char *e = std::getenv("VSPARSE_B200_SDDMM");
    if (e && !std::strcmp(e, "dense")) return true;
    if (e && !std::strcmp(e, "gather")) return false;
    const SddmmTimes t = sddmm_times(p, V, sm_count);
    return t.dense < 1.25 * t.gather;   // where the estimates are close, the one that long rows hold up least
}
// Small sampled products go to the one-kernel form.  lhs 512 x 256, rhs 2048 x 256, V = 4: 17.0 -> 7.8 us; 2048 x 512 x 256, V = 8,
// 90 % sparse: one 11.1 -> 5.1, eight 14.4 -> 10.2, sixteen 18.9 -> 18.4.  VSPARSE_B200_SDDMM = "dense" and "gather" force those,
// "direct" this one.
bool sddmm_direct_wanted(const SddmmParams &p, int V, const DeviceInfo *d) {
    const char *e = std::getenv("VSPARSE_B200_SDDMM");
    if (e) return !std::strcmp(e, "direct");
    const SddmmTimes t = sddmm_times(p, V, d->sm_count);
    return 1.07 * t.direct < (sddmm_use_dense(p, V, d->sm_count) ? t.dense : t.gather);
}

template <typename TOut, int V> int launch_sddmm_tc(const SddmmParams &p, cudaStream_t s) {
    DeviceInfo *d;
    int rc = device_info(&d);
    if (rc != VS_OK) return rc;
    if (sddmm_direct_wanted(p, V, d) && launch_sddmm_direct<TOut, V>(p, s, d, &rc)) return rc;
    const int chunks = (p.n + densesddmm::kChunk - 1) / densesddmm::kChunk;
    int64_t offsets_bytes = 0;
    const int64_t plan_bytes = sddmm_plan_bytes(p.m_vec, p.n, p.nnz_vec, &offsets_bytes);
    const size_t plan_smem = (size_t)2 * chunks * 4;
    const bool dense_ok = !t_no_scratch && p.n > 0 && p.m_vec > 0 && p.nnz_vec > 0 && p.k >= densesddmm::kBlockK && plan_bytes <= kMaxPlanBytes &&
                          plan_smem <= 40 * 1024 && aligned16(p.lhs) && aligned16(p.rhs) &&
                          (p.batch == 1 || ((p.stride_lhs * 2) % 16 == 0 && (p.stride_rhs * 2) % 16 == 0)) &&
                          sddmm_use_dense(p, V, d->sm_count);
    if (!dense_ok) return launch_sddmm_gather<TOut, V>(p, s, d);
    if (sddmm_pair_enabled() && launch_sddmm_pair<TOut, V>(p, s, d, &rc)) return rc;
    CUtensorMap map_l, map_r;
    if (make_tile_map(&map_l, p.lhs, false, (uint64_t)p.m_vec * V, (uint64_t)p.k, (uint64_t)p.batch, (uint64_t)p.stride_lhs, 64,
                      densesddmm::kTileM) != VS_OK ||
        make_tile_map(&map_r, p.rhs, false, (uint64_t)p.n, (uint64_t)p.k, (uint64_t)p.batch, (uint64_t)p.stride_rhs, 64,
                      densesddmm::kTileN) != VS_OK)
        return launch_sddmm_gather<TOut, V>(p, s, d);
    auto kernel = densesddmm::sddmm_dense_kernel<TOut, V>;
    static DeviceBits smem_set;
    rc = set_smem_once(kernel, densesddmm::kSmemBytes, smem_set);
    if (rc != VS_OK) return rc;
    uint8_t *plan = nullptr;
    PlanScratch scratch;
    if (scratch.take(d, s, (size_t)plan_bytes, reinterpret_cast<void **>(&plan)) != VS_OK)
        return launch_sddmm_gather<TOut, V>(p, s, d);
    int32_t *chunk_offsets = reinterpret_cast<int32_t *>(plan);
    uint2 *chunk_entries = reinterpret_cast<uint2 *>(plan + offsets_bytes);
    densesddmm::sddmm_plan_kernel<<<p.m_vec, densesddmm::kPlanThreads, plan_smem, s>>>(p.row_offsets, p.col_indices, p.n, chunks,
                                                                                   p.nnz_vec, chunk_offsets, chunk_entries);
    const int m_tiles = (p.m_vec * V + densesddmm::kTileM - 1) / densesddmm::kTileM;
    const int n_tiles = (p.n + densesddmm::kTileN - 1) / densesddmm::kTileN;
    const int64_t items = (int64_t)p.batch * m_tiles * n_tiles;
    const unsigned grid = (unsigned)(items < d->sm_count ? items : d->sm_count);   // one persistent CTA per SM
    rc = (int)cudaGetLastError();
    if (rc != VS_OK) return rc;
    return (int)launch_overlapped(kernel, grid, densesddmm::kThreads, densesddmm::kSmemBytes, s, p, map_l, map_r, chunk_offsets,
                                  chunk_entries, m_tiles, n_tiles, chunks, d->status);
}

// cudaSddmm with fp16 results: on the tensor cores like cudaSpmm's (spmm_cores_by_v), any contraction length that is a
// multiple of 8 (the tiles' last block is filled up with zeros by TMA).  The CUDA-core kernel, a group of lanes per
// vector-row or mask entry, is slower by 1.1 to 19 times at V > 1 (64 x 64 to 4096 x 2048, 60 and 95 % sparse); it takes the
// strides that tensor maps cannot address, and what sddmm_cores_wanted names.
// 159 x 577, 115 entries per row, k = 200, V = 8, 16 of them: 65 -> 18.5 us.
//
// Where the tensor cores do not pay, for V <= 2, whose tiles sample one or two values per look-up.  One 128-byte line per entry
// is little to gather: V = 1, 4096 x 4096, k = 64, 80 / 95 / 98 % sparse 144 / 44 / 21 us against 170 / 75 / 51; V = 2 at 98 % 23 against 26.
// Past k = 256 the CUDA-core kernel takes single entries and is not held up by long rows: 303 x 982, k = 296, V = 1, 80 %
// sparse 10.4 against 22.3, up to some 100 MB of gathered rows (1024 x 1024, k = 512, 54 / 107 / 215 MB: 12.5 / 18.7 / 31.9 against 13.1 /
// 16.9 / 23).
bool sddmm_cores_wanted(const SddmmParams &p, int V) {
    if (V == 1) return p.k <= 64 || (p.k > 256 && 2.0 * p.k * p.nnz_vec * p.batch < 1e8);
    return V == 2 && p.k <= 64 && p.nnz_vec < 0.03 * p.m_vec * p.n;
}
// And where the mask is sparse: the tensor-core forms multiply every tile, the CUDA-core kernels read a row per entry.  Their time (us, fitted
// to 64 x 64 to 16384 x 16384, k = 64 to 1504, 60 to 99.9 % sparse: 0.85 to 1.2 times the measured one): a launch, the bytes of
// the gathered rows, and up to k = 256 the longest chain, a row's entries one behind the other; beyond, where a group of lanes has one
// entry, its k.  16384 x 16384, k = 128, V = 4, 99.9 % sparse 182 us on tiles and 6.5 here; 4096 x 4096, k = 256, V = 8, 99 % 18 and 7.
double sddmm_cores_time(const SddmmParams &p, int V) {
    const int v = V == 1 ? 0 : V == 2 ? 1 : V == 4 ? 2 : 3;
    const double gathered = (double)p.nnz_vec * p.k * p.batch;
    if (p.k <= 256) {
        constexpr double launch[4] = {2.1, 2.1, 2.1, 3.7}, rows[4] = {2.04e-7, 2.32e-7, 2.84e-7, 3.69e-7}, chain[4] = {0.071, 0.087, 0.093, 0.119};
        return launch[v] + rows[v] * gathered + chain[v] * p.nnz_vec / std::max(p.m_vec, 1);
    }
    constexpr double rows[4] = {2.27e-7, 3.66e-7, 4.90e-7, 8.99e-7}, chain[4] = {2.8e-3, 3.1e-3, 2.9e-3, 1.0e-2};
    return 2.5 + rows[v] * gathered + chain[v] * p.k;
}
template <int V> int launch_sddmm_cores(const SddmmParams &p, cudaStream_t s) {
    DeviceInfo *d;
    int rc = device_info(&d);
    if (rc != VS_OK) return rc;
    const char *e = std::getenv("VSPARSE_B200_SDDMM");
    const bool force_cores = e && !std::strcmp(e, "gather"), force_dense = e && !std::strcmp(e, "dense"), force_direct = e && !std::strcmp(e, "direct");
    const bool strides = p.batch == 1 || ((p.stride_lhs * 2) % 16 == 0 && (p.stride_rhs * 2) % 16 == 0);
    const bool by_rule = !force_dense && !force_direct && sddmm_cores_wanted(p, V);
    if (!force_cores && !by_rule && strides && p.n > 0 && p.m_vec > 0) {
        const SddmmTimes t = sddmm_times(p, V, d->sm_count);
        const bool pair_ok = !t_no_scratch && sddmm_pair_enabled() && p.n <= pairsddmm::kMaxPlanColumns;
        const bool pair = pair_ok && !force_direct && (force_dense || t.dense < t.direct);
        // The tile forms' estimates are up to 1.7 times too high where they are long; below, what the CUDA-core kernel is taken for is a clear gain.
        const double tiled = pair ? t.dense : t.direct;
        const bool sparse = !force_dense && !force_direct && sddmm_cores_time(p, V) + 1.2 < (tiled < 30.0 ? 1.0 : V == 1 ? 0.9 : 0.6) * tiled;
        if (!sparse && pair && launch_sddmm_pair<__half, V>(p, s, d, &rc)) return rc;
        if (!sparse && !force_dense && launch_sddmm_direct<__half, V>(p, s, d, &rc)) return rc;
    }
    return launch_sddmm_cc<__half, __half, V>(p, s);
}
int sddmm_cores_by_v(int V, const SddmmParams &p, cudaStream_t s) {
    NoScratchScope scope(t_ws_set);   // as in spmm_cores_by_v
    switch (V) {
        case 1: return launch_sddmm_cores<1>(p, s);
        case 2: return launch_sddmm_cores<2>(p, s);
        case 4: return launch_sddmm_cores<4>(p, s);
        case 8: return launch_sddmm_cores<8>(p, s);
    }
    return VS_ERR_VEC_LENGTH;
}

template <typename TOut> int sddmm_tc_by_v(int V, const SddmmParams &p, cudaStream_t s) {
    switch (V) {
        case 2: return launch_sddmm_tc<TOut, 2>(p, s);
        case 4: return launch_sddmm_tc<TOut, 4>(p, s);
        case 8: return launch_sddmm_tc<TOut, 8>(p, s);
    }
    return VS_ERR_VEC_LENGTH;
}

template <typename T> int softmax_by_v(int V, const SoftmaxParams &p, cudaStream_t s) {
    const int64_t blocks = ((int64_t)p.m_vec * 32 + kCcThreads - 1) / kCcThreads;
    dim3 grid((unsigned)blocks, (unsigned)p.batch, 1);
    switch (V) {
        case 1: softmax_cvse_kernel<T, 1><<<grid, kCcThreads, 0, s>>>(p); break;
        case 2: softmax_cvse_kernel<T, 2><<<grid, kCcThreads, 0, s>>>(p); break;
        case 4: softmax_cvse_kernel<T, 4><<<grid, kCcThreads, 0, s>>>(p); break;
        case 8: softmax_cvse_kernel<T, 8><<<grid, kCcThreads, 0, s>>>(p); break;
        default: return VS_ERR_VEC_LENGTH;
    }
    return (int)cudaGetLastError();
}

template <typename T> int softmax_backward_by_v(int V, const SoftmaxBackwardParams &p, int batch, cudaStream_t s) {
    const int64_t blocks = ((int64_t)p.m_vec * 32 + kCcThreads - 1) / kCcThreads;
    dim3 grid((unsigned)blocks, (unsigned)batch, 1);
    switch (V) {
        case 1: softmax_cvse_backward_kernel<T, 1><<<grid, kCcThreads, 0, s>>>(p); break;
        case 2: softmax_cvse_backward_kernel<T, 2><<<grid, kCcThreads, 0, s>>>(p); break;
        case 4: softmax_cvse_backward_kernel<T, 4><<<grid, kCcThreads, 0, s>>>(p); break;
        case 8: softmax_cvse_backward_kernel<T, 8><<<grid, kCcThreads, 0, s>>>(p); break;
        default: return VS_ERR_VEC_LENGTH;
    }
    return (int)cudaGetLastError();
}

constexpr int kMaxBatch = 65535;  // grid.y of the CUDA-core kernels

}  // namespace

// =============================================================================================================

VS_EXPORT int vs_spmm_batched(int path, int in_dtype, int out_dtype, int m_vec, int vec_length, int k, int n,
                              const int32_t *row_indices, const int32_t *row_offsets, const int32_t *col_indices,
                              const void *values, const void *rhs_matrix, void *output_matrix, int batch,
                              int64_t stride_values, int64_t stride_rhs, int64_t stride_out, void *stream) {
    if (path != VS_PATH_TENSOR && path != VS_PATH_CUDA_CORE) return VS_ERR_ARG;
    if (path == VS_PATH_TENSOR ? !(vec_length == 2 || vec_length == 4 || vec_length == 8) : !valid_v(vec_length))
        return VS_ERR_VEC_LENGTH;
    const bool f16 = (in_dtype == VS_F16) && (out_dtype == VS_F16 || out_dtype == VS_F32);
    const bool f32 = (in_dtype == VS_F32) && (out_dtype == VS_F32) && path == VS_PATH_CUDA_CORE;
    if (!f16 && !f32) return VS_ERR_DTYPE;
    if (m_vec < 0 || k < 0 || n < 0) return VS_ERR_SHAPE;
    if (batch < 1 || batch > kMaxBatch) return VS_ERR_ARG;
    if (path == VS_PATH_TENSOR ? (k % 64 != 0) : (k % (in_dtype == VS_F16 ? 8 : 4) != 0)) return VS_ERR_SHAPE;
    if ((int64_t)m_vec * vec_length > 0x7fffffffll) return VS_ERR_SHAPE;
    if (m_vec == 0 || k == 0) return VS_OK;
    if (!row_indices || !row_offsets || !col_indices || !values || !rhs_matrix || !output_matrix) return VS_ERR_NULL;
    if (!aligned16(values) || !aligned16(rhs_matrix) || !aligned16(output_matrix)) return VS_ERR_ALIGN;
    if (!stride_ok(stride_values, in_dtype) || !stride_ok(stride_rhs, in_dtype) || !stride_ok(stride_out, out_dtype))
        return VS_ERR_ALIGN;
    if (batch > 1 && stride_out == 0) return VS_ERR_ARG;

    SpmmParams p;
    p.m_vec = m_vec; p.N = k; p.K = n; p.batch = batch;
    p.row_indices = row_indices; p.row_offsets = row_offsets; p.col_indices = col_indices;
    p.values = values; p.rhs = rhs_matrix; p.out = output_matrix;
    p.stride_values = stride_values; p.stride_rhs = stride_rhs; p.stride_out = stride_out;
    cudaStream_t s = static_cast<cudaStream_t>(stream);

    if (path == VS_PATH_TENSOR) {
        return out_dtype == VS_F16 ? spmm_tc_by_v<__half>(vec_length, p, s) : spmm_tc_by_v<float>(vec_length, p, s);
    }
    if (in_dtype == VS_F32) return spmm_cc_by_v<float, float>(vec_length, p, s);
    return out_dtype == VS_F16 ? spmm_cores_by_v(vec_length, p, s) : spmm_cc_by_v<__half, float>(vec_length, p, s);
}

VS_EXPORT int vs_spmm(int path, int in_dtype, int out_dtype, int m_vec, int vec_length, int k, int n,
                      const int32_t *row_indices, const int32_t *row_offsets, const int32_t *col_indices,
                      const void *values, const void *rhs_matrix, void *output_matrix, void *stream) {
    return vs_spmm_batched(path, in_dtype, out_dtype, m_vec, vec_length, k, n, row_indices, row_offsets,
                           col_indices, values, rhs_matrix, output_matrix, 1, 0, 0, 0, stream);
}

// ---- SpMM with the transposed sparse matrix ------------------------------------------------------------------
namespace {
// CUDA-core kernel.  With `plan_hdr` it is enqueued behind the dense kernel and returns at once unless that kernel
// left the call to it.
// `second`: another product of the same structure and sizes, served by the same launch (only behind the dense kernel).
template <typename TOut, int V>
int launch_spmm_t_cc(const spmmt::Params &p, cudaStream_t s, DeviceInfo *d, const int32_t *plan_hdr, int plan_checks, int redo = kPlanRedo,
                     const spmmt::Params *second = nullptr) {
    const int row_groups = (p.n + spmmt::kWarps - 1) / spmmt::kWarps;
    const int chunks = (p.N + spmmt::kChunk - 1) / spmmt::kChunk;
    const int64_t items = (int64_t)p.batch * chunks * row_groups;
    const int64_t cap = (int64_t)d->sm_count * 16;   // as many 128-thread CTAs as are resident at once; the rest by grid stride
                                                      // (behind the dense kernel the launch usually returns at once: 9472 CTAs
                                                      // took 14 us to do so, a quarter of them a quarter of that)
    const unsigned grid = (unsigned)(items < cap ? items : cap);
    auto kernel = spmmt::spmm_t_kernel<TOut, V>;
    if (second) {
        const int64_t half = cap / 2;
        return (int)launch_overlapped(spmmt::spmm_t_kernel<TOut, V, (V > 1)>, 2 * (unsigned)(items < half ? items : half), spmmt::kThreads, 0, s,
                                      p, *second, items, row_groups, chunks, plan_hdr, plan_checks, redo);
    }
    if (plan_hdr) return (int)launch_overlapped(kernel, grid, spmmt::kThreads, 0, s, p, p, items, row_groups, chunks, plan_hdr, plan_checks, redo);
    kernel<<<grid, spmmt::kThreads, 0, s>>>(p, p, items, row_groups, chunks, plan_hdr, plan_checks, redo);
    return (int)cudaGetLastError();
}

enum class SpmmTMode { kAuto, kDense, kGather };
SpmmTMode spmm_t_mode() {   // read at every call, so that a test can switch kernels inside one process
    const char *e = std::getenv("VSPARSE_B200_SPMM_T");
    if (e && !std::strcmp(e, "dense")) return SpmmTMode::kDense;
    if (e && !std::strcmp(e, "gather")) return SpmmTMode::kGather;
    return SpmmTMode::kAuto;
}

// Tensor path of the transposed product: A^T (n x m_vec * V) goes through the densifying SpMM kernel, its plan
// built straight from the transposed structure (dense_plan_kernel<true>), the values read where the forward
// operators keep them; a vector's V values land side by side in one row of the tile.  Costs for the choice, in the
// plan kernel's units (SM-cycles per 128 columns): the CUDA-core kernel ~5 per value (0.92 ms for 256 products of
// 2048 x 512, 90 % sparse, V = 8), the dense kernel ~1100 per stage plus ~1.5 per vector of fill work (0.170 ms on
// the same problem against 0.137 for the forward product with the same tiles).
struct Span {
    const void *at;
    int64_t elems;   // fp16, of each problem
};
// Whether two of them share memory.
bool overlap(const Span &x, const Span &y, int batch) {
    const uintptr_t a = reinterpret_cast<uintptr_t>(x.at), b = reinterpret_cast<uintptr_t>(y.at);
    return a < b + 2 * (uintptr_t)(y.elems * batch) && b < a + 2 * (uintptr_t)(x.elems * batch);
}
// `count` products (at most kPlanProducts) with the same structure, sizes and strides: one plan serves them.  `alone`: the caller has no other with that structure.
template <typename TOut, int V> int launch_spmm_t(const spmmt::Params *list, int count, int m_vec, cudaStream_t s, bool alone) {
    const spmmt::Params &p = list[0];
    DeviceInfo *d;
    int rc = device_info(&d);
    if (rc != VS_OK) return rc;
    const SpmmTMode mode = spmm_t_mode();
    const int shift = V == 8 ? 3 : V == 4 ? 2 : V == 2 ? 1 : 0;
    const int64_t M = (int64_t)m_vec * V;   // columns of A^T: the contraction
    SpmmParams q;
    q.m_vec = p.n; q.N = p.N; q.K = (int)M; q.batch = p.batch;
    q.row_indices = nullptr; q.row_offsets = p.t_offsets; q.col_indices = p.t_rows;
    q.values = p.values; q.rhs = p.rhs; q.out = p.out;
    q.stride_values = p.stride_values; q.stride_rhs = p.stride_rhs; q.stride_out = p.stride_out;
    const int k_blocks = (q.K + densespmm::kBlockK - 1) / densespmm::kBlockK;
    const int m_tiles = (q.m_vec + densespmm::kTileM - 1) / densespmm::kTileM;
    const int n_tiles = (q.N + densespmm::kTileN - 1) / densespmm::kTileN;
    const int groups = m_tiles * (densespmm::kTileM / densespmm::kGroupRows);
    const int plan_blocks = k_blocks * (densespmm::kBlockK / densespmm::kPlanCols);
    const int rows_per_group = densespmm::kGroupRows;
    int64_t capacity = 0, offsets_bytes = 0;
    const int64_t plan_bytes = spmm_t_plan_bytes(p.n, m_vec, V, q.batch, q.stride_values, &capacity, &offsets_bytes);
    const int checks = spmm_plan_checks(q.m_vec);
    const size_t plan_words = (size_t)(2 * plan_blocks + rows_per_group + 1), check_words = (size_t)densespmm::kPlanWarps * plan_blocks;
    const size_t plan_smem = (plan_words > check_words ? plan_words : check_words) * 4;
    auto by_cores = [&]() {
        for (int i = 0; i < count; ++i) {
            const int rc = launch_spmm_t_cc<TOut, V>(list[i], s, d, nullptr, 0);
            if (rc != VS_OK) return rc;
        }
        return (int)VS_OK;
    };
    // One small product, by the sizes of the whole call that it is a part of (the CUDA-core kernel adds up in another order than the tiles): plan, tiles and stand-by are 20 us at the least, and few tiles leave most SMs idle, where the CUDA-core kernel is one
    // launch of many warps.  The host does not know the number of entries, so the line is drawn where even a full matrix is small, and rows of A^T
    // are short (a warp walks one).  Forward and backward of a training product, tiles / entries, us (vector-rows first): 73 x 719 x 192, V = 4, 73 % sparse
    // 69 / 63; 462 x 174 x 64, V = 8, 60 % 94 / 74; 125 x 88 x 128, V = 4, 67 % 89 / 64; 229 x 94 x 1216, V = 2, 62 % 69 / 63; past the line
    // 182 x 1232 x 192, V = 8, 58 % 69 / 72, 154 x 926 x 512, V = 8, 52 % 71 / 81 and 367 x 847 x 192, V = 8, 53 % 74 / 99.
    const SpmmParams whole = whole_call(q);
    const bool small = mode == SpmmTMode::kAuto && alone && m_vec <= 512 && (double)M * p.n * whole.N * whole.batch <= 100e6;
    const bool dense_ok = !t_no_scratch && !small && mode != SpmmTMode::kGather && q.K > 0 && q.m_vec > 0 && plan_bytes <= kMaxPlanBytes &&
                          plan_smem <= 40 * 1024 && (q.batch == 1 || (q.stride_rhs * 2) % 16 == 0) &&
                          (q.batch == 1 || (q.stride_out * sizeof(TOut)) % 16 == 0);
    if (!dense_ok) return by_cores();

    constexpr bool kOutF32 = sizeof(TOut) == 4;
    CUtensorMap map[kPlanProducts], map_out[kPlanProducts], map_b4[kPlanProducts];
    int use_b4 = q.N % 64 == 0 ? 1 : 0;
    for (int i = 0; i < count; ++i) {
        if (make_tile_map(&map[i], list[i].rhs, false, (uint64_t)q.K, (uint64_t)q.N, (uint64_t)q.batch, (uint64_t)q.stride_rhs, 64, 64) != VS_OK ||
            make_tile_map(&map_out[i], list[i].out, kOutF32, (uint64_t)q.m_vec, (uint64_t)q.N, (uint64_t)q.batch, (uint64_t)q.stride_out,
                          densespmm::kStoreCols, 32) != VS_OK)
            return by_cores();
        map_b4[i] = map[i];
        if (use_b4 && make_blocked_map(&map_b4[i], list[i].rhs, (uint64_t)q.K, (uint64_t)q.N, (uint64_t)q.batch, (uint64_t)q.stride_rhs,
                                       densespmm::kTileN / 64) != VS_OK)
            use_b4 = 0;
    }
    auto kernel = densespmm::spmm_dense_kernel<TOut, V, true>;
    auto kernel_two = densespmm::spmm_dense_kernel<TOut, V, true, (V > 1)>;   // attention's vectors are longer than 1
    static DeviceBits smem_set, smem_set_two;
    rc = set_smem_once(kernel, densespmm::kSmemBytes, smem_set);
    if (rc == VS_OK && count == 2) rc = set_smem_once(kernel_two, densespmm::kSmemBytes, smem_set_two);
    if (rc != VS_OK) return rc;
    uint8_t *plan = nullptr;
    PlanScratch scratch;
    if (scratch.take(d, s, (size_t)plan_bytes, reinterpret_cast<void **>(&plan)) != VS_OK)
        return by_cores();
    int32_t *flag = reinterpret_cast<int32_t *>(plan);
    const int64_t header_bytes = spmm_plan_header_bytes(checks);
    int32_t *blk_offsets = reinterpret_cast<int32_t *>(plan + header_bytes);
    uint2 *blk_entries = reinterpret_cast<uint2 *>(plan + header_bytes + offsets_bytes);
    rc = (int)launch_overlapped(densespmm::dense_plan_kernel<true>, (unsigned)(groups + checks), densespmm::kPlanThreads, plan_smem, s,
                                p.t_offsets, p.t_rows, p.t_src, shift, q.m_vec, q.K, groups, rows_per_group, plan_blocks, blk_offsets,
                                blk_entries, capacity, mode == SpmmTMode::kDense ? 1 : 0, 1100.0f, 0.0f, 5.0f * V, 1.5f, flag);
    const int64_t items = (int64_t)q.batch * n_tiles * m_tiles;
    const unsigned grid = (unsigned)(items < d->sm_count ? items : d->sm_count);   // one persistent CTA per SM
    const bool pairs = (use_b4 || q.N % 64 != 0) && spmm_pair_takes(q.N, V, (int64_t)q.batch * m_tiles, d, true);
    if constexpr (V > 1) {
        // Half of the SMs each: never more waves than one product after the other.  Up to 128 columns wide that also beats pairs of CTAs
        // for one product after the other, in every size that the pairs took there: attention forward and backward of 12 heads x 2280,
        // d = 128, V = 8 244.4 -> 217.3 us, of 24 x 664, V = 4 116.2 -> 101.8, of one head of 2856, V = 8 92.4 -> 81.5.
        const char *forced = std::getenv("VSPARSE_B200_SPMM_PAIR");
        // Results that share memory are written one after the other.
        const int64_t elems = (int64_t)q.m_vec * q.N;
        if (count == 2 && (!pairs || (q.N <= 128 && !forced)) && d->sm_count > 1 && rc == VS_OK && !overlap({list[0].out, elems}, {list[1].out, elems}, q.batch)) {
            densespmm::Second<true> two;
            two.map_b = map[1]; two.map_out = map_out[1]; two.map_b4 = map_b4[1];
            two.values = list[1].values; two.rhs = list[1].rhs;
            const int64_t half = d->sm_count / 2;
            rc = (int)launch_overlapped(kernel_two, 2 * (unsigned)(items < half ? items : half), densespmm::kThreads, densespmm::kSmemBytes, s, q,
                                        map[0], map_out[0], map_b4[0], use_b4, blk_offsets, blk_entries, m_tiles, n_tiles, k_blocks, d->status,
                                        flag, checks, flag + kPlanRedo, two);
            if (rc == VS_OK) rc = launch_spmm_t_cc<TOut, V>(list[0], s, d, flag, checks, kPlanRedo, &list[1]);
            return rc;
        }
    }
    for (int i = 0; i < count && rc == VS_OK; ++i) {
        q.values = list[i].values; q.rhs = list[i].rhs; q.out = list[i].out;
        int rc_pair = VS_OK;
        if (pairs &&
            launch_spmm_pair<TOut, V, true>(q, s, d, map[i], map_out[i], map_b4[i], blk_offsets, blk_entries, m_tiles, k_blocks, flag, checks, flag + kPlanRedo + i, &rc_pair))
            rc = rc_pair;
        else
            rc = (int)launch_overlapped(kernel, grid, densespmm::kThreads, densespmm::kSmemBytes, s, q, map[i], map_out[i], map_b4[i], use_b4,
                                        blk_offsets, blk_entries, m_tiles, n_tiles, k_blocks, d->status, flag, checks, flag + kPlanRedo + i,
                                        densespmm::Second<false>());
        if (rc == VS_OK) rc = launch_spmm_t_cc<TOut, V>(list[i], s, d, flag, checks, kPlanRedo + i);
    }
    return rc;
}
template <typename TOut> int spmm_t_by_v(int V, const spmmt::Params *p, int count, int m_vec, cudaStream_t s, bool alone) {
    switch (V) {
        case 1: return launch_spmm_t<TOut, 1>(p, count, m_vec, s, alone);
        case 2: return launch_spmm_t<TOut, 2>(p, count, m_vec, s, alone);
        case 4: return launch_spmm_t<TOut, 4>(p, count, m_vec, s, alone);
        case 8: return launch_spmm_t<TOut, 8>(p, count, m_vec, s, alone);
    }
    return VS_ERR_VEC_LENGTH;
}
}  // namespace

namespace {
// Checks one batched product with the transposed matrix and fills in its parameters; *empty where there is nothing to compute.
int spmm_t_params(int in_dtype, int out_dtype, int m_vec, int vec_length, int k, int n, const int32_t *t_offsets, const int32_t *t_rows,
                  const int32_t *t_src, const void *values, const void *rhs_matrix, void *output_matrix, int batch, int64_t stride_values,
                  int64_t stride_rhs, int64_t stride_out, spmmt::Params &p, bool &empty) {
    empty = false;
    if (!valid_v(vec_length)) return VS_ERR_VEC_LENGTH;
    if (!(in_dtype == VS_F16 && (out_dtype == VS_F16 || out_dtype == VS_F32))) return VS_ERR_DTYPE;
    if (m_vec < 0 || k < 0 || n < 0 || k % 8 != 0) return VS_ERR_SHAPE;
    if ((int64_t)m_vec * vec_length > 0x7fffffffll) return VS_ERR_SHAPE;
    if (batch < 1 || batch > kMaxBatch) return VS_ERR_ARG;
    empty = n == 0 || k == 0;
    if (empty) return VS_OK;
    if (!t_offsets || !t_rows || !t_src || !values || !rhs_matrix || !output_matrix) return VS_ERR_NULL;
    if (!aligned16(values) || !aligned16(rhs_matrix) || !aligned16(output_matrix)) return VS_ERR_ALIGN;
    if (!stride_ok(stride_values, in_dtype) || !stride_ok(stride_rhs, in_dtype) || !stride_ok(stride_out, out_dtype))
        return VS_ERR_ALIGN;
    if (batch > 1 && stride_out == 0) return VS_ERR_ARG;
    p.n = n; p.N = k; p.batch = batch;
    p.t_offsets = t_offsets; p.t_rows = t_rows; p.t_src = t_src;
    p.values = static_cast<const __half *>(values); p.rhs = static_cast<const __half *>(rhs_matrix); p.out = output_matrix;
    p.stride_values = stride_values; p.stride_rhs = stride_rhs; p.stride_out = stride_out;
    return VS_OK;
}
}  // namespace

VS_EXPORT int vs_spmm_t_batched(int in_dtype, int out_dtype, int m_vec, int vec_length, int k, int n,
                                const int32_t *t_offsets, const int32_t *t_rows, const int32_t *t_src,
                                const void *values, const void *rhs_matrix, void *output_matrix, int batch,
                                int64_t stride_values, int64_t stride_rhs, int64_t stride_out, void *stream) {
    spmmt::Params p;
    bool empty;
    const int rc = spmm_t_params(in_dtype, out_dtype, m_vec, vec_length, k, n, t_offsets, t_rows, t_src, values, rhs_matrix, output_matrix, batch,
                                 stride_values, stride_rhs, stride_out, p, empty);
    if (rc != VS_OK || empty) return rc;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    return out_dtype == VS_F16 ? spmm_t_by_v<__half>(vec_length, &p, 1, m_vec, s, true) : spmm_t_by_v<float>(vec_length, &p, 1, m_vec, s, true);
}

VS_EXPORT int vs_spmm_t(int in_dtype, int out_dtype, int m_vec, int vec_length, int k, int n, const int32_t *t_offsets,
                        const int32_t *t_rows, const int32_t *t_src, const void *values, const void *rhs_matrix,
                        void *output_matrix, void *stream) {
    return vs_spmm_t_batched(in_dtype, out_dtype, m_vec, vec_length, k, n, t_offsets, t_rows, t_src, values, rhs_matrix,
                             output_matrix, 1, 0, 0, 0, stream);
}

VS_EXPORT int vs_sddmm_batched(int path, int in_dtype, int out_dtype, int m_vec, int k, int n, int nonzeros_vec,
                               const int32_t *row_indices, const int32_t *row_offsets, const int32_t *col_indices,
                               const void *lhs_matrix, const void *rhs_matrix, void *output_values,
                               int vec_length, int batch, int64_t stride_lhs, int64_t stride_rhs,
                               int64_t stride_out, void *stream, int algorithm) {
    if (path != VS_PATH_TENSOR && path != VS_PATH_CUDA_CORE) return VS_ERR_ARG;
    if (path == VS_PATH_TENSOR ? !(vec_length == 2 || vec_length == 4 || vec_length == 8) : !valid_v(vec_length))
        return VS_ERR_VEC_LENGTH;
    if (!(in_dtype == VS_F16 && (out_dtype == VS_F16 || out_dtype == VS_F32))) return VS_ERR_DTYPE;
    if (path == VS_PATH_TENSOR && (algorithm < 0 || algorithm > 3)) return VS_ERR_ARG;
    if (m_vec < 0 || k < 0 || n < 0 || nonzeros_vec < 0) return VS_ERR_SHAPE;
    if (batch < 1 || batch > kMaxBatch) return VS_ERR_ARG;
    if (path == VS_PATH_TENSOR ? (k % 64 != 0) : (k % 8 != 0)) return VS_ERR_SHAPE;
    if ((int64_t)nonzeros_vec * vec_length > 0x7fffffffll) return VS_ERR_SHAPE;
    if (m_vec == 0 || nonzeros_vec == 0) return VS_OK;
    if (!row_indices || !row_offsets || !col_indices || !lhs_matrix || !rhs_matrix || !output_values)
        return VS_ERR_NULL;
    if (!aligned16(lhs_matrix) || !aligned16(rhs_matrix) || !aligned16(output_values)) return VS_ERR_ALIGN;
    if (!stride_ok(stride_lhs, in_dtype) || !stride_ok(stride_rhs, in_dtype) || !stride_ok(stride_out, out_dtype))
        return VS_ERR_ALIGN;
    if (batch > 1 && stride_out == 0) return VS_ERR_ARG;

    SddmmParams p;
    p.m_vec = m_vec; p.k = k; p.n = n; p.nnz_vec = nonzeros_vec; p.batch = batch;
    p.row_indices = row_indices; p.row_offsets = row_offsets; p.col_indices = col_indices;
    p.lhs = lhs_matrix; p.rhs = rhs_matrix; p.out = output_values;
    p.stride_lhs = stride_lhs; p.stride_rhs = stride_rhs; p.stride_out = stride_out;
    cudaStream_t s = static_cast<cudaStream_t>(stream);

    if (k == 0) {  // empty contraction: every output is zero
        for (int b = 0; b < batch; ++b) {
            cudaError_t e = cudaMemsetAsync(static_cast<char *>(output_values) + (size_t)b * stride_out * elem_size(out_dtype),
                                            0, (size_t)nonzeros_vec * vec_length * elem_size(out_dtype), s);
            if (e != cudaSuccess) return (int)e;
        }
        return VS_OK;
    }
    if (path == VS_PATH_TENSOR) {
        return out_dtype == VS_F16 ? sddmm_tc_by_v<__half>(vec_length, p, s) : sddmm_tc_by_v<float>(vec_length, p, s);
    }
    return out_dtype == VS_F16 ? sddmm_cores_by_v(vec_length, p, s) : sddmm_cc_by_v<__half, float>(vec_length, p, s);
}

VS_EXPORT int vs_sddmm(int path, int in_dtype, int out_dtype, int m_vec, int k, int n, int nonzeros_vec,
                       const int32_t *row_indices, const int32_t *row_offsets, const int32_t *col_indices,
                       const void *lhs_matrix, const void *rhs_matrix, void *output_values, int vec_length,
                       void *stream, int algorithm) {
    return vs_sddmm_batched(path, in_dtype, out_dtype, m_vec, k, n, nonzeros_vec, row_indices, row_offsets,
                            col_indices, lhs_matrix, rhs_matrix, output_values, vec_length, 1, 0, 0, 0, stream,
                            algorithm);
}

VS_EXPORT int vs_softmax_cvse(int dtype, int m_vec, int vec_length, const int32_t *row_indices,
                              const int32_t *row_offsets, const void *scores, void *probs, float scale, int batch,
                              int64_t stride, void *stream) {
    (void)row_indices;  // rows are independent and equally cheap to reach: the order is not needed
    if (!valid_v(vec_length)) return VS_ERR_VEC_LENGTH;
    if (dtype != VS_F16 && dtype != VS_F32) return VS_ERR_DTYPE;
    if (m_vec < 0) return VS_ERR_SHAPE;
    if (batch < 1 || batch > kMaxBatch) return VS_ERR_ARG;
    if (m_vec == 0) return VS_OK;
    if (!row_offsets || !scores || !probs) return VS_ERR_NULL;
    if (stride < 0 || (batch > 1 && stride == 0)) return VS_ERR_ARG;
    {   // one entry (V values) is read and written as one vector of up to 16 bytes
        const size_t entry = (size_t)vec_length * elem_size(dtype), al = entry < 16 ? entry : 16;
        if (reinterpret_cast<uintptr_t>(scores) % al || reinterpret_cast<uintptr_t>(probs) % al ||
            ((size_t)stride * elem_size(dtype)) % al)
            return VS_ERR_ALIGN;
    }
    SoftmaxParams p;
    p.m_vec = m_vec; p.batch = batch; p.row_offsets = row_offsets; p.scores = scores; p.probs = probs;
    p.stride = stride; p.scale = scale;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    return dtype == VS_F16 ? softmax_by_v<__half>(vec_length, p, s) : softmax_by_v<float>(vec_length, p, s);
}

VS_EXPORT int vs_softmax_cvse_backward(int dtype, int m_vec, int vec_length, const int32_t *row_offsets, const void *probs,
                                       const void *grad_probs, void *grad_scores, float scale, int batch, int64_t stride,
                                       void *stream) {
    if (!valid_v(vec_length)) return VS_ERR_VEC_LENGTH;
    if (dtype != VS_F16 && dtype != VS_F32) return VS_ERR_DTYPE;
    if (m_vec < 0) return VS_ERR_SHAPE;
    if (batch < 1 || batch > kMaxBatch) return VS_ERR_ARG;
    if (m_vec == 0) return VS_OK;
    if (!row_offsets || !probs || !grad_probs || !grad_scores) return VS_ERR_NULL;
    if (stride < 0 || (batch > 1 && stride == 0)) return VS_ERR_ARG;
    {   // one entry (V values) is read and written as one vector of up to 16 bytes
        const size_t entry = (size_t)vec_length * elem_size(dtype), al = entry < 16 ? entry : 16;
        if (reinterpret_cast<uintptr_t>(probs) % al || reinterpret_cast<uintptr_t>(grad_probs) % al ||
            reinterpret_cast<uintptr_t>(grad_scores) % al || ((size_t)stride * elem_size(dtype)) % al)
            return VS_ERR_ALIGN;
    }
    SoftmaxBackwardParams p;
    p.m_vec = m_vec; p.row_offsets = row_offsets; p.probs = probs; p.grad_probs = grad_probs; p.grad_scores = grad_scores;
    p.stride = stride; p.scale = scale;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    return dtype == VS_F16 ? softmax_backward_by_v<__half>(vec_length, p, batch, s)
                           : softmax_backward_by_v<float>(vec_length, p, batch, s);
}

namespace {
// Attention in one kernel per direction (attention.cuh).
template <int D, int W, bool kBackward> int launch_attention(const attention::Params &p, int batch, cudaStream_t s) {
    constexpr int rows = attention::kThreads / (32 * W);
    attention::attention_kernel<D, W, kBackward><<<dim3((unsigned)((p.m_vec + rows - 1) / rows), (unsigned)batch), attention::kThreads, 0, s>>>(p);
    return (int)cudaGetLastError();
}
// Warps per vector-row: one where the rows fill the GPU three times over, which spares the exchange between them (128 heads, sequence
// 4096: 588 / 670 / 793 us with 1 / 2 / 4 warps); more where the rows are few (2 heads, sequence 1024, 154 keys: 12.6 / 9.3 / 8.5 us) and long enough
// for a chunk each.  VSPARSE_B200_ATTENTION_WARPS chooses.
template <int D, bool kBackward> int launch_attention_rows(const attention::Params &p, int batch, DeviceInfo *d, cudaStream_t s) {
    const int64_t rows = (int64_t)p.m_vec * std::max(batch, t_whole_batch), wave = (int64_t)d->sm_count * attention::kCtasPerSm<D, kBackward> * (attention::kThreads / 32);
    const int keys = p.nnz_vec / p.m_vec;
    const char *e = std::getenv("VSPARSE_B200_ATTENTION_WARPS");
    const int warps = e ? std::atoi(e) : rows >= 3 * wave || keys <= 32 ? 1 : 2 * rows >= 3 * wave || keys <= 64 ? 2 : 4;
    if (warps <= 1) return launch_attention<D, 1, kBackward>(p, batch, s);
    if (warps == 2) return launch_attention<D, 2, kBackward>(p, batch, s);
    return launch_attention<D, 4, kBackward>(p, batch, s);
}
// Whether the one-kernel form takes a call; what it does not take, and every refusal, is the operators' own.  Their steps read an operand for the
// last time before a later step writes (grad_q in the place of grad_out, out in the place of kmat): where a result lies on an operand, they stay.
// VSPARSE_B200_ATTENTION=steps|fused.
bool attention_fused(int path, int m_vec, int V, int n, int d, int nnz_vec, int batch, float scale, std::initializer_list<const void *> indices,
                     std::initializer_list<Span> sources, std::initializer_list<Span> results) {
    const char *e = std::getenv("VSPARSE_B200_ATTENTION");
    if (e && !std::strcmp(e, "steps")) return false;
    if (path != VS_PATH_TENSOR || !(V == 2 || V == 4 || V == 8) || (d != 64 && d != 128)) return false;
    if (!(scale > 0.f)) return false;   // it takes the maximum of scores ahead of the scale
    if ((int64_t)n * d > 0xffffffffll) return false;   // 32-bit offsets
    if (m_vec < 1 || n < 1 || nnz_vec < 1 || batch < 1 || batch > kMaxBatch || (int64_t)m_vec * V > 0x7fffffffll || (int64_t)nnz_vec * V > 0x7fffffffll) return false;
    // Gathering costs what the mask names, the operators' dense tiles cost the whole matrix, and the same for 2 queries as for 8: dense masks of short
    // vectors are theirs once there is enough work to fill the GPU, at 2048 columns more than at 4096.  us, operators / this, forward (backward alike): 32 heads,
    // sequence 2048, 20 % of the keys, d = 64: V = 2 257 / 344, V = 4 155 / 186, V = 8 137 / 99; d = 128: 266 / 652, 164 / 336, 147 / 178; 15 %: 235 / 255,
    // 141 / 139, 122 / 81; 244 / 488, 150 / 254, 129 / 148; 8 heads, 4096, 15 %: 319 / 267, 198 / 149, 196 / 74; 323 / 477, 231 / 537, 228 / 127; 128 heads, 1024,
    // 5 %, d = 128: 168 / 219, 136 / 114, 119 / 64; 4 heads, 2048, 20 %, d = 64: 80 / 61, 62 / 36, 54 / 20.
    const double named = (double)nnz_vec / ((double)m_vec * n), line = d == 64 ? (V == 2 ? 0.125 : V == 4 ? 0.145 : 1.0) : (V == 2 ? 0.04 : V == 4 ? 0.065 : 0.14);
    if (named > line * std::sqrt(std::max(1.0, n / 2048.0)) && (int64_t)nnz_vec * std::max(batch, t_whole_batch) * (d / 64) > 3000000 && !(e && !std::strcmp(e, "fused"))) return false;
    for (const void *x : indices)
        if (!x) return false;
    for (const Span &x : sources)   // read 32 bytes at a time
        if (!x.at || reinterpret_cast<uintptr_t>(x.at) % 32 != 0) return false;
    for (const Span &x : results) {
        if (!x.at || !aligned16(x.at)) return false;
        for (const Span &y : sources)
            if (overlap(x, y, batch)) return false;
    }
    return (int64_t)nnz_vec * V % 8 == 0;
}
}  // namespace

VS_EXPORT int vs_attention_cvse_backward(int path, int m_vec, int vec_length, int n, int d, int nonzeros_vec,
                                         const int32_t *row_indices, const int32_t *row_offsets, const int32_t *col_indices,
                                         const int32_t *t_offsets, const int32_t *t_rows, const int32_t *t_src, const void *q,
                                         const void *kmat, const void *vmat, const void *grad_out, void *grad_q, void *grad_k,
                                         void *grad_v, void *probs_workspace, void *grad_workspace, float scale, int batch,
                                         void *stream) {
    if ((!probs_workspace || !grad_workspace) && nonzeros_vec > 0) return VS_ERR_NULL;
    if (probs_workspace && probs_workspace == grad_workspace) return VS_ERR_ARG;
    const int64_t m = (int64_t)m_vec * vec_length;
    const int64_t s_ws = (int64_t)nonzeros_vec * vec_length;
    if ((s_ws * 2) % 16 != 0 && batch > 1) return VS_ERR_ALIGN;
    const int64_t s_q = m * d, s_k = (int64_t)n * d;
    if (nonzeros_vec == 0) {   // an empty mask: the output does not depend on q, k or v
        if (m_vec < 0 || n < 0 || d < 0 || batch < 1 || !valid_v(vec_length)) return VS_ERR_ARG;
        cudaStream_t st = static_cast<cudaStream_t>(stream);
        if (s_q > 0 && !grad_q) return VS_ERR_NULL;
        if (s_k > 0 && (!grad_k || !grad_v)) return VS_ERR_NULL;
        if (s_q > 0) VS_CUDA_TRY(cudaMemsetAsync(grad_q, 0, (size_t)batch * s_q * 2, st));
        if (s_k > 0) VS_CUDA_TRY(cudaMemsetAsync(grad_k, 0, (size_t)batch * s_k * 2, st));
        if (s_k > 0) VS_CUDA_TRY(cudaMemsetAsync(grad_v, 0, (size_t)batch * s_k * 2, st));
        return VS_OK;
    }
    if (attention_fused(path, m_vec, vec_length, n, d, nonzeros_vec, batch, scale, {row_indices, row_offsets, col_indices, t_offsets, t_rows, t_src},
                        {{q, s_q}, {kmat, s_k}, {vmat, s_k}, {grad_out, s_q}},
                        {{grad_q, s_q}, {grad_k, s_k}, {grad_v, s_k}, {probs_workspace, s_ws}, {grad_workspace, s_ws}})) {
        DeviceInfo *info = nullptr;
        int rc = device_info(&info);
        if (rc != VS_OK) return rc;
        attention::Params p;
        p.m_vec = m_vec; p.V = vec_length; p.n = n; p.nnz_vec = nonzeros_vec;
        p.row_offsets = row_offsets; p.col_indices = col_indices;
        p.q = static_cast<const __half *>(q); p.k = static_cast<const __half *>(kmat); p.v = static_cast<const __half *>(vmat);
        p.out = static_cast<__half *>(grad_q); p.probs = static_cast<__half *>(probs_workspace);
        p.grad_out = static_cast<const __half *>(grad_out); p.grad_scores = static_cast<__half *>(grad_workspace);
        p.scale = scale;
        cudaStream_t st = static_cast<cudaStream_t>(stream);
        rc = d == 64 ? launch_attention_rows<64, true>(p, batch, info, st) : launch_attention_rows<128, true>(p, batch, info, st);
        if (rc != VS_OK) return rc;
        // dV = P^T dO and dK = dS^T Q from one plan
        spmmt::Params both[2];
        bool empty;
        rc = spmm_t_params(VS_F16, VS_F16, m_vec, vec_length, d, n, t_offsets, t_rows, t_src, probs_workspace, grad_out, grad_v, batch, s_ws, s_q, s_k, both[0], empty);
        if (rc == VS_OK && !empty)
            rc = spmm_t_params(VS_F16, VS_F16, m_vec, vec_length, d, n, t_offsets, t_rows, t_src, grad_workspace, q, grad_k, batch, s_ws, s_q, s_k, both[1], empty);
        if (rc != VS_OK || empty) return rc;
        return spmm_t_by_v<__half>(vec_length, both, 2, m_vec, st, false);
    }
    // P = softmax(scale * Q K^T) at the mask, recomputed rather than kept from the forward pass
    int rc = vs_sddmm_batched(path, VS_F16, VS_F16, m_vec, d, n, nonzeros_vec, row_indices, row_offsets, col_indices, q, kmat,
                              probs_workspace, vec_length, batch, s_q, s_k, s_ws, stream, 0);
    if (rc != VS_OK) return rc;
    rc = vs_softmax_cvse(VS_F16, m_vec, vec_length, row_indices, row_offsets, probs_workspace, probs_workspace, scale, batch,
                         s_ws, stream);
    if (rc != VS_OK) return rc;
    // dV = P^T dO together with dK = dS^T Q, from one plan and (spmm_dense_kernel<kTwo>) in one launch, unless dQ or dK is to stand where
    // dO or P is still to be read, or shares dV's memory.  Forward and backward of 10 heads x 2152, d = 128, V = 4: 305.3 -> 277.2 us; 16 x 3400,
    // V = 2 658.7 -> 639.6.
    bool apart = false;
    for (const Span &x : {Span{grad_q, s_q}, Span{grad_k, s_k}})
        for (const Span &y : {Span{grad_out, s_q}, Span{probs_workspace, s_ws}, Span{grad_v, s_k}}) apart = apart || overlap(x, y, batch);
    spmmt::Params both[2];
    bool empty;
    rc = spmm_t_params(VS_F16, VS_F16, m_vec, vec_length, d, n, t_offsets, t_rows, t_src, probs_workspace, grad_out, grad_v, batch, s_ws, s_q, s_k,
                       both[0], empty);
    if (rc == VS_OK && !empty && apart) rc = spmm_t_by_v<__half>(vec_length, both, 1, m_vec, static_cast<cudaStream_t>(stream), false);
    if (rc != VS_OK) return rc;
    // dP = dO V^T at the mask; dS = scale * P o (dP - rowsum(P o dP))
    rc = vs_sddmm_batched(path, VS_F16, VS_F16, m_vec, d, n, nonzeros_vec, row_indices, row_offsets, col_indices, grad_out, vmat,
                          grad_workspace, vec_length, batch, s_q, s_k, s_ws, stream, 0);
    if (rc != VS_OK) return rc;
    rc = vs_softmax_cvse_backward(VS_F16, m_vec, vec_length, row_offsets, probs_workspace, grad_workspace, grad_workspace, scale,
                                  batch, s_ws, stream);
    if (rc != VS_OK) return rc;
    // dQ = dS K,  dK = dS^T Q
    rc = vs_spmm_batched(path, VS_F16, VS_F16, m_vec, vec_length, d, n, row_indices, row_offsets, col_indices, grad_workspace,
                         kmat, grad_q, batch, s_ws, s_k, s_q, stream);
    if (rc == VS_OK)
        rc = spmm_t_params(VS_F16, VS_F16, m_vec, vec_length, d, n, t_offsets, t_rows, t_src, grad_workspace, q, grad_k, batch, s_ws, s_q, s_k,
                           both[1], empty);
    if (rc != VS_OK || empty) return rc;
    return apart ? spmm_t_by_v<__half>(vec_length, both + 1, 1, m_vec, static_cast<cudaStream_t>(stream), false)
                 : spmm_t_by_v<__half>(vec_length, both, 2, m_vec, static_cast<cudaStream_t>(stream), false);
}

VS_EXPORT int vs_attention_cvse(int path, int m_vec, int vec_length, int n, int d, int nonzeros_vec,
                                const int32_t *row_indices, const int32_t *row_offsets, const int32_t *col_indices,
                                const void *q, const void *kmat, const void *vmat, void *out, void *workspace,
                                float scale, int batch, void *stream) {
    if (!workspace && nonzeros_vec > 0) return VS_ERR_NULL;
    const int64_t m = (int64_t)m_vec * vec_length;
    const int64_t s_ws = (int64_t)nonzeros_vec * vec_length;
    if ((s_ws * 2) % 16 != 0 && batch > 1) return VS_ERR_ALIGN;
    if (nonzeros_vec == 0) {   // an empty mask: no scores, no probabilities, every output row is zero
        if (m_vec < 0 || d < 0 || batch < 1 || !valid_v(vec_length)) return VS_ERR_ARG;
        if (m == 0 || d == 0) return VS_OK;
        if (!out) return VS_ERR_NULL;
        return (int)cudaMemsetAsync(out, 0, (size_t)batch * m * d * 2, static_cast<cudaStream_t>(stream));
    }
    if (attention_fused(path, m_vec, vec_length, n, d, nonzeros_vec, batch, scale, {row_indices, row_offsets, col_indices},
                        {{q, m * d}, {kmat, (int64_t)n * d}, {vmat, (int64_t)n * d}}, {{out, m * d}, {workspace, s_ws}})) {
        DeviceInfo *info = nullptr;
        const int rc = device_info(&info);
        if (rc != VS_OK) return rc;
        attention::Params p;
        p.m_vec = m_vec; p.V = vec_length; p.n = n; p.nnz_vec = nonzeros_vec;
        p.row_offsets = row_offsets; p.col_indices = col_indices;
        p.q = static_cast<const __half *>(q); p.k = static_cast<const __half *>(kmat); p.v = static_cast<const __half *>(vmat);
        p.out = static_cast<__half *>(out); p.probs = static_cast<__half *>(workspace);
        p.grad_out = nullptr; p.grad_scores = nullptr; p.scale = scale;
        cudaStream_t st = static_cast<cudaStream_t>(stream);
        return d == 64 ? launch_attention_rows<64, false>(p, batch, info, st) : launch_attention_rows<128, false>(p, batch, info, st);
    }
    int rc = vs_sddmm_batched(path, VS_F16, VS_F16, m_vec, d, n, nonzeros_vec, row_indices, row_offsets,
                              col_indices, q, kmat, workspace, vec_length, batch, m * d, (int64_t)n * d, s_ws,
                              stream, 0);
    if (rc != VS_OK) return rc;
    rc = vs_softmax_cvse(VS_F16, m_vec, vec_length, row_indices, row_offsets, workspace, workspace, scale, batch,
                         s_ws, stream);
    if (rc != VS_OK) return rc;
    return vs_spmm_batched(path, VS_F16, VS_F16, m_vec, vec_length, d, n, row_indices, row_offsets, col_indices,
                           workspace, vmat, out, batch, s_ws, (int64_t)n * d, m * d, stream);
}

// ---- attention without a caller workspace --------------------------------------------------------------------
//
// Scratch for vs_attention_cvse_static: the probabilities between its SDDMM, softmax and SpMM steps.  The array
// is part of the library image, so every GPU that loads the library carries these 8 MiB until the process exits.
// In host code the NAME below is only a handle; the device address comes from cudaGetSymbolAddress.
constexpr size_t kStaticScratchBytes = size_t(8) << 20;
static __device__ __align__(256) unsigned char g_attention_scratch[kStaticScratchBytes];

namespace {
void *g_attention_scratch_ptr[kMaxDevices];   // device address of the array, looked up once per device
std::mutex g_attention_scratch_mutex;

// Must run with the target device current.  The look-up is a runtime query, not an allocation.
int attention_scratch(void **out) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return (int)e;
    if (dev < 0 || dev >= kMaxDevices) return VS_ERR_ARG;
    std::lock_guard<std::mutex> lock(g_attention_scratch_mutex);
    if (!g_attention_scratch_ptr[dev]) {
        void *ptr = nullptr;
        e = cudaGetSymbolAddress(&ptr, g_attention_scratch);
        if (e != cudaSuccess) return (int)e;
        g_attention_scratch_ptr[dev] = ptr;
    }
    *out = g_attention_scratch_ptr[dev];
    return VS_OK;
}
}  // namespace

VS_EXPORT int vs_attention_cvse_static(int path, int m_vec, int vec_length, int n, int d, int nonzeros_vec,
                                       const int32_t *row_indices, const int32_t *row_offsets,
                                       const int32_t *col_indices, const void *q, const void *kmat, const void *vmat,
                                       void *out, float scale, int batch, void *stream) {
    if (batch < 1) return VS_ERR_ARG;
    if (nonzeros_vec < 0) return VS_ERR_SHAPE;
    if (!valid_v(vec_length)) return VS_ERR_VEC_LENGTH;
    const unsigned long long need = 2ull * (unsigned long long)batch * (unsigned long long)nonzeros_vec * (unsigned long long)vec_length;
    if (need > kStaticScratchBytes) {
        fprintf(stderr,
                "vs_attention_cvse_static: batch * nonzeros_vec * vec_length = %llu fp16 probabilities need %llu bytes, "
                "the built-in scratch holds %zu; use vs_attention_cvse with a workspace of your own\n",
                need / 2, need, kStaticScratchBytes);
        return VS_ERR_SHAPE;
    }
    void *scratch = nullptr;
    int rc = attention_scratch(&scratch);
    if (rc != VS_OK) return rc;
    NoScratchScope no_allocation;   // SDDMM and SpMM below: the formulations without plan scratch
    return vs_attention_cvse(path, m_vec, vec_length, n, d, nonzeros_vec, row_indices, row_offsets, col_indices, q, kmat,
                             vmat, out, scratch, scale, batch, stream);
}

// ---- host-buffer forms -------------------------------------------------------------------------------------

namespace {
struct DeviceBuffers {  // frees whatever was allocated when it goes out of scope
    void *ptr[8] = {nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr};
    int count = 0;
    cudaError_t alloc(void **out, size_t bytes) {
        cudaError_t e = cudaMalloc(out, bytes ? bytes : 16);
        if (e == cudaSuccess) ptr[count++] = *out;
        return e;
    }
    ~DeviceBuffers() {
        for (int i = 0; i < count; ++i) cudaFree(ptr[i]);
    }
};
}  // namespace

VS_EXPORT int vs_spmm_host(int path, int in_dtype, int out_dtype, int m_vec, int vec_length, int k, int n,
                           const int32_t *row_indices, const int32_t *row_offsets, const int32_t *col_indices,
                           const void *values, const void *rhs_matrix, void *output_matrix) {
    if (m_vec < 0 || k < 0 || n < 0) return VS_ERR_SHAPE;
    if (!valid_v(vec_length)) return VS_ERR_VEC_LENGTH;
    if ((in_dtype != VS_F16 && in_dtype != VS_F32) || (out_dtype != VS_F16 && out_dtype != VS_F32)) return VS_ERR_DTYPE;
    if (!row_indices || !row_offsets || !output_matrix) return VS_ERR_NULL;
    const int nnz_vec = row_offsets[m_vec];
    int rc = vs_cvse_validate(m_vec, n, nnz_vec, row_offsets, col_indices);
    if (rc != VS_OK) return rc;
    if (nnz_vec > 0 && (!values || !rhs_matrix)) return VS_ERR_NULL;
    const size_t si = elem_size(in_dtype), so = elem_size(out_dtype);
    const size_t b_idx = (size_t)m_vec * 4, b_off = (size_t)(m_vec + 1) * 4, b_col = (size_t)nnz_vec * 4;
    const size_t b_val = (size_t)nnz_vec * vec_length * si, b_rhs = (size_t)n * k * si;
    const size_t b_out = (size_t)m_vec * vec_length * k * so;
    DeviceBuffers bufs;
    int32_t *d_idx, *d_off, *d_col;
    void *d_val, *d_rhs, *d_out;
    VS_CUDA_TRY(bufs.alloc((void **)&d_idx, b_idx));
    VS_CUDA_TRY(bufs.alloc((void **)&d_off, b_off));
    VS_CUDA_TRY(bufs.alloc((void **)&d_col, b_col));
    VS_CUDA_TRY(bufs.alloc(&d_val, b_val));
    VS_CUDA_TRY(bufs.alloc(&d_rhs, b_rhs));
    VS_CUDA_TRY(bufs.alloc(&d_out, b_out));
    VS_CUDA_TRY(cudaMemcpy(d_idx, row_indices, b_idx, cudaMemcpyHostToDevice));
    VS_CUDA_TRY(cudaMemcpy(d_off, row_offsets, b_off, cudaMemcpyHostToDevice));
    if (b_col) VS_CUDA_TRY(cudaMemcpy(d_col, col_indices, b_col, cudaMemcpyHostToDevice));
    if (b_val) VS_CUDA_TRY(cudaMemcpy(d_val, values, b_val, cudaMemcpyHostToDevice));
    if (b_rhs) VS_CUDA_TRY(cudaMemcpy(d_rhs, rhs_matrix, b_rhs, cudaMemcpyHostToDevice));
    rc = vs_spmm(path, in_dtype, out_dtype, m_vec, vec_length, k, n, d_idx, d_off, d_col, d_val, d_rhs, d_out, nullptr);
    if (rc != VS_OK) return rc;
    VS_CUDA_TRY(cudaDeviceSynchronize());
    if (b_out) VS_CUDA_TRY(cudaMemcpy(output_matrix, d_out, b_out, cudaMemcpyDeviceToHost));
    return VS_OK;
}

VS_EXPORT int vs_sddmm_host(int path, int in_dtype, int out_dtype, int m_vec, int k, int n, int nonzeros_vec,
                            const int32_t *row_indices, const int32_t *row_offsets, const int32_t *col_indices,
                            const void *lhs_matrix, const void *rhs_matrix, void *output_values, int vec_length,
                            int algorithm) {
    if (m_vec < 0 || k < 0 || n < 0 || nonzeros_vec < 0) return VS_ERR_SHAPE;
    if (!valid_v(vec_length)) return VS_ERR_VEC_LENGTH;
    if ((in_dtype != VS_F16 && in_dtype != VS_F32) || (out_dtype != VS_F16 && out_dtype != VS_F32)) return VS_ERR_DTYPE;
    if (!row_indices || !row_offsets) return VS_ERR_NULL;
    int rc = vs_cvse_validate(m_vec, n, nonzeros_vec, row_offsets, col_indices);
    if (rc != VS_OK) return rc;
    if (nonzeros_vec > 0 && (!lhs_matrix || !rhs_matrix || !output_values)) return VS_ERR_NULL;
    const size_t si = elem_size(in_dtype), so = elem_size(out_dtype);
    const size_t b_idx = (size_t)m_vec * 4, b_off = (size_t)(m_vec + 1) * 4, b_col = (size_t)nonzeros_vec * 4;
    const size_t b_lhs = (size_t)m_vec * vec_length * k * si, b_rhs = (size_t)n * k * si;
    const size_t b_out = (size_t)nonzeros_vec * vec_length * so;
    DeviceBuffers bufs;
    int32_t *d_idx, *d_off, *d_col;
    void *d_lhs, *d_rhs, *d_out;
    VS_CUDA_TRY(bufs.alloc((void **)&d_idx, b_idx));
    VS_CUDA_TRY(bufs.alloc((void **)&d_off, b_off));
    VS_CUDA_TRY(bufs.alloc((void **)&d_col, b_col));
    VS_CUDA_TRY(bufs.alloc(&d_lhs, b_lhs));
    VS_CUDA_TRY(bufs.alloc(&d_rhs, b_rhs));
    VS_CUDA_TRY(bufs.alloc(&d_out, b_out));
    VS_CUDA_TRY(cudaMemcpy(d_idx, row_indices, b_idx, cudaMemcpyHostToDevice));
    VS_CUDA_TRY(cudaMemcpy(d_off, row_offsets, b_off, cudaMemcpyHostToDevice));
    if (b_col) VS_CUDA_TRY(cudaMemcpy(d_col, col_indices, b_col, cudaMemcpyHostToDevice));
    if (b_lhs) VS_CUDA_TRY(cudaMemcpy(d_lhs, lhs_matrix, b_lhs, cudaMemcpyHostToDevice));
    if (b_rhs) VS_CUDA_TRY(cudaMemcpy(d_rhs, rhs_matrix, b_rhs, cudaMemcpyHostToDevice));
    rc = vs_sddmm(path, in_dtype, out_dtype, m_vec, k, n, nonzeros_vec, d_idx, d_off, d_col, d_lhs, d_rhs, d_out,
                  vec_length, nullptr, algorithm);
    if (rc != VS_OK) return rc;
    VS_CUDA_TRY(cudaDeviceSynchronize());
    if (b_out) VS_CUDA_TRY(cudaMemcpy(output_values, d_out, b_out, cudaMemcpyDeviceToHost));
    return VS_OK;
}

VS_EXPORT int64_t vs_spmm_workspace_bytes(int m_vec, int vec_length, int n, int batch, int64_t stride_values) {
    if (m_vec <= 0 || n <= 0 || batch < 1 || !(vec_length == 2 || vec_length == 4 || vec_length == 8)) return 0;
    const int64_t bytes = spmm_plan_bytes(m_vec, vec_length, n, batch, stride_values, nullptr, nullptr);
    return bytes <= kMaxPlanBytes ? bytes : 0;
}

VS_EXPORT int64_t vs_spmm_t_workspace_bytes(int m_vec, int vec_length, int n, int batch, int64_t stride_values) {
    if (m_vec <= 0 || n <= 0 || batch < 1 || !valid_v(vec_length) || (int64_t)m_vec * vec_length > 0x7fffffffll) return 0;
    const int64_t bytes = spmm_t_plan_bytes(n, m_vec, vec_length, batch, stride_values, nullptr, nullptr);
    return bytes <= kMaxPlanBytes ? bytes : 0;
}

VS_EXPORT int64_t vs_sddmm_workspace_bytes(int m_vec, int n, int nonzeros_vec) {
    if (m_vec <= 0 || n <= 0 || nonzeros_vec <= 0) return 0;
    int64_t bytes = sddmm_plan_bytes(m_vec, n, nonzeros_vec, nullptr);   // of the single-CTA form
    if (bytes > kMaxPlanBytes) bytes = 0;
    const int64_t pair = sddmm_pair_plan_bytes(m_vec, n, nonzeros_vec, nullptr, nullptr);
    return n <= pairsddmm::kMaxPlanColumns && pair <= kMaxPlanBytes ? std::max(bytes, pair) : bytes;
}

VS_EXPORT int vs_set_workspace(void *workspace, int64_t bytes) {
    if (bytes < 0 || (workspace == nullptr && bytes != 0)) return VS_ERR_ARG;
    if (!aligned16(workspace)) return VS_ERR_ALIGN;
    t_ws_set = workspace != nullptr;
    t_ws_ptr = workspace;
    t_ws_bytes = bytes;
    return VS_OK;
}

VS_EXPORT int vs_set_part_of(int columns, int batch) {
    if (columns < 0 || batch < 0) return VS_ERR_ARG;
    t_whole_columns = columns;
    t_whole_batch = batch;
    return VS_OK;
}

VS_EXPORT int vs_release_scratch(void *stream, int every_stream) {
    DeviceInfo *d;
    int rc = device_info(&d);
    if (rc != VS_OK) return rc;
    std::vector<std::pair<cudaStream_t, std::shared_ptr<Scratch>>> released;
    {
        std::lock_guard<std::mutex> table(g_devices_mutex);
        if (every_stream) {
            for (auto &kv : d->scratch) released.emplace_back(kv.first.stream, std::move(kv.second));
            d->scratch.clear();
        } else {
            auto it = d->scratch.find(DeviceInfo::key_of(static_cast<cudaStream_t>(stream)));
            if (it != d->scratch.end()) {
                released.emplace_back(it->first.stream, std::move(it->second));
                d->scratch.erase(it);
            }
        }
    }
    for (auto &r : released) {
        std::lock_guard<std::mutex> use(r.second->use);   // behind the launches of a call in progress
        r.second->retired = true;
        if (r.second->ptr) (void)cudaFreeAsync(r.second->ptr, r.first);
    }
    int dev = 0;
    if (cudaGetDevice(&dev) == cudaSuccess) free_returned_scratch(dev, 0);   // what graphs that are gone have left
    return VS_OK;
}

VS_EXPORT int vs_sddmm_formulation(int m_vec, int k, int n, int nonzeros_vec, int vec_length) {
    if (m_vec <= 0 || n <= 0 || k < densesddmm::kBlockK || nonzeros_vec <= 0 || !(vec_length == 2 || vec_length == 4 || vec_length == 8))
        return 0;
    SddmmParams p{};
    p.m_vec = m_vec; p.k = k; p.n = n; p.nnz_vec = nonzeros_vec;
    p.batch = 4096;   // no batch is given and no device needed: the answer for as many products as fill a B200 many times over
    return sddmm_use_dense(p, vec_length, 148) ? 1 : 0;
}

VS_EXPORT int vs_kernel_timing(int enable, double *total_ms, int *launches) {
    KernelTiming &t = kernel_timing();
    std::vector<std::pair<cudaEvent_t, cudaEvent_t>> done;
    {
        std::lock_guard<std::mutex> g(t.lock);
        done.swap(t.pairs);
        t.on = enable != 0;
    }
    double ms = 0.0;
    int n = 0, rc = VS_OK;
    for (auto &pr : done) {
        float x = 0.0f;
        cudaError_t e = cudaEventSynchronize(pr.second);
        if (e == cudaSuccess) e = cudaEventElapsedTime(&x, pr.first, pr.second);
        if (e == cudaSuccess) { ms += x; ++n; } else { rc = (int)e; (void)cudaGetLastError(); }
        cudaEventDestroy(pr.first);
        cudaEventDestroy(pr.second);
    }
    if (total_ms) *total_ms = ms;
    if (launches) *launches = n;
    return rc;
}

VS_EXPORT int vs_measure_fp32_fma(double *tflops) {
    if (!tflops) return VS_ERR_NULL;
    DeviceInfo *d;
    int rc = device_info(&d);
    if (rc != VS_OK) return rc;
    const int iters = 1 << 14, blocks = d->sm_count * 8, threads = 256;
    cudaEvent_t e0, e1;
    VS_CUDA_TRY(cudaEventCreate(&e0));
    VS_CUDA_TRY(cudaEventCreate(&e1));
    float *sink = nullptr;
    fp32_fma_probe_kernel<<<blocks, threads>>>(iters, 1.0f, sink);   // warm-up
    double best = 0.0;
    for (int rep = 0; rep < 3; ++rep) {
        cudaEventRecord(e0);
        fp32_fma_probe_kernel<<<blocks, threads>>>(iters, 1.0f, sink);
        cudaEventRecord(e1);
        cudaError_t e = cudaEventSynchronize(e1);
        float ms = 0.0f;
        if (e == cudaSuccess) e = cudaEventElapsedTime(&ms, e0, e1);
        if (e != cudaSuccess) {
            cudaEventDestroy(e0);
            cudaEventDestroy(e1);
            return (int)e;
        }
        const double t = 2.0 * 8.0 * iters * (double)blocks * threads / (ms * 1e-3) / 1e12;
        if (t > best) best = t;
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    *tflops = best;
    return VS_OK;
}

VS_EXPORT int vs_device_status(int clear, uint32_t *status) {
    if (!status) return VS_ERR_NULL;
    DeviceInfo *d;
    int rc = device_info(&d);
    if (rc != VS_OK) return rc;
    VS_CUDA_TRY(cudaDeviceSynchronize());
    VS_CUDA_TRY(cudaMemcpy(status, d->status, sizeof(uint32_t), cudaMemcpyDeviceToHost));
    if (clear) VS_CUDA_TRY(cudaMemset(d->status, 0, sizeof(uint32_t)));
    return VS_OK;
}

VS_EXPORT int vs_selftest_gather4(const void *matrix, int rows, int cols, const int32_t *row_indices, int groups,
                                  int x, void *out, void *stream) {
    if (!matrix || !row_indices || !out) return VS_ERR_NULL;
    if (rows < 1 || cols < 64 || cols % 8 != 0 || groups < 1 || groups > 32 || x < 0 || x % 8 != 0) return VS_ERR_SHAPE;
    if (!aligned16(matrix) || !aligned16(out)) return VS_ERR_ALIGN;
    DeviceInfo *d;
    int rc = device_info(&d);
    if (rc != VS_OK) return rc;
    CUtensorMap map;
    rc = make_gather_map(&map, matrix, (uint64_t)rows, (uint64_t)cols);
    if (rc != VS_OK) return rc;
    const int smem = groups * 512 + 64 + 1024;
    tcselftest::gather4_kernel<<<1, 32, smem, static_cast<cudaStream_t>(stream)>>>(
        map, row_indices, groups, x, static_cast<uint8_t *>(out), d->status);
    return (int)cudaGetLastError();
}



namespace {
// Whether the 16 contraction elements x `rows` fp16 operand a shared-memory descriptor names lies inside an image
// of `image_bytes` (descriptor start relative to the image).  Only the layouts the kernels use are accepted:
// no swizzle or the 128-byte swizzle, either major.
bool selftest_operand_fits(uint64_t desc, int rows, bool mn_major, int image_bytes) {
    const int64_t start = (int64_t)(desc & 0x3fffu) << 4, lbo = (int64_t)((desc >> 16) & 0x3fffu) << 4,
                  sbo = (int64_t)((desc >> 32) & 0x3fffu) << 4;
    const unsigned swizzle = (unsigned)(desc >> 61) & 7u;
    if (swizzle != 0 && swizzle != 2) return false;
    if (rows < 8 || rows % 8 != 0) return false;
    int64_t end;
    if (swizzle == 2 && mn_major) {          // atoms of 64 rows x 8 contraction elements (1 KiB): LBO between atoms along the rows, SBO along the contraction
        if (rows % 64 != 0) return false;
        end = start + (rows / 64 - 1) * lbo + sbo + 1024;
    } else if (swizzle == 2) {               // rows of 128 bytes, eight to a 1 KiB block, SBO between blocks; the 32 bytes of a step stay inside a row
        if (start % 128 + 32 > 128) return false;
        end = start - start % 128 + (rows / 8 - 1) * sbo + 1024;
    } else {                                 // unswizzled: 128-byte core matrices, LBO between them along the contraction, SBO along the rows
        end = start + (rows / 8 - 1) * sbo + lbo + 128;
    }
    return start >= 0 && end <= image_bytes;
}
// Decodes what the self-test kernels rely on from an instruction descriptor; false for anything else.
bool selftest_idesc(uint32_t idesc, int max_m, int *M, int *N, bool *a_mn, bool *b_mn) {
    *N = (int)((idesc >> 17) & 0x3fu) << 3;
    *M = (int)((idesc >> 24) & 0x1fu) << 4;
    *a_mn = (idesc >> 15) & 1u;
    *b_mn = (idesc >> 16) & 1u;
    if ((idesc & ~((0x3fu << 17) | (0x1fu << 24) | (1u << 15) | (1u << 16))) != (1u << 4)) return false;   // fp16 x fp16 -> fp32 only
    return *M == max_m && *N >= 16 && *N <= 256 && *N % 16 == 0;
}
}  // namespace

VS_EXPORT int vs_selftest_mma(const void *image, int image_bytes, const uint64_t *descs_host, int n_mma,
                              uint32_t idesc, int ncols, float fill, float *out, void *stream) {
    if (!image || !descs_host || !out) return VS_ERR_NULL;
    if (image_bytes <= 0 || image_bytes > 128 * 1024 || n_mma < 1 || n_mma > 64) return VS_ERR_SHAPE;
    if (ncols < 8 || ncols > tcselftest::kTmemCols || ncols % 8 != 0) return VS_ERR_SHAPE;
    if (!aligned16(image)) return VS_ERR_ALIGN;
    int M, N;
    bool a_mn, b_mn;
    if (!selftest_idesc(idesc, 128, &M, &N, &a_mn, &b_mn) || N > ncols) return VS_ERR_SHAPE;
    for (int i = 0; i < n_mma; ++i)
        if (!selftest_operand_fits(descs_host[2 * i], M, a_mn, image_bytes) || !selftest_operand_fits(descs_host[2 * i + 1], N, b_mn, image_bytes))
            return VS_ERR_SHAPE;
    DeviceInfo *d;
    int rc = device_info(&d);
    if (rc != VS_OK) return rc;
    const int smem = ((image_bytes + 15) & ~15) + 16 + 1024;
    rc = set_smem(tcselftest::sandbox_kernel, smem);
    if (rc != VS_OK) return rc;
    tcselftest::DescList descs;
    std::memcpy(descs.d, descs_host, sizeof(uint64_t) * 2 * n_mma);
    tcselftest::sandbox_kernel<<<1, 128, smem, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const uint8_t *>(image), image_bytes, descs, n_mma, idesc, ncols, fill, out, d->status);
    return (int)cudaGetLastError();
}

VS_EXPORT int vs_selftest_mma_pair(const void *image0, const void *image1, int image_bytes, const uint64_t *descs_host,
                                   int n_mma, uint32_t idesc, int ncols, float fill, float *out, void *stream) {
    if (!image0 || !image1 || !descs_host || !out) return VS_ERR_NULL;
    if (image_bytes <= 0 || image_bytes > 128 * 1024 || n_mma < 1 || n_mma > 64) return VS_ERR_SHAPE;
    if (ncols < 8 || ncols > tcselftest::kPairTmemCols || ncols % 8 != 0) return VS_ERR_SHAPE;
    if (!aligned16(image0) || !aligned16(image1)) return VS_ERR_ALIGN;
    int M, N;
    bool a_mn, b_mn;
    if (!selftest_idesc(idesc, 256, &M, &N, &a_mn, &b_mn) || N > ncols || N % 32 != 0) return VS_ERR_SHAPE;
    for (int i = 0; i < n_mma; ++i)   // per CTA: 128 rows of A, N / 2 columns of B
        if (!selftest_operand_fits(descs_host[2 * i], 128, a_mn, image_bytes) || !selftest_operand_fits(descs_host[2 * i + 1], N / 2, b_mn, image_bytes))
            return VS_ERR_SHAPE;
    DeviceInfo *d;
    int rc = device_info(&d);
    if (rc != VS_OK) return rc;
    const int smem = ((image_bytes + 15) & ~15) + 16 + 1024;
    rc = set_smem(tcselftest::sandbox_pair_kernel, smem);
    if (rc != VS_OK) return rc;
    tcselftest::DescList descs;
    std::memcpy(descs.d, descs_host, sizeof(uint64_t) * 2 * n_mma);
    return (int)launch_pairs(tcselftest::sandbox_pair_kernel, 1, 128, (size_t)smem, static_cast<cudaStream_t>(stream), false,
                             static_cast<const uint8_t *>(image0), static_cast<const uint8_t *>(image1), image_bytes, descs, n_mma,
                             idesc, ncols, fill, out, d->status);
}
