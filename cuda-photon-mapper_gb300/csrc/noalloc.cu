// noalloc.cu -- k-nearest-neighbour queries over caller-provided points
// without any device allocation.
//
// Some callers of this library cannot call cudaMalloc: code that runs
// inside another framework's memory pool or stream-ordered allocator and
// must not step outside it, plug-ins whose host forbids device allocation
// after start-up, and real-time loops that may not risk an allocation
// stall or failure mid-frame. pm_knn_noalloc serves them: the caller
// passes only inputs and outputs, and the temporary memory the kd-tree
// build needs (the tree-ordered copy of the points, node boxes, counts)
// lives in one file-scope device array of fixed size.
//
// That array exists once per device for the life of the process (every GPU
// that loads the library holds it until exit). All calls share it and it
// keeps the last call's contents; each call overwrites everything it
// reads, so nothing has to start at zero. Calls that overlap on the GPU
// (different streams, or different host threads on the same device) race
// on the array and must be serialised by the caller.
#include <cuda.h>

#include <mutex>

#include "gather.cuh"
#include "kdtree.cuh"
#include "launch_count.cuh"
#include "pm.h"

namespace pm {
namespace {

constexpr uint32_t kMaxPoints = PM_KNN_NOALLOC_MAX_POINTS;
constexpr int kMaxDevices = 64;

// Byte layout of the scratch array (each part 256-byte aligned): the points
// with their index, their tree order, the node boxes, the build's scratch.
constexpr size_t align256(size_t b) { return (b + 255) & ~(size_t)255; }
constexpr size_t kNodes = (size_t)2 << 12;  // tree_nodes(kMaxPoints): depth 12 for 2^17 points
constexpr size_t kOffIpos = 0;
constexpr size_t kOffTpos = kOffIpos + align256(16 * kMaxPoints);
constexpr size_t kOffLo = kOffTpos + align256(16 * kMaxPoints);
constexpr size_t kOffHi = kOffLo + align256(16 * kNodes);
constexpr size_t kOffBuild = kOffHi + align256(16 * kNodes);
constexpr size_t kScratchBytes = PM_KNN_NOALLOC_SCRATCH_BYTES;
static_assert(kOffBuild < kScratchBytes, "the build's scratch needs the rest of the array");

__device__ __align__(256) unsigned char g_scratch[kScratchBytes];

// The scratch array's device address per device, valid for the CUDA
// context it was looked up in.
struct ScratchAddr {
    CUcontext ctx;
    unsigned char *addr;
};
std::mutex g_mu;
ScratchAddr g_addr[kMaxDevices] = {};
using CtxGetCurrentFn = CUresult (*)(CUcontext *);
CtxGetCurrentFn g_ctx_get_current = nullptr;

// Device address of g_scratch on the current device. In host code
// `g_scratch` names a host-side stand-in, not device memory, so kernels get
// this address instead. It is looked up (cudaGetSymbolAddress, with the
// device current) on the first call on each device, and again whenever the
// current context differs from the one it was looked up in (after a
// cudaDeviceReset, or under a context the caller made current through the
// driver API): an address from another context is not this one's memory.
cudaError_t scratch_address(unsigned char **out) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lk(g_mu);
    if (!g_ctx_get_current) {
        void *fn = nullptr;
        cudaDriverEntryPointQueryResult q;
        e = cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &fn, 12000, cudaEnableDefault, &q);
        if (e != cudaSuccess) return e;
        if (q != cudaDriverEntryPointSuccess || !fn) return cudaErrorSymbolNotFound;
        g_ctx_get_current = (CtxGetCurrentFn)fn;
    }
    CUcontext ctx = nullptr;
    if (g_ctx_get_current(&ctx) != CUDA_SUCCESS) return cudaErrorDeviceUninitialized;
    ScratchAddr &slot = g_addr[dev];
    if (!ctx || !slot.addr || slot.ctx != ctx) {
        // also makes the device's primary context current when no context is
        void *p = nullptr;
        e = cudaGetSymbolAddress(&p, g_scratch);
        if (e != cudaSuccess) return e;
        if (g_ctx_get_current(&ctx) != CUDA_SUCCESS || !ctx) return cudaErrorDeviceUninitialized;
        slot.addr = (unsigned char *)p;
        slot.ctx = ctx;
    }
    *out = slot.addr;
    return cudaSuccess;
}

constexpr int kPrepThreads = 256;

// Copies the points with their index in .w (the tie-break key) and combines
// their bounding box into the build's root box words (nullable; finite
// coordinates only, as the build's own boxes). Maxima of order-preserving
// words do not depend on the order they are taken in.
__global__ void __launch_bounds__(kPrepThreads) prepare_kernel(const float4 *__restrict__ pts, uint32_t n,
                                                               float4 *ipos, uint32_t *box) {
    __shared__ uint32_t red[6];
    if (threadIdx.x < 6) red[threadIdx.x] = 0u;
    __syncthreads();
    const uint32_t i = blockIdx.x * kPrepThreads + threadIdx.x;
    uint32_t w[6] = {0u, 0u, 0u, 0u, 0u, 0u};
    if (i < n) {
        const float4 p = pts[i];
        ipos[i] = make_float4(p.x, p.y, p.z, __uint_as_float(i));
        const float c[3] = {p.x, p.y, p.z};
#pragma unroll
        for (int a = 0; a < 3; ++a)
            if (isfinite(c[a])) {
                w[a] = ~kd_flip(c[a]);
                w[3 + a] = kd_flip(c[a]);
            }
    }
    if (!box) return;
#pragma unroll
    for (int a = 0; a < 6; ++a) {
        const uint32_t v = __reduce_max_sync(0xffffffffu, w[a]);
        if ((threadIdx.x & 31) == 0) atomicMax(&red[a], v);
    }
    __syncthreads();
    if (threadIdx.x < 6) atomicMax(&box[threadIdx.x], red[threadIdx.x]);
}

}  // namespace
}  // namespace pm

using namespace pm;

extern "C" pm_status pm_knn_noalloc(const float4 *points, uint32_t n, const float4 *queries,
                                    uint32_t nq, int k, float radius, uint32_t *idx_out,
                                    float *d2_out, cudaStream_t stream) {
    if (n > kMaxPoints) return PM_ERR_LIMIT;
    if (k < 1 || k > 128 || !(radius > 0.0f)) return PM_ERR_INVALID;
    if ((n && !points) || (nq && (!queries || !idx_out || !d2_out))) return PM_ERR_INVALID;
    unsigned char *base = nullptr;
    if (scratch_address(&base) != cudaSuccess) {
        cudaGetLastError();
        return PM_ERR_CUDA;
    }
    float4 *ipos = (float4 *)(base + kOffIpos);
    float4 *tpos = (float4 *)(base + kOffTpos);
    float4 *lo = (float4 *)(base + kOffLo);
    float4 *hi = (float4 *)(base + kOffHi);
    MapView m{};
    m.pos = tpos;
    m.pow = nullptr;
    m.lo = lo;
    m.hi = hi;
    m.n = n;
    m.depth = tree_depth(n);
    if (n > 0) {
        KdBuildArgs a;
        a.n = n;
        a.lo = make_float3(0.f, 0.f, 0.f);
        a.hi = make_float3(0.f, 0.f, 0.f);
        a.root_boxed = true;
        a.pos_in = ipos;
        a.pos_out = tpos;
        a.node_lo = lo;
        a.node_hi = hi;
        void *build = base + kOffBuild;
        if (kd_scratch_bytes(&a.n, &a.leaf_shift, 1) > kScratchBytes - kOffBuild) return PM_ERR_LIMIT;
        cudaError_t e = kd_clear_scratch(a, build, stream);
        if (e == cudaSuccess) {
            prepare_kernel<<<(n + kPrepThreads - 1) / kPrepThreads, kPrepThreads, 0, stream>>>(
                points, n, ipos, kd_root_box_words(a, build));
            note_launch();
            e = build_trees(&a, 1, build, stream);
        }
        if (e != cudaSuccess) {
            cudaGetLastError();
            return PM_ERR_CUDA;
        }
    }
    if (knn_query(m, 1, queries, nq, k, radius, idx_out, d2_out, stream) != cudaSuccess) {
        cudaGetLastError();
        return PM_ERR_CUDA;
    }
    return PM_OK;
}
