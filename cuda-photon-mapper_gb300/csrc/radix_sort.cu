// radix_sort.cu -- stable LSD radix sort and single-CTA exclusive scan.
#include "launch_count.cuh"
#include "radix_sort.cuh"

namespace pm {
namespace {

constexpr int kScanThreads = 1024;

__device__ __forceinline__ uint32_t lanemask_lt() {
    return (1u << (threadIdx.x & 31)) - 1u;
}

// Block-wide exclusive scan of one value per thread; returns this thread's
// prefix and writes the block total to *total. blockDim.x is a multiple of 32.
__device__ uint32_t block_exclusive_scan(uint32_t v, uint32_t *warp_sums, uint32_t *total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    uint32_t incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
    }
    if (lane == 31) warp_sums[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        uint32_t w = lane < nwarps ? warp_sums[lane] : 0u;
        uint32_t wi = w;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            uint32_t t = __shfl_up_sync(0xffffffffu, wi, o);
            if (lane >= o) wi += t;
        }
        if (lane < nwarps) warp_sums[lane] = wi - w;
        if (lane == 31) *total = wi;
    }
    __syncthreads();
    uint32_t r = warp_sums[warp] + incl - v;
    __syncthreads();
    return r;
}

__global__ void __launch_bounds__(kScanThreads) scan_kernel(const uint32_t *in, uint32_t *out,
                                                            uint32_t n, uint32_t *total_out) {
    __shared__ uint32_t warp_sums[32];
    __shared__ uint32_t total;
    const uint32_t per = (n + blockDim.x - 1) / blockDim.x;
    const uint32_t lo = threadIdx.x * per;
    const uint32_t hi = min(n, lo + per);
    uint32_t s = 0;
    for (uint32_t i = lo; i < hi; ++i) s += in[i];
    uint32_t run = block_exclusive_scan(s, warp_sums, &total);
    for (uint32_t i = lo; i < hi; ++i) {
        uint32_t v = in[i];
        out[i] = run;
        run += v;
    }
    if (threadIdx.x == 0 && total_out) *total_out = total;
}

constexpr int kSortWarps = kSortThreads / 32;

// The block's sum of v, on every thread.
__device__ __forceinline__ uint32_t block_sum(uint32_t v, uint32_t *warp_sums) {
    const int lane = threadIdx.x & 31;
    const uint32_t w = __reduce_add_sync(0xffffffffu, v);
    if (lane == 0) warp_sums[threadIdx.x >> 5] = w;
    __syncthreads();
    const uint32_t r = __reduce_add_sync(0xffffffffu, lane < kSortWarps ? warp_sums[lane] : 0u);
    __syncthreads();
    return r;
}

// Per-tile sums for the large scan (tile = kSortTile elements).
__global__ void __launch_bounds__(kSortThreads) tile_sum_kernel(const uint32_t *in, uint32_t n,
                                                                uint32_t *sums) {
    __shared__ uint32_t warp_sums[kSortWarps];
    const uint32_t base = blockIdx.x * kSortTile;
    uint32_t s = 0;
#pragma unroll
    for (int i = 0; i < kSortItems / 4; ++i) {
        const uint4 v = load_words4(in, base + 4 * ((uint32_t)i * kSortThreads + threadIdx.x), n);
        s += v.x + v.y + v.z + v.w;
    }
    s = block_sum(s, warp_sums);
    if (threadIdx.x == 0) sums[blockIdx.x] = s;
}

// A tile's scan, its first value from the tiles before it: offs holds their
// scan, or (raw) the tiles' sums, which the block adds up itself. With
// seg_tab (per tile: the first tile of its segment, the segment's tiles) each
// segment's scan starts at 0: the tile's offset less that of its segment's
// first tile. A warp scans 512 consecutive elements, 128 at a time in 16-byte
// loads and stores. Bound by them: 88M words 2 x 0.35 GB in 96 us (one thread
// per 16 consecutive words: 380).
__global__ void __launch_bounds__(kSortThreads) tile_scan_kernel(const uint32_t *in, uint32_t *out,
                                                                 uint32_t n, const uint32_t *offs, bool raw,
                                                                 uint32_t *total_out, const uint2 *seg_tab) {
    __shared__ uint32_t warp_sums[kSortWarps];
    constexpr int kRounds = kSortItems / 4;
    const bool aligned = (reinterpret_cast<uintptr_t>(out) & 15u) == 0;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t base = blockIdx.x * kSortTile + (uint32_t)warp * (32u * kSortItems) + 4u * lane;
    uint4 v[kRounds];
#pragma unroll
    for (int r = 0; r < kRounds; ++r) v[r] = load_words4(in, base + 128u * r, n);
    uint32_t first;
    if (raw) {
        uint32_t s = 0;
        for (uint32_t t = threadIdx.x; t < blockIdx.x; t += kSortThreads) s += offs[t];
        first = block_sum(s, warp_sums);
    } else {
        first = offs[blockIdx.x];
        if (seg_tab) first -= offs[seg_tab[blockIdx.x].x];
    }
    uint32_t pre[kRounds], run = 0;  // of this lane's words within the warp's
#pragma unroll
    for (int r = 0; r < kRounds; ++r) {
        const uint32_t s = v[r].x + v[r].y + v[r].z + v[r].w;
        uint32_t incl = s;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += t;
        }
        pre[r] = run + incl - s;
        run += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (lane == 0) warp_sums[warp] = run;
    __syncthreads();
    const uint32_t all = lane < kSortWarps ? warp_sums[lane] : 0u;
    first += __reduce_add_sync(0xffffffffu, lane < warp ? all : 0u);
    if (total_out && blockIdx.x == gridDim.x - 1 && threadIdx.x == kSortThreads - 1) *total_out = first + run;
#pragma unroll
    for (int r = 0; r < kRounds; ++r) {
        const uint32_t i = base + 128u * r, a = first + pre[r];
        const uint4 o = make_uint4(a, a + v[r].x, a + v[r].x + v[r].y, a + v[r].x + v[r].y + v[r].z);
        if (aligned && i + 4 <= n) {
            *reinterpret_cast<uint4 *>(out + i) = o;
        } else {
            if (i < n) out[i] = o.x;
            if (i + 1 < n) out[i + 1] = o.y;
            if (i + 2 < n) out[i + 2] = o.z;
            if (i + 3 < n) out[i + 3] = o.w;
        }
    }
}

// The launches of a scan of n words over its tiles, their sums in tmp. Up to
// kRawTiles tiles each block adds up the sums before its own (16 KB at most)
// instead of a launch of their scan.
constexpr uint32_t kRawTiles = 4096;
void scan_tiles(const uint32_t *in, uint32_t *out, uint32_t n, uint32_t *total, uint32_t *tmp, const uint2 *seg_tab,
                bool pooled, cudaStream_t stream) {
    const uint32_t tiles = scan_tile_count(n);
    const bool raw = !pooled && tiles <= kRawTiles;
    tile_sum_kernel<<<tiles, kSortThreads, 0, stream>>>(in, n, tmp); note_launch();
    if (!raw) {
        scan_kernel<<<1, kScanThreads, 0, stream>>>(tmp, tmp, tiles, total); note_launch();
    }
    tile_scan_kernel<<<tiles, kSortThreads, 0, stream>>>(in, out, n, tmp, raw, raw ? total : nullptr, seg_tab);
    note_launch();
}

// Position of the (digit d, tile t) count in the scanned array: digit-major;
// with seg_tab (per tile: its segment's first tile and tiles) segments one
// after another, digit-major inside a segment, so that the scan keeps every
// segment's items inside the segment.
__device__ __forceinline__ uint32_t count_at(uint32_t d, uint32_t t, uint32_t ntiles, const uint2 *seg_tab) {
    if (seg_tab) {
        const uint2 e = seg_tab[t];
        return e.x * 256u + d * e.y + (t - e.x);
    }
    return d * ntiles + t;
}

// A tile's digit counts: bound by latency in short sorts (5 tiles: 11 -> 4.7 us
// with the tile's loads issued together, 16 bytes each).
__global__ void __launch_bounds__(kSortThreads) hist_kernel(const uint32_t *keys, const uint32_t *n_dev,
                                                            int shift, uint32_t *hist,
                                                            uint32_t ntiles, const uint2 *seg_tab) {
    __shared__ uint32_t h[256];
    h[threadIdx.x] = 0;
    __syncthreads();
    const uint32_t n = *n_dev;
    const uint32_t base = blockIdx.x * kSortTile;
    uint4 v[kSortItems / 4];  // all loads in flight before the first count
#pragma unroll
    for (int i = 0; i < kSortItems / 4; ++i)
        v[i] = load_words4(keys, base + 4u * ((uint32_t)i * kSortThreads + threadIdx.x), n);
#pragma unroll
    for (int i = 0; i < kSortItems / 4; ++i) {
        const uint32_t idx = base + 4u * ((uint32_t)i * kSortThreads + threadIdx.x);
        if (idx < n) atomicAdd(&h[(v[i].x >> shift) & 255u], 1u);
        if (idx + 1 < n) atomicAdd(&h[(v[i].y >> shift) & 255u], 1u);
        if (idx + 2 < n) atomicAdd(&h[(v[i].z >> shift) & 255u], 1u);
        if (idx + 3 < n) atomicAdd(&h[(v[i].w >> shift) & 255u], 1u);
    }
    __syncthreads();
    hist[count_at(threadIdx.x, blockIdx.x, ntiles, seg_tab)] = h[threadIdx.x];
}

// A warp ranks its own 512 consecutive items of the tile against its own
// digit counters (no block barrier inside; the lanes of a digit by a ballot per
// bit); one pass over the warps' counters and a scan of the digits turn the
// ranks into places in the tile's sorted order, in which the keys and then the
// values are staged in the same shared memory, so that each digit's run leaves
// in consecutive writes. Bound by those writes: a run averages 64 bytes.
// Measured, four passes over the queries of a 512 x 512 frame: 301 us (the
// digit's lanes by match, 480; with both staged at once, 360; tiles of 8,192,
// 437); 41M pairs 396 -> 282 us a pass, 5 tiles 10 us (unstaged: 732, 30).
__global__ void __launch_bounds__(kSortThreads) scatter_kernel(
    const uint32_t *keys_in, const uint32_t *vals_in, uint32_t *keys_out, uint32_t *vals_out,
    const uint32_t *n_dev, int shift, const uint32_t *offs, uint32_t ntiles,
    const uint2 *seg_tab) {
    constexpr int kWarps = kSortThreads / 32;
    __shared__ uint32_t wcnt[kWarps][256];
    __shared__ uint32_t sk[kSortTile];
    __shared__ uint32_t gofs[256], warp_sums[32], total;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t n = *n_dev;
    if (blockIdx.x * kSortTile >= n) return;
    const uint32_t base = blockIdx.x * kSortTile + (uint32_t)warp * (32u * kSortItems) + (uint32_t)lane;
    uint32_t k[kSortItems], rank[kSortItems];
#pragma unroll
    for (int r = 0; r < kSortItems; ++r) k[r] = base + 32u * r < n ? keys_in[base + 32u * r] : 0u;
#pragma unroll
    for (int i = 0; i < 8; ++i) wcnt[warp][32 * i + lane] = 0u;
    __syncwarp();
#pragma unroll
    for (int r = 0; r < kSortItems; ++r) {
        const bool valid = base + 32u * r < n;
        const uint32_t d = valid ? ((k[r] >> shift) & 255u) : 256u;
        uint32_t peers = __ballot_sync(0xffffffffu, valid);
        if (!valid) peers = ~peers;
#pragma unroll
        for (int b = 0; b < 8; ++b) {
            const uint32_t set = __ballot_sync(0xffffffffu, (d >> b) & 1u);
            peers &= (d >> b) & 1u ? set : ~set;
        }
        const uint32_t before = valid ? wcnt[warp][d] : 0u;
        rank[r] = before + __popc(peers & lanemask_lt());
        __syncwarp();
        if (valid && (peers & lanemask_lt()) == 0u) wcnt[warp][d] = before + __popc(peers);
        __syncwarp();
    }
    __syncthreads();
    {
        // digit threadIdx.x: its items in the tile, its place among the
        // digits, the warps in order, and what takes a place to the output
        uint32_t c[kWarps], sum = 0;
#pragma unroll
        for (int w = 0; w < kWarps; ++w) {
            c[w] = wcnt[w][threadIdx.x];
            sum += c[w];
        }
        uint32_t run = block_exclusive_scan(sum, warp_sums, &total);
        gofs[threadIdx.x] = offs[count_at(threadIdx.x, blockIdx.x, ntiles, seg_tab)] - run;
#pragma unroll
        for (int w = 0; w < kWarps; ++w) {
            wcnt[w][threadIdx.x] = run;
            run += c[w];
        }
    }
    __syncthreads();
    uint32_t v[kSortItems];
#pragma unroll
    for (int r = 0; r < kSortItems; ++r)
        if (base + 32u * r < n) {
            rank[r] += wcnt[warp][(k[r] >> shift) & 255u];
            sk[rank[r]] = k[r];
            v[r] = vals_in[base + 32u * r];
        }
    __syncthreads();
    const uint32_t cnt = min((uint32_t)kSortTile, n - blockIdx.x * kSortTile);
    uint32_t to[kSortItems];
#pragma unroll
    for (int r = 0; r < kSortItems; ++r) {
        const uint32_t t = (uint32_t)r * kSortThreads + threadIdx.x;
        if (t < cnt) {
            const uint32_t key = sk[t];
            to[r] = gofs[(key >> shift) & 255u] + t;
            keys_out[to[r]] = key;
        }
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kSortItems; ++r)
        if (base + 32u * r < n) sk[rank[r]] = v[r];
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kSortItems; ++r) {
        const uint32_t t = (uint32_t)r * kSortThreads + threadIdx.x;
        if (t < cnt) vals_out[to[r]] = sk[t];
    }
}

}  // namespace

cudaError_t radix_sort_pairs_u32(uint32_t *keys, uint32_t *vals, uint32_t *keys_tmp, uint32_t *vals_tmp,
                                 const uint32_t *n_dev, uint32_t max_n, int begin_bit, int end_bit,
                                 uint32_t *hist, cudaStream_t stream, uint32_t **out_keys,
                                 uint32_t **out_vals, const uint2 *seg_tab) {
    uint32_t *kin = keys, *kout = keys_tmp;
    uint32_t *vin = vals, *vout = vals_tmp;
    uint32_t ntiles = (max_n + kSortTile - 1) / kSortTile;
    if (ntiles == 0) ntiles = 1;
    // The digit-count scan runs in three multi-CTA steps once the histogram
    // outgrows a few tiles (always for pooled segments, so that a pool's
    // launch sequence does not depend on its size); its tile partials live
    // past the histogram.
    const uint32_t hn = 256u * ntiles;
    uint32_t *partials = hist + hn;
    for (int shift = begin_bit; shift < end_bit; shift += 8) {
        hist_kernel<<<ntiles, kSortThreads, 0, stream>>>(kin, n_dev, shift, hist, ntiles, seg_tab); note_launch();
        if (hn <= kSortTile && !seg_tab) {
            scan_kernel<<<1, kScanThreads, 0, stream>>>(hist, hist, hn, nullptr); note_launch();
        } else {
            scan_tiles(hist, hist, hn, nullptr, partials, nullptr, seg_tab != nullptr, stream);
        }
        scatter_kernel<<<ntiles, kSortThreads, 0, stream>>>(kin, vin, kout, vout, n_dev, shift,
                                                               hist, ntiles, seg_tab); note_launch();
        uint32_t *tk = kin; kin = kout; kout = tk;
        uint32_t *tv = vin; vin = vout; vout = tv;
    }
    *out_keys = kin;
    *out_vals = vin;
    return cudaGetLastError();
}

uint32_t scan_tile_count(uint32_t n) {
    uint32_t t = (n + kSortTile - 1) / kSortTile;
    return t == 0 ? 1 : t;
}

cudaError_t exclusive_scan_u32_large(const uint32_t *in, uint32_t *out, uint32_t n,
                                     uint32_t *total, uint32_t *tmp, cudaStream_t stream) {
    if (n <= 65536) return exclusive_scan_u32(in, out, n, total, stream);
    scan_tiles(in, out, n, total, tmp, nullptr, false, stream);
    return cudaGetLastError();
}

cudaError_t exclusive_scan_u32_segmented(const uint32_t *in, uint32_t *out, uint32_t n, const uint2 *seg_tab,
                                         uint32_t *tmp, cudaStream_t stream) {
    if (n == 0) return cudaSuccess;
    scan_tiles(in, out, n, nullptr, tmp, seg_tab, true, stream);
    return cudaGetLastError();
}

cudaError_t exclusive_scan_u32(const uint32_t *in, uint32_t *out, uint32_t n, uint32_t *total,
                               cudaStream_t stream) {
    scan_kernel<<<1, kScanThreads, 0, stream>>>(in, out, n, total); note_launch();
    return cudaGetLastError();
}

}  // namespace pm
