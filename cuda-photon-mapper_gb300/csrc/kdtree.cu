// kdtree.cu -- photon-map kd-tree build.
//
// Implicit left-balanced kd-tree: node i has children 2i and 2i+1, leaves
// hold L = 32 << leaf_shift consecutive records (one or more warp-wide
// loads) at depth D, and the node at level l covers records
// [j*L*2^(D-l), (j+1)*L*2^(D-l)) of the final order (j = its index within
// the level), so no child pointers or ranges are stored.
//
// Top-down. A node is split at its median along the longest axis of its
// records' bounding box (the root: of the scene box): the coordinate is
// quantised to 16 bits of that box, a histogram over its upper bits finds the
// bin holding the median -- and one over the lower bits the part of that bin,
// where the bin holds more of the node than an even spread would put there --
// and one stable partition moves the records below that bin (or part) to the
// left child, those above it to the right, and its own records left until the
// left child is full, in their present order. The layout is therefore
// deterministic. It does not affect a query's result: the boxes that are
// tested are the exact bounds of each node's records.
//
// Nodes of more than 32,768 records take three launches per level over tiles
// of kTile records: bins and histogram, per-tile counts, partition (which
// also collects the children's boxes). Smaller nodes are split by a cluster
// of 8 CTAs in its shared memory, down to nodes of at most kSubMax records,
// and each of those is finished by one CTA: the remaining levels, the
// records and directions in tree order and the boxes of all its nodes; the
// last CTA of a map to finish combines the boxes of the nodes above.
//
// Against sorting every level (two 8-bit radix passes over 12-byte pairs
// and a key pass), a level moves each record once, 16 B read and written,
// and its 2-byte key three times. Measured (GB300, both maps): 2 x 8M records
// 15.7 -> 3.03 ms, 2 x 1M 2.75 -> 0.36 ms, 2 x 100,000 1.46 -> 0.10 ms, one map
// of 20,011 0.44 -> 0.06 ms (half of it in one clump: 0.074).
#include "launch_count.cuh"
#include "kdtree.cuh"

#include <algorithm>
#include <cooperative_groups.h>
#include <cstring>

namespace pm {
namespace {

constexpr uint32_t kFull = 0xffffffffu;

constexpr uint32_t kKeys = 65536;  // values of a split coordinate

// Split levels. 1024 bins: the records of the median's bin that go left by
// their order alone are 1/1024 of the node's extent thick, a few percent of
// a leaf's width at the root of an 8M-record map of even density, and less
// below; 4 KB of shared histogram. A bin that holds more than 1/64 of its node
// (16 times the even share) is cut into its 64 key values: the children of a
// node with a dense clump would overlap in the clump, level after level. Leaves
// within reach of a k = 100 query in a clump of 0.0003 of the box that holds a
// fifth of 262,144 records: 34.6 by 1024 bins alone, 16.2 (a clump of 0.0001
// with half of them: 120 and 19.9; even density 15.9 both; limits of 1/16 to
// 1/256 the same within 2 %); 65,536 such queries 2.91 -> 0.72 ms (5.09 -> 1.54).
constexpr int kBins = 1024;
constexpr int kSub = (int)kKeys / kBins, kSubShift = 6;
constexpr int kRow = kBins + kSub;     // words of a node's histograms
constexpr uint32_t kCrowd = 64;        // a bin of more than a node's records / kCrowd
static_assert(kSub == 1 << kSubShift && kSub == 64, "two values of a bin a lane");
constexpr uint32_t kTile = 4096;
constexpr int kTileThreads = 512;
constexpr int kTileWarps = kTileThreads / 32;
constexpr int kTileItems = (int)(kTile / kTileThreads);

// Subtrees.
constexpr int kSubMax = 2048;
// Split levels of a cluster of 8 CTAs, a tile of records each.
constexpr int kMidLevels = 4;
constexpr int kMidCtas = (kSubMax << kMidLevels) / (int)kTile;
static_assert(kMidCtas == 8, "the portable cluster size");
constexpr int kSubThreads = 512;
constexpr int kSubWarps = kSubThreads / 32;
constexpr int kSubItems = kSubMax / kSubThreads;
constexpr int kSubBins = 256;           // each of 256 key values
constexpr uint32_t kSubCrowd = 16;
constexpr uint32_t kMark = 0x80000000u;  // of a crowded bin
constexpr int kWarpSpan = kSubMax / kSubWarps;   // records of a warp: nodes this small are split by one warp
constexpr int kSubLeaves = kSubMax / 32;
static_assert(kWarpSpan == 128, "the warp-level splits sort 4 records per lane");

// Up to two maps as a kernel parameter.
struct Maps2 {
    KdMap m[2];
    int n;
    __device__ __forceinline__ const KdMap &of_tile(uint32_t t) const { return m[n > 1 && t >= m[1].tile0 ? 1 : 0]; }
    __device__ __forceinline__ const KdMap &of_mid(uint32_t c) const { return m[n > 1 && c >= m[1].mid0 ? 1 : 0]; }
    __device__ __forceinline__ const KdMap &of_sub(uint32_t b) const { return m[n > 1 && b >= m[1].sub0 ? 1 : 0]; }
};
// Any number of maps in device memory.
struct MapsN {
    const KdMap *m;
    const uint32_t *tile_map, *sub_first;
    int n;
    __device__ __forceinline__ const KdMap &of_tile(uint32_t t) const { return m[tile_map[t]]; }
    __device__ __forceinline__ const KdMap &of_mid(uint32_t c) const {
        int lo = 0, hi = n - 1;  // the last map whose first cluster <= c
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (m[mid].mid0 <= c) lo = mid; else hi = mid - 1;
        }
        return m[lo];
    }
    __device__ __forceinline__ const KdMap &of_sub(uint32_t b) const {
        int lo = 0, hi = n - 1;  // the last map whose first subtree <= b
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (sub_first[mid] <= b) lo = mid; else hi = mid - 1;
        }
        return m[lo];
    }
};

__device__ __forceinline__ float coord(float4 p, int a) { return a == 0 ? p.x : (a == 1 ? p.y : p.z); }

// Box words of a coordinate (kd_root_box_words): zero for a value that is
// not finite, which the box leaves out.
__device__ __forceinline__ uint32_t min_word(float x) { return isfinite(x) ? ~kd_flip(x) : 0u; }
__device__ __forceinline__ uint32_t max_word(float x) { return isfinite(x) ? kd_flip(x) : 0u; }

// Lane a's value is the warp's maximum of w[a] (a < N): one addition to a box
// then takes one atomic of N lanes.
template <int N>
__device__ __forceinline__ uint32_t box_lane(const uint32_t (&w)[N], int lane) {
    uint32_t mine = 0u;
#pragma unroll
    for (int a = 0; a < N; ++a) {
        const uint32_t x = __reduce_max_sync(0xffffffffu, w[a]);
        if (lane == a) mine = x;
    }
    return mine;
}

// The split axis, the box's lower side along it and key values per unit
// length. A box without finite records, or of no extent, gives every record
// key 0.
struct Cut {
    int axis;
    float lo, inv;
};
__device__ __forceinline__ Cut cut_of(float3 lo, float3 hi) {
    const float ex = hi.x - lo.x, ey = hi.y - lo.y, ez = hi.z - lo.z;
    Cut c;
    c.axis = (ex >= ey && ex >= ez) ? 0 : (ey >= ez ? 1 : 2);
    c.lo = c.axis == 0 ? lo.x : (c.axis == 1 ? lo.y : lo.z);
    const float e = c.axis == 0 ? ex : (c.axis == 1 ? ey : ez);
    c.inv = e > 0.0f ? (float)kKeys / e : 0.0f;
    return c;
}
__device__ __forceinline__ Cut cut_of_words(const uint32_t *w) {
    return cut_of(make_float3(kd_unflip(~w[0]), kd_unflip(~w[1]), kd_unflip(~w[2])),
                  make_float3(kd_unflip(w[3]), kd_unflip(w[4]), kd_unflip(w[5])));
}
// The key of a record. NaN and everything below the box: 0; +inf and above:
// the last.
__device__ __forceinline__ uint32_t key_of(const Cut &c, float4 p) {
    const float f = (coord(p, c.axis) - c.lo) * c.inv;
    return !(f > 0.0f) ? 0u : (f >= (float)(kKeys - 1u) ? kKeys - 1u : (uint32_t)f);
}
constexpr uint32_t kNoKey = 2u * kKeys - 1u;  // of no record: in no bin, beyond every key

// A node's split: its records with keys below lo (there are `less`) go first,
// then those with keys from lo to lo + span (`equal` of them), then the others,
// each in their present order. The left child ends among the middle ones.
struct Split {
    uint32_t lo, span, less, equal;
    // the place in the node of a record at pos, lb and eb of those before it
    // being below and in the middle
    __device__ __forceinline__ uint32_t place(bool below, bool middle, uint32_t pos, uint32_t lb, uint32_t eb) const {
        return below ? lb : (middle ? less + eb : less + equal + (pos - lb - eb));
    }
};

// The part of the median's bin that holds the median: lane l has the records
// a and b of the bin's values 2l and 2l + 1. less are below the bin.
__device__ __forceinline__ Split split_bin(uint32_t bin, uint32_t less, uint32_t half, uint32_t a, uint32_t b,
                                           int lane) {
    uint32_t incl = a + b;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(kFull, incl, o);
        if (lane >= o) incl += t;
    }
    const uint32_t before = less + incl - a - b;
    const unsigned at = __ballot_sync(kFull, before <= half && half < before + a + b);
    const int src = __ffs(at) - 1;  // one lane: half is within the bin's records
    const bool second = half >= before + a;
    Split sp;
    sp.lo = (bin << kSubShift) + 2u * (uint32_t)src + __shfl_sync(kFull, second ? 1u : 0u, src);
    sp.span = 0u;
    sp.less = __shfl_sync(kFull, second ? before + a : before, src);
    sp.equal = __shfl_sync(kFull, second ? b : a, src);
    return sp;
}
// The split at a whole bin.
__device__ __forceinline__ Split split_at(uint4 thr) {
    return Split{thr.x << kSubShift, (uint32_t)kSub - 1u, thr.y, thr.z};
}

// The buffer a split level reads: level 0 the input, then the partner
// buffer and the output in turn (level l writes the partner when l is even).
__device__ __forceinline__ const float4 *level_src(const KdMap &m, int l) {
    return l == 0 ? m.pos : ((l & 1) ? m.tmp : m.pos_out);
}
__device__ __forceinline__ float4 *level_dst(const KdMap &m, int l) { return (l & 1) ? m.pos_out : m.tmp; }

struct TileNode {
    uint32_t start, cnt;        // the tile's records within the map
    uint32_t nstart, ncnt, half;  // its node's
    uint32_t node;              // node words index
};
__device__ __forceinline__ TileNode tile_node(const KdMap &m, uint32_t t, int l) {
    TileNode n;
    const uint32_t span = (32u << m.leaf_shift) << (m.depth - l);
    n.start = (t - m.tile0) * kTile;
    n.cnt = min(kTile, m.n - n.start);
    const uint32_t j = n.start / span;
    n.nstart = j * span;
    n.ncnt = min(span, m.n - n.nstart);
    n.half = min(span >> 1, n.ncnt);
    n.node = m.node0 + (1u << l) + j;
    return n;
}

// Launch 1 of a split level: every record's key, and the node's histogram.
// Bound by the records' read (16 B each): 32 us for 8M records.
template <class Maps>
__global__ void __launch_bounds__(kTileThreads)
    kd_hist_kernel(const __grid_constant__ Maps maps, int level, const uint32_t *box, uint32_t *hist) {
    __shared__ uint32_t h[kBins];
    const KdMap &m = maps.of_tile(blockIdx.x);
    const TileNode n = tile_node(m, blockIdx.x, level);
    for (int i = threadIdx.x; i < kBins; i += kTileThreads) h[i] = 0;
    const Cut c = level == 0 && !m.root_boxed ? cut_of(m.root_lo, m.root_hi)
                                              : cut_of_words(box + 8 * (size_t)n.node);
    const float4 *src = level_src(m, level) + n.start;
    uint16_t *keys = m.keys + n.start;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kTileItems; ++i) {
        const uint32_t r = (uint32_t)i * kTileThreads + threadIdx.x;
        uint32_t b = kBins;
        if (r < n.cnt) {
            const uint32_t key = key_of(c, src[r]);
            keys[r] = (uint16_t)key;
            b = key >> kSubShift;
        }
        // records of one wall share a bin: one addition for a warp of them
        int all;
        __match_all_sync(kFull, b, &all);
        if (all) {
            if ((threadIdx.x & 31) == 0 && b < kBins) atomicAdd(&h[b], 32u);
        } else if (b < kBins) {
            atomicAdd(&h[b], 1u);
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < kBins; i += kTileThreads)
        if (h[i]) atomicAdd(&hist[(size_t)n.node * kRow + i], h[i]);
}

// Launch 2: the node's bin (every tile of the node finds the same one; its
// first tile writes it for launch 3) and the tile's records below the
// median's bin and in it: 12 us for 8M records (their keys, 2 B each). thr:
// {bin, records below it, its records}. Where the bin is crowded, also the
// bin's records by their key: the node's counts beside its histogram, and the
// tile's up to each of them.
__device__ __forceinline__ bool crowded(uint4 thr, uint32_t ncnt) { return (uint64_t)thr.z * kCrowd > ncnt; }

template <class Maps>
__global__ void __launch_bounds__(kTileThreads)
    kd_count_kernel(const __grid_constant__ Maps maps, int level, uint32_t *hist, uint4 *thr,
                    uint2 *tile_cnt, uint32_t *tile_sub) {
    constexpr int kPer = kBins / kTileThreads;
    __shared__ uint32_t wsum[kTileWarps];
    __shared__ uint4 split;
    __shared__ uint32_t sub[kSub];
    const KdMap &m = maps.of_tile(blockIdx.x);
    const TileNode n = tile_node(m, blockIdx.x, level);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t key[kTileItems];
#pragma unroll
    for (int i = 0; i < kTileItems; ++i) {
        const uint32_t r = (uint32_t)i * kTileThreads + threadIdx.x;
        key[i] = r < n.cnt ? m.keys[n.start + r] : kNoKey;
    }
    uint32_t v[kPer], s = 0;
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
        v[i] = hist[(size_t)n.node * kRow + threadIdx.x * kPer + i];
        s += v[i];
    }
    if (threadIdx.x == 0) split = make_uint4(kBins, n.ncnt, 0u, 0u);  // no right child: all below
    if (threadIdx.x < kSub) sub[threadIdx.x] = 0u;
    uint32_t incl = s;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(kFull, incl, o);
        if (lane >= o) incl += t;
    }
    if (lane == 31) wsum[warp] = incl;
    __syncthreads();
    const uint32_t before = __reduce_add_sync(kFull, lane < warp ? wsum[lane] : 0u);
    uint32_t run = before + incl - s;
    if (n.ncnt > n.half) {
#pragma unroll
        for (int i = 0; i < kPer; ++i) {
            if (run <= n.half && n.half < run + v[i])
                split = make_uint4(threadIdx.x * kPer + i, run, v[i], 0u);
            run += v[i];
        }
    }
    __syncthreads();
    const uint32_t tb = split.x;
    const bool crowd = crowded(split, n.ncnt);
    if (threadIdx.x == 0 && n.start == n.nstart) thr[n.node] = split;
    uint32_t less = 0, eq = 0;
#pragma unroll
    for (int i = 0; i < kTileItems; ++i) {
        less += key[i] >> kSubShift < tb ? 1u : 0u;
        eq += key[i] >> kSubShift == tb ? 1u : 0u;
    }
    if (crowd) {
#pragma unroll
        for (int i = 0; i < kTileItems; ++i) {  // records of one wall share a key too
            int all;
            __match_all_sync(kFull, key[i], &all);
            if (key[i] >> kSubShift == tb && (!all || lane == 0))
                atomicAdd(&sub[key[i] & (kSub - 1u)], all ? 32u : 1u);
        }
    }
    const uint32_t both = __reduce_add_sync(kFull, less | (eq << 16));  // at most 256 each
    __syncthreads();
    if (lane == 0) wsum[warp] = both;
    __syncthreads();
    if (warp == 0) {
        // 16-bit halves hold at most kTile
        const uint32_t t = __reduce_add_sync(kFull, lane < kTileWarps ? wsum[lane] : 0u);
        if (lane == 0) tile_cnt[blockIdx.x] = make_uint2(t & 0xffffu, t >> 16);
        if (crowd) {
            const uint32_t a = sub[2 * lane], b = sub[2 * lane + 1];
            uint32_t *node_sub = hist + (size_t)n.node * kRow + kBins;
            if (a) atomicAdd(&node_sub[2 * lane], a);
            if (b) atomicAdd(&node_sub[2 * lane + 1], b);
            uint32_t upto = a + b;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t x = __shfl_up_sync(kFull, upto, o);
                if (lane >= o) upto += x;
            }
            tile_sub[(size_t)blockIdx.x * (kSub / 2) + lane] = (upto - b) | (upto << 16);
        }
    }
}

// Launch 3: the stable partition. A warp moves 256 consecutive records; its
// first places come from the counts of the node's earlier tiles and of the
// block's earlier warps. Also the children's boxes when they are split
// again. Bound by the records' read and write (32 B each): 54 us for 8M
// records, 4.9 TB/s; the writes of a warp are runs of consecutive records.
template <class Maps>
__global__ void __launch_bounds__(kTileThreads)
    kd_split_kernel(const __grid_constant__ Maps maps, int level, const uint32_t *hist, const uint4 *thr,
                    const uint2 *tile_cnt, const uint32_t *tile_sub, uint32_t *box) {
    __shared__ uint32_t wcnt[kTileWarps], pre_l[kTileWarps], pre_e[kTileWarps];
    __shared__ uint32_t bb[12];
    const KdMap &m = maps.of_tile(blockIdx.x);
    const TileNode n = tile_node(m, blockIdx.x, level);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr int kPer = kTileItems;  // records per lane
    const uint32_t wfirst = n.start + (uint32_t)warp * (32u * kPer);
    const float4 *src = level_src(m, level);
    float4 *dst = level_dst(m, level);
    float4 p[kPer];
    uint32_t key[kPer];
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
        const uint32_t r = wfirst + 32u * i + lane;
        key[i] = r < m.n ? m.keys[r] : kNoKey;
        if (r < m.n) p[i] = src[r];
    }
    const uint4 bin = thr[n.node];
    const bool crowd = crowded(bin, n.ncnt);
    Split sp = split_at(bin);
    if (crowd) {
        const uint2 h = reinterpret_cast<const uint2 *>(hist + (size_t)n.node * kRow + kBins)[lane];
        sp = split_bin(bin.x, bin.y, n.half, h.x, h.y, lane);
    }
    const bool boxes = level + 1 < m.lf;  // split again, by launches or a cluster
    if (threadIdx.x < 12) bb[threadIdx.x] = 0u;
    // the node's earlier tiles
    uint32_t pl = 0, pe = 0;
    const uint32_t first = m.tile0 + n.nstart / kTile;
    for (uint32_t t = first + threadIdx.x; t < blockIdx.x; t += kTileThreads) {
        const uint2 c = tile_cnt[t];
        pl += c.x;
        if (crowd) {
            const uint16_t *u = reinterpret_cast<const uint16_t *>(tile_sub + (size_t)t * (kSub / 2));
            const uint32_t q = sp.lo & (kSub - 1u), below = q ? u[q - 1] : 0u;
            pl += below;
            pe += u[q] - below;
        } else {
            pe += c.y;
        }
    }
    pl = __reduce_add_sync(kFull, pl);
    pe = __reduce_add_sync(kFull, pe);
    if (lane == 0) {
        pre_l[warp] = pl;
        pre_e[warp] = pe;
    }
    uint32_t ml[kPer], me[kPer];
    uint32_t nl = 0, ne = 0;
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
        ml[i] = __ballot_sync(kFull, key[i] < sp.lo);
        me[i] = __ballot_sync(kFull, key[i] - sp.lo <= sp.span);
        nl += __popc(ml[i]);
        ne += __popc(me[i]);
    }
    if (lane == 0) wcnt[warp] = nl | (ne << 16);
    __syncthreads();
    uint32_t less, eq;
    {
        const uint32_t w = __reduce_add_sync(kFull, lane < warp ? wcnt[lane] : 0u);
        less = (w & 0xffffu) + __reduce_add_sync(kFull, lane < kTileWarps ? pre_l[lane] : 0u);
        eq = (w >> 16) + __reduce_add_sync(kFull, lane < kTileWarps ? pre_e[lane] : 0u);
    }
    const unsigned lt = (1u << lane) - 1u;
    uint32_t wl[6] = {0, 0, 0, 0, 0, 0}, wr[6] = {0, 0, 0, 0, 0, 0};
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
        const uint32_t r = wfirst + 32u * i + lane;
        if (r < m.n) {
            const uint32_t lb = less + __popc(ml[i] & lt), eb = eq + __popc(me[i] & lt);
            const bool is_l = (ml[i] >> lane) & 1u, is_e = (me[i] >> lane) & 1u;
            const uint32_t at = sp.place(is_l, is_e, r - n.nstart, lb, eb);
            const bool left = at < n.half;
            dst[n.nstart + at] = p[i];
            if (boxes) {
                const uint32_t c[6] = {min_word(p[i].x), min_word(p[i].y), min_word(p[i].z),
                                       max_word(p[i].x), max_word(p[i].y), max_word(p[i].z)};
#pragma unroll
                for (int a = 0; a < 6; ++a) {
                    if (left) wl[a] = max(wl[a], c[a]);
                    else wr[a] = max(wr[a], c[a]);
                }
            }
        }
        less += __popc(ml[i]);
        eq += __popc(me[i]);
    }
    if (!boxes) return;
    const uint32_t wb[12] = {wl[0], wl[1], wl[2], wl[3], wl[4], wl[5], wr[0], wr[1], wr[2], wr[3], wr[4], wr[5]};
    const uint32_t mine = box_lane(wb, lane);
    if (mine) atomicMax(&bb[lane], mine);
    __syncthreads();
    if (threadIdx.x < 12 && bb[threadIdx.x]) {
        const uint32_t j = n.node - m.node0, side = threadIdx.x / 6, a = threadIdx.x % 6;
        atomicMax(&box[8 * (size_t)(m.node0 + 2 * j + side) + a], bb[threadIdx.x]);
    }
}

struct MidScratch {
    float4 p[kTile];
    uint32_t hist[kBins];
    uint16_t key[kTile];
    uint32_t sub[2][kSub];  // the median's bin by its values where it is crowded: the node's, the earlier tiles'
    uint32_t box[2][6];  // a node's first CTA: its box, by the level's parity
    uint32_t bb[12];
    uint32_t wsum[kTileWarps], wcnt[kTileWarps], pre[kTileWarps];
    uint4 split;      // {lo, span, less, equal} of the node's split
    uint32_t earlier; // added to the earlier tiles' records below the split and in it (upper half)
};

extern __shared__ __align__(16) unsigned char mid_smem[];

// The split levels from a node of at most 32,768 records down to subtrees,
// by a cluster of 8 CTAs that hold a tile each: the same keys, medians and
// stable partition as the launches above (and so the same layout), with two
// cluster barriers a level in place of three launches. A CTA reads the
// node's other histograms in their shared memory and writes its records to
// their place there. Bound by latency: four levels of a small map in 23 us
// (launches: 19.5 us a level), of 2 x 8M records in 0.58 ms (0.82). Two CTAs
// an SM against one: 2 x 8M built in 3.30 / 3.64 ms, small maps the same;
// clusters of 16 CTAs and five levels: 100,000 records 5 us faster, 8M 0.3 ms
// slower.
template <class Maps>
__global__ void __cluster_dims__(kMidCtas, 1, 1) __launch_bounds__(kTileThreads, 2)
    kd_mid_kernel(const __grid_constant__ Maps maps, const uint32_t *box) {
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    MidScratch &ms = *reinterpret_cast<MidScratch *>(mid_smem);
    constexpr int kPer = kTileItems;          // records per lane
    constexpr int kBinPer = kBins / kTileThreads;
    const uint32_t id = blockIdx.x / kMidCtas;
    const KdMap &m = maps.of_mid(id);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned lt = (1u << lane) - 1u;
    const int q = (int)cluster.block_rank();
    const uint32_t c = id - m.mid0;
    const int levels = m.lf - m.ls;
    const uint32_t span0 = (uint32_t)kSubMax << levels;
    const uint32_t first = c * span0;          // the cluster's first record
    const uint32_t start = first + (uint32_t)q * kTile;
    const int cnt = q * (int)kTile < (int)span0 && start < m.n ? (int)min(kTile, m.n - start) : 0;
    const int wfirst = warp * 32 * kPer;
    float4 p[kPer];
    {
        const float4 *src = level_src(m, m.ls) + start;
#pragma unroll
        for (int i = 0; i < kPer; ++i)
            if (wfirst + 32 * i + lane < cnt) p[i] = src[wfirst + 32 * i + lane];
    }
    if (threadIdx.x < 12) (&ms.box[0][0])[threadIdx.x] = 0u;
    // zeroed before another CTA's records reach them: its first barrier
    for (int l = 0; l < levels; ++l) {
        const int span = (int)(span0 >> l), ctas = span / (int)kTile;
        const int f = q / ctas * ctas;          // the node's first CTA
        const uint32_t nstart = first + (uint32_t)f * kTile;
        const uint32_t ncnt = nstart < m.n ? min((uint32_t)span, m.n - nstart) : 0u;
        const uint32_t half = min((uint32_t)span >> 1, ncnt);
        const bool boxes = l + 1 < levels;
        Cut cut;
        if (l > 0) cut = cut_of_words(cluster.map_shared_rank(&ms.box[l & 1][0], f));
        else if (m.ls == 0 && !m.root_boxed) cut = cut_of(m.root_lo, m.root_hi);
        else cut = cut_of_words(box + 8 * (size_t)(m.node0 + (1u << m.ls) + c));
        for (int i = threadIdx.x; i < kBins; i += kTileThreads) ms.hist[i] = 0;
        if (threadIdx.x < 12) ms.bb[threadIdx.x] = 0u;
        if (threadIdx.x < 2 * kSub) (&ms.sub[0][0])[threadIdx.x] = 0u;
        __syncthreads();
#pragma unroll
        for (int i = 0; i < kPer; ++i) {
            const int at = wfirst + 32 * i + lane;
            uint32_t bin = kBins;
            if (at < cnt) {
                const uint32_t key = key_of(cut, p[i]);
                ms.key[at] = (uint16_t)key;
                bin = key >> kSubShift;
            }
            int all;
            __match_all_sync(kFull, bin, &all);
            if (all) {
                if (lane == 0 && bin < kBins) atomicAdd(&ms.hist[bin], 32u);
            } else if (bin < kBins) {
                atomicAdd(&ms.hist[bin], 1u);
            }
        }
        cluster.sync();  // histograms and keys complete; every record of the node is in registers
        uint32_t tot[kBinPer], pre[kBinPer], sum = 0;
#pragma unroll
        for (int i = 0; i < kBinPer; ++i) tot[i] = pre[i] = 0;
#pragma unroll 4
        for (int o = 0; o < ctas; ++o) {
            const uint2 v = reinterpret_cast<const uint2 *>(cluster.map_shared_rank(&ms.hist[0], f + o))[threadIdx.x];
            tot[0] += v.x;
            tot[1] += v.y;
            if (f + o < q) {
                pre[0] += v.x;
                pre[1] += v.y;
            }
        }
#pragma unroll
        for (int i = 0; i < kBinPer; ++i) sum += tot[i];
        if (threadIdx.x == 0) {
            ms.split = make_uint4(kKeys, 0u, ncnt, 0u);  // no right child: all below
            ms.earlier = 0u;
        }
        if (threadIdx.x < 6) ms.box[l & 1][threadIdx.x] = 0u;              // read before the barrier
        uint32_t incl = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(kFull, incl, o);
            if (lane >= o) incl += t;
        }
        if (lane == 31) ms.wsum[warp] = incl;
        __syncthreads();
        uint32_t run = __reduce_add_sync(kFull, lane < warp ? ms.wsum[lane] : 0u) + incl - sum;
        if (ncnt > half) {
#pragma unroll
            for (int i = 0; i < kBinPer; ++i) {
                if (run <= half && half < run + tot[i])
                    ms.split = make_uint4((threadIdx.x * kBinPer + i) << kSubShift, kSub - 1u, run, tot[i]);
                run += tot[i];
            }
        }
        __syncthreads();
        if (ms.split.w * kCrowd > ncnt) {
            // by the bin's values: each CTA reads the keys of all the node's,
            // without a barrier that the other nodes' CTAs would have to meet
            const uint32_t bin = ms.split.x >> kSubShift, below = ms.split.z;
#pragma unroll 1
            for (int o = f; o < f + ctas; ++o) {
                const uint32_t first_o = first + (uint32_t)o * kTile;
                const int n_o = first_o < m.n ? (int)min(kTile, m.n - first_o) - 8 * (int)threadIdx.x : 0;
                const uint4 w = reinterpret_cast<const uint4 *>(cluster.map_shared_rank(&ms.key[0], o))[threadIdx.x];
                const uint32_t k[4] = {w.x, w.y, w.z, w.w};
                uint32_t last = kNoKey, same = 0;  // a run of one key: records of one wall share it
#pragma unroll
                for (int i = 0; i < 9; ++i) {
                    const uint32_t v = i < 8 && i < n_o ? (k[(i >> 1) & 3] >> (16 * (i & 1))) & 0xffffu : kNoKey;
                    if (v != last && last >> kSubShift == bin) {
                        atomicAdd(&ms.sub[0][last & (kSub - 1u)], same);
                        if (o < q) atomicAdd(&ms.sub[1][last & (kSub - 1u)], same);
                    }
                    same = v == last ? same + 1u : 1u;
                    last = v;
                }
            }
            __syncthreads();
            if (warp == 0) {
                const Split sp = split_bin(bin, below, half, ms.sub[0][2 * lane], ms.sub[0][2 * lane + 1], lane);
                const uint32_t at = sp.lo & (kSub - 1u), x = 2u * lane, y = x + 1u, ex = ms.sub[1][x], ey = ms.sub[1][y];
                const uint32_t e = __reduce_add_sync(kFull, (x < at ? ex : (x == at ? 0u : 0u - (ex << 16))) +
                                                                (y < at ? ey : (y == at ? 0u : 0u - (ey << 16))) -
                                                                (x < at ? ex << 16 : 0u) - (y < at ? ey << 16 : 0u));
                if (lane == 0) {
                    ms.split = make_uint4(sp.lo, sp.span, sp.less, sp.equal);
                    ms.earlier = e;
                }
            }
            __syncthreads();
        }
        const Split sp{ms.split.x, ms.split.y, ms.split.z, ms.split.w};
        // records of the node's earlier tiles below the median's bin and in
        // it (at most 7 tiles of 4096: 16 bits each)
        uint32_t before = 0;
#pragma unroll
        for (int i = 0; i < kBinPer; ++i) {
            const uint32_t bin = threadIdx.x * kBinPer + i;
            before += bin < sp.lo >> kSubShift ? pre[i] : (bin == sp.lo >> kSubShift ? pre[i] << 16 : 0u);
        }
        before = __reduce_add_sync(kFull, before);
        uint32_t ml[kPer], me[kPer], own = 0;
#pragma unroll
        for (int i = 0; i < kPer; ++i) {
            const int at = wfirst + 32 * i + lane;
            const uint32_t key = at < cnt ? ms.key[at] : kNoKey;
            ml[i] = __ballot_sync(kFull, key < sp.lo);
            me[i] = __ballot_sync(kFull, key - sp.lo <= sp.span);
            own += __popc(ml[i]) | ((uint32_t)__popc(me[i]) << 16);
        }
        if (lane == 0) {
            ms.pre[warp] = before;
            ms.wcnt[warp] = own;
        }
        __syncthreads();
        uint32_t less, eq;
        {
            const uint32_t w = __reduce_add_sync(kFull, lane < warp ? ms.wcnt[lane] : 0u);
            const uint32_t t = __reduce_add_sync(kFull, lane < kTileWarps ? ms.pre[lane] : 0u) + ms.earlier;
            less = (w & 0xffffu) + (t & 0xffffu);
            eq = (w >> 16) + (t >> 16);
        }
        uint32_t wl[6] = {0, 0, 0, 0, 0, 0}, wr[6] = {0, 0, 0, 0, 0, 0};
#pragma unroll
        for (int i = 0; i < kPer; ++i) {
            const int r = wfirst + 32 * i + lane;
            if (r < cnt) {
                const uint32_t lb = less + __popc(ml[i] & lt), eb = eq + __popc(me[i] & lt);
                const bool is_l = (ml[i] >> lane) & 1u, is_e = (me[i] >> lane) & 1u;
                const uint32_t at = sp.place(is_l, is_e, (uint32_t)((q - f) * (int)kTile + r), lb, eb);
                const bool left = at < half;
                cluster.map_shared_rank(&ms.p[0], f + (int)(at / kTile))[at % kTile] = p[i];
                if (boxes) {
                    const uint32_t w[6] = {min_word(p[i].x), min_word(p[i].y), min_word(p[i].z),
                                           max_word(p[i].x), max_word(p[i].y), max_word(p[i].z)};
#pragma unroll
                    for (int a = 0; a < 6; ++a) {
                        if (left) wl[a] = max(wl[a], w[a]);
                        else wr[a] = max(wr[a], w[a]);
                    }
                }
            }
            less += __popc(ml[i]);
            eq += __popc(me[i]);
        }
        if (boxes) {
            const uint32_t wb[12] = {wl[0], wl[1], wl[2], wl[3], wl[4], wl[5], wr[0], wr[1], wr[2], wr[3], wr[4], wr[5]};
            const uint32_t mine = box_lane(wb, lane);
            if (mine) atomicMax(&ms.bb[lane], mine);
            __syncthreads();
            if (threadIdx.x < 12 && ms.bb[threadIdx.x]) {
                const int side = threadIdx.x / 6, a = threadIdx.x % 6;
                atomicMax(cluster.map_shared_rank(&ms.box[(l + 1) & 1][a], f + side * (ctas / 2)), ms.bb[threadIdx.x]);
            }
        }
        cluster.sync();  // records in place, boxes complete, histograms read
        if (boxes) {
#pragma unroll
            for (int i = 0; i < kPer; ++i)
                if (wfirst + 32 * i + lane < cnt) p[i] = ms.p[wfirst + 32 * i + lane];
        }
    }
    for (int r = threadIdx.x; r < cnt; r += kTileThreads) m.pos_out[start + r] = ms.p[r];
}

struct SubScratch {
    float4 p[kSubMax];
    union {
        struct {
            uint32_t hist[kSubMax / 256 * kSubBins];
            uint32_t bb[kSubMax / 256][6];
            uint4 thr[kSubMax / 256];
            uint32_t wcnt[kSubWarps];
        };
        struct {
            float4 lo[2 * kSubLeaves], hi[2 * kSubLeaves];
        } nb;
    };
    uint16_t ord[2][kSubMax];
    uint32_t last;
};

extern __shared__ __align__(16) unsigned char sub_smem[];

// Sorts 128 keys, element lane * 4 + r in k[r], ascending within blocks of
// kN (64 or 128) consecutive elements (bitonic; strides below 4 stay in the
// lane).
template <int kN>
__device__ __forceinline__ void warp_sort4(uint32_t (&k)[4], int lane) {
#pragma unroll
    for (int size = 2; size <= kN; size <<= 1) {
#pragma unroll
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            uint32_t o[4];
#pragma unroll
            for (int r = 0; r < 4; ++r)
                o[r] = stride >= 4 ? __shfl_xor_sync(kFull, k[r], stride >> 2) : k[r ^ (stride & 3)];
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const int e = lane * 4 + r;
                // the last merge of a block ascends whatever the block's place
                const bool up = size == kN || (e & size) == 0;
                k[r] = ((e & stride) == 0) == up ? min(k[r], o[r]) : max(k[r], o[r]);
            }
        }
    }
}

// The split of a warp's nodes of kN records (one of 128 or two of 64): its
// 128 places of ord from `base`, sorted along each node's longest axis by
// (16-bit coordinate, place).
template <int kN>
__device__ __forceinline__ void warp_split(SubScratch &ss, uint16_t *ord, int base, int cnt, int lane) {
    const unsigned mask = kN == 128 ? kFull : (lane < 16 ? 0x0000ffffu : 0xffff0000u);
    uint32_t w[6] = {0, 0, 0, 0, 0, 0};
    float4 p[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const int at = base + lane * 4 + r;
        if (at < cnt) {
            p[r] = ss.p[ord[at]];
            w[0] = max(w[0], min_word(p[r].x));
            w[1] = max(w[1], min_word(p[r].y));
            w[2] = max(w[2], min_word(p[r].z));
            w[3] = max(w[3], max_word(p[r].x));
            w[4] = max(w[4], max_word(p[r].y));
            w[5] = max(w[5], max_word(p[r].z));
        }
    }
#pragma unroll
    for (int a = 0; a < 6; ++a) w[a] = __reduce_max_sync(mask, w[a]);
    const Cut c = cut_of_words(w);
    uint32_t k[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const int e = lane * 4 + r;
        k[r] = base + e < cnt ? (key_of(c, p[r]) << 16) | (uint32_t)e : 0xffffff00u | (uint32_t)e;
    }
    warp_sort4<kN>(k, lane);
    // an empty place's key is above every record's, so the node's first
    // places keep holding its records
    uint16_t nw[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) nw[r] = base + lane * 4 + r < cnt ? ord[base + (int)(k[r] & 0x7fu)] : 0;
    __syncwarp();
#pragma unroll
    for (int r = 0; r < 4; ++r)
        if (base + lane * 4 + r < cnt) ord[base + lane * 4 + r] = nw[r];
    __syncwarp();
}

// The bin of a node's 256 (its row of the histograms, 8 consecutive bins a
// lane) that holds place `half`, `less` records lying below the row: {first +
// bin * step | mark, records below it, its records} into *thr by the lane that
// finds it, marked where it holds more than `many`. Returns (warp-uniform)
// whether it does.
__device__ __forceinline__ bool row_split(const uint32_t *row, uint32_t less, uint32_t half, uint32_t first,
                                          uint32_t step, uint32_t many, uint4 *thr, int lane) {
    uint32_t v[kSubBins / 32], s = 0;
#pragma unroll
    for (int i = 0; i < kSubBins / 32; i += 4) {
        const uint4 h = *reinterpret_cast<const uint4 *>(row + lane * (kSubBins / 32) + i);
        v[i] = h.x;
        v[i + 1] = h.y;
        v[i + 2] = h.z;
        v[i + 3] = h.w;
        s += (h.x + h.y) + (h.z + h.w);
    }
    uint32_t incl = s;
#pragma unroll
    for (int q = 1; q < 32; q <<= 1) {
        const uint32_t t = __shfl_up_sync(kFull, incl, q);
        if (lane >= q) incl += t;
    }
    uint32_t run = less + incl - s;
    bool crowd = false;
#pragma unroll
    for (int i = 0; i < kSubBins / 32; ++i) {
        if (run <= half && half < run + v[i]) {
            crowd = v[i] > many;
            *thr = make_uint4((first + (uint32_t)(lane * (kSubBins / 32) + i) * step) | (crowd ? kMark : 0u), run, v[i], 0u);
        }
        run += v[i];
    }
    return __any_sync(kFull, crowd);
}

// The crowded bins of a subtree's level: their records (keys b of this thread,
// node: this warp's, or -1) counted by the key's lower half, and the marked
// splits made by it (crowd: that of node `warp` is). Returns how many key
// values the middle of this warp's split has, less one. Out of line: the usual
// level keeps its registers.
__device__ __noinline__ uint32_t split_crowded(SubScratch &ss, int node, bool crowd, int span, int cnt, uint4 b) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t first = node >= 0 ? ss.thr[node].x : 0u;
    const uint32_t k[kSubItems] = {b.x, b.y, b.z, b.w};
    if (first & kMark) {
#pragma unroll
        for (int u = 0; u < kSubItems; ++u)
            if (k[u] >> 8 == (first & ~kMark) >> 8) atomicAdd(&ss.hist[node * kSubBins + (k[u] & 255u)], 1u);
    }
    __syncthreads();
    if (crowd) {
        const uint4 t = ss.thr[warp];
        const int half = min(span >> 1, cnt - warp * span);
        __syncwarp();
        row_split(&ss.hist[warp * kSubBins], t.y, (uint32_t)half, t.x & ~kMark, 1u, kKeys, &ss.thr[warp], lane);
    }
    __syncthreads();
    return first & kMark ? 0u : kSubBins - 1u;
}

// One subtree per CTA: the levels from a node of at most kSubMax records
// down to its leaves, the records in tree order and the boxes. Nodes of more
// than 128 records split as in the split levels, with a 256-bin shared
// histogram per node and five barriers per level (seven where a node's median
// lies in a bin of more than 1/16 of it, which is split by its 256 values);
// nodes of 128 and 64 are sorted by one warp in registers. Only the 2-byte
// places move; the records stay where they were loaded. Bound by latency
// (barriers, shared-memory round trips): 0.44 ms for 8M records (sorting every
// level of the subtree in shared memory: 2.27 ms), 28 us for a small map. 2 CTAs
// per SM at 64 registers (3 at 40, which spill: 0.50 ms and 31 us; 1: 8M slower
// by a quarter).
template <class Maps>
__global__ void __launch_bounds__(kSubThreads, 2) kd_finish_kernel(const __grid_constant__ Maps maps) {
    SubScratch &ss = *reinterpret_cast<SubScratch *>(sub_smem);
    const KdMap &m = maps.of_sub(blockIdx.x);
    const uint32_t j = blockIdx.x - m.sub0;
    const int leaf = 32 << m.leaf_shift;
    const int levels = m.depth - m.lf;          // below the subtree's root
    const int span0 = leaf << levels;
    const uint32_t start = j * (uint32_t)span0;
    const int cnt = start < m.n ? (int)min((uint32_t)span0, m.n - start) : 0;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const float inf = __int_as_float(0x7f800000);
    const float4 *src = m.lf == 0 ? m.pos : m.pos_out;
    for (int t = tid; t < cnt; t += kSubThreads) {
        ss.p[t] = src[start + t];
        ss.ord[0][t] = (uint16_t)t;
    }
    for (int i = tid; i < kSubMax / 256 * kSubBins; i += kSubThreads) ss.hist[i] = 0;
    for (int i = tid; i < kSubMax / 256 * 6; i += kSubThreads) (&ss.bb[0][0])[i] = 0;
    __syncthreads();
    int cur = 0, span = span0;
    for (; span > kWarpSpan && span > leaf; span >>= 1) {
        const int node = warp * kWarpSpan / span;
        const int nodes = (cnt + span - 1) / span;
        uint16_t o[kSubItems];
        float4 p[kSubItems];
        uint32_t w[6] = {0, 0, 0, 0, 0, 0};
#pragma unroll
        for (int u = 0; u < kSubItems; ++u) {
            const int at = warp * kWarpSpan + u * 32 + lane;
            if (at < cnt) {
                o[u] = ss.ord[cur][at];
                p[u] = ss.p[o[u]];
                w[0] = max(w[0], min_word(p[u].x));
                w[1] = max(w[1], min_word(p[u].y));
                w[2] = max(w[2], min_word(p[u].z));
                w[3] = max(w[3], max_word(p[u].x));
                w[4] = max(w[4], max_word(p[u].y));
                w[5] = max(w[5], max_word(p[u].z));
            }
        }
        if (warp * kWarpSpan < cnt) {
            const uint32_t mine = box_lane(w, lane);
            if (mine) atomicMax(&ss.bb[node][lane], mine);
        }
        __syncthreads();
        uint32_t b[kSubItems];
        if (warp * kWarpSpan < cnt) {
            const Cut c = cut_of_words(ss.bb[node]);
#pragma unroll
            for (int u = 0; u < kSubItems; ++u) {
                b[u] = kNoKey;
                if (warp * kWarpSpan + u * 32 + lane < cnt) {
                    b[u] = key_of(c, p[u]);
                    atomicAdd(&ss.hist[node * kSubBins + (b[u] >> 8)], 1u);
                }
            }
        }
        __syncthreads();
        // one warp per node; its split at a whole bin, or (crowded) the bin's
        // records counted by their key's lower half and split there
        bool crowd = false;
        if (warp < nodes) {
            const int ncnt = min(span, cnt - warp * span), half = min(span >> 1, ncnt);
            uint32_t *row = &ss.hist[warp * kSubBins];
            if (ncnt == half) {  // no right child: all below
                if (lane == 0) ss.thr[warp] = make_uint4(kKeys, (uint32_t)ncnt, 0u, 0u);
            } else {
                crowd = row_split(row, 0u, (uint32_t)half, 0u, 256u, (uint32_t)ncnt / kSubCrowd, &ss.thr[warp], lane);
            }
            if (crowd) {
#pragma unroll
                for (int i = 0; i < kSubBins; i += 32) row[i + lane] = 0u;
            }
        }
        uint32_t wide = kSubBins - 1u;  // the split's keys
        if (__syncthreads_or(crowd))
            wide = split_crowded(ss, warp * kWarpSpan < cnt ? node : -1, crowd, span, cnt, make_uint4(b[0], b[1], b[2], b[3]));
        uint32_t ml[kSubItems], me[kSubItems], tot = 0;
        uint4 sp = make_uint4(0u, 0u, 0u, 0u);
        if (warp * kWarpSpan < cnt) {
            sp = ss.thr[node];
#pragma unroll
            for (int u = 0; u < kSubItems; ++u) {
                ml[u] = __ballot_sync(kFull, b[u] < sp.x);
                me[u] = __ballot_sync(kFull, b[u] - sp.x <= wide);
                tot += __popc(ml[u]) | ((uint32_t)__popc(me[u]) << 16);
            }
        }
        if (lane == 0) ss.wcnt[warp] = tot;
        for (int i = 4 * tid; i < kSubMax / 256 * kSubBins; i += 4 * kSubThreads)
            *reinterpret_cast<uint4 *>(&ss.hist[i]) = make_uint4(0u, 0u, 0u, 0u);
        for (int i = tid; i < kSubMax / 256 * 6; i += kSubThreads) (&ss.bb[0][0])[i] = 0;
        __syncthreads();
        if (warp * kWarpSpan < cnt) {
            const int nwarp = node * span / kWarpSpan;  // the node's first warp
            const uint32_t pre = __reduce_add_sync(kFull, lane >= nwarp && lane < warp ? ss.wcnt[lane] : 0u);
            uint32_t less = pre & 0xffffu, eq = pre >> 16;
            const unsigned lt = (1u << lane) - 1u;
#pragma unroll
            for (int u = 0; u < kSubItems; ++u) {
                const int at = warp * kWarpSpan + u * 32 + lane;
                if (at < cnt) {
                    const bool lower = (ml[u] >> lane) & 1u, middle = (me[u] >> lane) & 1u;
                    const uint32_t lb = less + __popc(ml[u] & lt), eb = eq + __popc(me[u] & lt);
                    const uint32_t to = lower ? lb : (middle ? sp.y + eb : sp.y + sp.z + ((uint32_t)(at - node * span) - lb - eb));
                    ss.ord[cur ^ 1][node * span + (int)to] = o[u];
                }
                less += __popc(ml[u]);
                eq += __popc(me[u]);
            }
        }
        __syncthreads();
        cur ^= 1;
    }
    uint16_t *ord = ss.ord[cur];
    const int base = warp * kWarpSpan;
    if (base < cnt) {
        if (span == 128 && span > leaf) {
            warp_split<128>(ss, ord, base, cnt, lane);
            span = 64;
        }
        if (span == 64 && span > leaf) warp_split<64>(ss, ord, base, cnt, lane);
    }
    __syncthreads();
    // the records in tree order
    for (int t = tid; t < cnt; t += kSubThreads) {
        const float4 p = ss.p[ord[t]];
        m.pos_out[start + t] = p;
        if (m.pow) {
            const float4 pw = __ldg(&m.pow[__float_as_uint(p.w)]);
            m.pow_out[start + t] = pw;
            if (m.dir_out) {
                const v3 d = oct_decode(__float_as_uint(pw.w));
                m.dir_out[start + t] = make_float4(d.x, d.y, d.z, 0.0f);
            }
        }
    }
    // boxes: the leaves (empty ones inverted), then each level above
    const int leaves = 1 << levels;
    const uint32_t root = (1u << m.lf) + j;
    for (int f = warp; f < leaves; f += kSubWarps) {
        float lx = inf, ly = inf, lz = inf, hx = -inf, hy = -inf, hz = -inf;
        for (int c = 0; c < (1 << m.leaf_shift); ++c) {
            const int t = f * leaf + c * 32 + lane;
            if (t < cnt) {
                const float4 p = ss.p[ord[t]];
                lx = fminf(lx, p.x); ly = fminf(ly, p.y); lz = fminf(lz, p.z);
                hx = fmaxf(hx, p.x); hy = fmaxf(hy, p.y); hz = fmaxf(hz, p.z);
            }
        }
        const float4 lo = make_float4(kd_unflip(__reduce_min_sync(kFull, kd_flip(lx))),
                                      kd_unflip(__reduce_min_sync(kFull, kd_flip(ly))),
                                      kd_unflip(__reduce_min_sync(kFull, kd_flip(lz))), 0.0f);
        const float4 hi = make_float4(kd_unflip(__reduce_max_sync(kFull, kd_flip(hx))),
                                      kd_unflip(__reduce_max_sync(kFull, kd_flip(hy))),
                                      kd_unflip(__reduce_max_sync(kFull, kd_flip(hz))), 0.0f);
        if (lane == 0) {
            ss.nb.lo[leaves + f] = lo;
            ss.nb.hi[leaves + f] = hi;
        }
    }
    __syncthreads();
    for (int l = levels - 1; l >= 0; --l) {
        for (int i = tid; i < (1 << l); i += kSubThreads) {
            const int nd = (1 << l) + i;
            const float4 a = ss.nb.lo[2 * nd], b = ss.nb.lo[2 * nd + 1];
            const float4 c = ss.nb.hi[2 * nd], d = ss.nb.hi[2 * nd + 1];
            ss.nb.lo[nd] = make_float4(fminf(a.x, b.x), fminf(a.y, b.y), fminf(a.z, b.z), 0.0f);
            ss.nb.hi[nd] = make_float4(fmaxf(c.x, d.x), fmaxf(c.y, d.y), fmaxf(c.z, d.z), 0.0f);
        }
        __syncthreads();
    }
    for (int i = tid + 1; i < 2 * leaves; i += kSubThreads) {
        const int d = 31 - __clz(i);
        const uint32_t g = (root << d) + (uint32_t)(i - (1 << d));
        m.lo[g] = ss.nb.lo[i];
        m.hi[g] = ss.nb.hi[i];
    }
    if (m.lf == 0) return;
    // the last subtree of the map to get here combines the nodes above
    __threadfence();
    __syncthreads();
    if (tid == 0) ss.last = atomicAdd(m.done, 1u) == (1u << m.lf) - 1u ? 1u : 0u;
    __syncthreads();
    if (!ss.last) return;
    __threadfence();
    for (int l = m.lf - 1; l >= 0; --l) {
        for (uint32_t i = tid; i < (1u << l); i += kSubThreads) {
            const uint32_t nd = (1u << l) + i;
            const float4 a = __ldcg(&m.lo[2 * nd]), b = __ldcg(&m.lo[2 * nd + 1]);
            const float4 c = __ldcg(&m.hi[2 * nd]), d = __ldcg(&m.hi[2 * nd + 1]);
            __stcg(&m.lo[nd], make_float4(fminf(a.x, b.x), fminf(a.y, b.y), fminf(a.z, b.z), 0.0f));
            __stcg(&m.hi[nd], make_float4(fmaxf(c.x, d.x), fmaxf(c.y, d.y), fmaxf(c.z, d.z), 0.0f));
        }
        __syncthreads();
    }
}

template <class Maps>
__global__ void __launch_bounds__(kTileThreads) kd_pad_kernel(const __grid_constant__ Maps maps) {
    const KdMap &m = maps.of_tile(blockIdx.x);
    if (!m.pad_count) return;
    const uint32_t first = (blockIdx.x - m.tile0) * kTile, from = *m.pad_count;
    const float inf = __int_as_float(0x7f800000);
    for (uint32_t r = first + threadIdx.x; r < min(first + kTile, m.n); r += kTileThreads)
        if (r >= from) {
            const_cast<float4 *>(m.pos)[r] = make_float4(inf, inf, inf, __uint_as_float(r));
            const_cast<float4 *>(m.pow)[r] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        }
}

// The first level whose nodes hold at most kSubMax records.
int first_finish_level(int depth, uint32_t leaf) {
    int lf = depth;
    while (lf > 0 && ((uint64_t)leaf << (depth - (lf - 1))) <= (uint64_t)kSubMax) --lf;
    return lf;
}

uint32_t tiles_of(uint32_t n) { return (n + kTile - 1) / kTile; }

size_t align256(size_t b) { return (b + 255) & ~(size_t)255; }

// The level from which a map's nodes are split by clusters.
int mid_level(int lf) { return std::max(lf - kMidLevels, 0); }

// Scratch layout of a set of maps: the words zeroed by each build
// (histograms, boxes, finished-subtree counters), the splits, the tiles'
// counts, then the keys and the partner buffer of every map.
struct Layout {
    uint32_t tiles = 0, subs = 0, nodes = 0;
    size_t hist = 0, box = 0, done = 0, clear = 0, thr = 0, tile_cnt = 0, tile_sub = 0, keys = 0, tmp = 0, total = 0;
};

Layout layout_of(const uint32_t *n, const int *leaf_shift, int maps) {
    Layout L;
    size_t records = 0;
    for (int i = 0; i < maps; ++i) {
        const int D = tree_depth(n[i], leaf_shift[i]);
        const int lf = first_finish_level(D, 32u << leaf_shift[i]);
        if (n[i] == 0) continue;
        L.tiles += tiles_of(n[i]);
        L.subs += 1u << lf;
        if (lf == 0) continue;  // one subtree: no scratch
        L.nodes += 2u << mid_level(lf);  // down to those the clusters split
        if (mid_level(lf) > 0) records += (n[i] + 127u) & ~(size_t)127u;
    }
    L.box = align256(L.hist + sizeof(uint32_t) * kRow * (size_t)L.nodes);
    L.done = align256(L.box + sizeof(uint32_t) * 8 * (size_t)L.nodes);
    L.clear = align256(L.done + sizeof(uint32_t) * (size_t)std::max(maps, 1));
    L.thr = L.clear;
    L.tile_cnt = align256(L.thr + sizeof(uint4) * (size_t)L.nodes);
    L.tile_sub = align256(L.tile_cnt + sizeof(uint2) * (size_t)L.tiles);
    L.keys = align256(L.tile_sub + sizeof(uint16_t) * kSub * (size_t)L.tiles);
    L.tmp = align256(L.keys + sizeof(uint16_t) * records);
    L.total = align256(L.tmp + sizeof(float4) * records);
    return L;
}

int finish_level_of(const KdBuildArgs &a) {
    return first_finish_level(tree_depth(a.n, a.leaf_shift), 32u << a.leaf_shift);
}

// The kernel descriptors of maps a[idx[0..count)) (in that order), all with
// records.
void describe(const KdBuildArgs *a, const int *idx, int count, const Layout &L, void *scratch, KdMap *out) {
    unsigned char *base = (unsigned char *)scratch;
    uint32_t tile = 0, sub = 0, node = 0, mid = 0;
    size_t rec = 0;
    for (int i = 0; i < count; ++i) {
        const KdBuildArgs &b = a[idx[i]];
        KdMap &m = out[i];
        memset(&m, 0, sizeof(m));
        m.pos = b.pos_in;
        m.pow = b.pow_in;
        m.pos_out = b.pos_out;
        m.pow_out = b.pow_out;
        m.dir_out = b.dir_out;
        m.lo = b.node_lo;
        m.hi = b.node_hi;
        m.done = (uint32_t *)(base + L.done) + i;
        m.pad_count = b.pad_count;
        m.root_lo = b.lo;
        m.root_hi = b.hi;
        m.root_boxed = b.root_boxed ? 1 : 0;
        m.n = b.n;
        m.depth = tree_depth(b.n, b.leaf_shift);
        m.leaf_shift = b.leaf_shift;
        m.lf = first_finish_level(m.depth, 32u << b.leaf_shift);
        m.ls = mid_level(m.lf);
        m.tile0 = tile;
        m.sub0 = sub;
        m.node0 = node;
        m.mid0 = mid;
        tile += tiles_of(b.n);
        sub += 1u << m.lf;
        if (m.lf > 0) {
            mid += 1u << m.ls;
            node += 2u << m.ls;
        }
        if (m.ls > 0) {
            m.tmp = (float4 *)(base + L.tmp) + rec;
            m.keys = (uint16_t *)(base + L.keys) + rec;
            rec += (b.n + 127u) & ~(size_t)127u;
        }
    }
}

template <class Maps>
cudaError_t launch_build(const Maps &maps, const KdMap *host, int count, uint32_t subs, uint32_t *hist,
                         uint32_t *box, uint4 *thr, uint2 *tile_cnt, uint32_t *tile_sub, cudaStream_t s) {
    for (int l = 0; l < host[0].ls; ++l) {
        // the maps split at this level come first
        uint32_t t = 0;
        for (int i = 0; i < count && host[i].ls > l; ++i) t = host[i].tile0 + tiles_of(host[i].n);
        kd_hist_kernel<Maps><<<t, kTileThreads, 0, s>>>(maps, l, box, hist);
        kd_count_kernel<Maps><<<t, kTileThreads, 0, s>>>(maps, l, hist, thr, tile_cnt, tile_sub);
        kd_split_kernel<Maps><<<t, kTileThreads, 0, s>>>(maps, l, hist, thr, tile_cnt, tile_sub, box);
        note_launches(3);
    }
    cudaError_t e;
    uint32_t mids = 0;
    for (int i = 0; i < count && host[i].lf > 0; ++i) mids = host[i].mid0 + (1u << host[i].ls);
    if (mids) {
        const int smem = (int)sizeof(MidScratch);
        e = cudaFuncSetAttribute(kd_mid_kernel<Maps>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return e;
        kd_mid_kernel<Maps><<<mids * kMidCtas, kTileThreads, smem, s>>>(maps, box);
        note_launch();
    }
    const int smem = (int)sizeof(SubScratch);
    e = cudaFuncSetAttribute(kd_finish_kernel<Maps>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    kd_finish_kernel<Maps><<<subs, kSubThreads, smem, s>>>(maps);
    note_launch();
    return cudaGetLastError();
}

}  // namespace

int tree_depth(uint32_t n, int leaf_shift) {
    const uint32_t leaf = 32u << leaf_shift;
    uint32_t leaves = (uint32_t)(((uint64_t)n + leaf - 1) / leaf);
    int d = 0;
    while ((1u << d) < leaves) ++d;
    return d;
}

size_t tree_nodes(uint32_t n, int leaf_shift) { return (size_t)2 << tree_depth(n, leaf_shift); }

size_t kd_scratch_bytes(const uint32_t *n, const int *leaf_shift, int maps) {
    return layout_of(n, leaf_shift, maps).total;
}

namespace {
Layout layout_of_args(const KdBuildArgs *a, int maps) {
    uint32_t n[2] = {a[0].n, maps > 1 ? a[1].n : 0u};
    int ls[2] = {a[0].leaf_shift, maps > 1 ? a[1].leaf_shift : 0};
    return layout_of(n, ls, maps);
}
}  // namespace

uint32_t *kd_root_box_words(const KdBuildArgs &a, void *scratch) {
    const Layout L = layout_of_args(&a, 1);
    return L.nodes ? (uint32_t *)((unsigned char *)scratch + L.box) + 8 : nullptr;
}

cudaError_t kd_clear_scratch(const KdBuildArgs &a, void *scratch, cudaStream_t s) {
    const Layout L = layout_of_args(&a, 1);
    return L.nodes ? cudaMemsetAsync(scratch, 0, L.clear, s) : cudaSuccess;
}

cudaError_t build_trees(const KdBuildArgs *a, int maps, void *scratch, cudaStream_t s) {
    if (maps < 1 || maps > 2 || (maps == 2 && a[0].root_boxed)) return cudaErrorInvalidValue;
    int idx[2], count = 0;  // the map with the most split levels first
    for (int i = 0; i < maps; ++i)
        if (a[i].n > 0) idx[count++] = i;
    if (count == 0) return cudaSuccess;
    if (count == 2 && finish_level_of(a[1]) > finish_level_of(a[0])) std::swap(idx[0], idx[1]);
    const Layout L = layout_of_args(a, maps);
    if (L.nodes && !a[0].root_boxed) {
        cudaError_t e = cudaMemsetAsync(scratch, 0, L.clear, s);
        if (e != cudaSuccess) return e;
    }
    Maps2 m;
    memset(&m, 0, sizeof(m));
    m.n = count;
    describe(a, idx, count, L, scratch, m.m);
    unsigned char *base = (unsigned char *)scratch;
    return launch_build(m, m.m, count, L.subs, (uint32_t *)(base + L.hist), (uint32_t *)(base + L.box),
                        (uint4 *)(base + L.thr), (uint2 *)(base + L.tile_cnt), (uint32_t *)(base + L.tile_sub), s);
}

namespace {
template <typename T>
cudaError_t kd_alloc(T **p, size_t count) {
    *p = nullptr;
    return cudaMalloc((void **)p, sizeof(T) * (count ? count : 1));
}
}  // namespace

cudaError_t kd_multi_create(const std::vector<KdBuildArgs> &args, KdMulti *k) {
    *k = KdMulti();
    std::vector<int> idx, shift;  // maps with records, those with the most split levels first
    std::vector<uint32_t> n;
    for (int i = 0; i < (int)args.size(); ++i) {
        n.push_back(args[i].n);
        shift.push_back(args[i].leaf_shift);
        if (args[i].n > 0) idx.push_back(i);
    }
    std::stable_sort(idx.begin(), idx.end(),
                     [&](int x, int y) { return finish_level_of(args[x]) > finish_level_of(args[y]); });
    const Layout L = layout_of(n.data(), shift.data(), (int)n.size());
    cudaError_t e;
#define KM_TRY(x) do { e = (x); if (e != cudaSuccess) { kd_multi_free(*k); return e; } } while (0)
    KM_TRY(cudaMalloc(&k->scratch, std::max<size_t>(L.total, 256)));
    k->nmaps = (int)idx.size();
    k->maps.resize(k->nmaps);
    describe(args.data(), idx.data(), k->nmaps, L, k->scratch, k->maps.data());
    k->tiles = L.tiles;
    k->subs = L.subs;
    k->clear_bytes = L.nodes ? L.clear : 0;
    unsigned char *base = (unsigned char *)k->scratch;
    k->hist = (uint32_t *)(base + L.hist);
    k->box = (uint32_t *)(base + L.box);
    k->thr = (uint4 *)(base + L.thr);
    k->tile_cnt = (uint2 *)(base + L.tile_cnt);
    k->tile_sub = (uint32_t *)(base + L.tile_sub);
    std::vector<uint32_t> tile_map(std::max<uint32_t>(L.tiles, 1), 0), sub_first(k->nmaps + 1, 0);
    for (int i = 0; i < k->nmaps; ++i) {
        const KdMap &m = k->maps[i];
        for (uint32_t t = 0; t < tiles_of(m.n); ++t) tile_map[m.tile0 + t] = (uint32_t)i;
        sub_first[i] = m.sub0;
        if (m.pad_count) k->pad = true;
    }
    sub_first[k->nmaps] = L.subs;
    KM_TRY(kd_alloc(&k->desc, k->nmaps));
    KM_TRY(kd_alloc(&k->tile_map, tile_map.size()));
    KM_TRY(kd_alloc(&k->sub_first, sub_first.size()));
    if (k->nmaps) KM_TRY(cudaMemcpy(k->desc, k->maps.data(), sizeof(KdMap) * k->nmaps, cudaMemcpyHostToDevice));
    KM_TRY(cudaMemcpy(k->tile_map, tile_map.data(), sizeof(uint32_t) * tile_map.size(), cudaMemcpyHostToDevice));
    KM_TRY(cudaMemcpy(k->sub_first, sub_first.data(), sizeof(uint32_t) * sub_first.size(), cudaMemcpyHostToDevice));
#undef KM_TRY
    return cudaSuccess;
}

void kd_multi_free(KdMulti &k) {
    cudaFree(k.desc); cudaFree(k.tile_map); cudaFree(k.sub_first); cudaFree(k.scratch);
    k = KdMulti();
}

cudaError_t kd_multi_build(KdMulti &k, cudaStream_t s) {
    if (k.nmaps == 0) return cudaSuccess;
    MapsN m;
    m.m = k.desc;
    m.tile_map = k.tile_map;
    m.sub_first = k.sub_first;
    m.n = k.nmaps;
    if (k.clear_bytes) {
        cudaError_t e = cudaMemsetAsync(k.scratch, 0, k.clear_bytes, s);
        if (e != cudaSuccess) return e;
    }
    if (k.pad) {
        kd_pad_kernel<MapsN><<<k.tiles, kTileThreads, 0, s>>>(m);
        note_launch();
    }
    return launch_build(m, k.maps.data(), k.nmaps, k.subs, k.hist, k.box, k.thr, k.tile_cnt, k.tile_sub, s);
}

}  // namespace pm
