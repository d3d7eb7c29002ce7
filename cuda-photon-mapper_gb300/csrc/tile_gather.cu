// tile_gather.cu -- k-NN radiance estimates of a query list in spatial
// order, one candidate set per group of neighbouring queries, and the k-NN
// queries of points (pm_knn) by the same search.
//
// A warp takes chunks of 1, 2 or 4 consecutive groups of 32 queries (where
// queries are few, one group of 8) of the (map, Hilbert code) order. The k-th-neighbour distance d(x) (capped at the
// gather radius) is 1-Lipschitz in the query position, so exact distances d_j
// at points x_j bound it everywhere: d(x) <= min_j (d_j + |x - x_j|). A
// chunk's first group is bounded by its middle query, which is answered by
// itself first (single_bound, alone), every later group by the exact results
// of the group before it. A group's records are found once in the kd-tree --
// every record within the largest upper bound of the group's bounding box --
// and held in registers, kSlots positions to a lane. A query computes its
// squared distances to all of them and searches for the threshold that
// exactly k of them lie at or below (select_k), starting from its
// predecessor's.
//
// A group whose set does not fit the registers, or is not expected to
// (expected), is processed in segments: halves, down to single queries, each
// finished segment tightening the bounds of the queries after it. A single
// query whose set does not fit finds a radius of its own. Queries of the
// other map in a mixed group, and any result that contradicts its own upper
// bound, are deferred to a list-search launch after the pass. The selected
// set is exactly the list search's (ties broken by photon index) and the
// estimate's sum is order-independent (knn_core.cuh), so every value is
// bit-identical to the list search's.
//
// Bound by instructions and the latency between them (64 % of the issue slots
// with 7 warps a scheduler on preset 2, 58 % on preset 3); the selected
// records' flux comes from L1 and L2. Candidates in registers
// instead of shared memory make a query's distances and counts straight-line
// code without loads, need no lists of the certain and the doubtful
// candidates, and leave most of the L1 to the flux. Estimate pass (GB300, ms,
// presets 1 / 2 / 3 at seed 0x5EED0003: 11.0M, 46.0M and 20.8M queries):
// candidates in shared memory, scanned, the band between two bounds ranked,
// 16.9 / 113.0 / 45.4; in registers 12.0 / 76.0 / 34.5; Hilbert instead of
// Morton order, a lane per channel for the last rounding 10.0 / 64.0 / 29.9;
// expected set sizes instead of failed collections 9.8 / 62.6 / 29.7; the first
// bound found in the pass instead of a launch before it, 10 candidates per lane
// 10.0 / 59.8 / 25.9; now 10.2 / 60.0 / 24.7.
#include <algorithm>

#include "cache.cuh"
#include "eye_path.cuh"
#include "knn_core.cuh"
#include "launch_count.cuh"
#include "phys_state.cuh"

namespace pm {
namespace {

using namespace wknn;

constexpr int kTileWarps = 4;
// Blocks of 4 warps per SM (registers capped at 72) and candidates per lane:
// more candidates let a set serve more queries, more warps hide latency.
// Presets 1 / 2 / 3 (ms): 7 blocks with 8 slots 11.7 / 65.3 / 27.9, 9 slots
// 10.9 / 63.5 / 27.2, 10 slots 10.0 / 59.8 / 25.9, 11 slots 10.6 / 60.2 /
// 26.2, 12 slots 10.3 / 68.7 / 29.0; 8 blocks with 9 slots 10.7 / 59.7 / 26.3,
// 6 blocks with 10 slots 10.4 / 64.0 / 26.8.
constexpr int kTileBlocks = 7;
constexpr int kSlots = 10;
constexpr int kTileCap = 32 * kSlots;        // candidate records per warp
constexpr uint32_t kKnnLeft = 0xfffffffeu;   // mark of a query left to knn_rest_kernel (no record's index)
constexpr float kRel = 2e-4f;                // relative and absolute margins of the distance bounds
constexpr float kAbs = 1e-6f;
constexpr float kOuter = 1.000001f;          // collected beyond a squared bound: above the bound's rounding

// per-launch counters (pm_get_gather_stats)
enum TileStat { kStTiled, kStList, kStShrunk, kStViolations, kStGroups, kStCandidates, kStHalvings, kStCount };

struct TileScratch {
    uint32_t cat[kTileCap + kTileCap / kSlots];  // tree positions of the candidates (cat_at)
    union {
        uint32_t stack[kStackCap];  // the collection's node stack
        uint32_t sel[128];          // tree positions of the k selected candidates
    };
    float4 qx[32];           // the group's queries: position, upper bound of the k-th distance
    float4 qd[32];           // weight direction, query index bits
    float4 known[32];        // exact distances that bound the group: point, distance
    unsigned long long st[kStCount];  // counters, lane 0
};

// Place of candidate c in cat: a lane's kSlots consecutive candidates, lanes
// an odd number of words apart.
__device__ __forceinline__ int cat_at(int c) { return c + c / kSlots; }

// The parameters of the scene a warp is working on (per warp: in a launch
// over many scenes the warps of one block may serve different scenes).
struct TileArgs {
    MapView map[2];  // surface, volume
    float4 *out;
    uint32_t *defer;     // deferred query indices
    uint32_t *defer_sc;  // their scenes (launches over many scenes; nullable)
    uint32_t *defer_n;   // their count
    uint32_t scene;      // the scene's index in such a launch
    uint64_t cap;        // key bound of the gather radius
    float r2cap, rcap, g;
    int k;
    bool raw;
};

extern __shared__ __align__(16) unsigned char tile_smem[];
__shared__ __align__(16) unsigned char tile_args[kTileWarps * sizeof(TileArgs)];

__device__ __forceinline__ TileArgs &targs() {
    return reinterpret_cast<TileArgs *>(tile_args)[threadIdx.x >> 5];
}

// Lane 0 fills the warp's arguments; the warp then synchronises.
__device__ __forceinline__ void set_targs(const MapView &surf, const MapView &vol, float4 *out,
                                          uint32_t *defer, uint32_t *defer_sc, uint32_t *defer_n,
                                          uint32_t scene, float r2cap, float g, int k, bool raw) {
    if ((threadIdx.x & 31) == 0) {
        TileArgs &t = targs();
        t.map[0] = surf;
        t.map[1] = vol;
        t.out = out;
        t.defer = defer;
        t.defer_sc = defer_sc;
        t.defer_n = defer_n;
        t.scene = scene;
        t.cap = make_key(r2cap, 0xffffffffu);
        t.r2cap = r2cap;
        t.rcap = sqrtf(r2cap);
        t.g = g;
        t.k = k;
        t.raw = raw;
    }
    __syncwarp();
}

__device__ __forceinline__ TileScratch &scratch() {
    return reinterpret_cast<TileScratch *>(tile_smem)[threadIdx.x >> 5];
}

struct Query {
    v3 x;
    v3 dirv;       // facing normal (surface) or view direction wo (volume)
    int map;       // 0 surface, 1 volume
    uint32_t out;  // query index (destination)
};

// One query of the list: position, the weight direction and its map.
__device__ __forceinline__ Query load_query(const PScene &Sc, const float4 *qa, const float4 *qd,
                                            uint32_t i) {
    Query q;
    const float4 a = qa[i], d = qd[i];
    const int obj = __float_as_int(a.w);
    q.x = mk3(a.x, a.y, a.z);
    const v3 wo = mk3(d.x, d.y, d.z);
    q.map = obj != kNone ? 0 : 1;
    q.dirv = obj != kNone ? facing_normal(Sc, obj, q.x, wo) : wo;
    q.out = i;
    return q;
}

// Minimum and maximum of a float over the warp (NaN only when all are).
__device__ __forceinline__ float warp_min(float v) {
    float r;
    asm volatile("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}
__device__ __forceinline__ float warp_max(float v) {
    float r;
    asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}
// The hardware's approximate square root, for distances that only bound or
// steer (the bounds' margins are far above its error).
__device__ __forceinline__ float approx_sqrt(float v) {
    float r;
    asm("sqrt.approx.f32 %0, %1;" : "=f"(r) : "f"(v));
    return r;
}

// How far v lies outside [lo, hi]. NaN where a coordinate is: a record without
// one is in no set.
__device__ __forceinline__ float max_nan(float a, float b) {
    float r;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float gap(float lo, float hi, float v) { return max_nan(max_nan(lo - v, v - hi), 0.0f); }

__device__ __forceinline__ void count(int i, unsigned long long v = 1) {
    if ((threadIdx.x & 31) == 0) scratch().st[i] += v;
}

// Writes one estimate (lane 0): the flux sum and squared radius (raw; -1
// when nothing was found), or the normalised radiance estimate (the
// render's own expressions).
__device__ __forceinline__ float estimate_scale(float r2, bool surface) {
    return surface ? (1.0f / (3.14159265f * r2)) * 0.318309886f : 1.0f / (4.18879020f * r2 * sqrtf(r2));
}
__device__ __forceinline__ void write_estimate(float4 *out, uint32_t i, v3 e, int found, float r2,
                                               bool surface, bool raw) {
    float r2out = -1.0f;
    if (found > 0) {
        r2out = r2;
        if (!raw) e = e * estimate_scale(r2, surface);
    } else {
        e = mk3(0.f, 0.f, 0.f);
    }
    if ((threadIdx.x & 31) == 0) out[i] = make_float4(e.x, e.y, e.z, raw ? r2out : 0.0f);
}

// The same from the integer sums of the three channels: lanes 0, 1 and 2
// round one channel each (one pass through the 64-bit conversion instead of
// three), lane 3 has the squared radius.
__device__ __forceinline__ void write_sums(float4 *out, uint32_t i, const FixedSum &x, const FixedSum &y,
                                           const FixedSum &z, int found, float r2, bool surface, bool raw) {
    const int lane = threadIdx.x & 31;
    FixedSum f;
    f.sum = lane == 0 ? x.sum : (lane == 1 ? y.sum : z.sum);
    f.emax = lane == 0 ? x.emax : (lane == 1 ? y.emax : z.emax);
    float v = fixed_value(f);
    if (!raw) v = v * estimate_scale(r2, surface);
    if (found == 0) v = 0.0f;
    if (lane == 3) v = raw ? (found > 0 ? r2 : -1.0f) : 0.0f;
    if (lane < 4) reinterpret_cast<float *>(out + i)[lane] = v;
}

// Queues the queries (their indices on the lanes) of `mask` for the
// list-search launch.
__device__ __forceinline__ void defer(uint32_t out, unsigned mask) {
    const int lane = threadIdx.x & 31;
    uint32_t base = 0;
    if (lane == 0) base = atomicAdd(targs().defer_n, (uint32_t)__popc(mask));
    base = __shfl_sync(kFull, base, 0);
    if ((mask >> lane) & 1u) {
        const uint32_t at = base + __popc(mask & ((1u << lane) - 1u));
        targs().defer[at] = out;
        if (targs().defer_sc) targs().defer_sc[at] = targs().scene;
    }
    count(kStList, (unsigned long long)__popc(mask));
}

// The tree positions of every record of map `mid` within sqrt(rho2) of the
// box [lo, hi] into cat. Returns the count, or -1 when more than kTileCap qualify.
__device__ __noinline__ int collect(int mid, v3 lo, v3 hi, float rho2) {
    TileScratch &ts = scratch();
    const MapView &m = targs().map[mid];
    const int lane = threadIdx.x & 31;
    uint32_t *st = ts.stack;
    const unsigned lt = (1u << lane) - 1u;
    if (lane == 0) st[0] = 1u;
    __syncwarp();
    int top = 1, n = 0;
    const uint32_t first_leaf = 1u << m.depth;
    const int chunks = 1 << m.leaf_shift;
    while (top > 0) {
        --top;
        const uint32_t node = st[top];
        __syncwarp();
        const int dn = 31 - __clz(node);
        if (dn == m.depth) {
            for (int c = 0; c < chunks; ++c) {
                const uint32_t r = ((node - first_leaf) << (5 + m.leaf_shift)) + ((uint32_t)c << 5) + lane;
                bool in = false;
                if (r < m.n) {
                    const float4 p = __ldg(&m.pos[r]);
                    const float gx = gap(lo.x, hi.x, p.x), gy = gap(lo.y, hi.y, p.y),
                                gz = gap(lo.z, hi.z, p.z);
                    in = gx * gx + gy * gy + gz * gz <= rho2;
                }
                const unsigned mk = __ballot_sync(kFull, in);
                if (n + __popc(mk) > kTileCap) return -1;
                if (in) ts.cat[cat_at(n + __popc(mk & lt))] = r;
                n += __popc(mk);
            }
        } else {
            int w = (m.depth - dn) % 5;
            if (w == 0) w = 5;
            const int nc = 1 << w;
            const uint32_t child = (node << w) + lane;
            bool ok = false;
            if (lane < nc) {
                const float4 bl = __ldg(&m.lo[child]), bh = __ldg(&m.hi[child]);
                const float gx = fmaxf(fmaxf(bl.x - hi.x, lo.x - bh.x), 0.0f);
                const float gy = fmaxf(fmaxf(bl.y - hi.y, lo.y - bh.y), 0.0f);
                const float gz = fmaxf(fmaxf(bl.z - hi.z, lo.z - bh.z), 0.0f);
                ok = gx * gx + gy * gy + gz * gz <= rho2;
            }
            const unsigned mk = __ballot_sync(kFull, ok);
            const int rank = __popc(mk & lt);
            if (ok && top + rank < kStackCap) st[top + rank] = child;
            top = min(top + __popc(mk), kStackCap);
            __syncwarp();
        }
    }
    __syncwarp();
    return n;
}

// The k nearest of the warp's candidates, d2[s] their squared distances (bits;
// slots without a candidate above every other). A threshold with exactly k
// candidates at or below it is searched for: a count costs a compare and an
// addition per slot and one warp sum, the next threshold scales the last by
// the density it found (r^3 in the medium, r^2 on surfaces), and the last one
// or two candidates are stepped over one by one. Where the k-th distance
// occurs more than once the photon index decides, and those left out get a
// distance above all. t: the first guess, at most capb (the squared gather
// radius), the search's upper end; on return the threshold, with *own the
// candidates of this lane at or below it. Returns how many there are: k, or
// all within the cap when fewer.
__device__ __forceinline__ int select_k(uint32_t (&d2)[kSlots], uint32_t &t, uint32_t capb, int k, float expo,
                                        const MapView &m, int *own) {
    int lo = -1, hi = (int)capb + 1;  // at or below lo: fewer than k; hi: more than k, or past the cap
    for (int it = 0;; ++it) {
        int mine = 0;
#pragma unroll
        for (int s = 0; s < kSlots; ++s) mine += d2[s] <= t ? 1 : 0;
        const int c = (int)__reduce_add_sync(kFull, (uint32_t)mine);
        if (c == k || (c < k && t == capb)) {
            *own = mine;
            return c;
        }
        if (c < k) lo = (int)t; else hi = (int)t;
        if (hi - lo == 1) break;  // hi's distance occurs several times
        uint32_t nt = t;
        if (c < k && k - c <= 2) {
            for (int i = c; i < k; ++i) {
                uint32_t v = 0x7fffffffu;
#pragma unroll
                for (int s = 0; s < kSlots; ++s) v = min(v, d2[s] > nt ? d2[s] : 0x7fffffffu);
                nt = __reduce_min_sync(kFull, v);
            }
            nt = min(nt, capb);
        } else if (c > k && c - k <= 2) {
            for (int i = k; i < c; ++i) {
                uint32_t v = 0u;
#pragma unroll
                for (int s = 0; s < kSlots; ++s) v = max(v, d2[s] <= nt ? d2[s] : 0u);
                nt = __reduce_max_sync(kFull, v) - 1u;
            }
        } else if (it < 6) {
            nt = min(__float_as_uint(__uint_as_float(t) * __powf(__fdividef((float)k, (float)max(c, 1)), expo)), capb);
        } else {
            nt = 0u;  // halve
        }
        if ((int)nt <= lo || (int)nt >= hi) nt = (uint32_t)(lo + ((hi - lo) >> 1));
        t = nt;
    }
    // those nearer than hi, then those at hi by photon index
    t = (uint32_t)hi;
    const int lane = threadIdx.x & 31;
    uint32_t id[kSlots];
    int less = 0;
#pragma unroll
    for (int s = 0; s < kSlots; ++s) {
        id[s] = 0xffffffffu;
        if (d2[s] == t) {
            id[s] = __float_as_uint(__ldg(&m.pos[scratch().cat[cat_at(kSlots * lane + s)]]).w);
            d2[s] = 0xffffffffu;
        }
        less += d2[s] < t ? 1 : 0;
    }
    less = (int)__reduce_add_sync(kFull, (uint32_t)less);
    for (int i = less; i < k; ++i) {
        uint32_t w = 0xffffffffu;
#pragma unroll
        for (int s = 0; s < kSlots; ++s) w = min(w, id[s]);
        w = __reduce_min_sync(kFull, w);
#pragma unroll
        for (int s = 0; s < kSlots; ++s)
            if (id[s] == w) {
                d2[s] = t;
                id[s] = 0xffffffffu;
            }
    }
    int mine = 0;
#pragma unroll
    for (int s = 0; s < kSlots; ++s) mine += d2[s] <= t ? 1 : 0;
    *own = mine;
    return k;
}

// The candidate set of the queries of `mask` (this lane's at x, bounded by
// ub): every record within their largest bound of their box. Returns its
// size, -1 when it does not fit.
__device__ __forceinline__ int collect_for(v3 x, float ub, int mid, unsigned mask) {
    const bool member = (mask >> (threadIdx.x & 31)) & 1u;
    const float inf = __int_as_float(0x7f800000);
    const v3 lo = mk3(warp_min(member ? x.x : inf), warp_min(member ? x.y : inf), warp_min(member ? x.z : inf));
    const v3 hi = mk3(warp_max(member ? x.x : -inf), warp_max(member ? x.y : -inf), warp_max(member ? x.z : -inf));
    const float rho = warp_max(member ? ub : 0.0f);
    return collect(mid, lo, hi, rho * rho * kOuter);
}

// The positions of the n candidates in cat, kSlots consecutive ones
// (neighbours in the tree) to a lane; empty slots hold NaN, whose distance is
// above every other.
__device__ __forceinline__ void load_candidates(const MapView &m, int n, float (&px)[kSlots], float (&py)[kSlots],
                                                float (&pz)[kSlots]) {
    const TileScratch &ts = scratch();
    const int lane = threadIdx.x & 31;
    const float none = __int_as_float(0x7fffffff);
#pragma unroll
    for (int s = 0; s < kSlots; ++s) {
        px[s] = py[s] = pz[s] = none;
        if (kSlots * lane + s < n) {
            const float4 p = __ldg(&m.pos[ts.cat[cat_at(kSlots * lane + s)]]);
            px[s] = p.x;
            py[s] = p.y;
            pz[s] = p.z;
        }
    }
}

// The queries of `mask` (one map, lane order = spatial order) from the n
// candidates in cat, which hold every record within each query's bound.
// Sets d_lane to the capped k-th distance of the lane's query (-1 if it was
// deferred).
template <int S>
__device__ __noinline__ void tile_queries(int mid, int n, unsigned mask, float *d_lane) {
    TileScratch &ts = scratch();
    const int lane = threadIdx.x & 31;
    const int k = targs().k;
    const MapView &m = targs().map[mid];
    count(kStGroups);
    count(kStCandidates, (unsigned long long)n);
    float px[kSlots], py[kSlots], pz[kSlots];
    load_candidates(m, n, px, py, pz);
    const float r2cap = targs().r2cap, rcap = targs().rcap;
    const uint32_t capb = __float_as_uint(r2cap);
    const float expo = mid == 0 ? 1.0f : 0.6666667f;
    uint32_t guess = 0u;
    for (unsigned mm = mask; mm; mm &= mm - 1) {
        const int j = __ffs(mm) - 1;
        const float4 q = ts.qx[j];
        uint32_t d2[kSlots];
#pragma unroll
        for (int s = 0; s < kSlots; ++s) {
            const float dx = px[s] - q.x, dy = py[s] - q.y, dz = pz[s] - q.z;
            d2[s] = __float_as_uint(dx * dx + dy * dy + dz * dz);
        }
        if (guess == 0u) guess = __float_as_uint(q.w * q.w);
        uint32_t t = min(guess, capb);
        int own;
        const int found = select_k(d2, t, capb, k, expo, m, &own);
        // the selected ones' tree positions, in candidate order, and the
        // largest distance among them
        int at = own;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(kFull, at, o);
            if (lane >= o) at += v;
        }
        at -= own;
        uint32_t far = 0u;
#pragma unroll
        for (int s = 0; s < kSlots; ++s)
            if (d2[s] <= t) {
                far = max(far, d2[s]);
                ts.sel[at++] = ts.cat[cat_at(kSlots * lane + s)];
            }
        far = __reduce_max_sync(kFull, far);
        __syncwarp();
        // the set holds every record within the upper bound; a result
        // beyond it would mean the bound failed: defer to the list search
        const float kd2 = found == k ? __uint_as_float(far) : r2cap;
        if ((found == k && kd2 > q.w * q.w) || (found < k && q.w < rcap)) {
            count(kStViolations);
            defer(__float_as_uint(ts.qd[j].w), 1u);
            if (lane == j) *d_lane = -1.0f;
            guess = 0u;
            __syncwarp();
            continue;
        }
        guess = __float_as_uint(kd2);
        const float4 qd = ts.qd[j];
        const v3 dirv = mk3(qd.x, qd.y, qd.z);
        float tx[S], ty[S], tz[S];
#pragma unroll
        for (int s = 0; s < S; ++s) {
            tx[s] = ty[s] = tz[s] = 0.0f;
            const int e = lane + 32 * s;
            if (e < found) {
                const v3 t = flux_term(m, ts.sel[e], mid, dirv, targs().g);
                tx[s] = t.x;
                ty[s] = t.y;
                tz[s] = t.z;
            }
        }
        const FixedSum fx = warp_fixed_parts<S>(tx), fy = warp_fixed_parts<S>(ty), fz = warp_fixed_parts<S>(tz);
        write_sums(targs().out, __float_as_uint(qd.w), fx, fy, fz, found, kd2, mid == 0, targs().raw);
        __syncwarp();
        if (lane == j) *d_lane = found == k ? sqrtf(kd2) : rcap;
        count(kStTiled);
    }
}

// A radius around query j of the group that at least k and at most kTileCap
// records of map `mid` lie within (or the gather radius, when fewer do), at
// most `hi`; -1 when none turns up. The records are then in cat, *count of
// them. The first radius is that of k records at
// the density of the leaf nearest to the query (by volume, by area where the
// leaf is flat); it then grows by the density found and, between a radius
// that overflows and one with too few, is bisected in r^3. For points of any
// kind (kPoints) nothing is looked for beside four leaves that are one place,
// and far from the map (64 times the ball's radius) the radius grows and is
// bisected beyond the distance to the leaf.
template <bool kPoints>
__device__ __noinline__ float single_bound(int mid, int j, float hi, int *count) {
    const int k = targs().k, lane = threadIdx.x & 31;
    const MapView &m = targs().map[mid];
    const float4 q = scratch().qx[j];
    const v3 x = mk3(q.x, q.y, q.z);
    const float rcap = targs().rcap;
    uint32_t node = 1u;
    float dist = 0.0f;
    for (int dn = 0; dn < m.depth;) {
        int w = (m.depth - dn) % 5;
        if (w == 0) w = 5;
        const uint32_t child = (node << w) + lane;
        uint32_t d = 0xffffffffu;
        if (lane < (1 << w)) d = __float_as_uint(box_d2(__ldg(&m.lo[child]), __ldg(&m.hi[child]), x));
        const uint32_t best = __reduce_min_sync(kFull, d);
        const unsigned at = __ballot_sync(kFull, d == best);
        node = (node << w) + (uint32_t)(__ffs(at) - 1);
        dist = __uint_as_float(best);
        dn += w;
    }
    const float4 bl = __ldg(&m.lo[node]), bh = __ldg(&m.hi[node]);
    const float ex = bh.x - bl.x, ey = bh.y - bl.y, ez = bh.z - bl.z;
    const float f = (float)k / (float)(32 << m.leaf_shift);
    const float c = fminf(ex, fminf(ey, ez)), a = fmaxf(ex, fmaxf(ey, ez)), b = ex + ey + ez - a - c;
    float r = c > 0.25f * b ? cbrtf(f * a * b * c * 0.23873241f) : approx_sqrt(f * a * b * 0.31830989f);
    if (!(r > 0.0f)) r = 0.5f * f * a;  // records on a line
    if (kPoints && a == 0.0f && m.depth >= 2) {
        const float4 pl = __ldg(&m.lo[node >> 2]), ph = __ldg(&m.hi[node >> 2]);
        if (pl.x == ph.x && pl.y == ph.y && pl.z == ph.z) return -1.0f;
    }
    hi = fminf(hi, rcap);
    float base = 0.0f;
    if (kPoints) {
        const float d = approx_sqrt(dist);
        if (d > 64.0f * r && d < hi) base = d;
    }
    r = 1.18f * r + approx_sqrt(dist);
    r = r > 0.0f ? fminf(r, hi) : hi;  // and NaN
    float lo = 0.0f;
    bool over = false;
    for (int it = 0; it < (kPoints ? 20 : 32); ++it) {
        const int n = collect(mid, x, x, r * r * kOuter);
        if (n < 0) {
            hi = r;
            over = true;
        } else if (n < k && r < rcap) {
            lo = r;
        } else {
            *count = n;
            return r;
        }
        if (kPoints && base > 0.0f) {
            if (!over) r = fminf(base + 2.0f * (lo - base), hi);
            else r = base + (lo > base ? approx_sqrt((lo - base) * (hi - base)) : 0.25f * (hi - base));
            if (over && !(r < hi)) return -1.0f;
        } else if (over) r = lo > 0.0f ? cbrtf(0.5f * (lo * lo * lo + hi * hi * hi)) : 0.75f * hi;
        else r = fminf(lo * fminf(fmaxf(__powf(__fdividef(1.4f * (float)k, (float)max(n, 1)), mid == 0 ? 0.5f : 0.3333333f), 1.05f), 2.0f), hi);
        if (!(r > lo)) return -1.0f;
    }
    return -1.0f;
}

// The least of ub and what the exact distances of known[0..n) allow at x
// (entries with a negative distance say nothing).
__device__ __forceinline__ float bound_by(const float4 *known, int n, v3 x, float ub) {
    float u = 3.0e38f;
#pragma unroll 4
    for (int j = 0; j < n; ++j) {
        const float4 o = known[j];
        const float dx = x.x - o.x, dy = x.y - o.y, dz = x.z - o.z;
        const float v = o.w + approx_sqrt(dx * dx + dy * dy + dz * dz);
        u = fminf(u, o.w >= 0.0f ? v : u);
    }
    return fminf(ub, u * (1.0f + kRel) + kAbs);
}

// Query j of the group by itself, its bound found first (below ub); false:
// to be deferred.
template <int S>
__device__ __forceinline__ bool alone(float ub, int mid, int j, float *d_lane) {
    int n = 0;
    const float r = single_bound<false>(mid, j, __shfl_sync(kFull, ub, j), &n);
    if (!(r >= 0.0f)) return false;
    __syncwarp();
    // the bound of the set just collected: all records within r are in it
    if ((threadIdx.x & 31) == j) scratch().qx[j].w = r < targs().rcap ? r * (1.0f + kRel) : targs().rcap;
    __syncwarp();
    tile_queries<S>(mid, n, 1u << j, d_lane);
    return true;
}

// The records expected in the candidate set of the queries of `mask`: the
// volume within the largest bound of their box (for a surface map the area
// of its two longer sides) at the density of k records per ball of the mean
// known distance; 0 when that says nothing (nothing known, or the gather
// radius binds).
__device__ __forceinline__ float expected(v3 x, float ub, int mid, unsigned mask, float mean) {
    if (!(mean > 0.0f) || mean >= targs().rcap) return 0.0f;
    const bool member = (mask >> (threadIdx.x & 31)) & 1u;
    const float inf = __int_as_float(0x7f800000);
    const float a = warp_max(member ? x.x : -inf) - warp_min(member ? x.x : inf);
    const float b = warp_max(member ? x.y : -inf) - warp_min(member ? x.y : inf);
    const float c = warp_max(member ? x.z : -inf) - warp_min(member ? x.z : inf);
    const float r = warp_max(member ? ub : 0.0f);
    const float k = (float)targs().k;
    if (mid == 0) {
        const float lo = fminf(a, fminf(b, c)), hi = fmaxf(a, fmaxf(b, c)), md = a + b + c - lo - hi;
        return k * __fdividef(hi * md + 2.0f * (hi + md) * r + 3.1415927f * r * r, 3.1415927f * mean * mean);
    }
    const float v = a * b * c + 2.0f * (a * b + b * c + c * a) * r + 3.1415927f * (a + b + c) * r * r +
                    4.1887902f * r * r * r;
    return k * __fdividef(v, 4.1887902f * mean * mean * mean);
}

// One chunk (groups of W consecutive queries of the sorted order, from query
// chunk * W * groups) of a scene, with the warp's arguments set.
template <int S, uint32_t W>
__device__ __forceinline__ void tile_chunk(const PScene &Sc, const MapView &surf, const MapView &vol,
                                           const float4 *qa, const float4 *qd, const uint32_t *order,
                                           uint32_t n, uint32_t chunk, int groups,
                                           float r2cap, bool raw, float4 *out) {
    TileScratch &ts = scratch();
    const int lane = threadIdx.x & 31;
    const float rcap = sqrtf(r2cap);
    const uint32_t wfirst = chunk * (W * (uint32_t)groups);
    // exact distances known so far: those of the previous group
    int nknown = 0, wkind = -1;
    for (int g = 0; g < groups; ++g) {
        const uint32_t first = wfirst + W * (uint32_t)g;
        if (first >= n) break;
        const uint32_t cnt = min(W, n - first);
        Query q;
        q.x = q.dirv = mk3(0.f, 0.f, 0.f);
        q.map = 1;
        q.out = 0;
        if ((uint32_t)lane < cnt) q = load_query(Sc, qa, qd, order[first + lane]);
        const int gkind = __shfl_sync(kFull, q.map, 0);
        const unsigned valid = __ballot_sync(kFull, (uint32_t)lane < cnt);
        const unsigned members = __ballot_sync(kFull, (uint32_t)lane < cnt && q.map == gkind);
        const uint32_t mn = gkind == 0 ? surf.n : vol.n;
        float dnew = -1.0f;
        if (gkind != wkind) {
            nknown = 0;
            wkind = gkind;
        }
        __syncwarp();
        if (mn == 0) {
            // an empty map: nothing found
            if ((members >> lane) & 1u) out[q.out] = make_float4(0.f, 0.f, 0.f, raw ? -1.0f : 0.0f);
        } else {
            float ub = bound_by(ts.known, nknown, q.x, rcap);
            ts.qx[lane] = make_float4(q.x.x, q.x.y, q.x.z, ub);
            ts.qd[lane] = make_float4(q.dirv.x, q.dirv.y, q.dirv.z, __uint_as_float(q.out));
            __syncwarp();
            // segments of the members in spatial order: the whole group,
            // then halves of a segment whose set does not fit (or is not
            // expected to), down to single queries (growing again after a
            // fit); each finished segment tightens the bounds of the rest
            unsigned rem = members;
            int sz = 32;
            if (nknown == 0) {
                // nothing bounds the group yet: its middle query by itself first
                const int j = __fns(members, 0, (__popc(members) + 1) >> 1);
                if (alone<S>(ub, gkind, j, &dnew)) {
                    if (lane == j) ts.known[0] = make_float4(q.x.x, q.x.y, q.x.z, dnew);
                    __syncwarp();
                    nknown = 1;
                    ub = bound_by(ts.known, 1, q.x, ub);
                    ts.qx[lane].w = ub;
                    __syncwarp();
                } else {
                    defer(q.out, 1u << j);
                }
                rem &= ~(1u << j);
            }
            // the mean known distance: the density the sets are expected at
            const float kw = lane < nknown ? ts.known[lane].w : -1.0f;
            const int kn = __popc(__ballot_sync(kFull, kw >= 0.0f));
            float mean = kw >= 0.0f ? kw : 0.0f;
#pragma unroll
            for (int o = 16; o; o >>= 1) mean += __shfl_xor_sync(kFull, mean, o);
            mean = kn ? __fdividef(mean, (float)kn) : -1.0f;
            while (rem) {
                const unsigned seg = __popc(rem) <= sz ? rem : rem & ((1u << __fns(rem, 0, sz + 1)) - 1u);
                const int j = __ffs(seg) - 1;
                const bool big = expected(q.x, ub, gkind, seg, mean) > (float)kTileCap;
                if (big && __popc(seg) > 1) {
                    sz = __popc(seg) >> 1;
                    continue;
                }
                const int nc = big ? -1 : collect_for(q.x, ub, gkind, seg);
                if (nc < 0 && __popc(seg) > 1) {
                    count(kStHalvings);
                    sz = __popc(seg) >> 1;
                    continue;
                }
                bool done = nc >= 0;
                if (done) {
                    tile_queries<S>(gkind, nc, seg, &dnew);
                    sz = min(2 * sz, 32);
                } else {
                    done = alone<S>(ub, gkind, j, &dnew);
                    if (done) count(kStShrunk);
                    else defer(q.out, seg);
                }
                rem &= ~seg;
                if (rem && done) {
                    // the segment's exact distances, through the known list
                    const unsigned in = (seg >> lane) & 1u;
                    if (in) ts.known[__popc(seg & ((1u << lane) - 1u))] = make_float4(q.x.x, q.x.y, q.x.z, dnew);
                    __syncwarp();
                    ub = bound_by(ts.known, __popc(seg), q.x, ub);
                    ts.qx[lane].w = ub;
                    __syncwarp();
                }
            }
        }
        const unsigned odd = valid & ~members;
        if (odd) defer(q.out, odd);
        // this group's exact distances bound the next group
        ts.known[lane] = make_float4(q.x.x, q.x.y, q.x.z, ((members >> lane) & 1u) ? dnew : -1.0f);
        nknown = 32;
        __syncwarp();
    }
}

template <int S, uint32_t W>
__global__ void __launch_bounds__(kTileWarps * 32, kTileBlocks)
    query_knn_tile_kernel(PScene Sc, MapView surf, MapView vol, const float4 *qa, const float4 *qd,
                          const uint32_t *order, uint32_t n, const uint32_t *n_dev, int groups,
                          int k, float r2cap, bool raw, float4 *out,
                          uint32_t *defer_list, uint32_t *defer_n, uint32_t *chunk_counter,
                          unsigned long long *stats) {
    const int lane = threadIdx.x & 31;
    if (n_dev) n = min(n, *n_dev);
    set_targs(surf, vol, out, defer_list, nullptr, defer_n, 0u, r2cap, Sc.g, k, raw);
    TileScratch &ts = scratch();
    if (lane < kStCount) ts.st[lane] = 0;
    __syncwarp();
    const uint32_t nchunks = (n + W * (uint32_t)groups - 1u) / (W * (uint32_t)groups);
    // persistent warps: each takes the next chunk from the counter until
    // none is left, so a block's resources are never held by finished warps
    // waiting on a slow one
    for (;;) {
        uint32_t chunk = 0;
        if (lane == 0) chunk = atomicAdd(chunk_counter, 1u);
        chunk = __shfl_sync(kFull, chunk, 0);
        if (chunk >= nchunks) break;
        tile_chunk<S, W>(Sc, surf, vol, qa, qd, order, n, chunk, groups, r2cap, raw, out);
    }
    __syncwarp();
    if (stats && lane < kStCount && ts.st[lane]) atomicAdd(&stats[lane], ts.st[lane]);
}

// k nearest records of query points, sorted by (squared distance, index);
// one warp per query, each bounded and selected by itself as above. The
// selected records are put in order by their ranks: every lane counts the
// distances below its own, and where two are equal the indices decide. A
// query without a radius that fits its set (more records at one distance
// than the registers hold) is marked in its first index and left to
// knn_rest_kernel. Bound by instruction issue and the walk's L2 latency.
// Measured (GB300; the list search before): 262,144 queries, k = 100, 1M
// points 3.62 -> 1.59 ms; 32,768 queries, k = 32, 100,000 points 225 -> 110 us.
template <int S>
__global__ void __launch_bounds__(kTileWarps * 32, kTileBlocks)
    knn_kernel(MapView m, int mid, const float4 *q, uint32_t nq, int k, float r2cap, uint32_t *idx_out,
               float *d2_out) {
    const int lane = threadIdx.x & 31;
    const uint32_t qi = blockIdx.x * kTileWarps + (threadIdx.x >> 5);
    if (qi >= nq) return;
    set_targs(m, m, nullptr, nullptr, nullptr, nullptr, 0u, r2cap, 0.0f, k, true);
    TileScratch &ts = scratch();
    const float4 p = q[qi];
    if (lane == 0) ts.qx[0] = make_float4(p.x, p.y, p.z, targs().rcap);
    __syncwarp();
    uint32_t *idx = idx_out + (size_t)qi * k;
    float *dist = d2_out + (size_t)qi * k;
    int n = 0, found = 0;
    float r = targs().rcap;
    if (m.n > 0 && p.x == p.x && p.y == p.y && p.z == p.z) {  // nothing is near a NaN
        r = single_bound<true>(mid, 0, targs().rcap, &n);
        if (!(r >= 0.0f)) {
            if (lane == 0) idx[0] = kKnnLeft;
            return;
        }
        __syncwarp();
        if (n <= 32) {
            // A record a lane, its place by comparing with every other: 20,000
            // queries of 200,000 records with k = 1 49.5 -> 43.3 us, k = 12 68.4
            // -> 64.
            uint32_t *key = reinterpret_cast<uint32_t *>(ts.qd);
            uint32_t mine = 0xffffffffu, id = 0xffffffffu;
            if (lane < n) {
                const float4 c = __ldg(&m.pos[ts.cat[cat_at(lane)]]);
                const float dx = c.x - p.x, dy = c.y - p.y, dz = c.z - p.z;
                const uint32_t d2 = __float_as_uint(dx * dx + dy * dy + dz * dz);
                if (d2 <= __float_as_uint(r2cap)) {
                    mine = d2;
                    id = __float_as_uint(c.w);
                }
            }
            int rank = 0;
            for (int o = 0; o < n; ++o) {
                const uint32_t w = __shfl_sync(kFull, mine, o), i = __shfl_sync(kFull, id, o);
                rank += w < mine || (w == mine && i < id) ? 1 : 0;
            }
            found = min(k, __popc(__ballot_sync(kFull, mine != 0xffffffffu)));
            if (mine != 0xffffffffu && rank < k) {
                key[rank] = mine;
                ts.sel[rank] = id;
            }
            __syncwarp();
        } else {
            float px[kSlots], py[kSlots], pz[kSlots];
            load_candidates(m, n, px, py, pz);
            uint32_t d2[kSlots];
#pragma unroll
            for (int s = 0; s < kSlots; ++s) {
                const float dx = px[s] - p.x, dy = py[s] - p.y, dz = pz[s] - p.z;
                d2[s] = __float_as_uint(dx * dx + dy * dy + dz * dz);
            }
            const uint32_t capb = __float_as_uint(r2cap);
            const float expo = mid == 0 ? 1.0f : 0.6666667f;
            uint32_t t = min(__float_as_uint(r * r * __powf(__fdividef((float)k, (float)max(n, k)), expo)), capb);
            int own;
            found = select_k(d2, t, capb, k, expo, m, &own);
            int at = own;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(kFull, at, o);
                if (lane >= o) at += v;
            }
            at -= own;
            uint32_t *key = reinterpret_cast<uint32_t *>(ts.qd);  // 128 distances
#pragma unroll
            for (int s = 0; s < kSlots; ++s)
                if (d2[s] <= t) {
                    key[at] = d2[s];
                    ts.sel[at++] = ts.cat[cat_at(kSlots * lane + s)];
                }
            if (lane < 4 && found + lane < 128) key[found + lane] = 0xffffffffu;
            __syncwarp();
            uint32_t mine[S], id[S];
            int rank[S];
            uint32_t sum = 0;
#pragma unroll
            for (int s = 0; s < S; ++s) {
                const int e = lane + 32 * s;
                mine[s] = e < found ? key[e] : 0u;
                id[s] = e < found ? __float_as_uint(__ldg(&m.pos[ts.sel[e]]).w) : 0xffffffffu;
                rank[s] = 0;
            }
            for (int f = 0; f < found; f += 4) {
                const uint4 w = reinterpret_cast<const uint4 *>(key)[f >> 2];
#pragma unroll
                for (int s = 0; s < S; ++s)
                    rank[s] += (w.x < mine[s] ? 1 : 0) + (w.y < mine[s] ? 1 : 0) + (w.z < mine[s] ? 1 : 0) +
                               (w.w < mine[s] ? 1 : 0);
            }
#pragma unroll
            for (int s = 0; s < S; ++s) sum += lane + 32 * s < found ? (uint32_t)rank[s] : 0u;
            sum = __reduce_add_sync(kFull, sum);
            __syncwarp();
            if (sum != (uint32_t)(found * (found - 1) / 2)) {  // equal distances
#pragma unroll
                for (int s = 0; s < S; ++s)
                    if (lane + 32 * s < found) ts.sel[lane + 32 * s] = id[s];
                __syncwarp();
                for (int f = 0; f < found; ++f) {
                    const uint32_t w = key[f], o = ts.sel[f];
#pragma unroll
                    for (int s = 0; s < S; ++s) rank[s] += w == mine[s] && o < id[s] ? 1 : 0;
                }
                __syncwarp();
            }
#pragma unroll
            for (int s = 0; s < S; ++s)
                if (lane + 32 * s < found) {
                    key[rank[s]] = mine[s];
                    ts.sel[rank[s]] = id[s];
                }
            __syncwarp();
        }
    }
    // fewer than k of a radius's k records: their distance beside the gather
    // radius's rounding, or none at all (infinity less infinity); others may lie
    // beyond that radius
    if (found < k && r < targs().rcap) {
        if (lane == 0) idx[0] = kKnnLeft;
        return;
    }
#pragma unroll
    for (int s = 0; s < S; ++s) {
        const int e = lane + 32 * s;
        if (e < k) {
            idx[e] = e < found ? ts.sel[e] : 0xffffffffu;
            dist[e] = e < found ? __uint_as_float(reinterpret_cast<const uint32_t *>(ts.qd)[e]) : r2cap;
        }
    }
}

// One query by the list search.
template <int S>
__device__ __forceinline__ void list_query(const MapView &m, const float4 *q, size_t qi, int k, float r2cap,
                                           uint32_t *idx_out, float *d2_out, WarpScratch &ws, int lane) {
    const uint64_t cap = make_key(r2cap, 0xffffffffu);
    const float4 p = q[qi];
    Knn<S> kn;
    kn.reset(cap, k);
    knn_search<S>(m, mk3(p.x, p.y, p.z), kn, ws, lane, cap);
#pragma unroll
    for (int s = 0; s < S; ++s) {
        const int j = lane * S + s;
        if (j < k) {
            idx_out[qi * k + j] = (uint32_t)kn.key[s];
            d2_out[qi * k + j] = key_d2(kn.key[s]);
        }
    }
}

// The queries knn_kernel left, by the list search. A warp looks at the marks of
// 32 queries at a time, a grid of warps apart, so that queries left side by side
// (all of them, where the records are piles) go to different warps.
template <int S>
__global__ void __launch_bounds__(128) knn_rest_kernel(MapView m, const float4 *q, uint32_t nq, int k, float r2cap,
                                                       uint32_t *idx_out, float *d2_out) {
    __shared__ WarpScratch ws[4];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const uint64_t warps = (uint64_t)gridDim.x * 4;
    for (uint64_t base = (uint64_t)blockIdx.x * 4 + wib; base < nq; base += 32 * warps) {
        const uint64_t mine = base + lane * warps;
        unsigned left = __ballot_sync(kFull, mine < nq && idx_out[mine * k] == kKnnLeft);
        for (; left; left &= left - 1) {
            const uint64_t qi = base + (__ffs(left) - 1) * warps;
            list_query<S>(m, q, qi, k, r2cap, idx_out, d2_out, ws[wib], lane);
        }
    }
}

// Every query by the list search: thin maps.
template <int S>
__global__ void __launch_bounds__(128) knn_list_kernel(MapView m, const float4 *q, uint32_t nq, int k, float r2cap,
                                                       uint32_t *idx_out, float *d2_out) {
    __shared__ WarpScratch ws[4];
    const uint32_t qi = blockIdx.x * 4 + (threadIdx.x >> 5);
    if (qi < nq) list_query<S>(m, q, qi, k, r2cap, idx_out, d2_out, ws[threadIdx.x >> 5], threadIdx.x & 31);
}

// The scene of global chunk c: the last descriptor whose chunk_begin <= c.
__device__ __forceinline__ int scene_of_chunk(const TileScene *scenes, int nsc, uint32_t c) {
    int lo = 0, hi = nsc - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (scenes[mid].chunk_begin <= c) lo = mid; else hi = mid - 1;
    }
    return lo;
}

// The same pass over the chunks of many scenes (their descriptors in device
// memory, chunks numbered scene after scene): one persistent launch; a warp
// loads a scene's arguments when its next chunk belongs to another scene.
template <int S>
__global__ void __launch_bounds__(kTileWarps * 32, kTileBlocks)
    query_knn_tile_multi_kernel(const TileScene *scenes, int nsc, uint32_t total_chunks, int groups,
                                bool raw, uint32_t *defer_list,
                                uint32_t *defer_sc, uint32_t *defer_n, uint32_t *chunk_counter,
                                unsigned long long *stats) {
    const int lane = threadIdx.x & 31;
    TileScratch &ts = scratch();
    if (lane < kStCount) ts.st[lane] = 0;
    __syncwarp();
    int cur = -1;
    for (;;) {
        uint32_t chunk = 0;
        if (lane == 0) chunk = atomicAdd(chunk_counter, 1u);
        chunk = __shfl_sync(kFull, chunk, 0);
        if (chunk >= total_chunks) break;
        const int sidx = scene_of_chunk(scenes, nsc, chunk);
        const TileScene &d = scenes[sidx];
        if (sidx != cur) {
            set_targs(d.surf, d.vol, d.val, defer_list, defer_sc, defer_n, (uint32_t)sidx, d.r2cap, d.sc->g,
                      d.k, raw);
            cur = sidx;
        }
        tile_chunk<S, 32>(*d.sc, d.surf, d.vol, d.qa, d.qd, d.order, d.n, chunk - d.chunk_begin, groups,
                      d.r2cap, raw, d.val);
    }
    __syncwarp();
    if (stats && lane < kStCount && ts.st[lane]) atomicAdd(&stats[lane], ts.st[lane]);
}

// The deferred queries of many scenes (defer_sc: each one's scene).
template <int S>
__global__ void __launch_bounds__(128)
    deferred_multi_kernel(const TileScene *scenes, const uint32_t *defer_list, const uint32_t *defer_sc,
                          const uint32_t *defer_n, bool raw) {
    __shared__ WarpScratch ws[4];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const uint32_t total = *defer_n;
    for (uint32_t w = blockIdx.x * 4 + wib; w < total; w += gridDim.x * 4) {
        const TileScene &d = scenes[defer_sc[w]];
        const uint64_t cap = make_key(d.r2cap, 0xffffffffu);
        const Query q = load_query(*d.sc, d.qa, d.qd, defer_list[w]);
        const MapView &m = q.map == 0 ? d.surf : d.vol;
        v3 e = mk3(0.f, 0.f, 0.f);
        int found = 0;
        float r2 = d.r2cap;
        if (m.n > 0) {
            Knn<S> kn;
            kn.reset(cap, d.k);
            knn_search<S>(m, q.x, kn, ws[wib], lane, cap);
            e = flux_sum<S>(kn, m, lane, q.map, q.dirv, d.sc->g, cap, d.r2cap, &found, &r2);
        }
        write_estimate(d.val, q.out, e, found, r2, q.map == 0, raw);
    }
}

// The deferred queries, one warp each (grid-stride over the list).
template <int S>
__global__ void __launch_bounds__(128)
    deferred_kernel(PScene Sc, MapView surf, MapView vol, const float4 *qa, const float4 *qd,
                    const uint32_t *defer_list, const uint32_t *defer_n, int k, float r2cap, bool raw,
                    float4 *out) {
    __shared__ WarpScratch ws[4];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const uint32_t total = *defer_n;
    const uint64_t cap = make_key(r2cap, 0xffffffffu);
    for (uint32_t w = blockIdx.x * 4 + wib; w < total; w += gridDim.x * 4) {
        const Query q = load_query(Sc, qa, qd, defer_list[w]);
        const MapView &m = q.map == 0 ? surf : vol;
        v3 e = mk3(0.f, 0.f, 0.f);
        int found = 0;
        float r2 = r2cap;
        if (m.n > 0) {
            Knn<S> kn;
            kn.reset(cap, k);
            knn_search<S>(m, q.x, kn, ws[wib], lane, cap);
            e = flux_sum<S>(kn, m, lane, q.map, q.dirv, Sc.g, cap, r2cap, &found, &r2);
        }
        write_estimate(out, q.out, e, found, r2, q.map == 0, raw);
    }
}

}  // namespace

// The estimate pass's warps on the GPU at once.
static uint32_t tile_warps(int sm_count) { return (uint32_t)std::max(sm_count, 1) * kTileBlocks * kTileWarps; }

cudaError_t knn_values_tiles(const PScene &S, const MapView &surf, const MapView &vol,
                             const float4 *qa, const float4 *qd, const uint32_t *order, uint32_t n,
                             const uint32_t *n_dev, int k, float radius, bool raw, float4 *val,
                             const TileBuffers &buf, int sm_count, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    const int groups = tile_groups(n, sm_count);
    const float r2 = radius * radius;
    // Few queries: groups of 8, so that no warp waits for 32 of them while
    // others have none. 2^14 picks, k = 128, 1M records 1.22 -> 0.53 ms; 2^17,
    // k = 16, 20,000 records 0.49 -> 0.38; 2^18, k = 16 0.58 -> 0.55; 2^19 0.78 ->
    // 0.88, k = 128 2.61 -> 2.54.
    const bool few = n < 64u * tile_warps(sm_count);
    const uint32_t chunks = few ? (n + 7) / 8 : tile_chunks(n, groups);
    const dim3 grid((chunks + kTileWarps - 1) / kTileWarps), block(kTileWarps * 32);
    const int smem = (int)(kTileWarps * sizeof(TileScratch));
    const dim3 dgrid(std::max(sm_count, 1) * 8);
    // defer_n[0]: deferred queries, defer_n[1]: the chunk counter
    cudaError_t e = cudaMemsetAsync(buf.defer_n, 0, 2 * sizeof(uint32_t), s);
    if (e != cudaSuccess) return e;
    int per_sm = 1;
    // persistent tile launch: as many blocks as fit on the GPU at once
#define PM_TILE_KERNEL(SL, W)                                                                           \
    e = cudaFuncSetAttribute(query_knn_tile_kernel<SL, W>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem); \
    if (e != cudaSuccess) return e;                                                                     \
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, query_knn_tile_kernel<SL, W>, kTileWarps * 32, smem); \
    if (e != cudaSuccess) return e;                                                                     \
    query_knn_tile_kernel<SL, W><<<std::min<uint32_t>(grid.x, (uint32_t)std::max(sm_count, 1) * (uint32_t)std::max(per_sm, 1)), \
                                   block, smem, s>>>(S, surf, vol, qa, qd, order, n, n_dev, groups, k, \
                                                     r2, raw, val, buf.defer, buf.defer_n, buf.defer_n + 1, buf.stats)
#define PM_TILE_LAUNCH(SL)                                                                              \
    if (few) { PM_TILE_KERNEL(SL, 8); } else { PM_TILE_KERNEL(SL, 32); }                                \
    deferred_kernel<SL><<<dgrid, 128, 0, s>>>(S, surf, vol, qa, qd, buf.defer, buf.defer_n, k, r2, raw, val)
    switch ((k + 31) / 32) {
        case 1: PM_TILE_LAUNCH(1); break;
        case 2: PM_TILE_LAUNCH(2); break;
        case 3: PM_TILE_LAUNCH(3); break;
        default: PM_TILE_LAUNCH(4); break;
    }
#undef PM_TILE_LAUNCH
#undef PM_TILE_KERNEL
    note_launches(2);
    return cudaGetLastError();
}

cudaError_t knn_query(const MapView &m, int map, const float4 *q, uint32_t nq, int k, float radius,
                      uint32_t *idx, float *d2, cudaStream_t s, bool thin) {
    if (nq == 0) return cudaSuccess;
    const float r2 = radius * radius;
    const dim3 grid((nq + kTileWarps - 1) / kTileWarps), block(kTileWarps * 32);
    const dim3 rest(std::min<uint32_t>((nq + 3) / 4, 2432));  // 16 blocks on each of 152 SMs
    const int smem = (int)(kTileWarps * sizeof(TileScratch));
#define PM_KNN_LAUNCH(SL)                                                                 \
    if (thin) {                                                                           \
        knn_list_kernel<SL><<<(nq + 3) / 4, 128, 0, s>>>(m, q, nq, k, r2, idx, d2);       \
    } else {                                                                              \
        knn_kernel<SL><<<grid, block, smem, s>>>(m, map, q, nq, k, r2, idx, d2);          \
        knn_rest_kernel<SL><<<rest, 128, 0, s>>>(m, q, nq, k, r2, idx, d2);               \
    }
    switch ((k + 31) / 32) {
        case 1: PM_KNN_LAUNCH(1); break;
        case 2: PM_KNN_LAUNCH(2); break;
        case 3: PM_KNN_LAUNCH(3); break;
        default: PM_KNN_LAUNCH(4); break;
    }
#undef PM_KNN_LAUNCH
    note_launches(thin ? 1 : 2);
    return cudaGetLastError();
}

cudaError_t knn_values_tiles_multi(const TileScene *scenes, int nsc, uint32_t total_chunks, int groups,
                                   int slots, bool raw, const TileBuffers &buf, uint32_t *defer_sc,
                                   int sm_count, cudaStream_t s) {
    if (total_chunks == 0 || nsc == 0) return cudaSuccess;
    if (groups < 1 || groups > 4 || slots < 1 || slots > 4) return cudaErrorInvalidValue;
    const dim3 agrid((total_chunks + kTileWarps - 1) / kTileWarps), block(kTileWarps * 32);
    const int smem = (int)(kTileWarps * sizeof(TileScratch));
    const dim3 dgrid(std::max(sm_count, 1) * 8);
    cudaError_t e = cudaMemsetAsync(buf.defer_n, 0, 2 * sizeof(uint32_t), s);
    if (e != cudaSuccess) return e;
    int per_sm = 1;
#define PM_MULTI_LAUNCH(SL)                                                                              \
    e = cudaFuncSetAttribute(query_knn_tile_multi_kernel<SL>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem); \
    if (e != cudaSuccess) return e;                                                                     \
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, query_knn_tile_multi_kernel<SL>, kTileWarps * 32, smem); \
    if (e != cudaSuccess) return e;                                                                     \
    query_knn_tile_multi_kernel<SL><<<std::min<uint32_t>(agrid.x, (uint32_t)std::max(sm_count, 1) * (uint32_t)std::max(per_sm, 1)), \
                                      block, smem, s>>>(scenes, nsc, total_chunks, groups, raw, \
                                                        buf.defer, defer_sc, buf.defer_n, buf.defer_n + 1, buf.stats); \
    deferred_multi_kernel<SL><<<dgrid, 128, 0, s>>>(scenes, buf.defer, defer_sc, buf.defer_n, raw)
    switch (slots) {
        case 1: PM_MULTI_LAUNCH(1); break;
        case 2: PM_MULTI_LAUNCH(2); break;
        case 3: PM_MULTI_LAUNCH(3); break;
        default: PM_MULTI_LAUNCH(4); break;
    }
#undef PM_MULTI_LAUNCH
    note_launches(2);
    return cudaGetLastError();
}

uint32_t tile_chunks(uint32_t n, int groups) { return (n + 32u * groups - 1) / (32u * groups); }

// A chunk's first group costs a bound of its own, its later ones have the
// group before; the fewer chunks a warp gets, the longer the last ones leave
// the others idle. Measured (ms, 1 / 2 / 4 groups, per query count): 2.1M
// 2.4 / 2.6 / 3.3 (with 8 candidates a lane), 11M 12.5 / 11.5 / 11.4, 21M - /
// 25.4 / 25.9, 46M - / 62.6 / 59.8: four from 64 chunks a warp on, one below
// 8 chunks of two.
int tile_groups(uint64_t n, int sm_count) {
    const uint64_t warps = tile_warps(sm_count);
    if (n >= 128u * 64u * warps) return 4;
    return n >= 64u * 8u * warps ? 2 : 1;
}

}  // namespace pm
