// tile_gather.cu -- k-NN radiance estimates of a query list in spatial
// order, one candidate set per group of neighbouring queries.
//
// A warp takes 1 to 4 consecutive groups of 32 queries of the (map, Morton
// code) order. The k-th-neighbour distance d(x) (capped at the gather radius) is
// 1-Lipschitz in the query position, so exact distances d_j at points x_j
// bound it everywhere: d(x) <= min_j (d_j + |x - x_j|). The warp's first group
// is bounded by one anchor (an exact list search at one of its queries, done
// by a separate launch before), every later group by the exact results of the
// group before it. A group's records are found once in the kd-tree -- every
// record within the largest upper bound of the group's bounding box -- and
// held in registers, kSlots positions to a lane. A query computes its squared
// distances to all of them and searches for the threshold that exactly k of
// them lie at or below (select_k), starting from its predecessor's.
//
// A group whose set does not fit the registers is processed in segments:
// halves, down to single queries, each finished segment tightening the
// bounds of the queries after it. A single query whose set still does not
// fit, queries of the other map in a mixed group, and any result that
// contradicts its own upper bound, are deferred to a list-search launch
// after the pass. The selected set is exactly the list search's (ties
// broken by photon index) and the estimate's sum is order-independent
// (knn_core.cuh), so every value is bit-identical to the list search's.
//
// Bound by instruction issue; the selected records' flux comes from L1 and
// L2. Candidates in registers instead of shared memory make a query's
// distances and counts straight-line code without loads, need no lists of
// the certain and the doubtful candidates, and leave most of the L1 to the
// flux. Estimate pass (GB300; candidates in shared memory, scanned, the band
// between two bounds ranked, before): preset 2 113.0 -> 76.0 ms, preset 3
// 45.4 -> 34.5 ms, preset 1 16.9 -> 12.0 ms.
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
constexpr int kAnchorAt = 15;                // the anchor: query 15 of a warp's chunk
// Blocks of 4 warps per SM (registers capped at 64) and candidates per lane.
// Presets 2 / 3: 8 blocks and 8 slots 76.0 / 34.5 ms, 7 blocks 79.1 / 35.2,
// 6 blocks 82.8 / 36.2; 10 slots at 6 blocks 81.3 / 36.7.
constexpr int kTileBlocks = 8;
constexpr int kSlots = 8;
constexpr int kTileCap = 32 * kSlots;        // candidate records per warp
constexpr float kRel = 2e-4f;                // relative and absolute margins of the distance bounds
constexpr float kAbs = 1e-6f;

// per-launch counters (pm_get_gather_stats)
enum TileStat { kStTiled, kStList, kStShrunk, kStViolations, kStGroups, kStCandidates, kStHalvings, kStCount };

struct TileScratch {
    uint32_t cat[kTileCap];  // tree positions of the candidates
    union {
        uint32_t stack[kStackCap];  // the collection's node stack
        uint32_t sel[128];          // tree positions of the k selected candidates
    };
    float4 qx[32];           // the group's queries: position, upper bound of the k-th distance
    float4 qd[32];           // weight direction, query index bits
    float4 known[32];        // exact distances that bound the group: point, distance
    unsigned long long st[kStCount];  // counters, lane 0
};

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

__device__ __forceinline__ float gap(float lo, float hi, float v) {
    return fmaxf(fmaxf(lo - v, v - hi), 0.0f);
}

__device__ __forceinline__ void count(int i, unsigned long long v = 1) {
    if ((threadIdx.x & 31) == 0) scratch().st[i] += v;
}

// Writes one estimate (lane 0): the flux sum and squared radius (raw; -1
// when nothing was found), or the normalised radiance estimate (the
// render's own expressions).
__device__ __forceinline__ void write_estimate(float4 *out, uint32_t i, v3 e, int found, float r2,
                                               bool surface, bool raw) {
    float r2out = -1.0f;
    if (found > 0) {
        r2out = r2;
        if (!raw) {
            const float sc = surface ? (1.0f / (3.14159265f * r2)) * 0.318309886f
                                     : 1.0f / (4.18879020f * r2 * sqrtf(r2));
            e = e * sc;
        }
    } else {
        e = mk3(0.f, 0.f, 0.f);
    }
    if ((threadIdx.x & 31) == 0) out[i] = make_float4(e.x, e.y, e.z, raw ? r2out : 0.0f);
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
                if (in) ts.cat[n + __popc(mk & lt)] = r;
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
// occurs more than once the photon index decides. `t`: the first guess, at
// most capb (the squared gather radius), the search's upper end. Returns the
// mask of this lane's selected slots; *found: how many (k, or all within the
// cap when fewer).
__device__ __forceinline__ uint32_t select_k(const uint32_t (&d2)[kSlots], int n, uint32_t t, uint32_t capb, int k,
                                             float expo, const MapView &m, int *found) {
    int lo = -1, hi = (int)capb + 1;  // at or below lo: fewer than k; hi: more than k, or past the cap
    uint32_t mask;
    int c;
    for (int it = 0;; ++it) {
        c = 0;
#pragma unroll
        for (int s = 0; s < kSlots; ++s) c += d2[s] <= t ? 1 : 0;
        c = (int)__reduce_add_sync(kFull, (uint32_t)c);
        if (c == k || (c < k && t == capb)) break;
        if (c < k) lo = (int)t; else hi = (int)t;
        if (hi - lo == 1) break;  // hi's distance occurs several times
        uint32_t nt = t;
        if (c < k && k - c <= 2) {
            for (int i = c; i < k; ++i) {
                uint32_t v = 0x7f800000u;
#pragma unroll
                for (int s = 0; s < kSlots; ++s) v = min(v, d2[s] > nt ? d2[s] : 0x7f800000u);
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
    *found = min(c, k);
    mask = 0u;
#pragma unroll
    for (int s = 0; s < kSlots; ++s) mask |= d2[s] <= t ? 1u << s : 0u;
    if (hi - lo == 1 && c != k && !(c < k && t == capb)) {
        // those nearer than hi, then those at hi by photon index
        const uint32_t v = (uint32_t)hi;
        const int lane = threadIdx.x & 31;
        uint32_t id[kSlots];
        int less = 0;
        mask = 0u;
#pragma unroll
        for (int s = 0; s < kSlots; ++s) {
            id[s] = 0xffffffffu;
            if (d2[s] == v) id[s] = __float_as_uint(__ldg(&m.pos[scratch().cat[32 * s + lane]]).w);
            less += d2[s] < v ? 1 : 0;
            mask |= d2[s] < v ? 1u << s : 0u;
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
                    mask |= 1u << s;
                    id[s] = 0xffffffffu;
                }
        }
        *found = k;
    }
    return mask;
}

// The queries of `mask` (one map, lane order = spatial order; this lane's at
// x, bounded by ub) from one shared candidate set. Returns false when the
// set does not fit; otherwise sets d_lane to the capped k-th distance of the
// lane's query (-1 if it was deferred).
template <int S>
__device__ __noinline__ bool tile_queries(v3 x, float ub, int mid, unsigned mask, float *d_lane) {
    TileScratch &ts = scratch();
    const int lane = threadIdx.x & 31;
    const int k = targs().k;
    const MapView &m = targs().map[mid];
    const bool member = (mask >> lane) & 1u;
    const float inf = __int_as_float(0x7f800000);
    const v3 lo = mk3(warp_min(member ? x.x : inf), warp_min(member ? x.y : inf), warp_min(member ? x.z : inf));
    const v3 hi = mk3(warp_max(member ? x.x : -inf), warp_max(member ? x.y : -inf), warp_max(member ? x.z : -inf));
    const float rho = warp_max(member ? ub : 0.0f);
    const int n = collect(mid, lo, hi, rho * rho);
    if (n < 0) return false;
    count(kStGroups);
    count(kStCandidates, (unsigned long long)n);
    // the candidates, kSlots to a lane
    float px[kSlots], py[kSlots], pz[kSlots];
#pragma unroll
    for (int s = 0; s < kSlots; ++s) {
        px[s] = py[s] = pz[s] = inf;
        if (32 * s + lane < n) {
            const float4 p = __ldg(&m.pos[ts.cat[32 * s + lane]]);
            px[s] = p.x;
            py[s] = p.y;
            pz[s] = p.z;
        }
    }
    const float r2cap = targs().r2cap, rcap = targs().rcap;
    const uint32_t capb = __float_as_uint(r2cap);
    const float expo = mid == 0 ? 1.0f : 0.6666667f;
    const unsigned lt = (1u << lane) - 1u;
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
        int found;
        const uint32_t sm = select_k(d2, n, min(guess, capb), capb, k, expo, m, &found);
        uint32_t far = 0u;
#pragma unroll
        for (int s = 0; s < kSlots; ++s) far = max(far, (sm >> s) & 1u ? d2[s] : 0u);
        far = __reduce_max_sync(kFull, far);
        // the set holds every record within the upper bound; a result
        // beyond it would mean the bound failed: defer to the list search
        const float kd2 = found == k ? __uint_as_float(far) : r2cap;
        if ((found == k && kd2 > q.w * q.w) || (found < k && q.w < rcap)) {
            count(kStViolations);
            defer(__float_as_uint(ts.qd[j].w), 1u);
            if (lane == j) *d_lane = -1.0f;
            guess = 0u;
            continue;
        }
        guess = __float_as_uint(kd2);
        int at = 0;
#pragma unroll
        for (int s = 0; s < kSlots; ++s) {
            const bool in = (sm >> s) & 1u;
            const unsigned b = __ballot_sync(kFull, in);
            if (in) ts.sel[at + __popc(b & lt)] = ts.cat[32 * s + lane];
            at += __popc(b);
        }
        __syncwarp();
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
        const v3 e = mk3(warp_fixed_sum<S>(tx), warp_fixed_sum<S>(ty), warp_fixed_sum<S>(tz));
        write_estimate(targs().out, __float_as_uint(qd.w), e, found, kd2, mid == 0, targs().raw);
        __syncwarp();
        if (lane == j) *d_lane = found == k ? sqrtf(kd2) : rcap;
        count(kStTiled);
    }
    return true;
}

// The upper bound for the single query of lane j (at x) whose set within its
// bound *ub does not fit: the radius is bisected (in r^3) below the bound. A
// collection that overflows holds more than kTileCap >= k records, so its
// radius is an upper bound; one with fewer than k (and below the cap) is a
// lower bound; one in between holds the k nearest. Returns false when no
// such radius turns up.
__device__ __noinline__ bool shrink_single(int mid, int j, float *ub) {
    const int k = targs().k;
    const float4 q = scratch().qx[j];
    const v3 x = mk3(q.x, q.y, q.z);
    float lo = 0.0f, hi = fminf(q.w, targs().rcap);
    for (int it = 0; it < 24; ++it) {
        const float r = cbrtf(0.5f * (lo * lo * lo + hi * hi * hi));
        const int n = collect(mid, x, x, r * r);
        if (n < 0) {
            hi = r;
        } else if (n < k && r < targs().rcap) {
            lo = r;
        } else {
            *ub = r * (1.0f + kRel) + kAbs;
            return true;
        }
    }
    return false;
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

// One chunk (groups of 32 consecutive queries of the sorted order, from
// query chunk * 32 * groups) of a scene, with the warp's arguments set.
template <int S>
__device__ __forceinline__ void tile_chunk(const PScene &Sc, const MapView &surf, const MapView &vol,
                                           const float4 *qa, const float4 *qd, const uint32_t *order,
                                           uint32_t n, uint32_t chunk, float anchor, int groups,
                                           float r2cap, bool raw, float4 *out) {
    TileScratch &ts = scratch();
    const int lane = threadIdx.x & 31;
    const float rcap = sqrtf(r2cap);
    const uint32_t wfirst = chunk * (uint32_t)(32 * groups);
    // exact distances known so far: the anchor, later the previous group
    int nknown = 1, wkind;
    {
        const uint32_t ai = order[wfirst + min((uint32_t)kAnchorAt, n - 1 - wfirst)];
        const float4 a = qa[ai];
        wkind = __float_as_int(a.w) != kNone ? 0 : 1;
        if (lane == 0) ts.known[0] = make_float4(a.x, a.y, a.z, anchor);
    }
    for (int g = 0; g < groups; ++g) {
        const uint32_t first = wfirst + (uint32_t)(32 * g);
        if (first >= n) break;
        const uint32_t cnt = min(32u, n - first);
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
            // then halves of a segment whose set does not fit, down to
            // single queries (growing again after a fit); each finished
            // segment tightens the bounds of the rest
            unsigned rem = members;
            int sz = 32;
            while (rem) {
                const unsigned seg = __popc(rem) <= sz ? rem : rem & ((1u << __fns(rem, 0, sz + 1)) - 1u);
                const int j = __ffs(seg) - 1;
                bool done = tile_queries<S>(q.x, ub, gkind, seg, &dnew);
                if (!done && __popc(seg) > 1) {
                    count(kStHalvings);
                    sz = __popc(seg) >> 1;
                    continue;
                }
                if (done) {
                    sz = min(2 * sz, 32);
                } else {
                    float u = 0.0f;
                    if (shrink_single(gkind, j, &u)) {
                        __syncwarp();
                        if (lane == j) {
                            ub = u;
                            ts.qx[j].w = u;
                        }
                        __syncwarp();
                        done = tile_queries<S>(q.x, ub, gkind, seg, &dnew);
                    }
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

template <int S>
__global__ void __launch_bounds__(kTileWarps * 32, kTileBlocks)
    query_knn_tile_kernel(PScene Sc, MapView surf, MapView vol, const float4 *qa, const float4 *qd,
                          const uint32_t *order, uint32_t n, const uint32_t *n_dev, int groups,
                          const float *anchor_d, int k, float r2cap, bool raw, float4 *out,
                          uint32_t *defer_list, uint32_t *defer_n, uint32_t *chunk_counter,
                          unsigned long long *stats) {
    const int lane = threadIdx.x & 31;
    if (n_dev) n = min(n, *n_dev);
    set_targs(surf, vol, out, defer_list, nullptr, defer_n, 0u, r2cap, Sc.g, k, raw);
    TileScratch &ts = scratch();
    if (lane < kStCount) ts.st[lane] = 0;
    __syncwarp();
    const uint32_t nchunks = (n + 32u * (uint32_t)groups - 1u) / (32u * (uint32_t)groups);
    // persistent warps: each takes the next chunk from the counter until
    // none is left, so a block's resources are never held by finished warps
    // waiting on a slow one
    for (;;) {
        uint32_t chunk = 0;
        if (lane == 0) chunk = atomicAdd(chunk_counter, 1u);
        chunk = __shfl_sync(kFull, chunk, 0);
        if (chunk >= nchunks) break;
        tile_chunk<S>(Sc, surf, vol, qa, qd, order, n, chunk, anchor_d[chunk], groups, r2cap, raw, out);
    }
    __syncwarp();
    if (stats && lane < kStCount && ts.st[lane]) atomicAdd(&stats[lane], ts.st[lane]);
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
                                const float *anchor_d, bool raw, uint32_t *defer_list,
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
        tile_chunk<S>(*d.sc, d.surf, d.vol, d.qa, d.qd, d.order, d.n, chunk - d.chunk_begin, anchor_d[chunk],
                      groups, d.r2cap, raw, d.val);
    }
    __syncwarp();
    if (stats && lane < kStCount && ts.st[lane]) atomicAdd(&stats[lane], ts.st[lane]);
}

// Exact capped k-th distance of each warp chunk's anchor query (list search).
template <int S>
__global__ void __launch_bounds__(128)
    anchor_kernel(MapView surf, MapView vol, const float4 *qa, const uint32_t *order, uint32_t n,
                  const uint32_t *n_dev, int groups, int k, float r2cap, float *anchor_d) {
    __shared__ WarpScratch ws[4];
    if (n_dev) n = min(n, *n_dev);
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const uint32_t chunk = blockIdx.x * 4 + wib;
    const uint32_t wfirst = chunk * (uint32_t)(32 * groups);
    if (wfirst >= n) return;
    const float4 a = qa[order[wfirst + min((uint32_t)kAnchorAt, n - 1 - wfirst)]];
    const MapView &m = __float_as_int(a.w) != kNone ? surf : vol;
    const uint64_t cap = make_key(r2cap, 0xffffffffu);
    Knn<S> kn;
    kn.reset(cap, k);
    knn_search<S>(m, mk3(a.x, a.y, a.z), kn, ws[wib], lane, cap);
    if (lane == 0) anchor_d[chunk] = kn.worst < cap ? sqrtf(key_d2(kn.worst)) : sqrtf(r2cap);
}

// The anchors of the chunks of many scenes (global chunk numbering).
template <int S>
__global__ void __launch_bounds__(128)
    anchor_multi_kernel(const TileScene *scenes, int nsc, uint32_t total_chunks, int groups,
                        float *anchor_d) {
    __shared__ WarpScratch ws[4];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const uint32_t chunk = blockIdx.x * 4 + wib;
    if (chunk >= total_chunks) return;
    const TileScene &d = scenes[scene_of_chunk(scenes, nsc, chunk)];
    const uint32_t wfirst = (chunk - d.chunk_begin) * (uint32_t)(32 * groups);
    const float4 a = d.qa[d.order[wfirst + min((uint32_t)kAnchorAt, d.n - 1 - wfirst)]];
    const MapView &m = __float_as_int(a.w) != kNone ? d.surf : d.vol;
    const uint64_t cap = make_key(d.r2cap, 0xffffffffu);
    Knn<S> kn;
    kn.reset(cap, d.k);
    knn_search<S>(m, mk3(a.x, a.y, a.z), kn, ws[wib], lane, cap);
    if (lane == 0) anchor_d[chunk] = kn.worst < cap ? sqrtf(key_d2(kn.worst)) : sqrtf(d.r2cap);
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

cudaError_t knn_values_tiles(const PScene &S, const MapView &surf, const MapView &vol,
                             const float4 *qa, const float4 *qd, const uint32_t *order, uint32_t n,
                             const uint32_t *n_dev, int groups, int k, float radius, bool raw,
                             float4 *val, const TileBuffers &buf, int sm_count, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    if (groups < 1 || groups > 4) return cudaErrorInvalidValue;
    const float r2 = radius * radius;
    const uint32_t chunks = tile_chunks(n, groups);
    const dim3 grid((chunks + kTileWarps - 1) / kTileWarps), block(kTileWarps * 32);
    const int smem = (int)(kTileWarps * sizeof(TileScratch));
    const dim3 dgrid(std::max(sm_count, 1) * 8);
    // defer_n[0]: deferred queries, defer_n[1]: the chunk counter
    cudaError_t e = cudaMemsetAsync(buf.defer_n, 0, 2 * sizeof(uint32_t), s);
    if (e != cudaSuccess) return e;
    int per_sm = 1;
    // persistent tile launch: as many blocks as fit on the GPU at once
#define PM_TILE_LAUNCH(SL)                                                                              \
    anchor_kernel<SL><<<grid, block, 0, s>>>(surf, vol, qa, order, n, n_dev, groups, k, r2, buf.anchor_d); \
    e = cudaFuncSetAttribute(query_knn_tile_kernel<SL>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem); \
    if (e != cudaSuccess) return e;                                                                     \
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, query_knn_tile_kernel<SL>, kTileWarps * 32, smem); \
    if (e != cudaSuccess) return e;                                                                     \
    query_knn_tile_kernel<SL><<<std::min<uint32_t>(grid.x, (uint32_t)std::max(sm_count, 1) * (uint32_t)std::max(per_sm, 1)), \
                                block, smem, s>>>(S, surf, vol, qa, qd, order, n, n_dev, groups, buf.anchor_d, k, \
                                                  r2, raw, val, buf.defer, buf.defer_n, buf.defer_n + 1, buf.stats); \
    deferred_kernel<SL><<<dgrid, 128, 0, s>>>(S, surf, vol, qa, qd, buf.defer, buf.defer_n, k, r2, raw, val)
    switch ((k + 31) / 32) {
        case 1: PM_TILE_LAUNCH(1); break;
        case 2: PM_TILE_LAUNCH(2); break;
        case 3: PM_TILE_LAUNCH(3); break;
        default: PM_TILE_LAUNCH(4); break;
    }
#undef PM_TILE_LAUNCH
    note_launches(3);
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
    anchor_multi_kernel<SL><<<agrid, block, 0, s>>>(scenes, nsc, total_chunks, groups, buf.anchor_d);   \
    e = cudaFuncSetAttribute(query_knn_tile_multi_kernel<SL>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem); \
    if (e != cudaSuccess) return e;                                                                     \
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, query_knn_tile_multi_kernel<SL>, kTileWarps * 32, smem); \
    if (e != cudaSuccess) return e;                                                                     \
    query_knn_tile_multi_kernel<SL><<<std::min<uint32_t>(agrid.x, (uint32_t)std::max(sm_count, 1) * (uint32_t)std::max(per_sm, 1)), \
                                      block, smem, s>>>(scenes, nsc, total_chunks, groups, buf.anchor_d, raw, \
                                                        buf.defer, defer_sc, buf.defer_n, buf.defer_n + 1, buf.stats); \
    deferred_multi_kernel<SL><<<dgrid, 128, 0, s>>>(scenes, buf.defer, defer_sc, buf.defer_n, raw)
    switch (slots) {
        case 1: PM_MULTI_LAUNCH(1); break;
        case 2: PM_MULTI_LAUNCH(2); break;
        case 3: PM_MULTI_LAUNCH(3); break;
        default: PM_MULTI_LAUNCH(4); break;
    }
#undef PM_MULTI_LAUNCH
    note_launches(3);
    return cudaGetLastError();
}

uint32_t tile_chunks(uint32_t n, int groups) { return (n + 32u * groups - 1) / (32u * groups); }

}  // namespace pm
