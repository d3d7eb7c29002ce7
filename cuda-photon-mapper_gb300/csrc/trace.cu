// trace.cu -- photon emission, scattering and storage.
//
// One persistent launch: each warp keeps 32 live photon paths and, whenever
// some lanes' paths end (escape, Russian roulette, bounce limit), refills
// exactly those lanes from a global path counter with a single atomic per
// warp (ballot of the empty lanes, ranks by popcount). Warps therefore stay
// full while paths of very different lengths finish, and no path state is
// ever written to memory. A path's randomness is a Philox stream keyed by
// (seed) and counted by (path, event, slot, scene), so a path's trajectory
// does not depend on which warp or lane traced it.
//
// Two passes over the same deterministic paths: the counting pass stores
// nothing and stops issuing paths once both maps are full; a scan of the
// per-path counts then fixes every record's final index (records in path
// order, cut at the map's target), a compaction lists the ids of the paths
// the maps need (those with a record below a map's extent: about a tenth of
// the issued paths when one map fills much later than the other), and the
// writing pass retraces exactly those and writes each record straight into
// the SoA float4 map arrays, its power scaled by the number of paths the map
// drew from. No per-path staging memory, no compaction of records.
#include "launch_count.cuh"
#include "trace.cuh"
#include "radix_sort.cuh"

#include <algorithm>
#include <cstddef>

namespace pm {
namespace {

__device__ __forceinline__ uint32_t lanemask_lt() {
    return (1u << (threadIdx.x & 31)) - 1u;
}

// Direction bin of d and the bin's centre line (not normalised).
__device__ __forceinline__ int near_bin(v3 d) {
    const float ax = fabsf(d.x), ay = fabsf(d.y), az = fabsf(d.z);
    const int a = ax >= ay && ax >= az ? 0 : (ay >= az ? 1 : 2);
    const float m = a == 0 ? d.x : (a == 1 ? d.y : d.z);
    const float r = __fdividef(0.5f * (float)kNearFace, fabsf(m));
    const float u = (a == 0 ? d.y : (a == 1 ? d.z : d.x)) * r, v = (a == 0 ? d.z : (a == 1 ? d.x : d.y)) * r;
    const int iu = min(max((int)(u + 0.5f * (float)kNearFace), 0), kNearFace - 1);
    const int iv = min(max((int)(v + 0.5f * (float)kNearFace), 0), kNearFace - 1);
    return ((2 * a + (m < 0.0f ? 1 : 0)) * kNearFace + iu) * kNearFace + iv;
}
__device__ __forceinline__ v3 near_direction(int face, float u, float v) {
    const int a = face >> 1;
    const float m = face & 1 ? -1.0f : 1.0f;
    return a == 0 ? mk3(m, u, v) : (a == 1 ? mk3(v, m, u) : mk3(u, v, m));
}

// One warp per (cell, direction bin). The cell is taken as the ball around
// it, the bin as the cone around it, both enlarged beyond any rounding: a
// sphere is listed when its centre is within its radius plus the ball's of
// the cone.
__global__ void __launch_bounds__(256) near_list_kernel(const __grid_constant__ PScene S,
                                                        const __grid_constant__ NearLists N, uint32_t lists,
                                                        uint16_t *out) {
    const uint32_t l = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (l >= lists) return;
    const int lane = threadIdx.x & 31;
    const int bin = (int)(l % kNearDirs), cell = (int)(l / kNearDirs);
    const int c[3] = {cell % N.g, (cell / N.g) % N.g, cell / (N.g * N.g)};
    float mid[3], rho = 0.0f;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const float w = 1.0f / N.inv[a];
        mid[a] = N.lo[a] + ((float)c[a] + 0.5f) * w;
        rho += 0.2601f * w * w;  // half the diagonal and one part in fifty: origins a little outside
    }
    rho = sqrtf(rho);
    const int iv = bin % kNearFace, iu = (bin / kNearFace) % kNearFace, face = bin / (kNearFace * kNearFace);
    const float h = 1.0f / (float)kNearFace;
    const float uc = (2.0f * (float)iu + 1.0f) * h - 1.0f, vc = (2.0f * (float)iv + 1.0f) * h - 1.0f;
    const v3 axis = normalize(near_direction(face, uc, vc));
    float ct = 1.0f;
#pragma unroll
    for (int q = 0; q < 4; ++q)
        ct = fminf(ct, dot(axis, normalize(near_direction(face, uc + (q & 1 ? h : -h), vc + (q & 2 ? h : -h)))));
    ct = ct - 1e-3f;
    const float st = sqrtf(fmaxf(0.0f, 1.0f - ct * ct));
    uint32_t key[2];
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const int i = lane + 32 * r;
        key[r] = 0xffffu;
        if (i < S.ns) {
            const float4 s = S.sph[i];
            const v3 p = mk3(s.x - mid[0], s.y - mid[1], s.z - mid[2]);
            const float len = sqrtf(dot(p, p)), z = dot(p, axis);
            const float off = sqrtf(fmaxf(0.0f, len * len - z * z));
            const float reach = (s.w + rho) * 1.001f + 1e-4f * len;
            const float dist = z * ct + off * st <= 0.0f ? len : off * ct - z * st;
            const float least = len - reach;
            if (dist <= reach)
                key[r] = (uint32_t)i | ((uint32_t)fminf(fmaxf(least, 0.0f) / N.unit, 250.0f) << 8);
        }
    }
    // places by (distance, sphere)
    int at[2] = {0, 0}, n = 0;
    const uint32_t k0 = (key[0] >> 8) * 256u + (key[0] & 255u), k1 = (key[1] >> 8) * 256u + (key[1] & 255u);
    for (int j = 0; j < 32; ++j) {
        const uint32_t o0 = __shfl_sync(0xffffffffu, k0, j), o1 = __shfl_sync(0xffffffffu, k1, j);
        at[0] += (o0 < k0 ? 1 : 0) + (o1 < k0 ? 1 : 0);
        at[1] += (o0 < k1 ? 1 : 0) + (o1 < k1 ? 1 : 0);
    }
    n = __popc(__ballot_sync(0xffffffffu, key[0] != 0xffffu)) + __popc(__ballot_sync(0xffffffffu, key[1] != 0xffffu));
    uint16_t *row = out + (size_t)l * kNearList;
#pragma unroll
    for (int r = 0; r < 2; ++r)
        if (key[r] != 0xffffu && at[r] < kNearList - 1) row[at[r]] = (uint16_t)key[r];
    if (lane == 0) row[min(n, kNearList - 1)] = (uint16_t)(n > kNearList - 1 ? kNearMore : kNearEnd);
}

// intersect() through the lists (trace.cuh): the spheres of the origin's cell and the
// direction's bin by least distance, until the hit is nearer than the next.
// Equal distances keep the lower index, so the hit is intersect()'s. An origin
// outside the box, and a list that does not hold all its spheres, test every
// sphere. The lanes' rays differ, so a warp waits for its longest list: in the
// 64-sphere preset a lane tests 4 spheres, a warp's longest about 11, instead
// of 64. An entry is one 16-bit load a test ahead of its use (entries shifted
// out of registers, the distance as a float compared: 34.3 -> 33.3 ms for 8M
// records); whoever has more to test keeps the warp (lanes left walking while
// the others go on: 33.7).
__device__ __forceinline__ PHit intersect_near(const PScene &S, const PScene &U, const NearLists &N, v3 o, v3 d,
                                               float tmax) {
    PHit h;
    h.t = tmax;
    h.obj = kNone;
    const float f[3] = {(o.x - N.lo[0]) * N.inv[0], (o.y - N.lo[1]) * N.inv[1], (o.z - N.lo[2]) * N.inv[2]};
    const float top = (float)N.g + 0.01f;
    bool all = !(f[0] > -0.01f && f[1] > -0.01f && f[2] > -0.01f && f[0] < top && f[1] < top && f[2] < top);
    if (!all) {
        const int g1 = N.g - 1;
        const int cx = min(max((int)f[0], 0), g1), cy = min(max((int)f[1], 0), g1), cz = min(max((int)f[2], 0), g1);
        const uint16_t *at = reinterpret_cast<const uint16_t *>(N.list) +
                             ((size_t)((cz * N.g + cy) * N.g + cx) * kNearDirs + near_bin(d)) * kNearList;
        uint32_t e = __ldg(at), lim = 0xfe00u;  // entries from lim on are no nearer than the hit
        while (e < lim) {
            const uint32_t k = e & 255u;
            e = __ldg(++at);
            const float t = sphere_t(S.sph[k], o, d);
            if (t > kRayEps && (t < h.t || (t == h.t && h.obj != kNone && (int)k < h.obj))) {
                h.t = t;
                h.obj = (int)k;
                lim = ((uint32_t)fminf(t * N.inv_unit, 252.0f) + 1u) << 8;
            }
        }
        all = e == kNearMore;
    }
    if (all)
        for (int i = 0; i < S.ns; ++i) {
            const float t = sphere_t(S.sph[i], o, d);
            if (t > kRayEps && (t < h.t || (t == h.t && h.obj != kNone && i < h.obj))) { h.t = t; h.obj = i; }
        }
    plane_hits(U, o, d, h);
    return h;
}

struct Path {
    v3 o, d, thr;
    uint32_t id;
    int ev;
    bool glass;
    uint32_t ns, nv;
    uint32_t os, ov;  // writing pass: the path's first record index in each map
};

__device__ __forceinline__ void start_path(const TraceParams &P, uint32_t id, Path &p, const PScene &S) {
    pm_u32x4 r = philox(P.seed, id, 0u, 0u, P.scene_id);
    p.o = mk3(S.light[0], S.light[1], S.light[2]);
    p.d = sample_sphere(pm_u01(r.v[0]), pm_u01(r.v[1]));
    p.thr = mk3(1.0f, 1.0f, 1.0f);
    p.id = id;
    p.ev = 0;
    p.glass = false;
    p.ns = 0;
    p.nv = 0;
    if (P.store) {  // loaded now, used at the path's first stores
        p.os = P.off_s[id];
        p.ov = P.off_v[id];
    }
}

__device__ __forceinline__ void store(float4 *pos, float4 *pw, uint32_t j, v3 x, v3 thr, v3 d,
                                      float scale) {
    pos[j] = make_float4(x.x, x.y, x.z, __uint_as_float(j));
    pw[j] = make_float4(thr.x * scale, thr.y * scale, thr.z * scale, __uint_as_float(oct_encode(d)));
}

struct MapOut {
    uint32_t n, paths;
    float scale;
};

// One interaction of path p; returns false when the path ends. S is read at
// each lane's own object, U (the same scene) at one place by the whole warp.
//
// The instructions issued bound it, and how few lanes share them (15 of 32 in
// preset 3). So the lanes meet again after the hit and after the tracking,
// whose loop the compiler leaves in groups (39.1 -> 35.5 ms for 8M records of
// preset 3); a surface and the medium share the scattered direction's sine,
// frame and record, all kinds the last normalisation (with the planes' axes
// told apart by branches and read from the parameters 35.5 -> 34.3; preset 2,
// 1M records: 1.73 -> 1.63).
template <bool kNear>
__device__ __forceinline__ bool step_path(const PScene &S, const PScene &U, const TraceParams &P, Path &p,
                                          const MapOut &ms, const MapOut &mv) {
    p.ev += 1;
    pm_u32x4 r = philox(P.seed, p.id, (uint32_t)p.ev, 0u, P.scene_id);
    float u0 = pm_u01(r.v[0]), u1 = pm_u01(r.v[1]), u2 = pm_u01(r.v[2]), u3 = pm_u01(r.v[3]);
    // without lists a uniform loop over the spheres beats divergent walks
    // of a grid
    const unsigned together = __activemask();
    const PHit h = kNear ? intersect_near(S, U, P.near, p.o, p.d, 3.0e38f) : intersect(U, p.o, p.d, 3.0e38f);
    float seg = h.obj != kNone ? h.t : box_exit(U, p.o, p.d);
    __syncwarp(together);
    bool vol = false;
    v3 x = p.o;
    float ss = 0.0f, st = 1.0f;
    if (U.sigma_max > 0.0f && !p.glass) {
        if (U.het_res <= 0) {
            st = U.sigma_s + U.sigma_a;
            if (U.sigma_s > 0.0f) {
                float t = -pm_logf(1.0f - u0) / st;
                if (t < seg) {
                    vol = true;
                    x = p.o + p.d * t;
                    ss = U.sigma_s;
                }
            }
        } else {
            // Delta tracking against the majorant (Woodcock et al. 1965):
            // tentative collision j draws its distance and acceptance from
            // words 2(j % 2), 2(j % 2) + 1 of Philox block 1 + j / 2.
            float t = 0.0f;
            pm_u32x4 q;
            for (uint32_t j = 0; j < kMaxDeltaSteps; ++j) {
                if ((j & 1u) == 0u) q = philox(P.seed, p.id, (uint32_t)p.ev, 1u + (j >> 1), P.scene_id);
                const uint32_t ua = (j & 1u) ? q.v[2] : q.v[0], ub = (j & 1u) ? q.v[3] : q.v[1];
                t += -pm_logf(1.0f - pm_u01(ua)) * U.inv_sigma_max;
                if (!(t < seg)) break;
                v3 y = p.o + p.d * t;
                float s = sigma_s_at(U, y);
                float sty = s + U.sigma_a;
                if (pm_u01(ub) * U.sigma_max < sty) {
                    vol = true;
                    x = y;
                    ss = s;
                    st = sty;
                    break;
                }
            }
        }
    }
    __syncwarp(together);
    v3 n = mk3(0.0f, 0.0f, 0.0f);
    float dn = 0.0f;
    int kind = PM_MAT_DIFFUSE;
    if (!vol) {
        if (h.obj == kNone) return false;  // leaves through the open side
        x = p.o + p.d * h.t;
        n = outward_normal(S, h.obj, x);
        kind = material_kind(S, h.obj);
        dn = dot(n, p.d);
    }
    v3 v;  // the new direction, not normalised
    if (kind == PM_MAT_DIFFUSE) {  // or in the medium
        if (P.store) {
            const uint32_t j = vol ? p.ov + p.nv : p.os + p.ns;
            if (j < (vol ? mv.n : ms.n))
                store(vol ? P.vpos : P.spos, vol ? P.vpow : P.spow, j, x, p.thr, p.d, vol ? mv.scale : ms.scale);
        }
        p.nv += vol ? 1 : 0;
        p.ns += vol ? 0 : 1;
        if (!(u1 < P.rr)) return false;
        float r, z;
        v3 axis;
        if (vol) {
            p.thr = p.thr * ((ss / st) / P.rr);
            hg_cosine(S.g, u2, &z, &r);
            axis = p.d;
            p.o = x;
        } else {
            const v3 a = material_albedo(S, h.obj);
            p.thr = mk3(p.thr.x * a.x / P.rr, p.thr.y * a.y / P.rr, p.thr.z * a.z / P.rr);
            axis = dn < 0.0f ? n : n * -1.0f;
            r = sqrtf(u2);
            z = sqrtf(fmaxf(0.0f, 1.0f - u2));
            p.o = x + axis * kOffset;
        }
        float sn, cs;
        pm_sincos2pi(u3, &sn, &cs);
        v = from_local(axis, r * cs, r * sn, z);
    } else if (kind == PM_MAT_MIRROR) {
        v = p.d - n * (2.0f * dn);
        p.o = x + (dn < 0.0f ? n : n * -1.0f) * kOffset;
    } else {
        float ci = -dn;
        bool entering = ci > 0.0f;
        float ior = material_ior(S, h.obj);
        float eta = entering ? 1.0f / ior : ior;
        v3 nn = entering ? n : n * -1.0f;
        ci = fabsf(ci);
        float ct;
        float F = fresnel(ci, eta, &ct);
        if (u1 < F) {
            v = p.d + nn * (2.0f * ci);
            p.o = x + nn * kOffset;
        } else {
            v = p.d * eta + nn * (eta * ci - ct);
            p.o = x - nn * kOffset;
            p.glass = entering;
        }
    }
    p.d = normalize(v);
    return p.ev < P.max_bounces;
}

// Path ids come in blocks of kIdBlock per atomic. A warp always holds the
// next block's atomic in flight (issued when it takes the current one), so
// refilling lanes rarely waits for the counter; every block a warp takes is
// traced in full (the ids stay a gap-free prefix, which the record extents
// need), and the counting pass stops requesting blocks once both maps are
// full. The records of finished paths are counted in registers and added to
// the maps' counters once per block; the sums those atomics return, looked
// at when the warp takes its next block, say whether the maps are full. One
// addition per finished path instead puts three billion atomics a second on
// two addresses, which is about what one L2 sector serves: it, not the
// tracing, bounded scenes of few spheres (preset 2, 8.5M paths: 3.51 -> 1.72
// ms; preset 1, 1.1M paths: 0.54 -> 0.38 ms).
constexpr uint32_t kIdBlock = 32;

// The persistent per-warp loop of one scene: keep 32 live paths, refill
// empty lanes from the warp's pool of path ids until no ids are left.
template <bool kNear>
__device__ __forceinline__ void trace_loop(const PScene &S, const PScene &U, const TraceParams &P) {
    const int lane = threadIdx.x & 31;
    MapOut ms = {0u, 0u, 0.0f}, mv = {0u, 0u, 0.0f};
    uint32_t cap = P.path_cap;
    if (P.store) {
        ms.n = P.ext_s[0]; ms.paths = P.ext_s[1];
        mv.n = P.ext_v[0]; mv.paths = P.ext_v[1];
        ms.scale = ms.paths ? P.power / (float)ms.paths : 0.0f;
        mv.scale = mv.paths ? P.power / (float)mv.paths : 0.0f;
        cap = P.list ? *P.list_n : max(ms.paths, mv.paths);
    }
    Path p;
    bool live = false;
    // warp-uniform pool [pool, pool_end); lane 0 holds the prefetched block
    uint32_t pool = 0, pool_end = 0, pending = 0;
    uint32_t done_s = 0, done_v = 0;  // counting pass: this lane's records not yet added
    uint32_t seen_s = 0, seen_v = 0;  // lane 0: the counters after the warp's last addition
    bool has_pending = cap > 0;
    if (has_pending && lane == 0) pending = atomicAdd(P.path_counter, kIdBlock);
    for (;;) {
        const unsigned empty = __ballot_sync(0xffffffffu, !live);
        const uint32_t need = (uint32_t)__popc(empty);
        if (need && (pool < pool_end || has_pending)) {
            const uint32_t avail = pool_end - pool;
            uint32_t nb = 0;
            bool took = false;
            if (avail < need && has_pending) {
                nb = __shfl_sync(0xffffffffu, pending, 0);
                has_pending = false;
                took = true;
                bool more = nb < cap && cap - nb > kIdBlock;
                if (more && !P.store) {
                    const int full = seen_s >= P.target_s && seen_v >= P.target_v;
                    more = __shfl_sync(0xffffffffu, full, 0) == 0;
                    const uint32_t ns = __reduce_add_sync(0xffffffffu, done_s);
                    const uint32_t nv = __reduce_add_sync(0xffffffffu, done_v);
                    done_s = done_v = 0;
                    if (lane == 0) {
                        seen_s = atomicAdd(P.stored_s, ns) + ns;
                        seen_v = atomicAdd(P.stored_v, nv) + nv;
                    }
                }
                if (more) {
                    if (lane == 0) pending = atomicAdd(P.path_counter, kIdBlock);
                    has_pending = true;
                }
            }
            const uint32_t r = (uint32_t)__popc(empty & lanemask_lt());
            uint32_t id = cap;
            if (r < avail) id = pool + r;
            else if (took) id = nb + (r - avail);
            if (took) {
                const uint32_t used = need > avail ? need - avail : 0u;
                pool = nb + min(used, kIdBlock);
                pool_end = nb + kIdBlock;
                if (nb >= cap) pool = pool_end;  // nothing left below the cap
            } else {
                pool += min(need, avail);
            }
            if (!live && id < cap) {
                // the writing pass retraces only paths with a record in a map:
                // those of its list, or (without a list) the ids whose counts
                // are nonzero
                uint32_t pid = id;
                bool needed = true;
                if (P.store) {
                    if (P.list) pid = P.list[id];
                    else needed = (id < ms.paths && P.cnt_s[id] > 0u) || (id < mv.paths && P.cnt_v[id] > 0u);
                }
                if (needed) {
                    start_path(P, pid, p, S);
                    live = true;
                }
            }
        }
        if (!__any_sync(0xffffffffu, live)) {
            if (pool >= pool_end && !has_pending) break;
            continue;
        }
        if (live) {
            if (!step_path<kNear>(S, U, P, p, ms, mv)) {
                if (!P.store) {
                    uint32_t ns = min(p.ns, (uint32_t)P.max_bounces);
                    uint32_t nv = min(p.nv, (uint32_t)P.max_bounces);
                    P.cnt_s[p.id] = ns;
                    P.cnt_v[p.id] = nv;
                    done_s += ns;
                    done_v += nv;
                }
                live = false;
            }
        }
    }
}

// What the lanes read at their own objects (materials, normals, listed
// spheres) is read from shared memory: the constant bank serves one address at
// a time (preset 3, 87.6M paths: 57.8 -> 56.1 ms). Blocks per SM: the lists'
// loads want the ninth (56 registers; 32.3 -> 31.5 ms), small scenes have no
// use for it (0.37 / 0.38 ms in preset 1: more paths beyond the last needed).
constexpr int trace_blocks(bool near) { return near ? 9 : 8; }
template <bool kNear>
__global__ void __launch_bounds__(128, trace_blocks(kNear)) trace_kernel(const __grid_constant__ PScene S,
                                                                          const __grid_constant__ TraceParams P) {
    __shared__ PScene sS;
    const uint32_t *a = reinterpret_cast<const uint32_t *>(&S);
    uint32_t *b = reinterpret_cast<uint32_t *>(&sS);
    for (int i = threadIdx.x; i < (int)(offsetof(PScene, cell_mask) / 4); i += blockDim.x) b[i] = a[i];
    __syncthreads();
    trace_loop<kNear>(sS, S, P);
}

// Many scenes in one persistent launch: every block walks the scene list
// (starting at a different scene per block, so scenes are worked on side
// by side), stages the scene in shared memory and traces its paths with
// the single-scene loop until the scene's path ids run out. 64 registers for
// 8 blocks an SM, as the grid has (72: six scenes' frame 48.5 ms, 64: 48.0).
__global__ void __launch_bounds__(128, 8) trace_batch_kernel(const PScene *scenes,
                                                          const TraceParams *params, int n) {
    __shared__ PScene sS;
    __shared__ TraceParams sP;
    for (int j = 0; j < n; ++j) {
        const int sc = (int)((blockIdx.x + (unsigned)j) % (unsigned)n);
        __syncthreads();
        const uint32_t *a = reinterpret_cast<const uint32_t *>(&scenes[sc]);
        uint32_t *b = reinterpret_cast<uint32_t *>(&sS);
        for (int i = threadIdx.x; i < (int)(sizeof(PScene) / 4); i += blockDim.x) b[i] = a[i];
        const uint32_t *c = reinterpret_cast<const uint32_t *>(&params[sc]);
        uint32_t *d = reinterpret_cast<uint32_t *>(&sP);
        for (int i = threadIdx.x; i < (int)(sizeof(TraceParams) / 4); i += blockDim.x) d[i] = c[i];
        __syncthreads();
        trace_loop<false>(sS, sS, sP);
    }
}

// Smallest path count whose records reach the target (or all issued paths).
__device__ void find_extent(const uint32_t *off, const uint32_t *cnt, uint32_t issued, uint32_t total,
                            uint32_t target, uint32_t *extent) {
    if (target == 0) {
        extent[0] = 0;
        extent[1] = 0;
        return;
    }
    if (total <= target) {
        extent[0] = total;   // records
        extent[1] = issued;  // paths
        return;
    }
    uint32_t lo = 0, hi = issued;  // first p with off[p] + cnt[p] >= target
    while (lo < hi) {
        uint32_t mid = (lo + hi) >> 1;
        if (off[mid] + cnt[mid] >= target) hi = mid; else lo = mid + 1;
    }
    extent[0] = target;
    extent[1] = lo + 1;
}

__global__ void map_extent_kernel(const uint32_t *off, const uint32_t *cnt, uint32_t issued,
                                  const uint32_t *issued_dev, const uint32_t *total_p,
                                  uint32_t target, uint32_t *extent) {
    if (issued_dev) issued = min(*issued_dev, issued);
    find_extent(off, cnt, issued, *total_p, target, extent);
}

__global__ void map_extents_kernel(const ExtentJob *jobs, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const ExtentJob j = jobs[i];
    if (j.cap == 0) {
        j.extent[0] = 0;
        j.extent[1] = 0;
        return;
    }
    const uint32_t total = j.off[j.cap - 1] + j.cnt[j.cap - 1];
    *j.total = total;
    find_extent(j.off, j.cnt, min(*j.issued, j.cap), total, j.target, j.extent);
}

constexpr uint32_t kNeedTile = 1024;

// Needed paths per tile of kNeedTile ids, and a bit per id. Four ids a
// thread in 16-byte loads (87.8M paths, 0.7 GB of counts: 117 us; one id a thread: 293).
__global__ void __launch_bounds__(kNeedTile / 4) need_count_kernel(uint32_t issued, const uint32_t *cnt_s,
                                                                   const uint32_t *cnt_v, const uint32_t *ext_s,
                                                                   const uint32_t *ext_v, uint32_t *tile_cnt,
                                                                   uint32_t *bits) {
    __shared__ uint32_t warp_n[kNeedTile / 128];
    const int lane = threadIdx.x & 31;
    const uint32_t id = blockIdx.x * kNeedTile + 4u * threadIdx.x;
    const uint32_t ps = min(ext_s[1], issued), pv = min(ext_v[1], issued);
    const uint4 a = load_words4(cnt_s, id, ps), b = load_words4(cnt_v, id, pv);
    uint32_t w = ((a.x | b.x) ? 1u : 0u) | ((a.y | b.y) ? 2u : 0u) | ((a.z | b.z) ? 4u : 0u) | ((a.w | b.w) ? 8u : 0u);
    const uint32_t n = __reduce_add_sync(0xffffffffu, (uint32_t)__popc(w));
    w = __reduce_or_sync(0xffu << (lane & 24), w << (4 * (lane & 7)));
    if ((lane & 7) == 0) bits[id >> 5] = w;
    if (lane == 0) warp_n[threadIdx.x >> 5] = n;
    __syncthreads();
    if (threadIdx.x < 32) {
        const uint32_t v = __reduce_add_sync(0xffffffffu, lane < kNeedTile / 128 ? warp_n[lane] : 0u);
        if (lane == 0) tile_cnt[blockIdx.x] = v;
    }
}

// Each tile's needed ids, in order, at the tile's offset: a warp per tile,
// from its 32 words of bits (39 us; the counts read again: 393).
__global__ void __launch_bounds__(256) need_scatter_kernel(uint32_t tiles, const uint32_t *bits,
                                                           const uint32_t *tile_off, uint32_t *list) {
    const uint32_t tile = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (tile >= tiles) return;
    const int lane = threadIdx.x & 31;
    const uint32_t own = bits[tile * (kNeedTile / 32) + lane];
    uint32_t at = tile_off[tile];
    for (int i = 0; i < (int)(kNeedTile / 32); ++i) {
        const uint32_t w = __shfl_sync(0xffffffffu, own, i);
        if ((w >> lane) & 1u) list[at + __popc(w & lanemask_lt())] = tile * kNeedTile + 32u * i + lane;
        at += __popc(w);
    }
}

}  // namespace

uint32_t needed_tiles(uint32_t n) { return (n + kNeedTile - 1) / kNeedTile + 1; }
uint32_t needed_words(uint32_t n) { return needed_tiles(n) * (1u + kNeedTile / 32u); }

cudaError_t needed_paths(uint32_t issued, const uint32_t *cnt_s, const uint32_t *cnt_v,
                         const uint32_t *ext_s, const uint32_t *ext_v, uint32_t *tile_cnt,
                         uint32_t *tile_off, uint32_t *scan_tmp, uint32_t *list, uint32_t *list_n,
                         cudaStream_t s) {
    if (issued == 0) return cudaMemsetAsync(list_n, 0, sizeof(uint32_t), s);
    const uint32_t tiles = (issued + kNeedTile - 1) / kNeedTile;
    uint32_t *bits = tile_cnt + needed_tiles(issued);
    need_count_kernel<<<tiles, kNeedTile / 4, 0, s>>>(issued, cnt_s, cnt_v, ext_s, ext_v, tile_cnt, bits);
    note_launch();
    cudaError_t e = exclusive_scan_u32_large(tile_cnt, tile_off, tiles, list_n, scan_tmp, s);
    if (e != cudaSuccess) return e;
    need_scatter_kernel<<<(tiles + 7) / 8, 256, 0, s>>>(tiles, bits, tile_off, list);
    note_launch();
    return cudaGetLastError();
}

size_t near_lists_words(int g) { return (size_t)g * g * g * kNearDirs * (kNearList / 8); }

int near_lists_grid(int ns, uint32_t target) {
    // What the lists save grows with the spheres beyond about a dozen and with
    // the records; the table costs 0.3 (12 cells an axis), 0.7 (16) or 1.5 ms
    // (20) when the scene has changed, and every emission of 14M units or more
    // wins that back. Emission (ms) without the lists / with them and the table's
    // building / with a table kept, at 12 cells: 48 spheres, 300,000 records 1.99
    // / 1.95 / 1.65; 32, 500,000 2.44 / 2.49 / 2.22 and 1M 4.35 / 4.16 / 3.91;
    // 24, 1M 3.94 / 3.99 / 3.74; 16, 2M 5.94 / 6.04 / 5.79 and 4M 11.43 / 11.32 /
    // 11.08. 64 spheres: 1M 7.00, 5.21 / 4.85 at 12, 5.32 / 4.54 at 16, 5.90 /
    // 4.39 at 20; 8M 51.0, 33.4 / 32.6 at 16, 33.0 / 31.5 at 20, 33.5 / 30.9 at 24.
    const uint64_t units = ns > 12 ? (uint64_t)(ns - 12) * target : 0;
    if (units < 14000000ull) return 0;
    return units < 40000000ull ? 12 : (units < 160000000ull ? 16 : 20);
}

cudaError_t build_near_lists(const PScene &S, int g, uint4 *list, NearLists *out, cudaStream_t s) {
    NearLists N;
    N.list = list;
    N.g = g;
    float diag = 0.0f;
    for (int a = 0; a < 3; ++a) {
        const float ext = S.bmax[a] - S.bmin[a];
        N.lo[a] = S.bmin[a];
        N.inv[a] = (float)g / ext;
        diag += ext * ext;
    }
    N.unit = sqrtf(diag) / 250.0f;
    N.inv_unit = 1.00001f / N.unit;
    *out = N;
    const uint32_t lists = (uint32_t)g * g * g * kNearDirs;
    near_list_kernel<<<(lists + 7) / 8, 256, 0, s>>>(S, N, lists, reinterpret_cast<uint16_t *>(list)); note_launch();
    return cudaGetLastError();
}

cudaError_t trace_photons(const PScene &S, const TraceParams &P, int sm_count, cudaStream_t s) {
    if (P.near.list) trace_kernel<true><<<sm_count * trace_blocks(true), 128, 0, s>>>(S, P);
    else trace_kernel<false><<<sm_count * trace_blocks(false), 128, 0, s>>>(S, P);
    note_launch();
    return cudaGetLastError();
}

cudaError_t map_extent(uint32_t issued, const uint32_t *cnt, uint32_t *off, uint32_t *total,
                       uint32_t *scan_tmp, uint32_t target, uint32_t *extent, cudaStream_t s) {
    if (issued == 0) return cudaMemsetAsync(extent, 0, 2 * sizeof(uint32_t), s);
    cudaError_t e = exclusive_scan_u32_large(cnt, off, issued, total, scan_tmp, s);
    if (e != cudaSuccess) return e;
    map_extent_kernel<<<1, 1, 0, s>>>(off, cnt, issued, nullptr, total, target, extent); note_launch();
    return cudaGetLastError();
}

cudaError_t map_extent_dev(uint32_t cap, const uint32_t *issued_dev, const uint32_t *cnt,
                           uint32_t *off, uint32_t *total, uint32_t *scan_tmp, uint32_t target,
                           uint32_t *extent, cudaStream_t s) {
    if (cap == 0) return cudaMemsetAsync(extent, 0, 2 * sizeof(uint32_t), s);
    cudaError_t e = exclusive_scan_u32_large(cnt, off, cap, total, scan_tmp, s);
    if (e != cudaSuccess) return e;
    map_extent_kernel<<<1, 1, 0, s>>>(off, cnt, cap, issued_dev, total, target, extent); note_launch();
    return cudaGetLastError();
}

cudaError_t map_extents_multi(const ExtentJob *jobs, int n, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    map_extents_kernel<<<(n + 127) / 128, 128, 0, s>>>(jobs, n); note_launch();
    return cudaGetLastError();
}

cudaError_t trace_photons_batch(const PScene *scenes, const TraceParams *params, int n,
                                int sm_count, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    trace_batch_kernel<<<sm_count * 8, 128, 0, s>>>(scenes, params, n); note_launch();
    return cudaGetLastError();
}

namespace {

__global__ void pad_map_kernel(float4 *pos, float4 *pw, const uint32_t *n_dev, uint32_t cap) {
    const uint32_t n = *n_dev;
    const float inf = __int_as_float(0x7f800000);
    for (uint32_t i = n + blockIdx.x * blockDim.x + threadIdx.x; i < cap; i += gridDim.x * blockDim.x) {
        pos[i] = make_float4(inf, inf, inf, __uint_as_float(i));
        pw[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
}

}  // namespace

cudaError_t pad_map(float4 *pos, float4 *pw, const uint32_t *n_dev, uint32_t cap, cudaStream_t s) {
    if (cap == 0) return cudaSuccess;
    const uint32_t blocks = std::min<uint32_t>((cap + 255) / 256, 4096);
    pad_map_kernel<<<blocks, 256, 0, s>>>(pos, pw, n_dev, cap); note_launch();
    return cudaGetLastError();
}

}  // namespace pm
