// legacy.cu -- sm_103a kernels for the reference's voxel photon mapper.
//
// Arithmetic follows photonMappingKernel.cu operation for operation
// (single rounding per float operation, double precision where the
// reference's double literals promote an expression), so the grid and the
// image equal a serial run of the reference's own code. The structure is
// new: the unrolled specular recursion (:673-827) is one bounded loop,
// sphere animation is computed once on the host instead of by every
// thread, the random table is filled in parallel by jumping the generator
// ahead, and grid accumulation is a deterministic sort + ordered sum.
#include "launch_count.cuh"
#include "legacy.cuh"
#include "legacy_voxel.cuh"
#include "pm_vec.cuh"
#include "radix_sort.cuh"

#include <cmath>

namespace pm {
namespace {

constexpr int G = kLegacyGrid;

struct Scene {
    float sph[2][4];  // the two traced spheres (nrObjects = {2,5}, :61)
};

// planes[] (:66-72), folded into the unrolled loop over them
__device__ __forceinline__ int plane_axis(int i) { return i == 4 ? 2 : i & 1; }
__device__ __forceinline__ float plane_off(int i) {
    return i == 4 ? 6.0f : (i == 0 || i == 3 ? 1.5f : -1.5f);
}
__constant__ float c_vox_dim[3] = {0.09375f, 0.09375f, 0.1875f};  // getVoxelDim (:426-437)

__device__ __forceinline__ v3 light_pos() { return mk3(0.0f, 1.4f, 3.5f); }  // Light (:64)

struct Hit {
    float dist;
    int type, idx;
    bool hit;
};

__device__ __forceinline__ void consider(Hit &h, float t, int type, int idx) {  // :100-103
    if (t < h.dist && t > 0.0f) { h.type = type; h.idx = idx; h.dist = t; h.hit = true; }
}

// raytrace (:223-241) over the two spheres (:105-126) and five planes (:130-157).
__device__ void trace(const Scene &sc, v3 r, v3 o, Hit &h) {
    h.hit = false;
    h.dist = 999999.9f;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        v3 s = mk3(sc.sph[i][0], sc.sph[i][1], sc.sph[i][2]) - o;
        float rad = sc.sph[i][3];
        float A = dot(r, r);
        float B = -2.0f * dot(s, r);  // a power of two: exact, as in double
        float C = dot(s, s) - rad * rad;
        float D = B * B - (4.0f * A) * C;
        if (D > 0.0f) {
            float sign = C < -0.00001f ? 1.0f : -1.0f;  // no float lies between the constant and its double
            consider(h, (-B + sign * sqrtf(D)) / (2.0f * A), 0, i);
        }
    }
#pragma unroll
    for (int i = 0; i < 5; ++i) {
        float ra = axis_of(r, plane_axis(i));
        if (ra != 0.0f) consider(h, (plane_off(i) - axis_of(o, plane_axis(i))) / ra, 1, i);
    }
}

// surfaceNormal (:178-201).
__device__ v3 normal_at(const Scene &sc, int type, int idx, v3 p, v3 from) {
    if (type == 0) return normalize(p - mk3(sc.sph[idx][0], sc.sph[idx][1], sc.sph[idx][2]));
    v3 n = mk3(0.0f, 0.0f, 0.0f);
    set_axis(n, plane_axis(idx), axis_of(from, plane_axis(idx)) - plane_off(idx));
    return normalize(n);
}

__device__ v3 reflect_ray(const Scene &sc, v3 ray, v3 from, int type, int idx, v3 p) {  // :663-668
    v3 n = normal_at(sc, type, idx, p, from) * 1.0f;
    return normalize(ray - n * (2.0f * dot(ray, n)));
}

__device__ v3 refract_ray(const Scene &sc, v3 ray, int type, int idx, v3 p, float factor) {  // :620-659
    v3 n = normal_at(sc, type, idx, p, p) * factor;
    float eta = 1.0f / 1.3f;
    if (factor == -1.0f) eta = 1.0f;
    float cos_i = -dot(n, ray);
    float cos_t2 = (float)(1.0 - (double)(eta * eta) * (1.0 - (double)(cos_i * cos_i)));
    if (cos_t2 > 0.0f) return ray * eta + n * (eta * cos_i - sqrtf(cos_t2));
    return mk3(0.0f, 0.0f, 0.0f);
}

struct Chain {
    v3 ray, point;
    Hit h;
};

// Specular chain (:673-827): stages 1..8 alternate mirror reflection (odd)
// and glass refraction (even); a reflection continues when it lands on the
// glass sphere, a refraction when its exit ray lands on the mirror sphere.
__device__ void run_chain(const Scene &sc, Chain &c, int first, v3 from) {
    for (int st = first; st <= 8; ++st) {
        bool more;
        if (st & 1) {
            c.ray = reflect_ray(sc, c.ray, from, c.h.type, c.h.idx, c.point);
            trace(sc, c.ray, c.point, c.h);
            if (!c.h.hit) break;
            c.point = c.ray * c.h.dist + c.point;
            more = c.h.type == 0 && c.h.idx == 0;
        } else {
            c.ray = refract_ray(sc, c.ray, c.h.type, c.h.idx, c.point, 1.0f);
            c.point = c.ray * 0.00001f + c.point;
            trace(sc, c.ray, c.point, c.h);
            c.point = c.ray * c.h.dist + c.point;
            if (!(c.h.hit && c.h.type == 0 && c.h.idx == 0)) break;
            c.ray = refract_ray(sc, c.ray, c.h.type, c.h.idx, c.point, -1.0f);
            c.point = c.ray * 0.00001f + c.point;
            trace(sc, c.ray, c.point, c.h);
            c.point = c.ray * c.h.dist + c.point;
            more = c.h.type == 0 && c.h.idx == 1;
        }
        if (!more) break;
    }
}

struct I3 {
    int x, y, z;
};

__device__ __forceinline__ I3 voxel_of(v3 p) {  // getVoxelCoordinates (:254-261)
    I3 v;
    v.x = legacy_voxel_xy(p.x);
    v.y = legacy_voxel_xy(p.y);
    v.z = legacy_voxel_z(p.z);
    return v;
}

__device__ __forceinline__ v3 voxel_center(v3 p) {  // centerPoint + getWorldCoordinates (:263-268, 392-400)
    I3 v = voxel_of(p);
    v3 c = mk3(legacy_world_xy(v.x), legacy_world_xy(v.y), legacy_world_z(v.z));
    return c + mk3(0.046875f, 0.046875f, 0.09375f);
}

__device__ __forceinline__ int lo_edge(int c, int lo) { return (c - 3 >= lo) ? c - 3 : lo; }
__device__ __forceinline__ int hi_edge(int c, int hi) { return (c + 3 <= hi) ? c + 3 : hi; }
__device__ __forceinline__ int vox_index(int i, int j, int k) { return (i * G + j) * G + k; }

__device__ __forceinline__ v3 grid_at(const float4 *__restrict__ g, int i, int j, int k) {
    float4 q = __ldg(&g[vox_index(i, j, k)]);
    return mk3(q.x, q.y, q.z);
}

// integrate + computeEnergy (:286-389): the plane's wall-slab window.
__device__ v3 integrate_slab(const float4 *__restrict__ g, v3 e, I3 wp, int type, int id) {
    v3 acc = e;
    if (type != 1) return acc;
    int x0 = lo_edge(wp.x, 0), y0 = lo_edge(wp.y, 0), z0 = lo_edge(wp.z, 0);
    int x1 = hi_edge(wp.x, G), y1 = hi_edge(wp.y, G), z1 = hi_edge(wp.z, G);
    if (id == 0 || id == 2) {
        int i = id == 0 ? G - 1 : 0;
        for (int j = y0; j < y1; ++j)
            for (int k = z0; k < z1; ++k) acc = acc + grid_at(g, i, j, k) * 0.0005f;
    } else if (id == 1 || id == 3) {
        int j = id == 1 ? 0 : G - 1;
        for (int i = x0; i < x1; ++i)
            for (int k = z0; k < z1; ++k) acc = acc + grid_at(g, i, j, k) * 0.0005f;
    } else if (id == 4) {
        int k = G - 1;
        for (int i = x0; i < x1; ++i)
            for (int j = y0; j < y1; ++j) acc = acc + grid_at(g, i, j, k) * 0.0005f;
    }
    return acc;
}

__device__ __forceinline__ v3 lerp3(v3 a, v3 b, float t) {  // interpolate3f (:421-423)
    // 1 - t rounds to the same float as through double: the double is exact
    // unless t is below 2^-29, where both give 1
    return a * (1.0f - t) + b * t;
}

__device__ __forceinline__ float alpha_of(v3 p, v3 a, v3 b, int ax) {  // getAlpha (:404-418)
    return (axis_of(p, ax) - axis_of(a, ax)) / (axis_of(b, ax) - axis_of(a, ax));
}

// integrateVolumePhotons (:831-870) at voxel wp (getVoxelCoordinates of
// the march point).
__device__ v3 integrate_volume(const float4 *__restrict__ g, I3 wp) {
    v3 acc = mk3(0.0f, 0.0f, 0.0f);
    int x0 = lo_edge(wp.x, 1), y0 = lo_edge(wp.y, 1), z0 = lo_edge(wp.z, 1);
    int x1 = hi_edge(wp.x, G - 1), y1 = hi_edge(wp.y, G - 1), z1 = hi_edge(wp.z, G - 1);
    for (int i = x0; i < x1; ++i)
        for (int j = y0; j < y1; ++j) {
            // a row of the window is at most six voxels: all its loads together
            v3 g6[6];
#pragma unroll
            for (int k = 0; k < 6; ++k)
                if (z0 + k < z1) g6[k] = grid_at(g, i, j, z0 + k);
#pragma unroll
            for (int k = 0; k < 6; ++k)
                if (z0 + k < z1) acc = acc + g6[k];
        }
    return acc;
}

// Both window sums start from zero and depend only on integer voxel
// coordinates, so a frame computes each distinct window once -- in the loop
// order above, so the values are the same bits -- and the render looks them
// up. A coordinate's window is empty outside [kWinLo, kWinLo + kVolN) (volume)
// or [kWinLo, kWinLo + kSlabN) (slab).
constexpr int kWinLo = -2, kVolN = 36, kSlabN = 37;
constexpr int kVolWindows = kVolN * kVolN * kVolN, kSlabWindows = 5 * kSlabN * kSlabN;

__global__ void window_tables_kernel(const float4 *__restrict__ g, float4 *vol, float4 *slab) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < kVolWindows) {
        I3 wp;
        wp.z = t % kVolN + kWinLo;
        wp.y = (t / kVolN) % kVolN + kWinLo;
        wp.x = t / (kVolN * kVolN) + kWinLo;
        const v3 acc = integrate_volume(g, wp);
        vol[t] = make_float4(acc.x, acc.y, acc.z, 0.0f);
    } else if (t < kVolWindows + kSlabWindows) {
        const int u = t - kVolWindows;
        const int id = u / (kSlabN * kSlabN);
        const int a = (u / kSlabN) % kSlabN + kWinLo, b = u % kSlabN + kWinLo;
        // the plane's two free coordinates: (y, z) for 0 and 2, (x, z) for 1
        // and 3, (x, y) for 4; the fixed one does not enter the window
        I3 wp;
        wp.x = id == 0 || id == 2 ? 0 : a;
        wp.y = id == 0 || id == 2 ? a : (id == 4 ? b : 0);
        wp.z = id == 4 ? 0 : b;
        const v3 acc = integrate_slab(g, mk3(0.0f, 0.0f, 0.0f), wp, 1, id);
        slab[u] = make_float4(acc.x, acc.y, acc.z, 0.0f);
    }
}

__device__ __forceinline__ bool in_window_range(int c, int n) { return c >= kWinLo && c < kWinLo + n; }

// integrate_volume through the table.
__device__ __forceinline__ v3 volume_window(const float4 *__restrict__ vol, v3 p) {
    const I3 wp = voxel_of(p);
    if (!in_window_range(wp.x, kVolN) || !in_window_range(wp.y, kVolN) || !in_window_range(wp.z, kVolN))
        return mk3(0.0f, 0.0f, 0.0f);
    const float4 v = __ldg(&vol[((wp.x - kWinLo) * kVolN + (wp.y - kWinLo)) * kVolN + (wp.z - kWinLo)]);
    return mk3(v.x, v.y, v.z);
}

// integrate_slab(g, 0, wp, type, id) through the table.
__device__ __forceinline__ v3 slab_window(const float4 *__restrict__ slab, I3 wp, int type, int id) {
    if (type != 1 || id < 0 || id > 4) return mk3(0.0f, 0.0f, 0.0f);
    const int a = id == 0 || id == 2 ? wp.y : wp.x;
    const int b = id == 4 ? wp.y : wp.z;
    if (!in_window_range(a, kSlabN) || !in_window_range(b, kSlabN)) return mk3(0.0f, 0.0f, 0.0f);
    const float4 v = __ldg(&slab[(id * kSlabN + (a - kWinLo)) * kSlabN + (b - kWinLo)]);
    return mk3(v.x, v.y, v.z);
}

// interpolateEnergy + bilinearInterpolate (:442-583).
__device__ v3 interpolate_slab(const float4 *__restrict__ slab, v3 p, int type, int id) {
    v3 zero = mk3(0.0f, 0.0f, 0.0f);
    if (type != 1) return zero;
    int a1, a2;
    if (id == 0 || id == 2) { a1 = 2; a2 = 1; }
    else if (id == 1 || id == 3) { a1 = 0; a2 = 2; }
    else if (id == 4) { a1 = 0; a2 = 1; }
    else return zero;
    v3 p1 = voxel_center(p);
    v3 p2 = zero, p3 = zero, p4 = zero;
    float c1 = axis_of(p1, a1), d1 = c_vox_dim[a1];
    float s1 = axis_of(p, a1) > c1 ? c1 + d1 : c1 - d1;
    set_axis(p2, a1, s1); set_axis(p3, a1, s1); set_axis(p4, a1, c1);
    float c2 = axis_of(p1, a2), d2 = c_vox_dim[a2];
    float s2 = axis_of(p, a2) > c2 ? c2 + d2 : c2 - d2;
    set_axis(p2, a2, c2); set_axis(p3, a2, s2); set_axis(p4, a2, s2);
    v3 q1 = slab_window(slab, voxel_of(p1), type, id);
    v3 q2 = slab_window(slab, voxel_of(p2), type, id);
    v3 q3 = slab_window(slab, voxel_of(p3), type, id);
    v3 q4 = slab_window(slab, voxel_of(p4), type, id);
    float a = alpha_of(p, p1, p2, a1);
    v3 p12 = lerp3(p1, p2, a), q12 = lerp3(q1, q2, a);
    a = alpha_of(p, p3, p4, a1);
    v3 p34 = lerp3(p3, p4, a), q34 = lerp3(q3, q4, a);
    a = alpha_of(p, p12, p34, a2);
    return lerp3(q12, q34, a);
}

// ---- emission --------------------------------------------------------------

// A photon's path is traced by kPhotonLanes lanes together: the path is the
// same on each of them, a wall's splat window of up to 36 cells takes a cell
// per lane. 8 lanes: the path's arithmetic is repeated eight times, the
// window's is spread over them: 55 us (a thread per photon, which walks a
// bounce's 72 cells one by one: 121 us). One launch: a photon's deposits go to
// its own places and are closed up afterwards in 8 us, where a launch that
// only counted them took 37.
constexpr int kPhotonLanes = 8;
__device__ __forceinline__ int photon_lane() { return (int)(threadIdx.x & (kPhotonLanes - 1)); }
__device__ __forceinline__ unsigned photon_mask() {
    return ((1u << kPhotonLanes) - 1u) << (threadIdx.x & (31u & ~(kPhotonLanes - 1u)));
}

// Records a photon's grid deposits in the order the reference applies them,
// (voxel, value) from place `off` on.
struct Deposits {
    uint32_t *keys;
    float4 *vals;
    const float *inv;  // 1 / sqrt(i), i < kInvN
    uint32_t off, n;
    __device__ __forceinline__ void store(uint32_t at, int vox, v3 e) {
        keys[at] = (uint32_t)vox;
        vals[at] = make_float4(e.x, e.y, e.z, 0.0f);
    }
    // One deposit (the same on every lane).
    __device__ __forceinline__ void put(int vox, v3 e) {
        if (photon_lane() == 0) store(off + n, vox, e);
        ++n;
    }
    // One deposit on each lane with `on`, in lane order.
    __device__ __forceinline__ void put_lanes(bool on, int vox, v3 e) {
        const unsigned m = __ballot_sync(photon_mask(), on);
        if (on) store(off + n + __popc(m & ((1u << (threadIdx.x & 31)) - 1u)), vox, e);
        n += __popc(m);
    }
};

// Squared distances of a splat: two axes up to 3 cells, one up to 31.
constexpr int kInvN = 31 * 31 + 3 * 3 + 3 * 3 + 1;

// The voxel of p clamped to the grid. A coordinate beyond the fast range
// lies outside the grid: above it only a positive one clamps to the last
// voxel, NaN converts to 0 (a shadow photon that hits nothing is there).
__device__ __forceinline__ int clamped(float x, int v) {
    const int far = x >= kLegacyFastRange ? G - 1 : 0;
    return fabsf(x) < kLegacyFastRange ? min(max(v, 0), G - 1) : far;
}
__device__ __forceinline__ I3 clamped_voxel(v3 p) {
    const float r = kLegacyFastRange;
    I3 v;
    v.x = clamped(p.x, legacy_voxel_xy(fabsf(p.x) < r ? p.x : 0.0f));
    v.y = clamped(p.y, legacy_voxel_xy(fabsf(p.y) < r ? p.y : 0.0f));
    v.z = clamped(p.z, legacy_voxel_z(fabsf(p.z) < r ? p.z : 0.0f));
    return v;
}

// storePhoton + splatEnergy (:1074-1144, 1164-1183): the window's cells in
// the reference's row order, a cell per lane. A cell's value is the energy's
// twentieth over its distance (:1059-1071), whose reciprocal depends only on
// the squared distance in cells and is read from a table.
__device__ __forceinline__ void store_surface(Deposits &d, int type, int id, v3 loc, v3 e) {
    I3 c = clamped_voxel(loc);
    if (type != 0) d.put(vox_index(c.x, c.y, c.z), e);
    if (type != 1 || id < 0 || id > 4) return;
    // the wall's fixed coordinate and its two free ones, outer a, inner b
    const bool on_x = id == 0 || id == 2, on_y = id == 1 || id == 3;
    const int fixed = id == 1 || id == 2 ? 0 : G - 1;
    const int ca = on_x ? c.y : c.x, cb = on_x || on_y ? c.z : c.y, cf = on_x ? c.x : (on_y ? c.y : c.z);
    const int a0 = lo_edge(ca, 0), a1 = hi_edge(ca, G), b0 = lo_edge(cb, 0), b1 = hi_edge(cb, G);
    const int nb = b1 - b0, cells = (a1 - a0) * nb;  // 3 to 6 a side
    const v3 e20 = e * 0.05f;
    const int rcp = 65536 / nb + 1;  // t / nb for t < 64
    const int df = cf - fixed;
    for (int base = 0; base < cells; base += kPhotonLanes) {
        const int t = base + photon_lane();
        const int row = (t * rcp) >> 16, a = a0 + row, b = b0 + (t - row * nb);
        const int i = on_x ? fixed : a, j = on_y ? fixed : (on_x ? a : b), k = on_x || on_y ? b : fixed;
        const int da = ca - a, db = cb - b, d2 = da * da + db * db + df * df;
        const bool on = t < cells && d2 > 0;  // the photon's own cell is left out
        d.put_lanes(on, vox_index(i, j, k), e20 * (on ? d.inv[d2] : 0.0f));
    }
}

__device__ __forceinline__ v3 surface_color(v3 in, int type, int idx) {  // getColor (:605-617)
    v3 f = mk3(1.0f, 1.0f, 1.0f);
    if (type == 1 && idx == 0) f = mk3(0.0f, 1.0f, 0.0f);
    else if (type == 1 && idx == 2) f = mk3(1.0f, 0.0f, 0.0f);
    return mk3(fminf(f.x, in.x), fminf(f.y, in.y), fminf(f.z, in.z));
}

__device__ __forceinline__ uint32_t mulmod(uint64_t a, uint64_t b, uint64_t m) {
    return (uint32_t)((a * b) % m);
}

__host__ __device__ inline uint32_t mwc_jump(uint32_t state, uint64_t a, uint64_t m, uint64_t n) {
    uint64_t r = 1, base = a % m;
    while (n) {
        if (n & 1) r = (r * base) % m;
        base = (base * base) % m;
        n >>= 1;
    }
    return (uint32_t)((r * (uint64_t)state) % m);
}

struct Mwc {
    uint32_t z, w;
    __device__ __forceinline__ uint32_t next() {
        z = kMwcAz * (z & 65535u) + (z >> 16);
        w = kMwcAw * (w & 65535u) + (w >> 16);
        return (z << 16) + w;
    }
    __device__ __forceinline__ float uniform(float max) {  // randFloat (:1038-1051)
        float r = (float)(int)next() / 65535.0f;
        r = (r * 2.0f) * max;
        return r - max;
    }
};

// emitPhotons (:1215-1375) for photon `index`; the medium steps draw from
// the generator positioned at this photon's first draw.
__device__ void emit_one(const Scene &sc, const float4 *__restrict__ table, int index, bool media,
                         Mwc rng, Deposits &d) {
    int bounces = 1;
    v3 rgb = mk3(10.0f, 10.0f, 10.0f);
    float4 t = table[index];
    v3 ray = normalize(mk3(t.x, t.y, t.z));
    v3 first_ray = ray;
    v3 prev = light_pos();
    Chain c;
    c.point = mk3(0.0f, 0.0f, 0.0f);
    if (media) {
        for (int i = 0; i < 3; ++i) {
            rgb = sub_scalar(rgb, 1.0f);
            c.point = ray * 1.0f + prev;
            I3 v = clamped_voxel(c.point);
            d.put(vox_index(v.x, v.y, v.z), rgb * 0.00005f);
            float4 q = table[i];
            v3 rnd;
            rnd.x = rng.uniform(q.x);
            rnd.y = rng.uniform(q.y);
            rnd.z = rng.uniform(q.z);
            ray = normalize(rnd);
            prev = c.point;
        }
        ray = first_ray;
        prev = light_pos();
    }
    if (index < 100) {  // CAUSTICS_PHOTONS aim at the glass sphere (:1274-1278)
        ray = normalize(mk3(sc.sph[0][0], sc.sph[0][1], sc.sph[0][2]) - light_pos());
        ray = ray + normalize(mk3(t.x, t.y, t.z)) * 0.01f;
    }
    c.ray = ray;
    trace(sc, c.ray, prev, c.h);
    bool caustic = false, new_point = true;
    while (c.h.hit && bounces <= 5) {
        if (new_point) c.point = c.ray * c.h.dist + prev;
        if (caustic) {
            rgb = mk3(1.0f, 1.0f, 1.0f) * 10.0f;
            store_surface(d, c.h.type, c.h.idx, c.point, rgb);
        } else {
            rgb = div_scalar(surface_color(rgb, c.h.type, c.h.idx) * 1.0f, sqrtf((float)bounces)) * 5.0f;
            store_surface(d, c.h.type, c.h.idx, c.point, rgb);
            // shadowPhoton (:1185-1196)
            int st = c.h.type, si = c.h.idx;
            v3 bumped = c.point + c.ray * 0.00001f;
            trace(sc, c.ray, bumped, c.h);
            store_surface(d, c.h.type, c.h.idx, c.ray * c.h.dist + bumped, mk3(-0.25f, -0.25f, -0.25f));
            c.h.type = st;
            c.h.idx = si;
        }
        prev = c.point;
        if (c.h.type == 0 && c.h.idx == 1) {
            run_chain(sc, c, 1, prev);
            caustic = false; new_point = false;
        } else if (c.h.type == 0 && c.h.idx == 0) {
            run_chain(sc, c, 2, prev);
            caustic = true; new_point = false;
        } else {
            c.ray = reflect_ray(sc, c.ray, prev, c.h.type, c.h.idx, c.point);
            trace(sc, c.ray, c.point, c.h);
            caustic = false; new_point = true;
        }
        ++bounces;
    }
}

// base^(9 * 2^i) of both generator halves: photon p's medium loop starts
// 9p draws after the emission's first, p below 2^14.
constexpr int kJumpBits = 16;
static_assert(kLegacyPhotons <= 1 << kJumpBits && kJumpBits % kPhotonLanes == 0, "jump powers cover every photon");
struct JumpTable {
    uint32_t z[kJumpBits], w[kJumpBits];
};

// The generator 9p draws on: each lane of the photon multiplies the powers
// of its share of p's bits, three butterfly steps the rest.
__device__ __forceinline__ Mwc jump_photon(const JumpTable &J, uint32_t z0, uint32_t w0, int p) {
    uint32_t z = 1u, w = 1u;
#pragma unroll
    for (int i = 0; i < kJumpBits / kPhotonLanes; ++i) {
        const int bit = i * kPhotonLanes + photon_lane();
        if ((p >> bit) & 1) {
            z = mulmod(z, J.z[bit], kMwcMz);
            w = mulmod(w, J.w[bit], kMwcMw);
        }
    }
#pragma unroll
    for (int o = 1; o < kPhotonLanes; o <<= 1) {
        z = mulmod(z, __shfl_xor_sync(photon_mask(), z, o), kMwcMz);
        w = mulmod(w, __shfl_xor_sync(photon_mask(), w, o), kMwcMw);
    }
    Mwc r;
    r.z = mulmod(z, z0, kMwcMz);
    r.w = mulmod(w, w0, kMwcMw);
    return r;
}

// Bound by the latency of a photon's serial bounces and their arithmetic.
__global__ void __launch_bounds__(256) emit_kernel(Scene sc, const float4 *__restrict__ table, bool media,
                                                   uint32_t z0, uint32_t w0, JumpTable jump, uint32_t *counts,
                                                   uint32_t *keys, float4 *vals) {
    __shared__ float inv[kInvN];
    for (int i = threadIdx.x; i < kInvN; i += blockDim.x) inv[i] = 1.0f / sqrtf((float)i);
    __syncthreads();
    const int p = (int)((blockIdx.x * blockDim.x + threadIdx.x) / kPhotonLanes);
    if (p >= kLegacyPhotons) return;  // whole photons
    Mwc rng;
    rng.z = z0;
    rng.w = w0;
    if (media) rng = jump_photon(jump, z0, w0, p);
    Deposits d;
    d.keys = keys;
    d.vals = vals;
    d.inv = inv;
    d.off = (uint32_t)p * kLegacyMaxDepositsPerPhoton;
    d.n = 0;
    emit_one(sc, table, p, media, rng, d);
    if (photon_lane() == 0) counts[p] = d.n;
}

// The photons' deposits one after another: voxel and place, for the sort. A
// warp per photon; a block adds up the counts of the photons before its own.
constexpr int kClosePhotons = 32;
__global__ void __launch_bounds__(kClosePhotons * 32) close_up_kernel(const uint32_t *__restrict__ counts,
                                                                      const uint32_t *__restrict__ slots,
                                                                      uint32_t *keys, uint32_t *idx, uint32_t *total) {
    __shared__ uint32_t sums[kClosePhotons];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int first = blockIdx.x * kClosePhotons;
    uint32_t s = 0;
    for (int i = threadIdx.x; i < first; i += kClosePhotons * 32) s += counts[i];
    s = __reduce_add_sync(0xffffffffu, s);
    if (lane == 0) sums[warp] = s;
    const uint32_t c = first + lane < kLegacyPhotons ? counts[first + lane] : 0u;
    __syncthreads();
    const uint32_t off = __reduce_add_sync(0xffffffffu, sums[lane] + (lane < warp ? c : 0u));
    const uint32_t n = __shfl_sync(0xffffffffu, c, warp);
    const uint32_t from = (uint32_t)(first + warp) * kLegacyMaxDepositsPerPhoton;
    for (uint32_t i = lane; i < n; i += 32) {
        keys[off + i] = slots[from + i];
        idx[off + i] = from + i;
    }
    if (first + warp == kLegacyPhotons - 1 && lane == 0) *total = off + n;
}

// Deposit values in sorted order (one parallel gather), so that each
// voxel's sum below streams a contiguous range, and each voxel's first
// deposit (start[v] = the deposits below voxel v).
__global__ void gather_deposits_kernel(const uint32_t *__restrict__ skeys, const uint32_t *__restrict__ sidx,
                                       const float4 *__restrict__ vals, const uint32_t *total, float4 *sorted,
                                       uint32_t *start) {
    const uint32_t n = *total;
    const uint32_t first = blockIdx.x * blockDim.x + threadIdx.x, step = gridDim.x * blockDim.x;
    for (uint32_t j = first; j < n; j += step) {
        sorted[j] = vals[sidx[j]];
        const uint32_t v = skeys[j];
        for (uint32_t u = j ? skeys[j - 1] + 1u : 0u; u <= v; ++u) start[u] = j;
        if (j == n - 1)
            for (uint32_t u = v + 1u; u <= (uint32_t)kLegacyVoxels; ++u) start[u] = n;
    }
    if (n == 0)
        for (uint32_t u = first; u <= (uint32_t)kLegacyVoxels; u += step) start[u] = 0u;
}

// Sums each voxel's deposits in photon order and writes both grid layouts;
// one warp per voxel. The warp loads 128 consecutive deposits at a time
// (coalesced, the next 128 already in flight) and turns them into three rows
// in shared memory; lanes 0, 1 and 2 add a component each, four deposits
// per load: exactly the serial additions, bound by the chain of them in the
// voxels beside the light. 33 us a frame; broadcasting each deposit through
// three shuffles took 84 us, and 113 us with each voxel's range searched
// for instead of read.
constexpr int kSumWarps = 4;
constexpr int kSumItems = 128;
__global__ void __launch_bounds__(kSumWarps * 32) reduce_kernel(const uint32_t *__restrict__ start,
                                                                const float4 *__restrict__ sorted, float *grid3,
                                                                float4 *grid4) {
    __shared__ __align__(16) float row[kSumWarps][3][kSumItems + 4];  // rows a bank apart
    const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int v = blockIdx.x * kSumWarps + wib;
    if (v >= kLegacyVoxels) return;
    const uint32_t lo = start[v], hi = start[v + 1];
    const float4 zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    float4 e[kSumItems / 32];
#pragma unroll
    for (int i = 0; i < kSumItems / 32; ++i) {
        const uint32_t at = lo + 32u * i + lane;
        e[i] = at < hi ? __ldg(&sorted[at]) : zero;
    }
    float acc = 0.0f;
    for (uint32_t base = lo; base < hi; base += kSumItems) {
#pragma unroll
        for (int i = 0; i < kSumItems / 32; ++i) {
            row[wib][0][32 * i + lane] = e[i].x;
            row[wib][1][32 * i + lane] = e[i].y;
            row[wib][2][32 * i + lane] = e[i].z;
        }
#pragma unroll
        for (int i = 0; i < kSumItems / 32; ++i) {
            const uint32_t at = base + kSumItems + 32u * i + lane;
            e[i] = at < hi ? __ldg(&sorted[at]) : zero;
        }
        __syncwarp();
        if (lane < 3) {
            const float4 *r = reinterpret_cast<const float4 *>(row[wib][lane]);
            const int cnt = (int)min((uint32_t)kSumItems, hi - base);
            if (cnt == kSumItems) {
#pragma unroll
                for (int i = 0; i < kSumItems / 4; ++i) {
                    const float4 q = r[i];
                    acc = ((acc + q.x) + q.y) + q.z;
                    acc = acc + q.w;
                }
            } else {
                for (int i = 0; i < cnt; ++i) acc = acc + row[wib][lane][i];
            }
        }
        __syncwarp();
    }
    if (lane < 3) grid3[3 * v + lane] = acc;
    const float ay = __shfl_sync(0xffffffffu, acc, 1), az = __shfl_sync(0xffffffffu, acc, 2);
    if (lane == 0) grid4[v] = make_float4(acc, ay, az, 0.0f);
}

// init_random_numbers_kernel (:1483-1498): entry i holds draws 3i..3i+2
// after `base` earlier draws.
__global__ void table_kernel(float4 *table, uint32_t z0, uint32_t w0) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= kLegacyPhotons) return;
    Mwc rng;
    rng.z = mwc_jump(z0, kMwcAz, kMwcMz, 3ull * (uint64_t)i);
    rng.w = mwc_jump(w0, kMwcAw, kMwcMw, 3ull * (uint64_t)i);
    float x = rng.uniform(1.0f);
    float y = rng.uniform(1.0f);
    float z = rng.uniform(1.0f);
    table[i] = make_float4(x, y, z, 0.0f);
}

__global__ void grid_from_host_kernel(const float *grid3, float4 *grid4) {
    int v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v < kLegacyVoxels) grid4[v] = make_float4(grid3[3 * v], grid3[3 * v + 1], grid3[3 * v + 2], 0.0f);
}

// ---- render ----------------------------------------------------------------

// computePixelColor (:926-1017). The voxels of its up to ten march points and
// five interpolation corners are found in single precision
// (legacy_voxel.cuh): a 512 x 512 frame takes 38 us; in double precision,
// three divisions each, it took 366 us, bound by the double-precision units.
__device__ v3 shade_pixel(const Scene &sc, const float4 *__restrict__ vol,
                          const float4 *__restrict__ slab, float x, float y, bool interp, bool media) {
    v3 rgb = mk3(0.0f, 0.0f, 0.0f);
    v3 origin = mk3(0.0f, 0.0f, 0.0f);
    Chain c;
    // one rounding, in the difference: the double that held it was exact
    c.ray = mk3(x / 512.0f - 0.5f, -(y / 512.0f - 0.5f), 1.0f);
    c.h.hit = false;
    c.h.type = 0;
    c.h.idx = 0;
    if (media) {  // ten fixed steps of 0.6 along the unnormalised ray (:940-961)
        v3 at = origin;
        for (int i = 0; i < 10; ++i) {
            at = c.ray * 0.6f + at;
            rgb = rgb + volume_window(vol, at);
        }
    }
    trace(sc, c.ray, origin, c.h);
    if (!c.h.hit) return rgb;
    c.point = c.ray * c.h.dist;
    if (c.h.type == 0 && c.h.idx == 1) run_chain(sc, c, 1, origin);
    else if (c.h.type == 0 && c.h.idx == 0) run_chain(sc, c, 2, origin);
    if (!c.h.hit) return rgb;
    v3 e = interp ? interpolate_slab(slab, c.point, c.h.type, c.h.idx)
                  : slab_window(slab, voxel_of(c.point), c.h.type, c.h.idx);
    if (media) e = e * 0.15f;
    return rgb + e;
}

__global__ void __launch_bounds__(256) render_kernel(Scene sc, const float4 *__restrict__ vol,
                                                     const float4 *__restrict__ slab, uchar4 *out,
                                                     unsigned width, unsigned height, bool interp,
                                                     bool media, float *rgb_out) {
    unsigned index = blockIdx.x * blockDim.x + threadIdx.x;
    if (index >= width * height) return;
    unsigned x = index % width, y = index / width;
    v3 c = shade_pixel(sc, vol, slab, (float)x, (float)y, interp, media);
    if (rgb_out) {
        rgb_out[3 * index + 0] = c.x;
        rgb_out[3 * index + 1] = c.y;
        rgb_out[3 * index + 2] = c.z;
    }
    out[index] = make_uchar4(unit_to_u8(c.x), unit_to_u8(c.y), unit_to_u8(c.z), 0);
}

Scene make_scene(float anim_time) {
    Scene sc;
    legacy_position_spheres(anim_time, sc.sph);
    return sc;
}

}  // namespace

uint32_t mwc_jump_host(uint32_t state, uint64_t a, uint64_t m, uint64_t n) {
    return mwc_jump(state, a, m, n);
}

void legacy_position_spheres(float t, float out[2][4]) {
    out[0][0] = (float)(1.0 * (double)std::cos(t));
    out[0][1] = (float)(0.5 * std::sin(2.0 * (double)t));
    out[0][2] = (float)((double)std::sin(t) + 3.5);
    out[0][3] = 0.4f;
    out[1][0] = 0.0f;
    out[1][1] = (float)(std::sin(0.5 * (double)t + 5.0) - 0.25);
    out[1][2] = 3.5f;
    out[1][3] = 0.4f;
}

cudaError_t legacy_alloc(LegacyState &st) {
    cudaError_t e;
#define PM_ALLOC(ptr, bytes) \
    if ((e = cudaMalloc((void **)&(ptr), (bytes))) != cudaSuccess) { legacy_free(st); return e; }
    PM_ALLOC(st.table, sizeof(float4) * kLegacyPhotons);
    PM_ALLOC(st.grid3, sizeof(float) * 3 * kLegacyVoxels);
    PM_ALLOC(st.grid4, sizeof(float4) * kLegacyVoxels);
    PM_ALLOC(st.vol_win, sizeof(float4) * kVolWindows);
    PM_ALLOC(st.slab_win, sizeof(float4) * kSlabWindows);
    PM_ALLOC(st.counts, sizeof(uint32_t) * kLegacyPhotons);
    PM_ALLOC(st.total, sizeof(uint32_t));
    PM_ALLOC(st.start, sizeof(uint32_t) * (kLegacyVoxels + 1));
    PM_ALLOC(st.keys, sizeof(uint32_t) * kLegacyMaxDeposits);
    PM_ALLOC(st.keys_tmp, sizeof(uint32_t) * kLegacyMaxDeposits);
    PM_ALLOC(st.idx, sizeof(uint32_t) * kLegacyMaxDeposits);
    PM_ALLOC(st.idx_tmp, sizeof(uint32_t) * kLegacyMaxDeposits);
    PM_ALLOC(st.dep, sizeof(float4) * kLegacyMaxDeposits);
    PM_ALLOC(st.sdep, sizeof(float4) * kLegacyMaxDeposits);
    PM_ALLOC(st.hist, sizeof(uint32_t) * radix_sort_hist_words(kLegacyMaxDeposits));
#undef PM_ALLOC
    // A fresh module starts with a zero table and grid (static __device__
    // storage in the reference).
    if ((e = cudaMemset(st.table, 0, sizeof(float4) * kLegacyPhotons)) != cudaSuccess) return e;
    if ((e = cudaMemset(st.grid3, 0, sizeof(float) * 3 * kLegacyVoxels)) != cudaSuccess) return e;
    if ((e = cudaMemset(st.grid4, 0, sizeof(float4) * kLegacyVoxels)) != cudaSuccess) return e;
    st.rng_draws = 0;
    return cudaSuccess;
}

void legacy_free(LegacyState &st) {
    cudaFree(st.table); cudaFree(st.grid3); cudaFree(st.grid4); cudaFree(st.counts);
    cudaFree(st.vol_win); cudaFree(st.slab_win);
    cudaFree(st.total); cudaFree(st.start); cudaFree(st.keys); cudaFree(st.keys_tmp);
    cudaFree(st.idx); cudaFree(st.idx_tmp); cudaFree(st.dep); cudaFree(st.sdep); cudaFree(st.hist);
    st = LegacyState();
}

cudaError_t legacy_init_random(LegacyState &st, cudaStream_t s) {
    uint32_t z0 = mwc_jump_host(kMwcSeedZ, kMwcAz, kMwcMz, st.rng_draws);
    uint32_t w0 = mwc_jump_host(kMwcSeedW, kMwcAw, kMwcMw, st.rng_draws);
    table_kernel<<<(kLegacyPhotons + 255) / 256, 256, 0, s>>>(st.table, z0, w0); note_launch();
    st.rng_draws += 3ull * kLegacyPhotons;
    st.table_written = true;
    return cudaGetLastError();
}

cudaError_t legacy_emit(LegacyState &st, float anim_time, int flags, cudaStream_t s) {
    Scene sc = make_scene(anim_time);
    bool media = (flags & kLegacyMedia) != 0;
    uint32_t z0 = mwc_jump_host(kMwcSeedZ, kMwcAz, kMwcMz, st.rng_draws);
    uint32_t w0 = mwc_jump_host(kMwcSeedW, kMwcAw, kMwcMw, st.rng_draws);
    JumpTable jump;
    for (int i = 0; i < kJumpBits; ++i) {
        jump.z[i] = mwc_jump_host(1u, kMwcAz, kMwcMz, 9ull << i);
        jump.w[i] = mwc_jump_host(1u, kMwcAw, kMwcMw, 9ull << i);
    }
    const int blocks = (kLegacyPhotons * kPhotonLanes + 255) / 256;
    emit_kernel<<<blocks, 256, 0, s>>>(sc, st.table, media, z0, w0, jump, st.counts, st.keys_tmp, st.dep); note_launch();
    close_up_kernel<<<(kLegacyPhotons + kClosePhotons - 1) / kClosePhotons, kClosePhotons * 32, 0, s>>>(
        st.counts, st.keys_tmp, st.keys, st.idx, st.total);
    note_launch();
    uint32_t *sk = nullptr, *si = nullptr;
    cudaError_t e = radix_sort_pairs_u32(st.keys, st.idx, st.keys_tmp, st.idx_tmp, st.total, kLegacyMaxDeposits,
                             0, 16, st.hist, s, &sk, &si);
    if (e != cudaSuccess) return e;
    gather_deposits_kernel<<<512, 256, 0, s>>>(sk, si, st.dep, st.total, st.sdep, st.start); note_launch();
    reduce_kernel<<<(kLegacyVoxels + kSumWarps - 1) / kSumWarps, kSumWarps * 32, 0, s>>>(st.start, st.sdep, st.grid3,
                                                                                        st.grid4); note_launch();
    if (media) st.rng_draws += 9ull * kLegacyPhotons;
    return cudaGetLastError();
}

cudaError_t legacy_render(const LegacyState &st, uchar4 *out, unsigned width, unsigned height,
                          float anim_time, int flags, float *rgb_out, cudaStream_t s) {
    Scene sc = make_scene(anim_time);
    unsigned n = width * height;
    if (n == 0) return cudaSuccess;
    // the frame's window sums, from the current grid
    window_tables_kernel<<<(kVolWindows + kSlabWindows + 255) / 256, 256, 0, s>>>(st.grid4, st.vol_win,
                                                                                 st.slab_win);
    note_launch();
    render_kernel<<<(n + 255) / 256, 256, 0, s>>>(sc, st.vol_win, st.slab_win, out, width, height,
                                                  (flags & kLegacyInterpolate) != 0,
                                                  (flags & kLegacyMedia) != 0, rgb_out); note_launch();
    return cudaGetLastError();
}

cudaError_t legacy_upload_grid(LegacyState &st, const float *host_grid3, cudaStream_t s) {
    cudaError_t e = cudaMemcpyAsync(st.grid3, host_grid3, sizeof(float) * 3 * kLegacyVoxels,
                                    cudaMemcpyHostToDevice, s);
    if (e != cudaSuccess) return e;
    grid_from_host_kernel<<<(kLegacyVoxels + 255) / 256, 256, 0, s>>>(st.grid3, st.grid4); note_launch();
    return cudaGetLastError();
}

}  // namespace pm
