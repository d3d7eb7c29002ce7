// kdtree.cuh -- implicit median-split kd-tree over a photon map.
#pragma once
#include "phys_common.cuh"

#include <vector>

namespace pm {

// Depth D of the tree over n records (leaves of 32 << leaf_shift records at
// depth D, 2^D leaf slots).
int tree_depth(uint32_t n, int leaf_shift = 0);
// Node array length (index 0 unused, root at 1): 2^(D+1).
size_t tree_nodes(uint32_t n, int leaf_shift = 0);

struct KdBuildArgs {
    uint32_t n = 0;                  // records
    float3 lo, hi;                   // root cell (the scene box)
    bool root_boxed = false;         // the root cell is the box already in the node words
                                     // (kd_root_box_words): lo and hi are not read
    const float4 *pos_in = nullptr, *pow_in = nullptr;  // records in index order, pos.w the index (pow_in nullable)
    float4 *pos_out = nullptr, *pow_out = nullptr;      // records in tree order (pow_out with pow_in)
    float4 *dir_out = nullptr;       // nullable: decoded directions (xyz) in tree order
    float4 *node_lo = nullptr, *node_hi = nullptr;      // tree_nodes(n) boxes
    int leaf_shift = 0;              // leaves of 32 << leaf_shift records
    // plans only (nullable): the records from *pad_count to n are set to
    // infinity (position) and zero (power) before the build
    const uint32_t *pad_count = nullptr;
};

// One map of a build as the kernels read it.
struct KdMap {
    const float4 *pos, *pow;               // records in index order
    float4 *pos_out, *pow_out, *dir_out;   // tree order
    float4 *lo, *hi;                       // node boxes
    float4 *tmp;                           // n records: the other buffer of the split levels
    uint16_t *keys;                        // n: each record's split coordinate at the current level
    uint32_t *done;                        // finished subtrees (zero between builds)
    const uint32_t *pad_count;             // nullable
    float3 root_lo, root_hi;
    uint32_t n, tile0, mid0, sub0, node0;  // first tile, cluster, subtree and node words of this map in the launch
    int depth, leaf_shift, root_boxed;
    int ls, lf;                            // the first level split by clusters, the level of the subtrees
};

// Scratch of build_trees over these maps (one or two, built in shared
// launches), in bytes.
size_t kd_scratch_bytes(const uint32_t *n, const int *leaf_shift, int maps);
// Builds the trees of one or two maps. scratch: kd_scratch_bytes, 256-byte
// aligned.
cudaError_t build_trees(const KdBuildArgs *a, int maps, void *scratch, cudaStream_t s);
// A build of one map with root_boxed: the caller zeroes the scratch's words
// (kd_clear_scratch) and fills the root's box -- ~kd_flip of the minimum and
// kd_flip of the maximum per axis, combined with atomicMax, zero: no point
// (null: the tree needs no root box) -- before build_trees, which then
// leaves the clearing out.
uint32_t *kd_root_box_words(const KdBuildArgs &a, void *scratch);
cudaError_t kd_clear_scratch(const KdBuildArgs &a, void *scratch, cudaStream_t s);

// Order-preserving words of a coordinate: kd_flip grows with x; a box's
// minimum is kept as the complement so that both sides grow under atomicMax
// from zero.
__device__ __forceinline__ uint32_t kd_flip(float x) {
    const uint32_t u = __float_as_uint(x);
    return u ^ ((uint32_t)((int)u >> 31) | 0x80000000u);
}
__device__ __forceinline__ float kd_unflip(uint32_t f) {
    return __uint_as_float(f ^ ((f & 0x80000000u) ? 0x80000000u : 0xffffffffu));
}

// Several trees built together (a batch's maps): one plan, shared launches.
// Each tree comes out as build_trees makes it.
struct KdMulti {
    int nmaps = 0;
    std::vector<KdMap> maps;            // the most split levels first
    KdMap *desc = nullptr;
    uint32_t *tile_map = nullptr;       // per tile: its map
    uint32_t *sub_first = nullptr;      // per map: its first subtree (+ the total)
    uint32_t tiles = 0, subs = 0;
    bool pad = false;                   // some map pads its records
    void *scratch = nullptr;
    uint32_t *hist = nullptr;           // into scratch
    uint32_t *box = nullptr;
    uint4 *thr = nullptr;
    uint2 *tile_cnt = nullptr;
    uint32_t *tile_sub = nullptr;
    size_t clear_bytes = 0;             // of scratch, zeroed by each build
};
// Plans the build of the maps args[i] and allocates its tables and scratch.
// Maps with no records are left out.
cudaError_t kd_multi_create(const std::vector<KdBuildArgs> &args, KdMulti *k);
void kd_multi_free(KdMulti &k);
// The padding and the trees of every map.
cudaError_t kd_multi_build(KdMulti &k, cudaStream_t s);

}  // namespace pm
