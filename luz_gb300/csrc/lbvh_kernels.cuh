// lbvh_kernels.cuh — declarations of the LBVH build kernels (defined in lbvh.cu) and
// the segment descriptor they share, so that other translation units can launch the
// same kernels.
#pragma once
#include <algorithm>

#include "internal.cuh"

namespace luz {

// One mesh of a batched BLAS build: a contiguous run of primitives in the sort.
struct SegDesc {
    uint32_t prim_off;     // first primitive (global)
    uint32_t prim_count;
    uint32_t node_off;     // first internal node (global), max(n-1,1) nodes
    uint32_t pad;
    const luz_vertex* vertices;  // device copy, 48-B stride (BLAS only)
    const uint32_t* indices;
    float4* nodes;         // output nodes of this segment
    float4* tris;          // output triangles of this segment
    float4* nodes4;        // output 4-wide nodes (NULL: not built)
    uint32_t* morton;      // BLAS: output sorted 30-bit Morton codes of this segment
    uint32_t* order;       // BLAS: output primitive index of each leaf
};

// Onesweep radix sort geometry.
constexpr int kSortThreads = 256;
constexpr int kSortWarps = kSortThreads / 32;
constexpr int kSortItems = 8;
constexpr int kSortTile = kSortThreads * kSortItems;   // 2048 keys
constexpr int kRadix = 256;
constexpr int kMaxPasses = 6;
constexpr uint32_t kFlagAggregate = 1u << 30;
constexpr uint32_t kFlagPrefix = 2u << 30;
constexpr uint32_t kValueMask = (1u << 30) - 1;
constexpr uint32_t kLookbackSpinLimit = 1u << 22;
constexpr int kLookback = 8;      // tiles a look-back reads at a time

// Rows of 256 primitives one block of blas_bounds_kernel reduces (launch 256 threads and
// ceil(total / (256 * rows)) blocks), and blocks of blas_morton_kernel: about four blocks per
// SM, up to 16 rows each / four keys a thread at least.
inline uint32_t bounds_rows(uint32_t total) { return std::min(std::max(total / (256u * 608u), 1u), 16u); }
inline uint32_t morton_blocks(uint32_t total) { return std::min((total + 1023u) / 1024u, 1216u); }
__global__ void __launch_bounds__(256) blas_bounds_kernel(const SegDesc* segs, const uint32_t* seg_prim_off,
                                                          int nseg, uint32_t total, uint32_t rows, uint32_t* seg_bounds);
__global__ void __launch_bounds__(256) blas_morton_kernel(const SegDesc* segs, const uint32_t* seg_prim_off, int nseg,
                                                          uint32_t total, const uint32_t* seg_bounds,
                                                          unsigned long long* keys, uint32_t* vals, int passes,
                                                          uint32_t* hist);
__global__ void __launch_bounds__(kSortThreads)
onesweep_pass_kernel(const unsigned long long* __restrict__ kin, const uint32_t* __restrict__ vin,
                     unsigned long long* __restrict__ kout, uint32_t* __restrict__ vout, uint32_t n, int shift,
                     const uint32_t* __restrict__ pass_hist, uint32_t* __restrict__ pass_offsets, uint32_t* tile_status,
                     uint32_t* tile_counter, uint32_t* dev_status);

// Leaves per block of the hierarchy kernels (one thread each), at most; blocks start near
// the multiples of kMergeStep.
constexpr uint32_t kMergeLeaves = 512, kMergeStep = kMergeLeaves / 2;
inline uint32_t merge_blocks(uint32_t total) { return (total - 1 + kMergeStep / 2) / kMergeStep + 1; }   // total > 0
// What the merges of a build meet in (lbvh.cu).
struct MergeArgs {
    const unsigned long long* keys;   // sorted
    uint32_t* node_parent;            // (parent << 1) | side of each node, per segment (NULL: not kept)
    uint2* ends[2];                   // (far end, prefix there + 1) of the two sides of the merge after each leaf
    uint32_t* flags;                  // arrivals at the merge after each leaf (zero)
    uint32_t* status;                 // device status word
    uint32_t total;
};
__global__ void __launch_bounds__(kMergeLeaves) blas_tree_kernel(const SegDesc* segs, const uint32_t* seg_prim_off, int nseg,
                                                                 const uint32_t* vals, MergeArgs A);
__global__ void empty_segments_kernel(const SegDesc* segs, int nseg, uint32_t* node_parent);
__global__ void blas_radius_kernel(const SegDesc* segs, const uint32_t* seg_prim_off, int nseg,
                                   uint32_t total);

}  // namespace luz
