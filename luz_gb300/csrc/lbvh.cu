// lbvh.cu — device-built two-level LBVH: BLAS over triangles (batched over many
// meshes as sort segments) and TLAS over instances.
//
// Pipeline (each step a kernel on the context stream):
//   bounds   : centroid bounds per segment (order-preserving uint atomics, exact)
//   morton   : 64-bit key = segment << 30 | morton30(centroid), value = primitive
//   sort     : LSD radix sort, 8-bit digits, the histograms of all passes counted with
//              the keys + one "onesweep" kernel per pass (tile-local warp multi-split
//              ranking, decoupled look-back across tiles). Stable.
//   tree     : triangles / instances gathered into leaf order, padded leaf boxes, and the
//              radix tree of T. Karras, "Maximizing Parallelism in the Construction of BVHs,
//              Octrees, and k-d Trees", HPG 2012, built bottom-up with its boxes;
//              duplicate codes split by index (delta = 32 + clz(i ^ j)).
//   bfs      : (TLAS) breadth-first relayout so that the top of the tree is a prefix
//              of the node array, staged into shared memory by the traversal.
// Replaces the driver builds behind vkw::CmdBuildBLAS / vkw::CmdBuildTLAS
// (source/Graphics/VulkanWrapper.cpp:1089-1139).
#include <algorithm>
#include <cstring>
#include <vector>

#include "internal.cuh"
#include "lbvh_device.cuh"

namespace luz {

// ---------------------------------------------------------------- helpers

__device__ __forceinline__ int find_seg(const uint32_t* offs, int nseg, uint32_t g) {
    int lo = 0, hi = nseg - 1;
    while (lo < hi) {
        int mid = (lo + hi + 1) >> 1;
        if (offs[mid] <= g) lo = mid; else hi = mid - 1;
    }
    return lo;
}

__device__ __forceinline__ V3 load_pos(const luz_vertex* v, uint32_t i) {
    const float* p = v[i].position;
    return V3{p[0], p[1], p[2]};
}

__device__ __forceinline__ void tri_box(V3 a, V3 b, V3 c, V3& lo, V3& hi) {
    lo = V3{fmin_(fmin_(a.x, b.x), c.x), fmin_(fmin_(a.y, b.y), c.y), fmin_(fmin_(a.z, b.z), c.z)};
    hi = V3{fmax_(fmax_(a.x, b.x), c.x), fmax_(fmax_(a.y, b.y), c.y), fmax_(fmax_(a.z, b.z), c.z)};
}

// Leaf padding of a triangle box (relative 2^-20 of the coordinate magnitude).
__device__ __forceinline__ float leaf_pad(float lo, float hi) {
    return fmax_(fabsf(lo), fabsf(hi)) * 0x1p-20f + 0x1p-100f;
}

// ---------------------------------------------------------------- bounds + morton
// seg_bounds: 6 ordered uints per segment (min xyz, max xyz); init min=~0, max=0.
// A block walks `rows` rows of 256 consecutive primitives. Per row, a warp whose
// lanes all belong to one segment reduces its ordered centroid keys (redux.sync) and
// lane 0 merges them into a running min/max of that segment, which goes to the global
// words (six atomics) only when the segment changes; a warp that straddles a segment
// boundary issues per-lane atomics. At the end of the block's range the warps' running
// values are merged first where they are of one segment. Min and max do not
// depend on the order, so the result is the one of any reduction order. Bound by latency:
// few rows where that still gives blocks for the chip (81,920 triangles: 13.7 us with 16
// rows and six atomics per warp, 3.1 with one).
__global__ void __launch_bounds__(256) blas_bounds_kernel(const SegDesc* segs, const uint32_t* seg_prim_off,
                                                          int nseg, uint32_t total, uint32_t rows, uint32_t* seg_bounds) {
    chain_wait();
    __shared__ int s_seg[8];
    __shared__ uint32_t s_acc[8][6];
    const uint32_t full = 0xFFFFFFFFu;
    const bool leader = (threadIdx.x & 31) == 0;
    int acc_s = -1;
    uint32_t acc[6] = {0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu, 0u, 0u, 0u};
    auto flush = [&]() {
        if (acc_s < 0) return;
        uint32_t* b = seg_bounds + 6 * acc_s;
        for (int a = 0; a < 3; ++a) if (acc[a] != 0xFFFFFFFFu) atomicMin(b + a, acc[a]);
        for (int a = 3; a < 6; ++a) if (acc[a] != 0u) atomicMax(b + a, acc[a]);
    };
    const uint32_t base = blockIdx.x * (blockDim.x * rows);
    for (uint32_t it = 0; it < rows; ++it) {
        const uint32_t row = base + it * blockDim.x;
        if (row >= total) break;   // uniform across the block
        const uint32_t g = row + threadIdx.x;
        const bool in = g < total;
        const int s = in ? find_seg(seg_prim_off, nseg, g) : -1;
        uint32_t k[6] = {0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu, 0u, 0u, 0u};
        if (in) {
            const SegDesc sd = segs[s];
            const uint32_t p = g - sd.prim_off;
            const uint32_t i0 = sd.indices[3 * p], i1 = sd.indices[3 * p + 1], i2 = sd.indices[3 * p + 2];
            V3 lo, hi;
            tri_box(load_pos(sd.vertices, i0), load_pos(sd.vertices, i1), load_pos(sd.vertices, i2), lo, hi);
            V3 c = V3{(lo.x + hi.x) * 0.5f + 0.0f, (lo.y + hi.y) * 0.5f + 0.0f, (lo.z + hi.z) * 0.5f + 0.0f};
            if (finite3(c)) {
                k[0] = k[3] = float_to_ordered(c.x);
                k[1] = k[4] = float_to_ordered(c.y);
                k[2] = k[5] = float_to_ordered(c.z);
            }
        }
        const int s0 = __shfl_sync(full, s, 0);
        if (__all_sync(full, s == s0 || s < 0)) {
            uint32_t r[6];
            for (int a = 0; a < 3; ++a) r[a] = __reduce_min_sync(full, k[a]);
            for (int a = 3; a < 6; ++a) r[a] = __reduce_max_sync(full, k[a]);
            if (leader && s0 >= 0) {
                if (s0 != acc_s) {
                    flush();
                    acc_s = s0;
                    for (int a = 0; a < 3; ++a) { acc[a] = 0xFFFFFFFFu; acc[a + 3] = 0u; }
                }
                for (int a = 0; a < 3; ++a) acc[a] = min(acc[a], r[a]);
                for (int a = 3; a < 6; ++a) acc[a] = max(acc[a], r[a]);
            }
        } else if (s >= 0 && k[0] != 0xFFFFFFFFu) {
            uint32_t* b = seg_bounds + 6 * s;
            for (int a = 0; a < 3; ++a) atomicMin(b + a, k[a]);
            for (int a = 3; a < 6; ++a) atomicMax(b + a, k[a]);
        }
    }
    if (leader) {
        const uint32_t w = threadIdx.x >> 5;
        s_seg[w] = acc_s;
        for (int a = 0; a < 6; ++a) s_acc[w][a] = acc[a];
    }
    __syncthreads();
    bool same = true;   // of the warps that have a running value
    for (int w = 0; w < 8; ++w) same = same && (s_seg[w] == s_seg[0] || s_seg[w] < 0);
    if (!same) {
        if (leader) flush();
    } else if (threadIdx.x < 6 && s_seg[0] >= 0) {
        uint32_t v = s_acc[0][threadIdx.x];
        for (int w = 1; w < 8; ++w) v = threadIdx.x < 3 ? min(v, s_acc[w][threadIdx.x]) : max(v, s_acc[w][threadIdx.x]);
        uint32_t* b = seg_bounds + 6 * s_seg[0] + threadIdx.x;
        if (threadIdx.x < 3) { if (v != 0xFFFFFFFFu) atomicMin(b, v); }
        else if (v != 0u) atomicMax(b, v);
    }
}

// The sort's digit histograms: a block counts its keys in shared memory and adds what it
// found. Used by the kernels that make the keys, so that they are not read again.
struct BlockHist {
    uint32_t (*h)[kRadix];
    int passes;
    __device__ __forceinline__ void clear() const {
        for (int i = threadIdx.x; i < passes * kRadix; i += blockDim.x) (&h[0][0])[i] = 0u;
        __syncthreads();
    }
    __device__ __forceinline__ void count(unsigned long long key) const {
        for (int p = 0; p < passes; ++p) atomicAdd(&h[p][(key >> (8 * p)) & 0xFF], 1u);
    }
    __device__ __forceinline__ void add(uint32_t* hist) const {
        __syncthreads();
        for (int i = threadIdx.x; i < passes * kRadix; i += blockDim.x) {
            const uint32_t v = (&h[0][0])[i];
            if (v) atomicAdd(hist + i, v);
        }
    }
};

__global__ void __launch_bounds__(256) blas_morton_kernel(const SegDesc* segs, const uint32_t* seg_prim_off, int nseg,
                                                          uint32_t total, const uint32_t* seg_bounds,
                                                          unsigned long long* keys, uint32_t* vals, int passes,
                                                          uint32_t* hist) {
    chain_wait();
    __shared__ uint32_t s_hist[kMaxPasses][kRadix];
    const BlockHist H{s_hist, passes};
    H.clear();
    for (uint32_t g = blockIdx.x * blockDim.x + threadIdx.x; g < total; g += gridDim.x * blockDim.x) {
        int s = find_seg(seg_prim_off, nseg, g);
        const SegDesc sd = segs[s];
        uint32_t p = g - sd.prim_off;
        uint32_t i0 = sd.indices[3 * p], i1 = sd.indices[3 * p + 1], i2 = sd.indices[3 * p + 2];
        V3 lo, hi;
        tri_box(load_pos(sd.vertices, i0), load_pos(sd.vertices, i1), load_pos(sd.vertices, i2), lo, hi);
        V3 cmin, ext;
        decode_bounds(seg_bounds + 6 * s, cmin, ext);
        const unsigned long long key = ((unsigned long long)s << 30) | morton30(lo, hi, cmin, ext);
        keys[g] = key;
        vals[g] = g;
        H.count(key);
    }
    H.add(hist);
}

// ---------------------------------------------------------------- onesweep radix sort
// Block-wide exclusive scan of one value per thread (blockDim.x == 256).
__device__ __forceinline__ uint32_t block_excl_scan_256(uint32_t v, uint32_t* s_tmp /*8*/,
                                                        uint32_t* total) {
    int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t x = v;
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) s_tmp[warp] = x;
    __syncthreads();
    uint32_t wsum = 0, all = 0;
    for (int w = 0; w < 8; ++w) {
        uint32_t t = s_tmp[w];
        if (w < warp) wsum += t;
        all += t;
    }
    __syncthreads();
    if (total) *total = all;
    return wsum + x - v;
}

__device__ __forceinline__ uint32_t ld_volatile_u32(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.volatile.global.u32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ void st_volatile_u32(uint32_t* p, uint32_t v) {
    asm volatile("st.volatile.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

__global__ void __launch_bounds__(kSortThreads)
onesweep_pass_kernel(const unsigned long long* __restrict__ kin, const uint32_t* __restrict__ vin,
                     unsigned long long* __restrict__ kout, uint32_t* __restrict__ vout, uint32_t n,
                     int shift, const uint32_t* __restrict__ pass_hist, uint32_t* __restrict__ pass_offsets,
                     uint32_t* tile_status, uint32_t* tile_counter, uint32_t* dev_status) {
    chain_wait();
    __shared__ uint32_t s_tile;
    __shared__ uint32_t s_warp_hist[kSortWarps][kRadix];
    __shared__ uint32_t s_digit_excl[kRadix];
    __shared__ uint32_t s_global_base[kRadix];
    __shared__ uint32_t s_tmp[8];
    __shared__ unsigned long long s_keys[kSortTile];
    __shared__ uint32_t s_vals[kSortTile];

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // Tiles in the order the blocks start, so that a look-back waits only on blocks that run,
    // however few of them the chip has room for beside other streams' kernels.
    if (tid == 0) s_tile = atomicAdd(tile_counter, 1u);
    for (int i = tid; i < kSortWarps * kRadix; i += kSortThreads) (&s_warp_hist[0][0])[i] = 0;
    __syncthreads();
    const uint32_t tile = s_tile;
    const uint32_t base = tile * kSortTile;

    unsigned long long key[kSortItems];
    uint32_t val[kSortItems], dig[kSortItems], rank[kSortItems];
#pragma unroll
    for (int k = 0; k < kSortItems; ++k) {
        uint32_t idx = base + warp * (32 * kSortItems) + k * 32 + lane;
        bool valid = idx < n;
        key[k] = valid ? kin[idx] : 0ull;
        val[k] = valid ? vin[idx] : 0u;
        dig[k] = valid ? (uint32_t)((key[k] >> shift) & 0xFF) : 256u;
    }
    const uint32_t lt_mask = (1u << lane) - 1u;
#pragma unroll
    for (int k = 0; k < kSortItems; ++k) {
        uint32_t d = dig[k];
        uint32_t peers = __match_any_sync(0xFFFFFFFFu, d);
        uint32_t before = peers & lt_mask;
        uint32_t cnt = (d < 256) ? s_warp_hist[warp][d] : 0u;
        rank[k] = cnt + __popc(before);
        __syncwarp();
        if (d < 256 && before == 0) s_warp_hist[warp][d] = cnt + __popc(peers);
        __syncwarp();
    }
    __syncthreads();
    // Digit `tid`: exclusive scan across warps and tile total.
    uint32_t tile_count = 0;
#pragma unroll
    for (int w = 0; w < kSortWarps; ++w) {
        uint32_t c = s_warp_hist[w][tid];
        s_warp_hist[w][tid] = tile_count;
        tile_count += c;
    }
    // Decoupled look-back for digit `tid`.
    uint32_t* my_status = tile_status + (size_t)tile * kRadix + tid;
    uint32_t global_base;
    if (tile == 0) {
        // the pass's digit offsets: the exclusive scan of its histogram
        global_base = block_excl_scan_256(pass_hist[tid], s_tmp, nullptr);
        pass_offsets[tid] = global_base;
        st_volatile_u32(my_status, kFlagPrefix | (global_base + tile_count));
    } else {
        st_volatile_u32(my_status, kFlagAggregate | tile_count);
        uint32_t excl = 0;
        int j = (int)tile - 1;
        uint32_t spins = 0;
        bool done = false;
        while (!done) {
            // kLookback words of earlier tiles in flight at a time (tile 0 ends every look-back)
            uint32_t w[kLookback];
#pragma unroll
            for (int k = 0; k < kLookback; ++k)
                w[k] = j - k >= 0 ? ld_volatile_u32(tile_status + (size_t)(j - k) * kRadix + tid) : 0u;
            int used = 0;
#pragma unroll
            for (int k = 0; k < kLookback; ++k) {
                if (done || used != k) continue;
                const uint32_t flag = w[k] & ~kValueMask;
                if (flag == 0) continue;
                excl += w[k] & kValueMask;
                done = flag == kFlagPrefix;
                ++used;
            }
            j -= used;
            if (!done && used == 0 && ++spins > kLookbackSpinLimit) {
                atomicOr(dev_status, (uint32_t)LUZ_DEV_SORT_LOOKBACK_TIMEOUT);
                done = true;
            }
        }
        global_base = excl;
        st_volatile_u32(my_status, kFlagPrefix | (excl + tile_count));
    }
    s_global_base[tid] = global_base;
    s_digit_excl[tid] = block_excl_scan_256(tile_count, s_tmp, nullptr);
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kSortItems; ++k) {
        uint32_t d = dig[k];
        if (d < 256) {
            uint32_t pos = s_digit_excl[d] + s_warp_hist[warp][d] + rank[k];
            s_keys[pos] = key[k];
            s_vals[pos] = val[k];
        }
    }
    __syncthreads();
    uint32_t tile_n = min((uint32_t)kSortTile, n - base);
    for (uint32_t i = tid; i < tile_n; i += kSortThreads) {
        unsigned long long k = s_keys[i];
        uint32_t d = (uint32_t)((k >> shift) & 0xFF);
        uint32_t out = s_global_base[d] + (i - s_digit_excl[d]);
        if (out < n) {   // always true unless a look-back timed out (status word raised)
            kout[out] = k;
            vout[out] = s_vals[i];
        }
    }
}

// ---------------------------------------------------------------- hierarchy + refit
// The radix tree bottom-up, boxes and all, in one kernel (the scheme of C. Apetrei, "Fast and
// Simple Agglomerative LBVH Construction", CGVC 2014): a thread per leaf climbs; a range
// [l, r] of leaves merges with the neighbour it shares the longer prefix with, and the
// second of the two to arrive goes on with the union. The tree is the one of T. Karras
// (HPG 2012), and so is its numbering: a node that is a left child has the index of its
// last leaf, a right child that of its first, the root 0.
//
// A block takes a span of consecutive leaves. Merges whose union lies inside them happen
// in shared memory; whether one does follows from the prefix lengths between the block's
// leaves alone: the union of a merge at prefix length d ends inside the block on either side
// where that side has a shorter prefix. Other merges, and all above them, meet in device
// memory: each side stores its node, then its far end with the prefix there, then counts
// itself with an acquire-release atomic, and the second reads the sibling's box from its node. Bound by the
// latency of those climbs. 81,920 triangles: 32 us against 51 (a search per node for its range and
// split, leaves, and a refit through device memory: 11.9 + 4.4 + 34.6 us).
// The leaves of a block: from the place with the shortest prefix in a window of kMergeStep
// leaves around kMergeStep * block to that of the next block, 511 at most. The merges that
// cross a block's ends are the ancestors of the nodes split there: a split high up in the
// tree has few, one at a fixed distance as many as any node (81,920 triangles: 54 us with
// blocks of 512 leaves).
struct MergeSpan {
    uint32_t first, count;
};

struct MergeShared {
    float box[kMergeLeaves][2][6];    // per merge position: the two sides' boxes
    uint32_t end[kMergeLeaves][2];
    uint32_t flag[kMergeLeaves];
    int8_t delta[kMergeLeaves + 1];   // prefix length between leaf b0 - 1 + k and the next (-1: none)
    int8_t before[kMergeLeaves], after[kMergeLeaves];   // least delta of the pairs before / after a position's
    int8_t warp_min[kMergeLeaves / 32];
    uint32_t cut[kMergeLeaves / 32];
};

// Called by whole blocks of kMergeLeaves = 2 kMergeStep threads: half of them look at either end.
__device__ __forceinline__ MergeSpan merge_span(MergeShared& S, const unsigned long long* keys, uint32_t total) {
    const uint32_t tid = threadIdx.x, t = blockIdx.x + tid / kMergeStep, i = tid % kMergeStep;
    const uint32_t at = t * kMergeStep + i - kMergeStep / 2;   // (t = 0 is the first leaf)
    uint32_t key = 0xFFFFFFFFu;
    if (t > 0 && at < total) {
        const unsigned long long a = keys[at - 1], b = keys[at];
        key = ((a == b ? 64u + __clz((at - 1) ^ at) : (uint32_t)__clzll((long long)(a ^ b))) << 16) | i;
    }
    key = __reduce_min_sync(0xFFFFFFFFu, key);
    if ((tid & 31) == 0) S.cut[tid >> 5] = key;
    __syncthreads();
    uint32_t end[2];
#pragma unroll
    for (uint32_t h = 0; h < 2; ++h) {
        uint32_t k = 0xFFFFFFFFu;
#pragma unroll
        for (uint32_t w = 0; w < kMergeStep / 32; ++w) k = min(k, S.cut[h * (kMergeStep / 32) + w]);
        const uint32_t b = blockIdx.x + h;
        end[h] = b == 0 ? 0u : (k == 0xFFFFFFFFu ? total : b * kMergeStep + (k & 0xFFFFu) - kMergeStep / 2);
    }
    return MergeSpan{end[0], end[1] - end[0]};
}

// Prefix length between leaf g and g + 1 of all segments' leaves (-1 across a segment's end).
__device__ __forceinline__ int pair_delta(const SegDesc& sd, const unsigned long long* keys, uint32_t g) {
    if (g < sd.prim_off || g - sd.prim_off + 1 >= sd.prim_count) return -1;   // (g may be prim_off - 1)
    const uint32_t a = (uint32_t)keys[g] & 0x3FFFFFFFu, b = (uint32_t)keys[g + 1] & 0x3FFFFFFFu;
    if (a != b) return __clz(a ^ b);
    const uint32_t i = g - sd.prim_off;
    return 32 + __clz(i ^ (i + 1));
}

// The leaf of thread t is span.first + t (in: it is of the span), of segment sd with box
// [lo, hi]; called by whole blocks of kMergeLeaves threads. leaf_box(j, lo, hi): the box of leaf j of the segment,
// written before by the thread of that leaf.
template <typename LeafBox>
__device__ __forceinline__ void merge_block(MergeShared& S, const MergeArgs& A, MergeSpan span, const SegDesc& sd, bool in,
                                            float4 lo, float4 hi, const LeafBox& leaf_box) {
    const uint32_t full = 0xFFFFFFFFu, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t b0 = span.first, g = b0 + tid;
    S.flag[tid] = 0u;
    const int dg = in ? pair_delta(sd, A.keys, g) : 127;   // past the span: no bound
    S.delta[tid + 1] = (int8_t)dg;
    if (tid == 0) S.delta[0] = (int8_t)(in && g > 0 ? pair_delta(sd, A.keys, g - 1) : -1);
    // least deltas of the pairs after / before each position's pair, inside the block (the
    // pair before its first leaf counts)
    int up = dg, down = dg;   // inclusive within the warp
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(full, up, o), v = __shfl_down_sync(full, down, o);
        if (lane >= (uint32_t)o) up = min(up, u);
        if (lane + o < 32) down = min(down, v);
    }
    if (lane == 31) S.warp_min[warp] = (int8_t)up;
    __syncthreads();
    {
        int u = __shfl_up_sync(full, up, 1), v = __shfl_down_sync(full, down, 1);
        if (lane == 0) u = 127;
        if (lane == 31) v = 127;
        u = min(u, (int)S.delta[0]);
        for (uint32_t w = 0; w < kMergeLeaves / 32; ++w) {
            if (w < warp) u = min(u, (int)S.warp_min[w]);
            if (w > warp) v = min(v, (int)S.warp_min[w]);
        }
        S.before[tid] = (int8_t)u;
        S.after[tid] = (int8_t)v;
    }
    __syncthreads();
    const bool climbs = in && sd.prim_count >= 2;
    const uint32_t off = sd.prim_off, last = off + sd.prim_count - 1;
    uint32_t l = g, r = g;
    int dl = S.delta[tid], dr = S.delta[tid + 1];   // prefixes before and after [l, r]
    bool go = climbs;                               // still on its way at the end of the local merges
    if (climbs) {
        while (l != off || r != last) {             // every pass widens [l, r]
            const bool left = dr > dl;
            const uint32_t m = left ? r : l - 1, k = m - b0;   // the merge: between leaf m and m + 1
            const int d = max(dl, dr);
            if (!(m >= b0 && k < kMergeLeaves && (int)S.before[k] < d && (int)S.after[k] < d)) break;
            const uint32_t side = left ? 0u : 1u;
            float* slot = S.box[k][side];
            slot[0] = lo.x; slot[1] = lo.y; slot[2] = lo.z;
            slot[3] = hi.x; slot[4] = hi.y; slot[5] = hi.z;
            S.end[k][side] = left ? l : r;
            __threadfence_block();
            if (atomicAdd(&S.flag[k], 1u) == 0u) { go = false; break; }
            __threadfence_block();
            const float* c0 = S.box[k][0];
            const float* c1 = S.box[k][1];
            lo = make_float4(fmin_(c0[0], c1[0]), fmin_(c0[1], c1[1]), fmin_(c0[2], c1[2]), 0.f);
            hi = make_float4(fmax_(c0[3], c1[3]), fmax_(c0[4], c1[4]), fmax_(c0[5], c1[5]), 0.f);
            l = S.end[k][0];
            r = S.end[k][1];
            if (l < b0 || r - b0 >= kMergeLeaves || l > m || r <= m) {   // (never for sorted keys)
                atomicOr(A.status, (uint32_t)LUZ_DEV_KARRAS_RANGE);
                go = false;
                break;
            }
            dl = S.delta[l - b0];
            dr = S.delta[r - b0 + 1];
        }
    }
    __syncthreads();
    // the nodes completed in shared memory, one per merge position
    auto put_node = [&](const SegDesc& seg, uint32_t nl, uint32_t nr, uint32_t m, int el, int er, float4 lo0, float4 hi0,
                        float4 lo1, float4 hi1) {
        const uint32_t o = seg.prim_off;
        const bool top = nl == o && nr == o + seg.prim_count - 1;
        // its own side, and so its index, from the prefixes around it
        const uint32_t node = top ? 0u : (er > el ? nr : nl) - o;
        const int c0 = nl == m ? ~(int)(m - o) : (int)(m - o);
        const int c1 = nr == m + 1 ? ~(int)(m + 1 - o) : (int)(m + 1 - o);
        float4* q = seg.nodes + (size_t)node * kNodeF4;
        q[0] = make_float4(lo0.x, hi0.x, lo0.y, hi0.y);
        q[1] = make_float4(lo1.x, hi1.x, lo1.y, hi1.y);
        q[2] = make_float4(lo0.z, hi0.z, lo1.z, hi1.z);
        q[3] = make_float4(__int_as_float(c0), __int_as_float(c1), 0.f, 0.f);
        if (A.node_parent) {
            uint32_t* parent = A.node_parent + seg.node_off;
            if (c0 >= 0) parent[c0] = node << 1;
            if (c1 >= 0) parent[c1] = (node << 1) | 1u;
            if (top) parent[0] = 0xFFFFFFFFu;
        }
    };
    if (in && S.flag[tid] == 2u) {   // a merge position lies in the segment of its leaf
        const uint32_t nl = S.end[tid][0], nr = S.end[tid][1];
        const float* c0 = S.box[tid][0];
        const float* c1 = S.box[tid][1];
        if (nl >= b0 && nr - b0 < kMergeLeaves)
            put_node(sd, nl, nr, g, S.delta[nl - b0], S.delta[nr - b0 + 1], make_float4(c0[0], c0[1], c0[2], 0.f),
                     make_float4(c0[3], c0[4], c0[5], 0.f), make_float4(c1[0], c1[1], c1[2], 0.f),
                     make_float4(c1[3], c1[4], c1[5], 0.f));
    }
    __syncthreads();   // the block's nodes before its first merge in device memory
    while (go && (l != off || r != last)) {
        const bool left = dr > dl;
        const uint32_t m = left ? r : l - 1;
        (left ? A.ends[0] : A.ends[1])[m] = left ? make_uint2(l, (uint32_t)(dl + 1)) : make_uint2(r, (uint32_t)(dr + 1));
        if (atomic_add_acq_rel_gpu(A.flags + m, 1u) == 0u) break;
        // the sibling's far end and the prefix there, and both that it may be, its leaf and its
        // node, in flight together
        const uint32_t sib = (left ? m + 1 : m) - off;
        const float4* q = sd.nodes + (size_t)min(sib, sd.prim_count - 2u) * kNodeF4;
        const uint2 far = __ldcg((left ? A.ends[1] : A.ends[0]) + m);
        const uint32_t oend = far.x;
        const float4 n0 = __ldcg(q), n1 = __ldcg(q + 1), n2 = __ldcg(q + 2);
        float4 olo, ohi;
        leaf_box(sib, olo, ohi);
        if (oend != sib + off) {
            olo = make_float4(fmin_(n0.x, n1.x), fmin_(n0.z, n1.z), fmin_(n2.x, n2.z), 0.f);
            ohi = make_float4(fmax_(n0.y, n1.y), fmax_(n0.w, n1.w), fmax_(n2.y, n2.w), 0.f);
        }
        if (left ? oend <= m || oend > last : oend > m || oend < off) {   // (never for sorted keys)
            atomicOr(A.status, (uint32_t)LUZ_DEV_KARRAS_RANGE);
            break;
        }
        const float4 lo0 = left ? lo : olo, hi0 = left ? hi : ohi, lo1 = left ? olo : lo, hi1 = left ? ohi : hi;
        if (left) { r = oend; dr = (int)far.y - 1; }
        else { l = oend; dl = (int)far.y - 1; }
        put_node(sd, l, r, m, dl, dr, lo0, hi0, lo1, hi1);
        lo = make_float4(fmin_(lo0.x, lo1.x), fmin_(lo0.y, lo1.y), fmin_(lo0.z, lo1.z), 0.f);
        hi = make_float4(fmax_(hi0.x, hi1.x), fmax_(hi0.y, hi1.y), fmax_(hi0.z, hi1.z), 0.f);
    }
}

// The padded box of a triangle.
__device__ __forceinline__ void leaf_tri_box(V3 a, V3 b, V3 c, float4& lo, float4& hi) {
    V3 l, h;
    tri_box(a, b, c, l, h);
    const float px = leaf_pad(l.x, h.x), py = leaf_pad(l.y, h.y), pz = leaf_pad(l.z, h.z);
    lo = make_float4(l.x - px, l.y - py, l.z - pz, 0.f);
    hi = make_float4(h.x + px, h.y + py, h.z + pz, 0.f);
}

// The node of a segment without leaves or with one (leaf 0, box [lo, hi]).
__device__ __forceinline__ void write_single_node(const SegDesc& sd, uint32_t* node_parent, float4 lo, float4 hi) {
    write_inverted_slot(sd.nodes, 0);
    write_inverted_slot(sd.nodes, 1);
    if (sd.prim_count == 1) write_slot(sd.nodes, 0, lo, hi);
    sd.nodes[3] = make_float4(__int_as_float(sd.prim_count == 1 ? ~0 : kEmptyChild), __int_as_float(kEmptyChild), 0.f, 0.f);
    if (node_parent) node_parent[sd.node_off] = 0xFFFFFFFFu;
}

// The nodes of the segments without a leaf (the others' are written with their leaves).
__global__ void empty_segments_kernel(const SegDesc* segs, int nseg, uint32_t* node_parent) {
    chain_wait();
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s < nseg && segs[s].prim_count == 0) write_single_node(segs[s], node_parent, float4{}, float4{});
}

// BLAS: triangles gathered into leaf order, sorted morton/order into the segment's own
// arrays, and the hierarchy over them.
__global__ void __launch_bounds__(kMergeLeaves) blas_tree_kernel(const SegDesc* segs, const uint32_t* seg_prim_off, int nseg,
                                                                 const uint32_t* vals, MergeArgs A) {
    chain_wait();
    __shared__ MergeShared S;
    const MergeSpan span = merge_span(S, A.keys, A.total);
    const uint32_t g = span.first + threadIdx.x;
    const bool in = threadIdx.x < span.count;
    SegDesc sd{};
    float4 lo = make_float4(0.f, 0.f, 0.f, 0.f), hi = lo;
    if (in) {
        sd = segs[find_seg(seg_prim_off, nseg, g)];
        const uint32_t j = g - sd.prim_off, prim = vals[g] - sd.prim_off;
        sd.morton[j] = (uint32_t)A.keys[g] & 0x3FFFFFFFu;
        sd.order[j] = prim;
        const uint32_t i0 = sd.indices[3 * prim], i1 = sd.indices[3 * prim + 1], i2 = sd.indices[3 * prim + 2];
        const V3 a = load_pos(sd.vertices, i0), b = load_pos(sd.vertices, i1), c = load_pos(sd.vertices, i2);
        float4* t = sd.tris + (size_t)j * kTriF4;
        t[0] = make_float4(a.x, a.y, a.z, __int_as_float((int)prim));
        t[1] = make_float4(b.x, b.y, b.z, 0.f);
        t[2] = make_float4(c.x, c.y, c.z, 0.f);
        leaf_tri_box(a, b, c, lo, hi);
        if (sd.prim_count == 1) write_single_node(sd, A.node_parent, lo, hi);
    }
    const float4* tris = sd.tris;
    merge_block(S, A, span, sd, in, lo, hi, [tris](uint32_t j, float4& l, float4& h) {
        const float4* t = tris + (size_t)j * kTriF4;
        const float4 a = __ldcg(t), b = __ldcg(t + 1), c = __ldcg(t + 2);
        leaf_tri_box(V3{a.x, a.y, a.z}, V3{b.x, b.y, b.z}, V3{c.x, c.y, c.z}, l, h);
    });
}

// ---------------------------------------------------------------- bounding sphere

// Bounding sphere of every BLAS about its root box centre: the largest squared
// distance of a triangle vertex from the centre, kept as float bits in the root
// node's spare word n3.z (zero after the hierarchy pass; positive floats order like their
// bits, so atomicMax on the bits is a float max). Runs after the refit. The TLAS
// build intersects each instance's transformed root box with the transformed sphere.
__global__ void blas_radius_kernel(const SegDesc* segs, const uint32_t* seg_prim_off, int nseg,
                                   uint32_t total) {
    chain_wait();
    uint32_t g = blockIdx.x * blockDim.x + threadIdx.x;
    bool in = g < total;
    int s = in ? find_seg(seg_prim_off, nseg, g) : -1;
    uint32_t r2 = 0u;
    float4* root = nullptr;
    if (in) {
        const SegDesc sd = segs[s];
        root = sd.nodes;
        V3 c = root_centre(__ldcg(root + 0), __ldcg(root + 1), __ldcg(root + 2));
        const float4* t = sd.tris + (size_t)(g - sd.prim_off) * kTriF4;
        for (int k = 0; k < 3; ++k) {
            float4 v = t[k];
            float dx = v.x - c.x, dy = v.y - c.y, dz = v.z - c.z;
            float d2 = dx * dx + dy * dy + dz * dz;
            r2 = max(r2, __float_as_uint(d2));
        }
    }
    const uint32_t full = 0xFFFFFFFFu;
    int s0 = __shfl_sync(full, s, 0);
    bool uniform = __all_sync(full, s == s0 || s < 0);
    // one atomic per block where it is of one segment (320 instead of 2560 to one word)
    __shared__ int s_seg;
    __shared__ uint32_t s_max;
    if (threadIdx.x == 0) {
        s_seg = s0;
        s_max = 0u;
    }
    __syncthreads();
    if (__syncthreads_and(uniform && (s0 == s_seg || s0 < 0))) {
        const uint32_t r = __reduce_max_sync(full, r2);
        if ((threadIdx.x & 31) == 0) atomicMax(&s_max, r);
        __syncthreads();
        if (threadIdx.x == 0 && s >= 0) atomicMax((uint32_t*)&root[3].z, s_max);
    } else if (uniform) {
        uint32_t r = __reduce_max_sync(full, r2);
        float4* root0 = (float4*)__shfl_sync(full, (unsigned long long)root, 0);
        if ((threadIdx.x & 31) == 0 && s0 >= 0) atomicMax((uint32_t*)&root0[3].z, r);
    } else if (s >= 0) {
        atomicMax((uint32_t*)&root[3].z, r2);
    }
}

// ---------------------------------------------------------------- 4-wide collapse
// Every binary node at even depth becomes a 4-wide node whose slots are its
// grandchildren (or its children, where a child is a leaf). Numbering: the rank of
// the node among its segment's even-depth nodes in binary-node order (root first).

// flags[q] = 1 when internal node q lies at even depth in its segment's tree.
__global__ void even_depth_kernel(const SegDesc* segs, const uint32_t* seg_node_off, int nseg, uint32_t total_nodes,
                                  const uint32_t* node_parent, uint32_t* flags) {
    chain_wait();
    uint32_t q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= total_nodes) return;
    int s = find_seg(seg_node_off, nseg, q);
    const uint32_t off = segs[s].node_off;
    uint32_t d = 0, p = node_parent[q];
    for (uint32_t guard = 0; p != 0xFFFFFFFFu && guard < 4096; ++guard) {
        ++d;
        p = node_parent[off + (p >> 1)];
    }
    flags[q] = (d & 1u) == 0u;
}

// Chunked exclusive scan of u32 (chunks of 1024 = 256 threads x 4).
__global__ void __launch_bounds__(256) chunk_sum_kernel(const uint32_t* in, uint32_t n, uint32_t* sums) {
    chain_wait();
    __shared__ uint32_t s_tmp[8];
    uint32_t base = blockIdx.x * 1024 + threadIdx.x * 4, c = 0;
    for (int k = 0; k < 4; ++k) c += base + k < n ? in[base + k] : 0u;
    for (int o = 16; o > 0; o >>= 1) c += __shfl_down_sync(0xFFFFFFFFu, c, o);
    if ((threadIdx.x & 31) == 0) s_tmp[threadIdx.x >> 5] = c;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t t = 0;
        for (int w = 0; w < 8; ++w) t += s_tmp[w];
        sums[blockIdx.x] = t;
    }
}

__global__ void __launch_bounds__(1024) chunk_scan_kernel(uint32_t* sums, uint32_t chunks) {
    chain_wait();
    __shared__ uint32_t s_warp[32];
    __shared__ uint32_t s_carry;
    int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) s_carry = 0;
    __syncthreads();
    for (uint32_t base = 0; base < chunks; base += 1024) {
        uint32_t i = base + threadIdx.x;
        uint32_t v = i < chunks ? sums[i] : 0u, x = v;
        for (int o = 1; o < 32; o <<= 1) {
            uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) s_warp[warp] = x;
        __syncthreads();
        uint32_t pre = 0, all = 0;
        for (int w = 0; w < 32; ++w) {
            if (w < warp) pre += s_warp[w];
            all += s_warp[w];
        }
        uint32_t carry = s_carry;
        if (i < chunks) sums[i] = carry + pre + x - v;
        __syncthreads();
        if (threadIdx.x == 0) s_carry = carry + all;
        __syncthreads();
    }
}

__global__ void __launch_bounds__(256) chunk_apply_kernel(const uint32_t* in, uint32_t n, const uint32_t* offs,
                                                          uint32_t* out) {
    chain_wait();
    __shared__ uint32_t s_tmp[8];
    uint32_t base = blockIdx.x * 1024 + threadIdx.x * 4;
    uint32_t v[4], c = 0;
    for (int k = 0; k < 4; ++k) { v[k] = base + k < n ? in[base + k] : 0u; c += v[k]; }
    int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t x = c;
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) s_tmp[warp] = x;
    __syncthreads();
    uint32_t pre = 0;
    for (int w = 0; w < warp; ++w) pre += s_tmp[w];
    uint32_t run = offs[blockIdx.x] + pre + x - c;
    for (int k = 0; k < 4; ++k) {
        if (base + k < n) out[base + k] = run;
        run += v[k];
    }
}




// idx4[q]: exclusive prefix of the even-depth flags over all segments' nodes.
__global__ void bvh4_emit_kernel(const SegDesc* segs, const uint32_t* seg_node_off, int nseg, uint32_t total_nodes,
                                 const uint32_t* flags, const uint32_t* idx4) {
    chain_wait();
    uint32_t q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= total_nodes || !flags[q]) return;
    int s = find_seg(seg_node_off, nseg, q);
    const SegDesc sd = segs[s];
    if (!sd.nodes4) return;
    const uint32_t base4 = idx4[sd.node_off];
    const float4* n2 = sd.nodes + (size_t)(q - sd.node_off) * kNodeF4;
    float4 n3 = n2[3];
    int c[2] = {__float_as_int(n3.x), __float_as_int(n3.y)};
    Slot4 s4;
    s4.k = 0;
    for (int side = 0; side < 2; ++side) {
        if (c[side] < 0) {
            slot4_put(s4, n2, side, c[side]);
            continue;
        }
        const float4* m = sd.nodes + (size_t)c[side] * kNodeF4;
        float4 m3 = m[3];
        int g[2] = {__float_as_int(m3.x), __float_as_int(m3.y)};
        for (int s2 = 0; s2 < 2; ++s2)
            slot4_put(s4, m, s2, g[s2] < 0 ? g[s2] : (int)(idx4[sd.node_off + g[s2]] - base4));
    }
    slot4_store(s4, sd.nodes4 + (size_t)(idx4[q] - base4) * kNode4F4);
}


// ---------------------------------------------------------------- TLAS

// Ordered keys of a box centre's bounds (an empty range where there is none), reduced over
// the warp and merged by its first lane.
__device__ __forceinline__ void merge_bounds(bool have, V3 c, uint32_t* bounds) {
    uint32_t k[6] = {0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu, 0u, 0u, 0u};
    if (have) {
        k[0] = k[3] = float_to_ordered(c.x);
        k[1] = k[4] = float_to_ordered(c.y);
        k[2] = k[5] = float_to_ordered(c.z);
    }
#pragma unroll
    for (int a = 0; a < 6; ++a)
        k[a] = a < 3 ? __reduce_min_sync(0xFFFFFFFFu, k[a]) : __reduce_max_sync(0xFFFFFFFFu, k[a]);
    if ((threadIdx.x & 31) == 0) {
#pragma unroll
        for (int a = 0; a < 3; ++a) atomicMin(bounds + a, k[a]);
#pragma unroll
        for (int a = 3; a < 6; ++a) atomicMax(bounds + a, k[a]);
    }
}

// seg_bounds: NULL where the next kernel takes the bounds from the boxes.
__global__ void tlas_instance_kernel(const DevInstanceInput* in, uint32_t n, float4* inst_box,
                                     DevShadeInstance* shade, uint32_t* seg_bounds) {
    chain_wait();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    V3 c;
    const bool have = i < n && tlas_instance_one(in, i, inst_box, shade, c);
    if (seg_bounds) merge_bounds(have, c, seg_bounds);
}

__global__ void tlas_setup_kernel(uint32_t* bounds, SegDesc* seg, SegDesc value) {
    chain_wait();
    if (threadIdx.x < 6) bounds[threadIdx.x] = threadIdx.x < 3 ? 0xFFFFFFFFu : 0u;
    if (threadIdx.x == 0) *seg = value;
}

__global__ void __launch_bounds__(256) tlas_morton_kernel(const float4* inst_box, uint32_t n, const uint32_t* seg_bounds,
                                                          unsigned long long* keys, uint32_t* vals, int passes,
                                                          uint32_t* hist) {
    chain_wait();
    __shared__ uint32_t s_hist[kMaxPasses][kRadix];
    const BlockHist H{s_hist, passes};
    H.clear();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) {
        float4 l = inst_box[2 * i], h = inst_box[2 * i + 1];
        V3 cmin, ext;
        decode_bounds(seg_bounds, cmin, ext);
        keys[i] = morton30(V3{l.x, l.y, l.z}, V3{h.x, h.y, h.z}, cmin, ext);
        vals[i] = i;
        H.count(keys[i]);
    }
    H.add(hist);
}

// Instance records in leaf order, leaf boxes, sorted codes and order, and the hierarchy
// over them (seg: the one segment, at least two leaves).
__global__ void __launch_bounds__(kMergeLeaves) tlas_tree_kernel(const SegDesc* seg, const DevInstanceInput* in_instances,
                                                                 const float4* inst_box, const uint32_t* vals,
                                                                 DevInstance* inst_out, float4* leaf_boxes,
                                                                 uint32_t* morton_out, uint32_t* order_out, MergeArgs A) {
    chain_wait();
    __shared__ MergeShared S;
    const MergeSpan span = merge_span(S, A.keys, A.total);
    const uint32_t g = span.first + threadIdx.x;
    const bool in = threadIdx.x < span.count;
    const SegDesc sd = *seg;
    float4 lo = make_float4(0.f, 0.f, 0.f, 0.f), hi = lo;
    if (in) {
        const uint32_t i = vals[g];
        tlas_emit_leaf(inst_box, g, A.keys[g], i, leaf_boxes, morton_out, order_out);
        tlas_emit_record(in_instances, g, i, inst_out);
        lo = inst_box[2 * i];
        hi = inst_box[2 * i + 1];
    }
    merge_block(S, A, span, sd, in, lo, hi, [leaf_boxes](uint32_t j, float4& l, float4& h) {
        l = __ldcg(leaf_boxes + 2 * j);
        h = __ldcg(leaf_boxes + 2 * j + 1);
    });
}

__global__ void tlas_record_kernel(const DevInstanceInput* in, const uint32_t* order, uint32_t n, DevInstance* inst_out) {
    chain_wait();
    uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j < n) tlas_emit_record(in, j, order[j], inst_out);
}

constexpr uint32_t kTlasLevels = 64;   // above the depth of 30-bit codes split by index

// Breadth-first relayout and 4-wide collapse of a tree too large for tlas_fused_kernel. A
// node's place is its level's start plus its rank among the level's node indices: one pass
// of the radix sort over (depth, node), stable and with the depth as its digit, gives the
// order, and the digits' offsets are the level table. Every step takes the whole chip
// (8000 instances: relayout and collapse by one block, level by level, 119 us; these kernels
// and their sort pass 27).
__global__ void __launch_bounds__(256) tlas_depth_kernel(const uint32_t* node_parent, uint32_t m, unsigned long long* keys,
                                                         uint32_t* vals, uint32_t* hist) {
    chain_wait();
    __shared__ uint32_t s_hist[1][kRadix];
    const BlockHist H{s_hist, 1};
    H.clear();
    const uint32_t q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q < m) {
        uint32_t d = 0, p = node_parent[q];
        while (p != 0xFFFFFFFFu && d + 1 < kTlasLevels) {
            ++d;
            p = node_parent[p >> 1];
        }
        keys[q] = d;
        vals[q] = q;
        H.count(d);
    }
    H.add(hist);
}

// Level table {L, start_0, ..., start_L}, and the inverse of the order.
__global__ void tlas_newidx_kernel(const uint32_t* order, uint32_t m, const uint32_t* offsets, uint32_t* newidx,
                                   uint32_t* levels) {
    chain_wait();
    const uint32_t b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b < m) newidx[order[b]] = b;
    if (b < kTlasLevels && offsets[b] < m) {
        levels[1 + b] = offsets[b];
        if (offsets[b + 1] == m) {
            levels[0] = b + 1;
            levels[2 + b] = m;
        }
    }
}

__global__ void __launch_bounds__(128) tlas_relayout_kernel(const float4* __restrict__ src,
                                                            const unsigned long long* __restrict__ depth,
                                                            const uint32_t* __restrict__ order,
                                                            const uint32_t* __restrict__ newidx, uint32_t m,
                                                            const uint32_t* __restrict__ levels, float4* dst, float4* nodes4) {
    chain_wait();
    __shared__ uint32_t s_start[kTlasLevels + 1], s_even[kTlasLevels];
    const uint32_t L = levels[0];
    if (threadIdx.x <= L) s_start[threadIdx.x] = levels[1 + threadIdx.x];
    __syncthreads();
    if (threadIdx.x < L) {
        uint32_t acc = 0;
        for (uint32_t l = 0; l < threadIdx.x; l += 2) acc += s_start[l + 1] - s_start[l];
        s_even[threadIdx.x] = acc;   // 4-wide nodes before this level
    }
    __syncthreads();
    const uint32_t b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= m) return;
    const uint32_t d = (uint32_t)depth[b];
    const float4* s = src + (size_t)order[b] * kNodeF4;
    const float4 n0 = s[0], n1 = s[1], n2 = s[2], n3 = s[3];
    const int c[2] = {__float_as_int(n3.x), __float_as_int(n3.y)};
    float4* o = dst + (size_t)b * kNodeF4;
    o[0] = n0;
    o[1] = n1;
    o[2] = n2;
    o[3] = make_float4(__int_as_float(c[0] < 0 ? c[0] : (int)newidx[c[0]]),
                       __int_as_float(c[1] < 0 ? c[1] : (int)newidx[c[1]]), 0.f, 0.f);
    if (d & 1u) return;
    Slot4 s4;
    s4.k = 0;
    for (int side = 0; side < 2; ++side) {
        if (c[side] < 0) {
            slot4_put(s4, s, side, c[side]);
            continue;
        }
        const float4* k = src + (size_t)c[side] * kNodeF4;
        const float4 k3 = k[3];
        const int g[2] = {__float_as_int(k3.x), __float_as_int(k3.y)};
        for (int t = 0; t < 2; ++t)
            slot4_put(s4, k, t, g[t] < 0 ? g[t] : (int)(s_even[d + 2] + newidx[g[t]] - s_start[d + 2]));
    }
    slot4_store(s4, nodes4 + (size_t)(s_even[d] + b - s_start[d]) * kNode4F4);
}

// Shared memory of tlas_fused_kernel for n instances: sort keys (their space holds the
// arrival flags later), the nodes' own boxes, children, parents, breadth-first ranks and
// depths. 43 bytes an instance: 172 KB at kFusedTlasMax.
struct TlasShared {
    uint32_t keys;       // power of two, at least a warp
    uint32_t nodes;
    size_t box, child, parent, leaf_parent, rank, depth, bytes;
};
__host__ __device__ inline TlasShared tlas_shared(uint32_t n) {
    TlasShared s;
    s.keys = 32;
    while (s.keys < n) s.keys <<= 1;
    s.nodes = n > 2 ? n - 1 : 1;
    s.box = (size_t)s.keys * 8;
    s.child = s.box + (size_t)s.nodes * 24;
    s.parent = s.child + (size_t)s.nodes * 4;
    s.leaf_parent = s.parent + (size_t)s.nodes * 2;
    s.rank = s.leaf_parent + (size_t)n * 2;
    s.depth = s.rank + (size_t)s.nodes * 2;
    s.bytes = s.depth + s.nodes;
    return s;
}
constexpr uint32_t kTlasOneBlock = 768;

// The whole TLAS build of up to kFusedTlasMax instances as one block: the same results as
// the kernels of the larger builds, bit for bit. Bound by latency: a few dozen steps that
// each wait for the one before, so the tree lives in shared memory and only records that
// outlive the build go to device memory. Three things keep the steps few: the sort network's
// distances below a warp run in registers (34 barriers for 4096 keys instead of 78); a
// node's place in breadth-first order is its level's start plus its rank among the level's
// node indices (the ranges of a level are disjoint and a node's index lies in its own), one
// stable counting sort by depth in place of a pass per level; and a node's box is kept
// once, as its own box, so that the refit, the relayout and the 4-wide collapse read
// shared memory. 65 instances: 36 -> 15 us; 201: 52 -> 19; 1024: 85 -> 42
// (three kernels); 4096: 264 -> 153 (the same build with the tree in device memory, a pass
// per level).
//
// kTreeOnly: the instance boxes are there, and the records are written from the order
// by a kernel after this one; both take the whole chip, where one block is bound by its own
// loads and inverses. Three kernels from kTlasOneBlock on: 500 instances 28.8 us and two
// gaps of 2.5 against 29.0, 700 36.6 and the gaps against 38.4, 1024 42.3 against 50.4.
template <bool kTreeOnly>
__global__ void __launch_bounds__(1024) tlas_fused_kernel(TlasBuildArgs A, uint32_t* dev_status) {
    chain_wait();
    extern __shared__ unsigned long long s_keys[];
    __shared__ uint32_t s_bounds[6], s_total[kTlasLevels], s_start[kTlasLevels + 1], s_even[kTlasLevels + 1];
    __shared__ uint16_t s_count[32][kTlasLevels];
    const uint32_t full = 0xFFFFFFFFu, tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t n = A.n;
    const TlasShared L = tlas_shared(n);
    const uint32_t P = L.keys, m = L.nodes;
    char* base = reinterpret_cast<char*>(s_keys);
    float* s_box = reinterpret_cast<float*>(base + L.box);   // [6][m]
    short2* s_child = reinterpret_cast<short2*>(base + L.child);
    uint16_t* s_parent = reinterpret_cast<uint16_t*>(base + L.parent);
    uint16_t* s_leaf_parent = reinterpret_cast<uint16_t*>(base + L.leaf_parent);
    uint16_t* s_rank = reinterpret_cast<uint16_t*>(base + L.rank);
    uint8_t* s_depth = reinterpret_cast<uint8_t*>(base + L.depth);
    uint32_t* s_flag = reinterpret_cast<uint32_t*>(s_keys);

    if (tid < 6) s_bounds[tid] = tid < 3 ? 0xFFFFFFFFu : 0u;
    for (uint32_t q = tid; q < m; q += nt) s_parent[q] = 0xFFFFu;
    for (uint32_t g = tid; g < n; g += nt) s_leaf_parent[g] = 0xFFFFu;
    __syncthreads();
    // instance boxes and the bounds of their centres
    for (uint32_t i = tid; i < P; i += nt) {
        V3 c;
        bool have = false;
        if (i < n) {
            if (kTreeOnly) {
                const float4 l = A.inst_box[2 * i], h = A.inst_box[2 * i + 1];
                c = V3{(l.x + h.x) * 0.5f + 0.0f, (l.y + h.y) * 0.5f + 0.0f, (l.z + h.z) * 0.5f + 0.0f};
                have = finite3(c);
            } else {
                have = tlas_instance_one(A.in, i, A.inst_box, A.shade, c);
            }
        }
        merge_bounds(have, c, s_bounds);
    }
    __syncthreads();
    // (Morton code, index) sorted: the stable order of the radix sort. Steps of 32 keys and
    // more exchange through shared memory, shorter ones between the lanes of a warp.
    {
        V3 cmin, ext;
        decode_bounds(s_bounds, cmin, ext);
        for (uint32_t i = tid; i < P; i += nt) {
            unsigned long long v = ~0ull;
            if (i < n) {
                const float4 l = A.inst_box[2 * i], h = A.inst_box[2 * i + 1];
                const unsigned long long code = morton30(V3{l.x, l.y, l.z}, V3{h.x, h.y, h.z}, cmin, ext);
                v = (code << 32) | i;
            }
#pragma unroll
            for (uint32_t k = 2; k <= 32; k <<= 1)
#pragma unroll
                for (uint32_t j = k >> 1; j > 0; j >>= 1) {
                    const unsigned long long o = __shfl_xor_sync(full, v, j);
                    v = ((i & j) == 0) == ((i & k) == 0) ? min(v, o) : max(v, o);
                }
            s_keys[i] = v;
        }
    }
    __syncthreads();
    for (uint32_t k = 64; k <= P; k <<= 1) {
        for (uint32_t j = k >> 1; j >= 32; j >>= 1) {
            for (uint32_t t = tid; t < P / 2; t += nt) {
                const uint32_t i = 2 * t - (t & (j - 1));
                const unsigned long long a = s_keys[i], b = s_keys[i + j];
                if ((a > b) == ((i & k) == 0)) { s_keys[i] = b; s_keys[i + j] = a; }
            }
            __syncthreads();
        }
        for (uint32_t i = tid; i < P; i += nt) {
            unsigned long long v = s_keys[i];
#pragma unroll
            for (uint32_t j = 16; j > 0; j >>= 1) {
                const unsigned long long o = __shfl_xor_sync(full, v, j);
                v = ((i & j) == 0) == ((i & k) == 0) ? min(v, o) : max(v, o);
            }
            s_keys[i] = v;
        }
        __syncthreads();
    }
    // leaves, and the hierarchy
    for (uint32_t j = tid; j < n; j += nt) {
        const uint32_t i = (uint32_t)s_keys[j];
        tlas_emit_leaf(A.inst_box, j, s_keys[j] >> 32, i, A.leaf_box, A.morton_out, A.order_out);
        if (!kTreeOnly) tlas_emit_record(A.in, j, i, A.inst_out);
    }
    if (n == 1) {
        if (tid == 0) {
            const float inf = __int_as_float(0x7f800000);
            const float4 lo = A.leaf_box[0], hi = A.leaf_box[1];
            A.nodes_out[0] = make_float4(lo.x, hi.x, lo.y, hi.y);
            A.nodes_out[1] = make_float4(inf, -inf, inf, -inf);
            A.nodes_out[2] = make_float4(lo.z, hi.z, inf, -inf);
            A.nodes_out[3] = make_float4(__int_as_float(~0), __int_as_float(kEmptyChild), 0.f, 0.f);
            Slot4 s4;
            s4.k = 0;
            slot4_put(s4, lo, hi, ~0);
            slot4_store(s4, A.nodes4);
            A.levels[0] = 1u;
            A.levels[1] = 0u;
            A.levels[2] = 1u;
        }
        return;
    }
    for (uint32_t i = tid; i < m; i += nt) {
        int lo, hi, gamma;
        if (!karras_range([](int j) { return (uint32_t)(s_keys[j] >> 32); }, (int)n, (int)i, lo, hi, gamma, dev_status))
            continue;
        const int c0 = lo == gamma ? ~gamma : gamma, c1 = hi == gamma + 1 ? ~(gamma + 1) : gamma + 1;
        (c0 < 0 ? s_leaf_parent : s_parent)[gamma] = (uint16_t)(i << 1);
        (c1 < 0 ? s_leaf_parent : s_parent)[gamma + 1] = (uint16_t)((i << 1) | 1u);
        s_child[i] = make_short2((short)c0, (short)c1);
    }
    __syncthreads();
    // breadth-first ranks: a stable counting sort of the node indices by depth
    for (uint32_t q = tid; q < m; q += nt) {
        uint32_t d = 0, p = s_parent[q];
        while (p != 0xFFFFu && d + 1 < kTlasLevels) {
            ++d;
            p = s_parent[p >> 1];
        }
        s_depth[q] = (uint8_t)d;
        s_flag[q] = 0u;   // the keys have been read
    }
    for (uint32_t l = tid; l < kTlasLevels; l += nt) s_total[l] = 0u;
    for (uint32_t b = 0; b < m; b += nt) {
        for (uint32_t k = tid; k < (nt >> 5) * kTlasLevels; k += nt) (&s_count[0][0])[k] = 0u;
        __syncthreads();
        const uint32_t q = b + tid, d = q < m ? s_depth[q] : kTlasLevels;
        const uint32_t peers = __match_any_sync(full, d), before = __popc(peers & ((1u << lane) - 1u));
        if (q < m && before == 0) s_count[warp][d] = (uint16_t)__popc(peers);
        __syncthreads();
        for (uint32_t l = tid; l < kTlasLevels; l += nt) {
            uint32_t run = s_total[l];
            for (uint32_t w = 0; w < nt >> 5; ++w) {
                const uint32_t t = s_count[w][l];
                s_count[w][l] = (uint16_t)run;
                run += t;
            }
            s_total[l] = run;
        }
        __syncthreads();
        if (q < m) s_rank[q] = (uint16_t)(s_count[warp][d] + before);
        __syncthreads();
    }
    if (tid == 0) {
        uint32_t at = 0, even = 0, l = 0;
        for (; l < kTlasLevels && s_total[l]; ++l) {
            s_start[l] = at;
            s_even[l] = even;
            A.levels[1 + l] = at;
            at += s_total[l];
            if (!(l & 1u)) even += s_total[l];
        }
        A.levels[0] = l;
        A.levels[1 + l] = at;
    }
    __syncthreads();
    // refit: the second child to arrive at a node completes it
    auto box_of = [&](int c, float4& lo, float4& hi) {
        if (c < 0) {
            lo = A.leaf_box[2 * ~c];
            hi = A.leaf_box[2 * ~c + 1];
        } else {
            lo = make_float4(s_box[c], s_box[m + c], s_box[2 * m + c], 0.f);
            hi = make_float4(s_box[3 * m + c], s_box[4 * m + c], s_box[5 * m + c], 0.f);
        }
    };
    for (uint32_t g = tid; g < n; g += nt) {
        float4 lo = A.leaf_box[2 * g], hi = A.leaf_box[2 * g + 1];
        uint32_t p = s_leaf_parent[g];
        while (p != 0xFFFFu) {   // at most the tree's depth
            const uint32_t i = p >> 1;
            __threadfence_block();
            if (atomicAdd(s_flag + i, 1u) != 1u) break;
            __threadfence_block();
            const short2 c = s_child[i];
            float4 lo0 = lo, hi0 = hi, lo1 = lo, hi1 = hi;
            if (p & 1u) box_of(c.x, lo0, hi0);
            else box_of(c.y, lo1, hi1);
            lo = make_float4(fmin_(lo0.x, lo1.x), fmin_(lo0.y, lo1.y), fmin_(lo0.z, lo1.z), 0.f);
            hi = make_float4(fmax_(hi0.x, hi1.x), fmax_(hi0.y, hi1.y), fmax_(hi0.z, hi1.z), 0.f);
            s_box[i] = lo.x; s_box[m + i] = lo.y; s_box[2 * m + i] = lo.z;
            s_box[3 * m + i] = hi.x; s_box[4 * m + i] = hi.y; s_box[5 * m + i] = hi.z;
            float4* node = A.nodes_out + (size_t)(s_start[s_depth[i]] + s_rank[i]) * kNodeF4;
            const int c0 = c.x < 0 ? c.x : (int)(s_start[s_depth[c.x]] + s_rank[c.x]);
            const int c1 = c.y < 0 ? c.y : (int)(s_start[s_depth[c.y]] + s_rank[c.y]);
            node[0] = make_float4(lo0.x, hi0.x, lo0.y, hi0.y);
            node[1] = make_float4(lo1.x, hi1.x, lo1.y, hi1.y);
            node[2] = make_float4(lo0.z, hi0.z, lo1.z, hi1.z);
            node[3] = make_float4(__int_as_float(c0), __int_as_float(c1), 0.f, 0.f);
            p = s_parent[i];
        }
    }
    __syncthreads();
    // 4-wide nodes: the even levels, a slot per grandchild (or child, where that is a leaf)
    for (uint32_t i = tid; i < m; i += nt) {
        const uint32_t d = s_depth[i];
        if (d & 1u) continue;
        Slot4 s4;
        s4.k = 0;
        auto put = [&](int c) {
            float4 lo, hi;
            box_of(c, lo, hi);
            slot4_put(s4, lo, hi, c < 0 ? c : (int)(s_even[s_depth[c]] + s_rank[c]));
        };
        const short2 c = s_child[i];
        if (c.x < 0) put(c.x);
        else { const short2 k = s_child[c.x]; put(k.x); put(k.y); }
        if (c.y < 0) put(c.y);
        else { const short2 k = s_child[c.y]; put(k.x); put(k.y); }
        slot4_store(s4, A.nodes4 + (size_t)(s_even[d] + s_rank[i]) * kNode4F4);
    }
}

// ---------------------------------------------------------------- host drivers
static inline uint32_t cdiv(uint64_t a, uint64_t b) { return (uint32_t)((a + b - 1) / b); }

static int passes_for(int nseg) {
    int bits = 30;
    int sb = 0;
    while ((1 << sb) < nseg) ++sb;
    return (bits + sb + 7) / 8;
}

struct SortBuffers {
    unsigned long long* keys[2];
    uint32_t* vals[2];
    uint32_t* hist;       // passes * 256
    uint32_t* offsets;    // passes * 256
    uint32_t* tile_status;  // passes * tiles * 256
    uint32_t* tile_counter; // passes
    uint32_t tiles;
};

static size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

// Bytes of scratch for a sort of n keys with `passes` passes.
static size_t sort_scratch_bytes(uint32_t n, int passes) {
    uint32_t tiles = std::max(1u, cdiv(n, kSortTile));
    return 2 * align256((size_t)n * 8) + 2 * align256((size_t)n * 4) +
           2 * align256((size_t)passes * 256 * 4) +
           align256((size_t)passes * tiles * 256 * 4) + align256((size_t)passes * 4);
}

static char* carve_sort(char* p, uint32_t n, int passes, SortBuffers& sb) {
    sb.tiles = std::max(1u, cdiv(n, kSortTile));
    sb.keys[0] = (unsigned long long*)p; p += align256((size_t)n * 8);
    sb.keys[1] = (unsigned long long*)p; p += align256((size_t)n * 8);
    sb.vals[0] = (uint32_t*)p; p += align256((size_t)n * 4);
    sb.vals[1] = (uint32_t*)p; p += align256((size_t)n * 4);
    sb.hist = (uint32_t*)p; p += align256((size_t)passes * 256 * 4);
    sb.offsets = (uint32_t*)p; p += align256((size_t)passes * 256 * 4);
    sb.tile_status = (uint32_t*)p; p += align256((size_t)passes * sb.tiles * 256 * 4);
    sb.tile_counter = (uint32_t*)p; p += align256((size_t)passes * 4);
    return p;
}

// Clears what a sort counts in (its buffers from hist to tile_counter are consecutive),
// before the kernel that makes the keys and counts their digits.
static luz_status clear_sort(luz_ctx* ctx, SortBuffers& sb, int passes) {
    LUZ_CUDA(ctx, cudaMemsetAsync(sb.hist, 0, (char*)(sb.tile_counter + passes) - (char*)sb.hist, ctx->stream));
    return LUZ_OK;
}

// Sorts sb.keys[0]/vals[0], whose digits are counted; returns the index (0/1) of the buffer
// holding the result. n: at most what sb was carved for.
static luz_status run_sort(luz_ctx* ctx, SortBuffers& sb, uint32_t n, int passes, int& result) {
    const uint32_t tiles = cdiv(n, kSortTile);
    int cur = 0;
    for (int p = 0; p < passes; ++p) {
        chain(onesweep_pass_kernel, tiles, kSortThreads, 0, ctx->stream, sb.keys[cur], sb.vals[cur], sb.keys[cur ^ 1],
              sb.vals[cur ^ 1], n, 8 * p, sb.hist + p * 256, sb.offsets + p * 256,
              sb.tile_status + (size_t)p * sb.tiles * 256, sb.tile_counter + p, ctx->d_status);
        LUZ_LAUNCHED(ctx, "onesweep_pass_kernel");
        cur ^= 1;
    }
    result = cur;
    return LUZ_OK;
}

luz_status build_blas_batch(luz_ctx* ctx, uint32_t count, const luz_blas_desc* descs,
                            luz_blas** out) {
    // Validate on the host (indices in range, sizes) before any device work.
    std::vector<SegDesc> segs(count);
    std::vector<uint32_t> prim_off(count), node_off(count);
    uint64_t total_prims = 0, total_nodes = 0, total_verts = 0;
    bool has_empty = false;
    for (uint32_t s = 0; s < count; ++s) {
        const luz_blas_desc& d = descs[s];
        if (d.index_count % 3 != 0)
            return set_error(ctx, LUZ_ERR_INVALID, "index_count is not a multiple of 3");
        if (d.vertex_stride < 12 || (d.vertex_count > 0 && !d.vertices) ||
            (d.index_count > 0 && !d.indices))
            return set_error(ctx, LUZ_ERR_INVALID, "bad vertex/index buffer description");
        for (uint32_t k = 0; k < d.index_count; ++k)
            if (d.indices[k] >= d.vertex_count)
                return set_error(ctx, LUZ_ERR_INVALID, "index out of range of the vertex buffer");
        uint32_t n = d.index_count / 3;
        has_empty = has_empty || n == 0;
        prim_off[s] = (uint32_t)total_prims;
        node_off[s] = (uint32_t)total_nodes;
        total_prims += n;
        total_nodes += std::max(n, 2u) - 1;
        total_verts += d.vertex_count;
    }
    if (total_prims >= (1ull << 30) - 1)
        return set_error(ctx, LUZ_ERR_LIMIT, "more than 2^30 triangles in one batch");
    cudaStream_t st = ctx->stream;
    // Persistent arena: per BLAS nodes | 4-wide nodes | tris | morton | order | vertices | indices.
    std::vector<size_t> off_nodes(count), off_tris(count), off_mort(count), off_ord(count),
        off_vtx(count), off_idx(count), off_nodes4(count);
    size_t arena_bytes = 0;
    for (uint32_t s = 0; s < count; ++s) {
        uint32_t n = descs[s].index_count / 3;
        uint32_t m = std::max(n, 2u) - 1;
        off_nodes[s] = arena_bytes; arena_bytes += align256((size_t)m * 64);
        off_nodes4[s] = arena_bytes; arena_bytes += align256((size_t)m * 128);
        off_tris[s] = arena_bytes; arena_bytes += align256((size_t)std::max(n, 1u) * 48);
        off_mort[s] = arena_bytes; arena_bytes += align256((size_t)std::max(n, 1u) * 4);
        off_ord[s] = arena_bytes; arena_bytes += align256((size_t)std::max(n, 1u) * 4);
        off_vtx[s] = arena_bytes; arena_bytes += align256((size_t)std::max(descs[s].vertex_count, 1u) * sizeof(luz_vertex));
        off_idx[s] = arena_bytes; arena_bytes += align256((size_t)std::max(descs[s].index_count, 3u) * 4);
    }
    Arena* arena = new Arena();
    cudaError_t e = cudaMalloc(&arena->base, arena_bytes);
    if (e != cudaSuccess) { delete arena; return cuda_error(ctx, e, "cudaMalloc(BLAS arena)"); }
    char* ab = (char*)arena->base;
    // Upload vertices (repacked to 48-B luz_vertex when the stride differs) and indices.
    for (uint32_t s = 0; s < count; ++s) {
        const luz_blas_desc& d = descs[s];
        luz_vertex* dv = (luz_vertex*)(ab + off_vtx[s]);
        if (d.vertex_stride == sizeof(luz_vertex)) {
            if (d.vertex_count)
                LUZ_CUDA(ctx, cudaMemcpyAsync(dv, d.vertices, (size_t)d.vertex_count * 48,
                                              cudaMemcpyHostToDevice, st));
        } else {
            std::vector<luz_vertex> tmp(d.vertex_count);
            for (uint32_t v = 0; v < d.vertex_count; ++v) {
                memset(&tmp[v], 0, sizeof(luz_vertex));
                memcpy(tmp[v].position, (const char*)d.vertices + (size_t)v * d.vertex_stride, 12);
                if (d.vertex_stride >= 24)
                    memcpy(tmp[v].normal, (const char*)d.vertices + (size_t)v * d.vertex_stride + 12, 12);
            }
            if (d.vertex_count)
                LUZ_CUDA(ctx, cudaMemcpy(dv, tmp.data(), (size_t)d.vertex_count * 48,
                                         cudaMemcpyHostToDevice));
        }
        if (d.index_count)
            LUZ_CUDA(ctx, cudaMemcpyAsync(ab + off_idx[s], d.indices, (size_t)d.index_count * 4,
                                          cudaMemcpyHostToDevice, st));
        SegDesc& sd = segs[s];
        sd.prim_off = prim_off[s];
        sd.prim_count = d.index_count / 3;
        sd.node_off = node_off[s];
        sd.pad = 0;
        sd.vertices = dv;
        sd.indices = (const uint32_t*)(ab + off_idx[s]);
        sd.nodes = (float4*)(ab + off_nodes[s]);
        sd.tris = (float4*)(ab + off_tris[s]);
        sd.nodes4 = (float4*)(ab + off_nodes4[s]);
        sd.morton = (uint32_t*)(ab + off_mort[s]);
        sd.order = (uint32_t*)(ab + off_ord[s]);
    }
    // Scratch: segs | prim_off | node_off | bounds | sort | parents | merges' flags and far
    // ends | 4-wide collapse indices.
    uint32_t N = (uint32_t)total_prims, M = (uint32_t)total_nodes;
    int passes = passes_for((int)count);
    size_t need = align256(count * sizeof(SegDesc)) + 2 * align256(count * 4) +
                  align256(count * 24) + sort_scratch_bytes(std::max(N, 1u), passes) +
                  align256((size_t)M * 4) + align256((size_t)std::max(N, 1u) * 4) + 2 * align256((size_t)std::max(N, 1u) * 8) +
                  2 * align256((size_t)M * 4) +
                  align256((size_t)(M / 1024 + 1) * 4);
    luz_status stt = ensure_scratch(ctx, need);
    if (stt != LUZ_OK) { cudaFree(arena->base); delete arena; return stt; }
    char* p = (char*)ctx->d_scratch;
    SegDesc* d_segs = (SegDesc*)p; p += align256(count * sizeof(SegDesc));
    uint32_t* d_prim_off = (uint32_t*)p; p += align256(count * 4);
    uint32_t* d_node_off = (uint32_t*)p; p += align256(count * 4);
    uint32_t* d_bounds = (uint32_t*)p; p += align256(count * 24);
    SortBuffers sb;
    p = carve_sort(p, std::max(N, 1u), passes, sb);
    uint32_t* d_node_parent = (uint32_t*)p; p += align256((size_t)M * 4);
    uint32_t* d_flags = (uint32_t*)p; p += align256((size_t)std::max(N, 1u) * 4);
    uint2* d_ends[2];
    for (uint2*& e : d_ends) { e = (uint2*)p; p += align256((size_t)std::max(N, 1u) * 8); }
    uint32_t* d_even = (uint32_t*)p; p += align256((size_t)M * 4);
    uint32_t* d_idx4 = (uint32_t*)p; p += align256((size_t)M * 4);
    uint32_t* d_sums = (uint32_t*)p; p += align256((size_t)(M / 1024 + 1) * 4);

    LUZ_CUDA(ctx, cudaMemcpyAsync(d_segs, segs.data(), count * sizeof(SegDesc), cudaMemcpyHostToDevice, st));
    LUZ_CUDA(ctx, cudaMemcpyAsync(d_prim_off, prim_off.data(), count * 4, cudaMemcpyHostToDevice, st));
    LUZ_CUDA(ctx, cudaMemcpyAsync(d_node_off, node_off.data(), count * 4, cudaMemcpyHostToDevice, st));
    std::vector<uint32_t> binit(count * 6);
    for (uint32_t s = 0; s < count; ++s)
        for (int k = 0; k < 6; ++k) binit[s * 6 + k] = k < 3 ? 0xFFFFFFFFu : 0u;
    LUZ_CUDA(ctx, cudaMemcpyAsync(d_bounds, binit.data(), count * 24, cudaMemcpyHostToDevice, st));
    LUZ_CUDA(ctx, cudaEventRecord(ctx->build_ev[0], st));   // device pipeline starts here
    LUZ_CUDA(ctx, cudaMemsetAsync(d_flags, 0, (size_t)std::max(N, 1u) * 4, st));
    if (N > 0) {
        if ((stt = clear_sort(ctx, sb, passes)) != LUZ_OK) { cudaFree(arena->base); delete arena; return stt; }
        const uint32_t rows = bounds_rows(N);
        chain(blas_bounds_kernel, cdiv(N, 256 * rows), 256, 0, st, d_segs, d_prim_off, count, N, rows, d_bounds);
        LUZ_LAUNCHED(ctx, "blas_bounds_kernel");
        chain(blas_morton_kernel, morton_blocks(N), 256, 0, st, d_segs, d_prim_off, count, N, d_bounds, sb.keys[0],
              sb.vals[0], passes, sb.hist);
        LUZ_LAUNCHED(ctx, "blas_morton_kernel");
        int res = 0;
        stt = run_sort(ctx, sb, N, passes, res);
        if (stt != LUZ_OK) { cudaFree(arena->base); delete arena; return stt; }
        const MergeArgs A{sb.keys[res], d_node_parent, {d_ends[0], d_ends[1]}, d_flags, ctx->d_status, N};
        chain(blas_tree_kernel, merge_blocks(N), kMergeLeaves, 0, st, d_segs, d_prim_off, count, sb.vals[res], A);
        LUZ_LAUNCHED(ctx, "blas_tree_kernel");
    }
    // Every segment has at least one node, also one without a primitive.
    if (has_empty) {
        chain(empty_segments_kernel, cdiv(count, 128), 128, 0, st, d_segs, count, d_node_parent);
        LUZ_LAUNCHED(ctx, "empty_segments_kernel");
    }
    if (N > 0) {
        chain(blas_radius_kernel, cdiv(N, 256), 256, 0, st, d_segs, d_prim_off, count, N);
        LUZ_LAUNCHED(ctx, "blas_radius_kernel");
    }
    // 4-wide collapse of every segment's tree (the traversal structure of the
    // shadow/AO rays; the binary tree stays the parity-checked structure).
    {
        uint32_t chunks = cdiv(M, 1024);
        chain(even_depth_kernel, cdiv(M, 256), 256, 0, st, d_segs, d_node_off, count, M, d_node_parent, d_even);
        LUZ_LAUNCHED(ctx, "even_depth_kernel");
        chain(chunk_sum_kernel, chunks, 256, 0, st, d_even, M, d_sums);
        LUZ_LAUNCHED(ctx, "chunk_sum_kernel");
        chain(chunk_scan_kernel, 1, 1024, 0, st, d_sums, chunks);
        LUZ_LAUNCHED(ctx, "chunk_scan_kernel");
        chain(chunk_apply_kernel, chunks, 256, 0, st, d_even, M, d_sums, d_idx4);
        LUZ_LAUNCHED(ctx, "chunk_apply_kernel");
        chain(bvh4_emit_kernel, cdiv(M, 256), 256, 0, st, d_segs, d_node_off, count, M, d_even, d_idx4);
        LUZ_LAUNCHED(ctx, "bvh4_emit_kernel");
    }
    LUZ_CUDA(ctx, cudaEventRecord(ctx->build_ev[1], st));
    ctx->build_timed = true;
    LUZ_CUDA(ctx, cudaStreamSynchronize(st));
    uint32_t bits = 0;
    LUZ_CUDA(ctx, cudaMemcpy(&bits, ctx->d_status, 4, cudaMemcpyDeviceToHost));
    if (bits) {
        cudaFree(arena->base);
        delete arena;
        return set_error(ctx, LUZ_ERR_DEVICE, "BLAS build kernel raised the device status word");
    }
    for (uint32_t s = 0; s < count; ++s) {
        luz_blas* b = new luz_blas();
        b->ctx = ctx;
        b->arena = arena;
        arena->refs++;
        b->nodes = segs[s].nodes;
        b->nodes4 = segs[s].nodes4;
        b->memory.nodes = off_nodes4[s] - off_nodes[s];
        b->memory.wide_nodes = off_tris[s] - off_nodes4[s];
        b->memory.leaves = off_mort[s] - off_tris[s];
        b->memory.other = (s + 1 < count ? off_nodes[s + 1] : arena_bytes) - off_mort[s];
        b->tris = segs[s].tris;
        b->morton = (uint32_t*)(ab + off_mort[s]);
        b->order = (uint32_t*)(ab + off_ord[s]);
        b->vertices = (luz_vertex*)(ab + off_vtx[s]);
        b->indices = (uint32_t*)(ab + off_idx[s]);
        b->prims = segs[s].prim_count;
        b->vertex_count = descs[s].vertex_count;
        out[s] = b;
    }
    return LUZ_OK;
}

// TLAS scratch layout (allocated once per luz_tlas for max_instances).
static size_t tlas_tmp_bytes(uint32_t cap) {
    uint32_t m = std::max(cap, 2u) - 1;
    return align256((size_t)cap * 32) + align256(24) + sort_scratch_bytes(std::max(cap, 1u), 4) +
           align256((size_t)cap * 32) + align256((size_t)m * 4) + align256((size_t)cap * 4) +
           align256((size_t)m * 4) + align256((size_t)m * 64) + 2 * align256((size_t)m * 4) +
           align256(sizeof(SegDesc)) + 2 * align256((size_t)cap * 8);
}

luz_status launch_tlas_build(luz_ctx* ctx, luz_tlas* t);
luz_status launch_tlas_kernels(luz_ctx* ctx, luz_tlas* t);

luz_status tlas_alloc(luz_ctx* ctx, luz_tlas* t) {
    uint32_t cap = std::max(t->max_instances, 1u);
    uint32_t m = std::max(cap, 2u) - 1;
    LUZ_CUDA(ctx, cudaMalloc(&t->nodes, (size_t)m * 64));
    LUZ_CUDA(ctx, cudaMalloc(&t->nodes4, (size_t)m * 128));
    LUZ_CUDA(ctx, cudaMalloc(&t->levels, 66 * 4));
    LUZ_CUDA(ctx, cudaMalloc(&t->instances, (size_t)cap * sizeof(DevInstance)));
    LUZ_CUDA(ctx, cudaMalloc(&t->shade, (size_t)cap * sizeof(DevShadeInstance)));
    LUZ_CUDA(ctx, cudaMalloc(&t->d_input, (size_t)cap * sizeof(DevInstanceInput)));
    LUZ_CUDA(ctx, cudaMallocHost(&t->h_input, (size_t)cap * sizeof(DevInstanceInput)));
    LUZ_CUDA(ctx, cudaMalloc(&t->morton, (size_t)cap * 4));
    LUZ_CUDA(ctx, cudaMalloc(&t->order, (size_t)cap * 4));
    t->tmp_bytes = tlas_tmp_bytes(cap);
    LUZ_CUDA(ctx, cudaMalloc(&t->tmp, t->tmp_bytes));
    return LUZ_OK;
}

// Host part of a TLAS build: validates the instances and packs them into the pinned
// staging buffer (the buffer must not be in use by an earlier build's copy).
luz_status pack_tlas_input(luz_ctx* ctx, luz_tlas* t, const luz_instance* inst, uint32_t n) {
    if (n > t->max_instances)
        return set_error(ctx, LUZ_ERR_LIMIT, "instance count exceeds the TLAS max_instances");
    for (uint32_t i = 0; i < n; ++i) {
        const luz_blas* b = inst[i].blas;
        if (!b) return set_error(ctx, LUZ_ERR_INVALID, "instance without a BLAS");
        DevInstanceInput& d = t->h_input[i];
        memcpy(d.o2w, inst[i].transform, 48);
        d.nodes = b->nodes;
        d.tris = b->tris;
        d.vertices = b->vertices;
        d.indices = b->indices;
        d.custom_index = inst[i].custom_index;
        d.mask = inst[i].mask;
        d.blas_prims = b->prims;
        d.pad = 0;
        d.nodes4 = b->nodes4;
    }
    t->count = n;
    t->node_count = std::max(n, 2u) - 1;
    return LUZ_OK;
}

luz_status build_tlas(luz_ctx* ctx, luz_tlas* t, const luz_instance* inst, uint32_t n) {
    luz_status s = pack_tlas_input(ctx, t, inst, n);
    if (s != LUZ_OK) return s;
    return launch_tlas_build(ctx, t);
}

// The TLAS's scratch buffer (t->tmp) carved for a build of up to max_instances.
struct TlasScratch {
    TlasBuildArgs a;
    uint32_t* bounds;
    SortBuffers sb;
    SegDesc* d_seg;
    uint2* ends[2];
};

static TlasScratch carve_tlas(luz_tlas* t) {
    TlasScratch s;
    uint32_t cap = std::max(t->max_instances, 1u);
    uint32_t mcap = std::max(cap, 2u) - 1;
    char* p = (char*)t->tmp;
    TlasBuildArgs& a = s.a;
    a.in = t->d_input;
    a.n = t->count;
    a.shade = t->shade;
    a.inst_box = (float4*)p; p += align256((size_t)cap * 32);
    s.bounds = (uint32_t*)p; p += align256(24);
    p = carve_sort(p, cap, 4, s.sb);
    a.keys = s.sb.keys[0];
    a.vals = s.sb.vals[0];
    a.leaf_box = (float4*)p; p += align256((size_t)cap * 32);
    a.node_parent = (uint32_t*)p; p += align256((size_t)mcap * 4);
    a.leaf_parent = (uint32_t*)p; p += align256((size_t)cap * 4);
    a.flags = (uint32_t*)p; p += align256((size_t)mcap * 4);
    a.karras_nodes = (float4*)p; p += align256((size_t)mcap * 64);
    a.queue = (uint32_t*)p; p += align256((size_t)mcap * 4);
    a.newidx = (uint32_t*)p; p += align256((size_t)mcap * 4);
    s.d_seg = (SegDesc*)p; p += align256(sizeof(SegDesc));
    for (uint2*& e : s.ends) { e = (uint2*)p; p += align256((size_t)cap * 8); }
    a.inst_out = t->instances;
    a.morton_out = t->morton;
    a.order_out = t->order;
    a.nodes_out = t->nodes;
    a.levels = t->levels;
    a.nodes4 = t->nodes4;
    return s;
}

TlasBuildArgs tlas_build_args(luz_tlas* t) { return carve_tlas(t).a; }
const float4* tlas_leaf_boxes(const luz_tlas* t) { return carve_tlas(const_cast<luz_tlas*>(t)).a.leaf_box; }

// Device part of a TLAS build from the packed staging buffer: one host-to-device copy
// from pinned memory and the LBVH kernels; no host synchronisation (graph-capturable).
luz_status launch_tlas_build(luz_ctx* ctx, luz_tlas* t) {
    if (t->count)
        LUZ_CUDA(ctx, cudaMemcpyAsync(t->d_input, t->h_input, (size_t)t->count * sizeof(DevInstanceInput),
                                      cudaMemcpyHostToDevice, ctx->stream));
    return launch_tlas_kernels(ctx, t);
}

// The kernels alone, over the instances on the device.
luz_status launch_tlas_kernels(luz_ctx* ctx, luz_tlas* t) {
    cudaStream_t st = ctx->stream;
    const uint32_t n = t->count;
    if (n == 0) return LUZ_OK;
    const uint32_t m = std::max(n, 2u) - 1;
    TlasScratch ts = carve_tlas(t);
    const TlasBuildArgs& A = ts.a;
    float4* inst_box = A.inst_box;
    uint32_t* bounds = ts.bounds;
    SortBuffers& sb = ts.sb;
    float4* leaf_box = A.leaf_box;
    uint32_t* node_parent = A.node_parent;
    uint32_t* flags = A.flags;
    float4* karras_nodes = A.karras_nodes;
    uint32_t* newidx = A.newidx;
    SegDesc* d_seg = ts.d_seg;

    if (n <= kFusedTlasMax) {
        static DeviceSetup setup;   // the kernel's shared-memory limit
        luz_status s = device_setup(setup, setup_generation(), 1, [&]() -> luz_status {
            for (const void* fn : {(const void*)tlas_fused_kernel<false>, (const void*)tlas_fused_kernel<true>})
                LUZ_CUDA(ctx, cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                   (int)tlas_shared(kFusedTlasMax).bytes));
            return LUZ_OK;
        });
        if (s != LUZ_OK) return s;
        const uint32_t threads = std::min(std::max((n + 31u) & ~31u, 64u), 1024u);
        prof_begin(ctx, LUZ_KERNEL_TLAS_BUILD);
        if (n <= kTlasOneBlock) {
            chain(tlas_fused_kernel<false>, 1, threads, tlas_shared(n).bytes, st, A, ctx->d_status);
            LUZ_LAUNCHED(ctx, "tlas_fused_kernel");
        } else {
            chain(tlas_instance_kernel, cdiv(n, 64), 64, 0, st, A.in, n, A.inst_box, A.shade, nullptr);
            LUZ_LAUNCHED(ctx, "tlas_instance_kernel");
            chain(tlas_fused_kernel<true>, 1, threads, tlas_shared(n).bytes, st, A, ctx->d_status);
            LUZ_LAUNCHED(ctx, "tlas_fused_kernel<tree>");
            chain(tlas_record_kernel, cdiv(n, 64), 64, 0, st, A.in, A.order_out, n, A.inst_out);
            LUZ_LAUNCHED(ctx, "tlas_record_kernel");
        }
        prof_end(ctx);
        return LUZ_OK;
    }
    SegDesc sd{};
    sd.prim_off = 0;
    sd.prim_count = n;
    sd.node_off = 0;
    sd.nodes = karras_nodes;
    // Bounds initialiser and segment descriptor are written by a kernel from its
    // parameters: a copy from host memory would, inside a CUDA graph, re-read a
    // host address that no longer holds them.
    chain(tlas_setup_kernel, 1, 32, 0, st, bounds, d_seg, sd);
    LUZ_LAUNCHED(ctx, "tlas_setup_kernel");
    LUZ_CUDA(ctx, cudaMemsetAsync(flags, 0, (size_t)m * 4, st));
    luz_status s = clear_sort(ctx, sb, 4);
    if (s != LUZ_OK) return s;
    chain(tlas_instance_kernel, cdiv(n, 128), 128, 0, st, t->d_input, n, inst_box, t->shade, bounds);
    LUZ_LAUNCHED(ctx, "tlas_instance_kernel");
    chain(tlas_morton_kernel, cdiv(n, 256), 256, 0, st, inst_box, n, bounds, sb.keys[0], sb.vals[0], 4, sb.hist);
    LUZ_LAUNCHED(ctx, "tlas_morton_kernel");
    int res = 0;
    if ((s = run_sort(ctx, sb, n, 4, res)) != LUZ_OK) return s;
    const MergeArgs merge{sb.keys[res], node_parent, {ts.ends[0], ts.ends[1]}, flags, ctx->d_status, n};
    chain(tlas_tree_kernel, merge_blocks(n), kMergeLeaves, 0, st, d_seg, t->d_input, inst_box, sb.vals[res],
          t->instances, leaf_box, t->morton, t->order, merge);
    LUZ_LAUNCHED(ctx, "tlas_tree_kernel");
    if ((s = clear_sort(ctx, sb, 1)) != LUZ_OK) return s;
    chain(tlas_depth_kernel, cdiv(m, 256), 256, 0, st, node_parent, m, sb.keys[0], sb.vals[0], sb.hist);
    LUZ_LAUNCHED(ctx, "tlas_depth_kernel");
    if ((s = run_sort(ctx, sb, m, 1, res)) != LUZ_OK) return s;
    chain(tlas_newidx_kernel, cdiv(m, 128), 128, 0, st, sb.vals[res], m, sb.offsets, newidx, t->levels);
    LUZ_LAUNCHED(ctx, "tlas_newidx_kernel");
    chain(tlas_relayout_kernel, cdiv(m, 128), 128, 0, st, karras_nodes, sb.keys[res], sb.vals[res], newidx, m, t->levels,
                                                       t->nodes, t->nodes4);
    LUZ_LAUNCHED(ctx, "tlas_relayout_kernel");
    return LUZ_OK;
}

}  // namespace luz
