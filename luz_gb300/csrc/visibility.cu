// visibility.cu — the persistent wavefront kernel that traces every shadow and AO ray
// of a frame (light.frag:86-135) and writes the hit/miss bit planes; and its batched
// form, one launch over the rays of many scenes.
//
// A frame's rays are first resolved in groups: shafts.cuh culls whole (light, patch)
// groups of shadow rays, aocull.cuh AO rays above their patch's horizon. What is left is
// generated on full warps, tested against the boxes its group's list starts at, and
// written as compact records. The traversal kernel keeps one ray per lane as an explicit
// state; after every few steps a warp counts its idle lanes with a ballot and, when enough
// are idle, one lane takes that many records with a single atomic and the idle lanes pick
// theirs by rank. 1080p two-level frame (64 x 81,920 triangles, 1024 instances, 41 lights,
// 16 AO rays; 18.4 M rays to trace): ray generation and lists 0.59 -> 0.83 ms, traversal
// 2.27 -> 0.97 ms (BLAS node visits 121 M -> 40 M, TLAS 7.8 M -> 1.6 M) against tracing
// every ray from the leaves its 32 neighbours' capsule reaches; 4K, 4096 instances, 145
// lights, 64 AO rays: 18.5 + 94.2 ms -> 27 + 44 ms.
//
// Traversal runs over 4-wide nodes (the even-depth collapse of the binary LBVH):
// one step tests four child boxes, with the near and far planes picked per ray by
// the direction's signs. Nodes and triangles come through 16-B vector loads (the
// TLAS top can also be staged in shared memory); the stack is warp-interleaved in
// shared memory (entry k of lane l at [k][l]) with a local-memory tail for rare deep
// paths. Only the state a node step needs stays in registers; the rest of a ray
// (world origin and direction, output bit, watertight shear) sits in shared memory,
// which keeps the kernel at 64 registers and 4 CTAs per SM without spills.
#include <algorithm>
#include <cstring>
#include <type_traits>

#include "aocull.cuh"
#include "shafts.cuh"
#include "vis_trace.cuh"

namespace luz {

// Ray generation of the shadow rays: warps take up to kRaygenTake consecutive active groups
// (shafts.cuh) at a time, fewer when there are not enough for two rounds of the grid; lane
// = pixel of the group's patch, over the samples of its virtual light. Separated from
// traversal so the long arithmetic of light.frag's sampling and the tests against the
// group's list, the same leaves for all lanes, run on full warps. A ray that enters none
// of the leaves is unoccluded and leaves no record. Bound by latency, hence four blocks per
// SM, and the list of a group held by the lanes: 0.25 ms for the 5.2 M samples that the
// shafts of a 1080p frame leave (three blocks 0.28, five 0.26; lists read per sample and
// leaf 0.29), 4K 13.0 -> 10.95 ms; the traversal that found the same on partly filled warps
// took 0.28 ms longer.
constexpr uint32_t kRaygenTake = 4;
// kLong: with lists of more than kListShort leaves.
template <bool kLong>
__global__ void __launch_bounds__(256, 4) shadow_raygen_kernel(SceneVis S, VisCommon C, Entries E,
                                                               const uint4* __restrict__ active,
                                                               const uint32_t* __restrict__ active_count,
                                                               uint32_t* tickets, RayOut R) {
    chain_wait();
    __shared__ float s_ray[8][kLong ? kStageWords : kStageWords - 1][kStageRays];
    const uint32_t full = 0xFFFFFFFFu;
    const uint32_t lit = *S.lit_count, lane = threadIdx.x & 31, n = *active_count;
    RayStage stage{s_ray[threadIdx.x >> 5], 0u};
    const uint32_t take = max(min(n / (2u * gridDim.x * (blockDim.x >> 5)), kRaygenTake), 1u);
    for (;;) {
        uint32_t g0 = 0;
        if (lane == 0) g0 = atomicAdd(tickets, take);
        g0 = __shfl_sync(full, g0, 0);
        if (g0 >= n) break;
        for (uint32_t g = g0; g < min(g0 + take, n); ++g) {
            const uint4 a = __ldg(active + g);
            const uint32_t first = a.y & 0xFFFFu, samples = a.y >> 16, j = a.z * kPatch + lane;
            const uint32_t* list = E.lists + (size_t)a.x * kEntryWords;
            const uint32_t cnt = __ldg(list);
            // lane k: leaf k of the list and its cut
            const bool has = cnt != kListAll && lane < cnt;
            const bool longer = kLong && cnt != kListAll && cnt > kListShort;
            // (of a long list the leaves from the 33rd on in place of the cuts)
            const uint32_t my_leaf = has ? __ldg(list + 1 + lane) : 0u;
            const uint32_t my_cut = (longer ? lane + 32 < cnt : has) ? __ldg(list + kEntryCuts + (longer ? 1u : 0u) + lane) : 0u;
            for (uint32_t s = 0; s < samples; ++s) {
                V3 wo{0.f, 0.f, 0.f}, wd{0.f, 0.f, 1.f};
                float tmin = 0.f, tmax = 0.f;
                uint32_t* out;
                bool record_hit = true;
                uint32_t pix = 0;
                const bool ok = j < lit && gen_ray(S, C, first + s, j, wo, wd, tmin, tmax, out, record_hit, pix);
                uint32_t mask = cnt == kListAll ? kFromRoot : 0u, more = 0u;
                if (cnt != kListAll && __any_sync(full, ok)) {
                    LaneRay r;
                    r.tmin = tmin;
                    r.tmax = tmax;
                    r.idir = safe_inv(wd);
                    set_origin(r, wo);
                    near_planes(r);
                    if (longer) {   // leaf boxes alone
                        more = kLongList;
                        for (uint32_t k = 0; k < cnt; ++k) {
                            const uint32_t leaf = __shfl_sync(full, k < 32 ? my_leaf : my_cut, k & 31);
                            if (ok && leaf_overlaps(r, S.leaf_box, leaf)) (k < 31 ? mask : more) |= 1u << (k < 31 ? k : k - 31);
                        }
                    }
                    for (uint32_t k = 0; k < cnt && !longer; ++k) {
                        const uint32_t leaf = __shfl_sync(full, my_leaf, k), cut = __shfl_sync(full, my_cut, k);
                        if (ok && leaf_overlaps(r, S.leaf_box, leaf) &&
                            (cnt > E.cut_cap || leaf_enters(S.instances + leaf, cut ? E.cuts + (size_t)(cut - 1u) * kNode4F4 : nullptr, wo, wd,
                                        tmin, tmax)))
                            mask |= 1u << k;
                    }
                }
                stage_rays<kLong>(stage, R, lane, ok && (mask | (more & ~kLongList)) != 0u, wo, tmax, wd, pix, a.x, first + s, mask, more);
            }
        }
    }
    if (stage.n) stage_flush<kLong>(stage, R, lane);
}

// The rays of a frame that have something to trace (the counting trace's figure: shafts
// and horizons resolve most of them without a record).
__global__ void __launch_bounds__(256) count_rays_kernel(SceneVis S, VisCommon C, unsigned long long* stats) {
    chain_wait();
    const uint32_t lit = *S.lit_count;
    const unsigned long long total = (unsigned long long)lit * (S.shadow_slots + S.ao_samples);
    uint32_t n = 0;
    for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; i < total;
         i += (unsigned long long)gridDim.x * blockDim.x) {
        V3 wo, wd;
        float tmin, tmax;
        uint32_t* out;
        bool record_hit;
        uint32_t pix;
        const uint32_t slot = (uint32_t)(i / lit);
        n += gen_ray(S, C, slot, (uint32_t)(i - (unsigned long long)slot * lit), wo, wd, tmin, tmax, out, record_hit, pix);
    }
    n = __reduce_add_sync(0xFFFFFFFFu, n);
    if ((threadIdx.x & 31) == 0) atomicAdd(stats, (unsigned long long)n);
}

// Traversal of one chunk's ray records (one scene; the TLAS top may be staged in shared
// memory). Shared memory: staged TLAS nodes, then the stacks, then the cold ray state.
// kLong: with lists of more than kListShort leaves.
template <bool kStats, bool kStaged, bool kLong = true>
__global__ void __launch_bounds__(kVisThreads, LUZ_VIS_MIN_BLOCKS)
visibility_kernel(SceneVis S, VisCommon C, Entries E, RayOut R, unsigned long long* stats) {
    chain_wait();
    extern __shared__ float4 smem[];
    const uint32_t staged = min(S.tlas_node_count, C.smem_nodes);
    for (uint32_t i = threadIdx.x; i < staged * kNode4F4; i += blockDim.x) smem[i] = __ldg(S.tlas_nodes + i);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t* stack_base = reinterpret_cast<uint32_t*>(smem + staged * kNode4F4);
    uint32_t* s_stack = stack_base + warp * (kSmemStack * 32) + lane;
    const Cold c{reinterpret_cast<float*>(stack_base + kVisThreads * kSmemStack) + threadIdx.x};
    int lstack[kLocalStack];
    __syncthreads();
    const uint32_t full = 0xFFFFFFFFu, lt_mask = (1u << lane) - 1u;
    const uint32_t n = *R.count;
    uint32_t err = 0;
    TraceCounters cnt{0, 0, 0, 0};
    LaneRay r{};
    bool active = false, exhausted = n == 0;
    for (;;) {
        uint32_t idle = __ballot_sync(full, !active);
        if (!exhausted && __popc(idle) >= (int)C.refill) {
            int leader = __ffs(idle) - 1;
            unsigned long long base = 0;
            if (lane == leader) base = atomicAdd(C.work_counter, (unsigned long long)__popc(idle));
            base = __shfl_sync(full, base, leader);
            if (base + __popc(idle) >= n) exhausted = true;
            const unsigned long long k = base + __popc(idle & lt_mask);
            if (!active && k < n) {
                const float4 a = __ldg(R.a + k), b = __ldg(R.b + k);
                const uint4 q = __ldg(R.c + k);
                const bool sh = q.y < S.shadow_slots;
                const uint32_t pix = __float_as_uint(b.w);
                start_ray(r, c, S, V3{a.x, a.y, a.z}, V3{b.x, b.y, b.z}, sh ? 0.001f : S.ao_min, a.w,
                          (sh ? S.shadow_bits + (size_t)q.y * S.words : S.ao_bits + (size_t)(q.y - S.shadow_slots) * S.words) +
                              (pix >> 5),
                          sh, pix);
                active = true;
                if (q.z != kFromRoot) {
                    // The leaves its tests left, the nearest first: it starts at the nearest,
                    // the others stacked.
                    c[kList] = __uint_as_float(q.x);
                    const uint32_t flag = kEntryFlag | (kLong && q.w ? kEntryLong : 0u);
                    uint32_t lo = q.z, hi = kLong ? q.w & ~kLongList : 0u;
                    r.node = ~(int)(flag | (lo ? (uint32_t)__ffs(lo) : 31u + (uint32_t)__ffs(hi)));
                    if (lo) lo &= lo - 1u;
                    else hi &= hi - 1u;
                    while (lo | hi) {
                        uint32_t top;
                        if (hi) { top = 63u - __clz(hi); hi ^= 1u << (top - 32u); }
                        else { top = 32u - __clz(lo); lo ^= 1u << (top - 1u); }
                        const int e = ~(int)(flag | top);
                        if (r.sp < kSmemStack) s_stack[r.sp * 32] = (uint32_t)e;
                        else lstack[r.sp - kSmemStack] = e;
                        ++r.sp;
                    }
                }
            }
        }
        if (exhausted && __ballot_sync(full, active) == 0) break;
        run_steps<kStats, kStaged, kLong ? 2 : 1>(r, c, active, smem, staged, S.tlas_nodes, S.instances, s_stack, lstack,
                                         C.steps, C.step_cap, err, cnt, E);
    }
    if (err) atomicOr(C.status, err);
    if (kStats) flush_stats(stats, 0u, cnt);
}

// The rays of many scenes traced from their TLAS roots in one counting launch: item g
// belongs to the scene s with offsets[s] <= g < offsets[s+1]; each lane carries its scene's
// TLAS and outputs.
__global__ void __launch_bounds__(kVisThreads, LUZ_VIS_MIN_BLOCKS)
visibility_count_kernel(const SceneVis* __restrict__ scenes, uint32_t n, const unsigned long long* __restrict__ offsets,
                        VisCommon C, unsigned long long* stats) {
    extern __shared__ float4 smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t* stack_base = reinterpret_cast<uint32_t*>(smem);
    uint32_t* s_stack = stack_base + warp * (kSmemStack * 32) + lane;
    const Cold c{reinterpret_cast<float*>(stack_base + kVisThreads * kSmemStack) + threadIdx.x};
    int lstack[kLocalStack];
    const uint32_t full = 0xFFFFFFFFu, lt_mask = (1u << lane) - 1u;
    const unsigned long long total = offsets[n];
    uint32_t err = 0, rays = 0;
    TraceCounters cnt{0, 0, 0, 0};
    LaneRay r{};
    bool active = false, exhausted = false;
    for (;;) {
        uint32_t idle = __ballot_sync(full, !active);
        if (!exhausted && __popc(idle) >= (int)C.refill) {
            int leader = __ffs(idle) - 1;
            unsigned long long base = 0;
            if (lane == leader) base = atomicAdd(C.work_counter, (unsigned long long)__popc(idle));
            base = __shfl_sync(full, base, leader);
            if (base + __popc(idle) >= total) exhausted = true;
            if (!active) {
                unsigned long long item = base + __popc(idle & lt_mask);
                if (item < total) {
                    uint32_t lo = 0, hi = n - 1;
                    while (lo < hi) {
                        uint32_t mid = (lo + hi + 1) >> 1;
                        if (offsets[mid] <= item) lo = mid; else hi = mid - 1;
                    }
                    const SceneVis& S = scenes[lo];
                    uint32_t lit = *S.lit_count;
                    unsigned long long local = item - offsets[lo];
                    uint32_t slot = (uint32_t)(local / lit);
                    uint32_t j = (uint32_t)(local - (unsigned long long)slot * lit);
                    active = setup_ray(r, c, S, C, slot, j);
                    if (active) ++rays;
                }
            }
        }
        if (exhausted && __ballot_sync(full, active) == 0) break;
        run_steps<true, false>(r, c, active, nullptr, 0u, r.tlas, r.insts, s_stack, lstack, C.steps, C.step_cap, err,
                                 cnt);
    }
    if (err) atomicOr(C.status, err);
    flush_stats(stats, rays, cnt);
}

// offsets[s] = rays of scenes 0..s-1 (lit pixels x samples), read after the
// G-buffer passes have counted the lit pixels.
__global__ void batch_offsets_kernel(const SceneVis* scenes, uint32_t n, unsigned long long* offsets) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    unsigned long long acc = 0;
    for (uint32_t s = 0; s < n; ++s) {
        offsets[s] = acc;
        acc += (unsigned long long)(*scenes[s].lit_count) * (scenes[s].shadow_slots + scenes[s].ao_samples);
    }
    offsets[n] = acc;
}

// ---------------------------------------------------------------- host side
// Default launch shapes. Batches' frame kernels generate their rays in the traversal: 24 idle
// lanes to a refill, 8 steps between checks. A single scene's records hold only rays that
// enter a BLAS, which are short: a check every 4 steps and a refill at 16 idle lanes (refill
// {4..28} x steps {2,4,8,16}: 1080p two-level frame 0.966 ms against 1.009 at 24 / 8, 4K
// scene 43.8 against 46.0). Staging the TLAS top in shared memory does not pay: L1 holds it.
static const VisTuning g_tuning{0, 16, 4, 4, 1}, g_batch_tuning{0, 24, 8, 4, 1};

const VisTuning& vis_tuning(const luz_ctx* ctx) { return ctx->vis_tuning.set ? ctx->vis_tuning : g_tuning; }
const VisTuning& batch_tuning(const luz_ctx* ctx) { return ctx->vis_tuning.set ? ctx->vis_tuning : g_batch_tuning; }

SceneVis make_scene_vis(const luz_frame* f, const luz_tlas* t, int frame_index) {
    SceneVis S;
    // 4-wide nodes; node_count (the binary count) bounds the 4-wide count and the
    // size of the nodes4 buffer, so staging that many stays inside it.
    S.tlas_nodes = t->nodes4;
    S.tlas_node_count = t->count ? t->node_count : 0;
    S.instance_count = t->count;
    S.instances = t->instances;
    S.surf = f->surf;
    S.lit_count = f->lit_count;
    S.lights = f->d_lights;
    S.slot_table = f->d_slot_table;
    S.shadow_slots = f->shadow_slots;
    S.ao_samples = f->ao_samples;
    memcpy(S.cam, f->h_scene.cam_pos, 12);
    S.ao_min = f->h_scene.ao_min;
    S.ao_max = f->h_scene.ao_max;
    S.sampler = f->h_scene.sampler;
    S.frame = frame_index;
    S.width = f->width;
    S.words = f->words;
    S.shadow_bits = f->shadow_bits;
    S.ao_bits = f->ao_bits;
    S.cull = f->shadow_cull ? 1 : 0;
    S.leaf_box = nullptr;
    return S;
}

VisCommon make_vis_common(luz_ctx* ctx, const VisTuning& tu, unsigned long long* work_counter) {
    VisCommon C;
    C.blue_noise = ctx->d_blue_noise;
    C.bn_size = ctx->blue_noise_size;
    C.work_counter = work_counter;
    C.status = ctx->d_status;
    C.refill = tu.refill;
    C.steps = tu.steps;
    C.smem_nodes = tu.smem_nodes;
    C.step_cap = ctx->debug_step_cap ? ctx->debug_step_cap : kRayStepCap;
    return C;
}

luz_status clear_visibility(luz_ctx* ctx, luz_frame* f) {
    cudaStream_t st = ctx->stream;
    if (f->shadow_slots)
        LUZ_CUDA(ctx, cudaMemsetAsync(f->shadow_bits, 0, (size_t)f->shadow_slots * f->words * 4, st));
    if (f->ao_samples)
        LUZ_CUDA(ctx, cudaMemsetAsync(f->ao_bits, 0, (size_t)f->ao_samples * f->words * 4, st));
    return LUZ_OK;
}


// Sizes of a frame's traces: every pixel lit and no ray resolved before the traversal.
struct VisSizes {
    uint32_t patches, supers;
    uint32_t pairs, ao_patches;      // per chunk
    uint32_t records;                // per chunk
    uint32_t shadow_chunks, ao_chunks, chunks;
};

static_assert(((kRayChunkMin / kPatch) >> 2) % kSuper == 0, "chunks of whole blocks of pairs");
// Chunks over the largest possible counts; what lies past the frame's actual counts
// returns at once on the device. Without instances no shadow ray has anything to hit.
static VisSizes vis_sizes(const luz_frame* f, const luz_tlas* t, uint32_t ray_chunk) {
    VisSizes z{};
    z.patches = (f->pixels + kPatch - 1) / kPatch;
    z.supers = (z.patches + kSuper - 1) / kSuper;
    const uint32_t shift = f->vlight_shift;
    const unsigned long long max_pairs = t->count > 0 ? (unsigned long long)z.supers * kSuper * f->vlight_count : 0ull;
    z.pairs = (uint32_t)std::min<unsigned long long>(max_pairs, (ray_chunk / kPatch) >> shift);   // whole blocks
    if (f->ao_samples) z.ao_patches = std::min(z.patches, std::max(ray_chunk / 2 / (kPatch * f->ao_samples), 1u));
    z.records = ((z.pairs * kPatch) << shift) + z.ao_patches * kPatch * f->ao_samples;
    z.shadow_chunks = z.pairs ? (uint32_t)((max_pairs + z.pairs - 1) / z.pairs) : 0u;
    z.ao_chunks = z.ao_patches ? (z.patches + z.ao_patches - 1) / z.ao_patches : 0u;
    z.chunks = std::max(z.shadow_chunks, z.ao_chunks);
    return z;
}

// A trace's buffers: of a chunk (shafts.cuh) the patch bounds (the patches', then their
// blocks'), start lists per (virtual light, patch) and per AO patch, the lists' cuts, the
// shadow groups to trace and the ray records (RayOut), and the chunks' counters.
struct VisBuffers {
    PatchRec* patches;
    uint32_t* start_lists;
    float4* cuts;
    uint4* active;
    VisCounters* counters;
    float4* rays_a;
    float4* rays_b;
    uint4* rays_c;
    size_t bytes[4];   // of the scratch's blocks: all but the rays, the rays' three arrays
};
static VisBuffers carve_vis(const VisScratch& v, const VisSizes& z) {
    VisBuffers b{};
    uintptr_t at = (uintptr_t)v.block[0];
    auto take = [&](auto*& p, size_t count, int k) {
        if (k && v.block[k]) at = (uintptr_t)v.block[k];   // (else after the arrays before it)
        p = reinterpret_cast<std::remove_reference_t<decltype(p)>>(at);
        const size_t n = (count * sizeof(*p) + 255) & ~(size_t)255;
        b.bytes[k] += n;
        at += n;
    };
    take(b.patches, (size_t)z.patches + z.supers, 0);
    take(b.start_lists, ((size_t)z.pairs + z.ao_patches) * kEntryWords, 0);
    take(b.cuts, (size_t)z.pairs * kCutsPerPair * kNode4F4, 0);
    take(b.active, z.pairs, 0);
    take(b.counters, z.chunks, 0);
    take(b.rays_a, z.records, 1);
    take(b.rays_b, z.records, 2);
    take(b.rays_c, z.records, 3);
    return b;
}

static size_t total_bytes(const size_t (&n)[4]) { return n[0] + n[1] + n[2] + n[3]; }

size_t visibility_bytes(const luz_frame* f, const luz_tlas* t, uint32_t ray_chunk) {
    const VisSizes z = vis_sizes(f, t, ray_chunk);
    return z.chunks ? total_bytes(carve_vis(VisScratch{}, z).bytes) : 0;
}

// The blocks for a trace of f over t, in smaller chunks where there is no memory for larger
// ones; z: the sizes it then has. One allocation: a new frame object's first frame at 640x360
// takes 297 us, with one per buffer 490 (its second 190); at 4K 2665 and 2985 (2450). Up to
// kVisPooled four: cudaMalloc serves those out of what it holds (frames of 96x64 made and
// dropped in turn, first frame and preparation: 1090 us, with one block 1285).
constexpr size_t kVisPooled = 1 << 20;
static luz_status ensure_vis_buffers(luz_ctx* ctx, VisScratch& v, const luz_frame* f, const luz_tlas* t, VisSizes& z) {
    for (;;) {
        z = vis_sizes(f, t, v.ray_chunk);
        if (!z.chunks) return LUZ_OK;
        size_t need[4];
        memcpy(need, carve_vis(VisScratch{}, z).bytes, sizeof need);
        bool fits = true, pooled = true;
        if (!v.block[1]) fits = total_bytes(need) <= v.bytes[0];
        for (int k = 0; k < 4; ++k) {
            fits = fits && (!v.block[1] || need[k] <= v.bytes[k]);
            pooled = pooled && need[k] <= kVisPooled;
        }
        if (fits) return LUZ_OK;
        LUZ_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
        v.release();
        cudaError_t e = cudaSuccess;
        for (int k = 0; k < (pooled ? 4 : 1) && e == cudaSuccess; ++k) {
            v.bytes[k] = pooled ? need[k] : total_bytes(need);
            e = cudaMalloc(&v.block[k], std::max<size_t>(v.bytes[k], 256));
        }
        if (e == cudaSuccess) return LUZ_OK;
        cudaGetLastError();
        v.release();
        if (e != cudaErrorMemoryAllocation || v.ray_chunk <= kRayChunkMin) return cuda_error(ctx, e, "trace buffers");
        v.ray_chunk /= 2;
    }
}

luz_status reserve_visibility(luz_ctx* ctx, const luz_frame* f, const luz_tlas* t, VisScratch& scratch) {
    VisSizes z;
    return ensure_vis_buffers(ctx, scratch, f, t, z);
}

luz_status launch_visibility(luz_ctx* ctx, luz_frame* f, const luz_tlas* t, int frame_index,
                             unsigned long long* d_stats, VisScratch& v) {
    luz_status s = ensure_lit_list(ctx, f);
    if (s != LUZ_OK) return s;
    if (f->shadow_slots + f->ao_samples == 0) return LUZ_OK;
    cudaStream_t st = ctx->stream;
    SceneVis S = make_scene_vis(f, t, frame_index);
    const VisTuning& tu = vis_tuning(ctx);
    VisCommon C = make_vis_common(ctx, tu, nullptr);
    uint32_t staged = std::min<uint32_t>(S.tlas_node_count, tu.smem_nodes);
    size_t smem = (size_t)staged * kNode4F4 * 16 + kStackBytes + kColdBytes;
    static DeviceSetup setup;   // the traversal kernels' shared-memory limit
    s = device_setup(setup, setup_generation(), smem, [&]() -> luz_status {
        const void* fns[5] = {(const void*)visibility_kernel<false, false, false>, (const void*)visibility_kernel<false, false>, (const void*)visibility_kernel<true, false>,
                              (const void*)visibility_kernel<false, true>, (const void*)visibility_kernel<true, true>};
        for (const void* fn : fns)
            LUZ_CUDA(ctx, cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        return LUZ_OK;
    });
    if (s != LUZ_OK) return s;
    uint32_t grid = (uint32_t)ctx->sm_count * tu.ctas_per_sm;
    VisSizes z;
    if ((s = ensure_vis_buffers(ctx, v, f, t, z)) != LUZ_OK) return s;
    const uint32_t shadow_chunks = z.shadow_chunks, ao_chunks = z.ao_chunks;
    if (d_stats) LUZ_CUDA(ctx, cudaMemsetAsync(d_stats, 0, 5 * sizeof(unsigned long long), st));
    if (!shadow_chunks && (s = clear_visibility(ctx, f)) != LUZ_OK) return s;   // else by patch_kernel
    if (z.chunks == 0) return LUZ_OK;
    const VisBuffers buf = carve_vis(v, z);
    VisCounters* counters = buf.counters;
    if (!shadow_chunks) LUZ_CUDA(ctx, cudaMemsetAsync(counters, 0, (size_t)z.chunks * sizeof(VisCounters), st));
    if (t->count) S.leaf_box = tlas_leaf_boxes(t);
    if (ctx->raygen_blocks == 0) {   // resident blocks per SM: the persistent grids are one wave
        int a = 0, b = 0;
        LUZ_CUDA(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&a, cull_kernel<true, false>, kCullThreads, 0));
        LUZ_CUDA(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, shadow_raygen_kernel<true>, 256, 0));
        ctx->cull_blocks = std::max(a, 1);
        ctx->raygen_blocks = std::max(b, 1);
    }
    const uint32_t sms = (uint32_t)ctx->sm_count;
    const Entries entries{buf.start_lists, buf.cuts, cut_cap(t->count)};
    prof_begin(ctx, LUZ_KERNEL_RAYGEN);
    PatchRec* patches = buf.patches;
    if (shadow_chunks) {
        chain(patch_kernel, std::min(z.supers, sms * 8), kSuper * 32, 0, st, S, patches, patches + z.patches, counters,
                                                                          z.chunks);
        LUZ_LAUNCHED(ctx, "patch_kernel");
    }
    if (d_stats) {
        chain(count_rays_kernel, sms * 4, 256, 0, st, S, C, d_stats);
        LUZ_LAUNCHED(ctx, "count_rays_kernel");
    }
    for (uint32_t k = 0; k < z.chunks; ++k) {
        if (k) prof_begin(ctx, LUZ_KERNEL_RAYGEN);
        VisCounters* n = counters + k;
        C.work_counter = &n->traversed;
        const RayOut R{buf.rays_a, buf.rays_b, buf.rays_c, &n->records};
        const bool shadow = k < shadow_chunks, ao = k < ao_chunks;
        const ShaftOut A{patches, patches + z.patches, f->d_vlights, f->vlight_count, (unsigned long long)k * z.pairs,
                         shadow ? z.pairs : 0u, list_cap(t->count), entries.cut_cap, super_cap(t->count), buf.start_lists, buf.cuts, buf.active, &n->groups};
        const AoOut O{k * z.ao_patches, ao ? std::min(z.ao_patches, z.patches - k * z.ao_patches) : 0u,
                      f->ao_samples < kAoMinSamples ? 0u : std::min(kAoStepsPerSample * f->ao_samples, kAoSteps),
                      buf.start_lists + (size_t)z.pairs * kEntryWords, z.pairs, R};
        const uint32_t shaft_work = A.cap / kSuper, max_grid = sms * ctx->cull_blocks;
        auto cull_grid = [&](uint32_t warps) { return std::min((warps + kCullWarps - 1) / kCullWarps, max_grid); };
        if (shadow && ao && f->pixels <= kCullTogether) {
            chain(cull_kernel<true, true>, cull_grid(shaft_work + O.patches), kCullThreads, 0, st, S, C, A, O, n->cull_tickets);
            LUZ_LAUNCHED(ctx, "cull_kernel");
        } else {
            if (shadow) {
                chain(cull_kernel<false, true>, cull_grid(shaft_work), kCullThreads, 0, st, S, C, A, O, n->cull_tickets);
                LUZ_LAUNCHED(ctx, "cull_kernel<shadow>");
            }
            if (ao) {
                chain(cull_kernel<true, false>, cull_grid(O.patches), kCullThreads, 0, st, S, C, A, O, n->cull_tickets + 1);
                LUZ_LAUNCHED(ctx, "cull_kernel<ao>");
            }
        }
        if (shadow) {
            chain(A.list_cap > kListShort ? shadow_raygen_kernel<true> : shadow_raygen_kernel<false>, std::min((z.pairs + 7) / 8, sms * ctx->raygen_blocks), 256, 0, st, S, C, entries, buf.active, &n->groups, &n->raygen_tickets, R);
            LUZ_LAUNCHED(ctx, "shadow_raygen_kernel");
        }
        prof_end(ctx);
        if (d_stats) {
            if (staged) chain(visibility_kernel<true, true>, grid, 256, smem, st, S, C, entries, R, d_stats);
            else chain(visibility_kernel<true, false>, grid, 256, smem, st, S, C, entries, R, d_stats);
            LUZ_LAUNCHED(ctx, "visibility_kernel<stats>");
        } else {
            prof_begin(ctx, LUZ_KERNEL_TRAVERSAL);
            if (staged) chain(visibility_kernel<false, true>, grid, 256, smem, st, S, C, entries, R, nullptr);
            else chain(A.list_cap > kListShort ? visibility_kernel<false, false, true> : visibility_kernel<false, false, false>, grid,
                       256, smem, st, S, C, entries, R, nullptr);
            prof_end(ctx);
            LUZ_LAUNCHED(ctx, "visibility_kernel");
        }
    }
    return LUZ_OK;
}

luz_status launch_visibility_count(luz_ctx* ctx, const SceneVis* d_scenes, uint32_t n, unsigned long long* d_offsets,
                                   unsigned long long* work_counter, unsigned long long* d_stats) {
    cudaStream_t st = ctx->stream;
    batch_offsets_kernel<<<1, 32, 0, st>>>(d_scenes, n, d_offsets);
    LUZ_LAUNCHED(ctx, "batch_offsets_kernel");
    LUZ_CUDA(ctx, cudaMemsetAsync(work_counter, 0, 8, st));
    LUZ_CUDA(ctx, cudaMemsetAsync(d_stats, 0, 5 * sizeof(unsigned long long), st));
    const VisTuning& tu = batch_tuning(ctx);
    VisCommon C = make_vis_common(ctx, tu, work_counter);
    visibility_count_kernel<<<(uint32_t)ctx->sm_count * tu.ctas_per_sm, 256, kStackBytes + kColdBytes, st>>>(
        d_scenes, n, d_offsets, C, d_stats);
    LUZ_LAUNCHED(ctx, "visibility_count_kernel");
    return LUZ_OK;
}

}  // namespace luz

extern "C" luz_status luz_ctx_set_vis_tuning(luz_ctx* ctx, const luz_vis_tuning* t) {
    using namespace luz;
    if (!ctx || !t) return LUZ_ERR_INVALID;
    if (t->smem_nodes == 0 && t->refill == 0 && t->steps == 0 && t->ctas_per_sm == 0) {
        ++ctx->vis_tuning_changes;
        ctx->vis_tuning = VisTuning{0, 0, 0, 0, 0};
        return LUZ_OK;
    }
    if (t->smem_nodes > 1024 || t->refill < 1 || t->refill > 32 || t->steps < 1 || t->steps > 1024 ||
        t->ctas_per_sm < 1 || t->ctas_per_sm > 16)
        return set_error(ctx, LUZ_ERR_INVALID, "visibility tuning outside its documented ranges");
    ++ctx->vis_tuning_changes;
    ctx->vis_tuning = VisTuning{t->smem_nodes, t->refill, t->steps, t->ctas_per_sm, 1};
    return LUZ_OK;
}

extern "C" luz_status luz_ctx_get_vis_tuning(const luz_ctx* ctx, luz_vis_tuning* t) {
    using namespace luz;
    if (!ctx || !t) return LUZ_ERR_INVALID;
    const VisTuning& tu = vis_tuning(ctx);
    *t = luz_vis_tuning{tu.smem_nodes, tu.refill, tu.steps, tu.ctas_per_sm};
    return LUZ_OK;
}

namespace luz {

luz_status frame_lit_count(luz_ctx* ctx, luz_frame* f, uint32_t* count) {
    LUZ_CUDA(ctx, cudaMemcpyAsync(&f->h_lit_count, f->lit_count, 4, cudaMemcpyDeviceToHost, ctx->stream));
    LUZ_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    *count = f->h_lit_count;
    return LUZ_OK;
}

}  // namespace luz
