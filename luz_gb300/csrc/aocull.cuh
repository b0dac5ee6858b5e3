// aocull.cuh — ray generation of the AO rays, one patch (32 lit pixels, shafts.cuh) per
// warp, with most rays resolved by the patch's horizon; and the kernel that runs it beside
// the shadow shafts.
//
// All AO rays of a patch start in the small box of its ray origins, are at most aoMax
// long, and leave into the hemispheres of its pixels' normals. The horizon is the largest
// elevation over the plane normal to the patch's mean normal n at which any geometry
// within reach is seen from the patch: for a point x of a BVH box,
// dot(n, x - o) / |x - o| is at most (the box's largest dot with n less the least dot of
// the origins) / (distance of the box to the origins' box). A ray with
// dot(n, d) / |d| above the horizon hits nothing and is recorded as a miss at once. The
// horizon is found by descending the BVH from the instances around the patch, eight nodes
// (32 child boxes) at a time, leaving out boxes that are out of reach or below the horizon
// found so far; when the step budget or the node stack runs out, what is left counts with
// its own bounds, so the horizon only gets higher.
//
// The rays below it that reach the box of an instance around the patch become records,
// which start the traversal at the patch's list of those instances.
#pragma once
#include "shafts.cuh"

namespace luz {

constexpr uint32_t kAoStack = 192;           // nodes of a warp's descent
constexpr uint32_t kAoInstances = 16;        // instances a horizon descends at most
// A horizon costs about as much as tracing a patch's rays of one or two samples, so one is
// sought from kAoMinSamples on, with a budget that grows with the samples it can resolve.
constexpr uint32_t kAoMinSamples = 4, kAoStepsPerSample = 4, kAoSteps = 64;
constexpr float kAoFloor = 0x1p-6f;          // horizons start here: lower rays are traced

struct AoOut {
    uint32_t patch0, patches;    // patches [patch0, patch0 + patches) of the frame (0: no AO here)
    uint32_t steps;              // node-stack steps of one horizon (0: no horizon)
    uint32_t* lists;             // start lists (kEntryWords), one per patch of the chunk
    uint32_t list0;              // index of the first of them
    RayOut rays;
};

// An instance around the patch, in its object space: the origins' box (centre, half
// extents), the scaled normal n' and its offset (dot(n, x - o) <= n' . x' - on for every
// origin o), an upper bound of the world-to-object stretch (a distance in object space
// over it bounds the world-space one from below), the reach in object space, squared, and
// the BLAS.
struct __align__(16) AoInstance {
    float c[3], on;
    float h[3], scale;
    float n[3], reach2;
    const float4* nodes;
    uint32_t leaf, pad;
};
static_assert(sizeof(AoInstance) == 64, "AoInstance layout");

// Bound of the elevation of a box seen from the origins' box (c, h): false when the box
// is out of reach (squared, in the space of the boxes). e <= 0: below the plane of every
// origin; far above 1 where the boxes touch.
__device__ __forceinline__ bool elevation(const float c[3], const float h[3], const float n[3], float on, float scale,
                                          float reach2, const float lo[3], const float hi[3], float& e) {
    float d2 = 0.f, sup = 0.f;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float d = fmaxf(fmaxf(lo[k] - (c[k] + h[k]), (c[k] - h[k]) - hi[k]), 0.0f);
        d2 = __fmaf_rn(d, d, d2);
        sup += fmaxf(n[k] * lo[k], n[k] * hi[k]);
    }
    float r;   // 1 / sqrt(d2) to 2^-22, +inf for 0
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d2));
    const float num = sup - on;   // NaN where an infinite plane meets a zero of n, or the box has one: no bound
    e = num <= 0.0f ? -1.0f : fminf(num * (r * scale), 1e9f);
    return d2 <= reach2;
}

// Object-space record of the instance at a TLAS leaf; false when it cannot be used (a
// transform that is singular or not finite): the horizon then covers everything.
__device__ __forceinline__ bool ao_instance(const DevInstance* I, uint32_t leaf, const float c[3], const float h[3],
                                            V3 n, float on, float reach, AoInstance& o) {
    const float4* wp = reinterpret_cast<const float4*>(I->w2o);
    const float4 q0 = __ldg(wp), q1 = __ldg(wp + 1), q2 = __ldg(wp + 2);
    const float w[3][4] = {{q0.x, q0.y, q0.z, q0.w}, {q1.x, q1.y, q1.z, q1.w}, {q2.x, q2.y, q2.z, q2.w}};
    float wm = 0.f, norm2 = 0.f, t = 0.f;
#pragma unroll
    for (int r = 0; r < 3; ++r) {
        const float a0 = fabsf(w[r][0]), a1 = fabsf(w[r][1]), a2 = fabsf(w[r][2]);
        const float m = a0 * fabsf(c[0]) + a1 * fabsf(c[1]) + a2 * fabsf(c[2]) + fabsf(w[r][3]);
        o.c[r] = w[r][0] * c[0] + w[r][1] * c[1] + w[r][2] * c[2] + w[r][3];
        o.h[r] = (a0 * h[0] + a1 * h[1] + a2 * h[2]) * (1.0f + 0x1p-18f) + 0x1p-18f * m + 0x1p-60f;
        wm = fmaxf(wm, fmaxf(a0, fmaxf(a1, a2)));
        t += fabsf(w[r][3]);
        // |W|^2 <= the largest absolute row sum of W W^T
        float s = 0.f;
#pragma unroll
        for (int k = 0; k < 3; ++k) s += fabsf(w[r][0] * w[k][0] + w[r][1] * w[k][1] + w[r][2] * w[k][2]);
        norm2 = fmaxf(norm2, s);
    }
    const V3 r0 = V3{w[0][0], w[0][1], w[0][2]}, r1 = V3{w[1][0], w[1][1], w[1][2]}, r2 = V3{w[2][0], w[2][1], w[2][2]};
    const V3 c0 = cross(r1, r2), c1 = cross(r2, r0), c2 = cross(r0, r1);
    const float det = dot(r0, c0), inv = 1.0f / fabsf(det);
    const float sg = det < 0.0f ? -inv : inv;
    // n' . (W x + t) = n . x + n' . t; rounding as in object_shaft, over |det|
    o.n[0] = sg * dot(c0, n); o.n[1] = sg * dot(c1, n); o.n[2] = sg * dot(c2, n);
    const float nt = o.n[0] * w[0][3] + o.n[1] * w[1][3] + o.n[2] * w[2][3];
    const float mo = fmaxf(fabsf(o.c[0]) + o.h[0], fmaxf(fabsf(o.c[1]) + o.h[1], fabsf(o.c[2]) + o.h[2]));
    o.on = (on + nt) - (0x1p-16f * (wm * wm) * (wm * fabsf(on) + mo + t) * inv + 0x1p-60f);
    o.scale = __fsqrt_rn(norm2) * (1.0f + 0x1p-10f);
    o.reach2 = (reach * o.scale) * (reach * o.scale);
    o.leaf = leaf;
    o.nodes = I->nodes4;
    o.pad = 0;
    const float big = 1e30f;
    return fabsf(o.c[0]) <= big && fabsf(o.c[1]) <= big && fabsf(o.c[2]) <= big && o.h[0] <= big && o.h[1] <= big &&
           o.h[2] <= big && fabsf(o.on) <= big && fabsf(o.n[0]) <= big && fabsf(o.n[1]) <= big &&
           fabsf(o.n[2]) <= big && o.scale <= big;
}

// One warp's shared memory.
struct AoShared {
    AoInstance inst[kAoInstances];
    uint32_t node[kAoStack];
    float e[kAoStack];
    unsigned char slot[kAoStack];        // the nodes' instances
    float ray[kStageWords - 1][kStageRays];
};

// The AO rays of patch A.patch0 + local; called by a whole warp.
__device__ __forceinline__ void ao_patch(const SceneVis& S, const VisCommon& C, const AoOut& A, uint32_t lit, uint32_t local,
                                         AoShared& sm, RayStage& stage) {
    const uint32_t full = 0xFFFFFFFFu, lane = threadIdx.x & 31, lt_mask = (1u << lane) - 1u;
    const V3 cam = V3{S.cam[0], S.cam[1], S.cam[2]};
    const uint32_t patch = A.patch0 + local;
    const uint32_t j = patch * kPatch + lane;
    const bool in = j < lit;
    const float4* sp4 = S.surf + 2 * (size_t)(in ? j : patch * kPatch);
    const float4 s0 = __ldg(sp4), s1 = __ldg(sp4 + 1);
    const V3 p = V3{s0.x, s0.y, s0.z}, N = V3{s1.x, s1.y, s1.z};
    const uint32_t pix = __float_as_uint(s0.w), pxy = __float_as_uint(s1.w);
    const float bias = length(p - cam) * 0.01f;          // ao_ray's origin
    const V3 o = p + N * bias;
    const bool any = S.instance_count > 0 && S.ao_min <= S.ao_max;

    // ---- bounds of the origins, the reach of the rays (|d| <= max(|N|, |N|^2): d is a unit
    // vector of the basis (T, N x T, N) with |T| <= |N|) and the mean normal
    float c[3], h[3];
    const float ov[3] = {o.x, o.y, o.z};
    float mag = 0.f;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float lo = warp_min(ov[k]), hi = warp_max(ov[k]);
        c[k] = 0.5f * (lo + hi);
        h[k] = 0.5f * (hi - lo);
        mag = fmaxf(mag, fmaxf(fabsf(lo), fabsf(hi)));
    }
    const float grow = 0x1p-16f * mag + 0x1p-60f;
#pragma unroll
    for (int k = 0; k < 3; ++k) h[k] = h[k] * (1.0f + 0x1p-10f) + grow;
    const float nl = length(N);
    const float reach = S.ao_max * warp_max(fmaxf(nl, nl * nl)) * (1.0f + 0x1p-9f) + grow;
    V3 n = normalize(V3{warp_sum(in ? N.x : 0.f), warp_sum(in ? N.y : 0.f), warp_sum(in ? N.z : 0.f)});
    const bool flat = !finite3(n);                       // no mean normal: no horizon
    if (flat) n = V3{0.f, 0.f, 0.f};
    const float on = warp_min(dot(n, o)) - 4.0f * grow;
    const float nn[3] = {n.x, n.y, n.z};

    const float reach2 = (reach * (1.0f + 0x1p-10f)) * (reach * (1.0f + 0x1p-10f));

    // ---- the TLAS leaves within reach, eight nodes at a time
    uint32_t* node_st = sm.node;
    float* e_st = sm.e;
    const uint32_t g = lane >> 2, ch_i = lane & 3;
    uint32_t* list = A.lists + (size_t)local * kEntryWords;
    uint32_t leaves = 0;
    bool all = !any || !(reach <= 1e18f) || !(fabsf(c[0]) + fabsf(c[1]) + fabsf(c[2]) <= 1e18f);
    float horizon = kAoFloor;
    bool open = A.steps > 0 && !flat;                    // a horizon is being sought
    if (!all) {
        uint32_t sp = 1;
        if (lane == 0) node_st[0] = 0u;
        __syncwarp();
        for (uint32_t it = 0; sp > 0 && it < kTraversalCap; ++it) {
            const uint32_t take = min(sp, 8u);
            sp -= take;
            int ch = kEmptyChild;
            bool hit = false, odd = false;
            float e = -1.0f;
            if (g < take) {
                const float* f = reinterpret_cast<const float*>(S.tlas_nodes + (size_t)node_st[sp + g] * kNode4F4) + ch_i;
                const float lo[3] = {__ldg(f), __ldg(f + 8), __ldg(f + 16)}, hi[3] = {__ldg(f + 4), __ldg(f + 12), __ldg(f + 20)};
                ch = __float_as_int(__ldg(f + 24));
                hit = ch != kEmptyChild && elevation(c, h, nn, on, 1.0f + 0x1p-10f, reach2, lo, hi, e);
                odd = box_has_nan(lo, hi);
            }
            if (__any_sync(full, odd)) { all = true; break; }   // its other boxes may not nest: the rays start at the root
            __syncwarp();
            const uint32_t lb = __ballot_sync(full, hit && ch < 0), nb = __ballot_sync(full, hit && ch >= 0);
            const uint32_t lpos = leaves + __popc(lb & lt_mask), npos = sp + __popc(nb & lt_mask);
            if (hit && ch < 0 && lpos < kEntryCuts - 1) {
                list[1 + lpos] = (uint32_t)~ch;
                list[kEntryCuts + lpos] = 0u;           // entered at the BLAS root
                if (lpos < kAoInstances) sm.inst[lpos].leaf = (uint32_t)~ch;
            }
            if (hit && ch >= 0 && npos < kAoStack) node_st[npos] = (uint32_t)ch;
            leaves += __popc(lb);
            sp += __popc(nb);
            if (leaves > kListShort || sp > kAoStack) { all = true; break; }
            __syncwarp();
        }
    }
    if (all) leaves = 0;
    if (lane == 0) list[0] = all ? kListAll : leaves;
    __syncwarp();

    // ---- the horizon over those instances
    if (all || leaves > kAoInstances) open = false;
    if (open && leaves) {
        bool good = true, use = false;
        if (lane < leaves) {
            const uint32_t leaf = sm.inst[lane].leaf;
            const DevInstance* I = S.instances + leaf;
            const uint4 meta = __ldg(reinterpret_cast<const uint4*>(&I->custom_index));
            use = (meta.y & 0xFFu) != 0 && meta.w > 0;
            AoInstance rec;
            good = blas_nests(I) && ao_instance(I, leaf, c, h, n, on, reach, rec);
            if (use && good) sm.inst[lane] = rec;
        }
        if (__any_sync(full, use && !good)) open = false;
        const uint32_t ub = __ballot_sync(full, use);
        uint32_t sp = __popc(ub);
        unsigned char* slot_st = sm.slot;
        if (use) {
            const uint32_t pos = __popc(ub & lt_mask);
            node_st[pos] = 0u;
            slot_st[pos] = (unsigned char)lane;
            e_st[pos] = 1e9f;
        }
        __syncwarp();
        uint32_t it = 0;
        for (; open && sp > 0 && it < A.steps; ++it) {
            const uint32_t take = min(sp, 8u);
            sp -= take;
            int ch = kEmptyChild;
            bool hit = false;
            float e = -1.0f;
            uint32_t slot = 0;
            if (g < take && e_st[sp + g] > horizon) {
                slot = slot_st[sp + g];
                const AoInstance& I = sm.inst[slot];
                const float* f = reinterpret_cast<const float*>(I.nodes + (size_t)node_st[sp + g] * kNode4F4) + ch_i;
                const float lo[3] = {__ldg(f), __ldg(f + 8), __ldg(f + 16)}, hi[3] = {__ldg(f + 4), __ldg(f + 12), __ldg(f + 20)};
                ch = __float_as_int(__ldg(f + 24));
                hit = ch != kEmptyChild && elevation(I.c, I.h, I.n, I.on, I.scale, I.reach2, lo, hi, e) && e > horizon;
            }
            // triangles raise the horizon (positive floats order like their bits)
            const float top = __uint_as_float(__reduce_max_sync(full, hit && ch < 0 ? __float_as_uint(e) : 0u));
            horizon = fmaxf(horizon, top);
            const bool push = hit && ch >= 0 && e > horizon;
            const uint32_t nb = __ballot_sync(full, push);
            const uint32_t pos = sp + __popc(nb & lt_mask);
            const bool fits = pos < kAoStack;
            if (push && fits) {
                node_st[pos] = (uint32_t)ch;
                slot_st[pos] = (unsigned char)slot;
                e_st[pos] = e;
            }
            if (sp + __popc(nb) > kAoStack) {   // no room: those boxes count as they are
                horizon = fmaxf(horizon, __uint_as_float(__reduce_max_sync(full, push && !fits ? __float_as_uint(e) : 0u)));
                sp = kAoStack;
            } else {
                sp += __popc(nb);
            }
            if (horizon >= 1.0f) open = false;
            __syncwarp();
        }
        // out of steps: what is left counts as it is
        float rest = 0.f;
        for (uint32_t k = lane; k < sp; k += 32) rest = fmaxf(rest, e_st[k]);
        horizon = fmaxf(horizon, __uint_as_float(__reduce_max_sync(full, __float_as_uint(rest))));
    }
    if (!open) horizon = 2.0f;
    const float h2 = horizon < 1.0f ? horizon * horizon * (1.0f + 0x1p-9f) : 4.0f;

    // ---- the rays. Runs of lanes whose pixels follow each other in one word of a bit plane
    // write their misses with one atomic.
    const uint32_t prev = __shfl_up_sync(full, pix, 1);
    const uint32_t starts = __ballot_sync(full, lane == 0 || pix != prev + 1u || (pix >> 5) != (prev >> 5));
    const uint32_t after = lane == 31 ? 0u : starts & (0xFFFFFFFEu << lane);
    const uint32_t run = (after ? (uint32_t)__ffs(after) - 1u : 32u) - lane;   // lanes of the run that starts here
    const uint32_t run_mask = run >= 32u ? full : (1u << run) - 1u;
    const bool lead = (starts >> lane) & 1u;
    uint32_t* word = S.ao_bits + (pix >> 5);
    const AoPixel px = ao_pixel(C, S.sampler, pxy & 0xFFFFu, pxy >> 16);
    for (uint32_t s = 0; s < S.ao_samples; ++s) {
        V3 wo, wd;
        const bool ok = in && ao_gen(S, px, s, p, N, cam, wo, wd);
        const float el = dot(n, wd), dd = dot(wd, wd);
        const bool clear = !ok || (leaves == 0 && !all) || (el > 0.0f && el * el > h2 * dd);
        uint32_t mask = all ? kFromRoot : 0u;
        if (!all && __any_sync(full, !clear)) {
            LaneRay r;
            r.tmin = S.ao_min;
            r.tmax = S.ao_max;
            r.idir = safe_inv(wd);
            set_origin(r, wo);
            near_planes(r);
            for (uint32_t k = 0; k < leaves; ++k)
                if (leaf_overlaps(r, S.leaf_box, list[1 + k])) mask |= 1u << k;
        }
        const bool trace = !clear && mask != 0u;
        const uint32_t misses = (__ballot_sync(full, !trace && in) >> lane) & run_mask;
        if (lead && misses) atomicOr(word + (size_t)s * S.words, misses << (pix & 31u));
        stage_rays(stage, A.rays, lane, trace, wo, S.ao_max, wd, pix, A.list0 + local, S.shadow_slots + s, mask);
    }
}

// ---------------------------------------------------------------- the kernel
// AO patches and blocks of shadow pairs of a chunk, taken by ticket by the warps of a
// persistent grid. Both are chains of dependent loads. On a small frame neither fills the
// chip and one launch runs both (96x64 frame: 16 us against 11 + 16 in two; 512x512: 57
// against 62); on a large one each has its own launch with the registers it needs (1080p:
// 335 + 216 us against 573, 4K: 15.0 ms against 16.2).
constexpr int kCullThreads = 128, kCullWarps = kCullThreads / 32;
constexpr uint32_t kCullTogether = 1u << 19;   // pixels up to which one launch runs both
union CullShared {
    AoShared ao;
    ShaftShared shaft;
    __device__ CullShared() {}
};

template <bool kAo, bool kShaft>
__global__ void __launch_bounds__(kCullThreads, kAo ? (kShaft ? 4 : 6) : 5)
cull_kernel(SceneVis S, VisCommon C, ShaftOut A, AoOut O, uint32_t* tickets) {
    chain_wait();
    __shared__ CullShared s_mem[kCullWarps];
    const uint32_t full = 0xFFFFFFFFu, lane = threadIdx.x & 31;
    CullShared& sm = s_mem[threadIdx.x >> 5];
    const uint32_t lit = *S.lit_count, patches = (lit + kPatch - 1) / kPatch;
    const uint32_t ao = kAo ? min(O.patches, patches - min(O.patch0, patches)) : 0u;
    const uint32_t blocks = kShaft ? shaft_blocks(A, patches) : 0u;
    RayStage stage{sm.ao.ray, 0u};
    for (;;) {
        uint32_t t = 0;
        if (lane == 0) t = atomicAdd(tickets, 1u);
        t = __shfl_sync(full, t, 0);
        if (kAo && t < ao) {
            ao_patch(S, C, O, lit, t, sm.ao, stage);
        } else {
            if (kAo && stage.n) stage_flush(stage, O.rays, lane);   // its memory is the shafts' from here on
            if (t - ao >= blocks) break;
            if (kShaft) shaft_block(S, A, patches, t - ao, sm.shaft);
        }
        __syncwarp();
    }
}

}  // namespace luz
