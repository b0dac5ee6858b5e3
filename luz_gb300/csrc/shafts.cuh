// shafts.cuh — culling of whole groups of shadow rays before they are generated.
//
// A patch is 32 consecutive lit pixels (an 8x4 block of the image in the list's tile
// order). Every shadow ray from a patch to one light starts in the box of the patch's
// ray origins and ends in a box around the light's disk, so the point of any of them at
// parameter t lies in the linear blend of the two boxes: a shaft, bounded per axis by two
// lines in t, and along the patch's mean normal by one more. A box that no t in [0, 1]
// brings into reach of all seven bounds cannot be touched by any ray of the group.
// A warp per light and block of eight patches descends the TLAS with that test, then four
// lanes per patch the BLAS of each leaf it reaches, and keeps per leaf the up to four nodes of the BLAS
// that the shaft still touches as a 4-wide node of their own (a cut). A leaf without any
// is dropped; a group without leaves has only unoccluded rays: their bits stay 0 and
// neither a ray record nor a traversal step is spent on them. The normal bound is what
// makes that common: rays leave a surface upwards, and a patch's shaft clears the surface
// it starts on.
//
// The result is that of tracing every ray from the TLAS root: boxes are conservative, and
// the shaft's boxes are grown past the rounding of the ray origins, ends and transforms.
// A start below the root also needs every box to lie inside those above it. Unions with a
// NaN (a vertex or a transform that is none) can lose a box, so that a trace from the root
// never comes to it: where a NaN is met among the TLAS's boxes, or the mesh has a vertex that
// is not finite, the rays start at that root instead.
#pragma once
#include "raygen.cuh"
#include "traverse.cuh"
#include "vis_trace.cuh"
#include "visibility.cuh"

namespace luz {

// ---------------------------------------------------------------- ray records
// A generated ray that the traversal has to trace: (origin, tMax), (direction, pixel) and
// (start list, slot, leaves, more leaves): the entries of the list (Entries) that the ray's
// own tests leave, bit k = leaf k + 1, or all bits for a start at the TLAS root; of a long
// list, the second word's bit k = leaf k + 32 and kLongList. Slots of the
// AO samples follow those of the shadow samples. Warps stage records in shared memory and
// append them kStageFlush at a time, so one atomic reserves whole lines.
struct RayOut {
    float4* a;
    float4* b;
    uint4* c;
    uint32_t* count;
};
constexpr uint32_t kFromRoot = 0xFFFFFFFFu;
constexpr uint32_t kStageFlush = 64, kStageRays = kStageFlush + 32, kStageWords = 12;
constexpr uint32_t kLongList = 0x80000000u;

// Device counters of one chunk, zero before its launches.
struct VisCounters {
    unsigned long long traversed;    // records taken by the traversal
    uint32_t records;                // written by ray generation
    uint32_t groups;                 // shadow groups left by the shafts
    uint32_t cull_tickets[2], raygen_tickets, pad;
};

struct RayStage {
    float (*w)[kStageRays];   // kStageWords rows of the warp's shared memory
    uint32_t n;
};

// kMore: with the second word of leaves.
template <bool kMore = false>
__device__ __forceinline__ void stage_flush(RayStage& st, const RayOut& R, uint32_t lane) {
    __syncwarp();
    const uint32_t n = min(st.n, kStageFlush);
    uint32_t base = 0;
    if (lane == 0) base = atomicAdd(R.count, n);
    base = __shfl_sync(0xFFFFFFFFu, base, 0);
    for (uint32_t k = lane; k < n; k += 32) {
        const size_t at = (size_t)base + k;
        R.a[at] = make_float4(st.w[0][k], st.w[1][k], st.w[2][k], st.w[3][k]);
        R.b[at] = make_float4(st.w[4][k], st.w[5][k], st.w[6][k], st.w[7][k]);
        R.c[at] = make_uint4(__float_as_uint(st.w[8][k]), __float_as_uint(st.w[9][k]), __float_as_uint(st.w[10][k]),
                             kMore ? __float_as_uint(st.w[kMore ? 11 : 0][k]) : 0u);
    }
    const uint32_t left = st.n - n;   // fewer than 32
    constexpr uint32_t rows = kMore ? kStageWords : kStageWords - 1;
    float keep[rows];
    if (lane < left)
#pragma unroll
        for (uint32_t q = 0; q < rows; ++q) keep[q] = st.w[q][kStageFlush + lane];
    __syncwarp();
    if (lane < left)
#pragma unroll
        for (uint32_t q = 0; q < rows; ++q) st.w[q][lane] = keep[q];
    st.n = left;
    __syncwarp();
}

// Appends the rays of the lanes with `live` set; every lane of the warp calls it.
template <bool kMore = false>
__device__ __forceinline__ void stage_rays(RayStage& st, const RayOut& R, uint32_t lane, bool live, V3 o, float tmax,
                                           V3 d, uint32_t pix, uint32_t list, uint32_t slot, uint32_t leaves,
                                           uint32_t more = 0u) {
    const uint32_t m = __ballot_sync(0xFFFFFFFFu, live);
    if (m == 0u) return;
    if (live) {
        const uint32_t k = st.n + __popc(m & ((1u << lane) - 1u));
        st.w[0][k] = o.x; st.w[1][k] = o.y; st.w[2][k] = o.z; st.w[3][k] = tmax;
        st.w[4][k] = d.x; st.w[5][k] = d.y; st.w[6][k] = d.z; st.w[7][k] = __uint_as_float(pix);
        st.w[8][k] = __uint_as_float(list);
        st.w[9][k] = __uint_as_float(slot);
        st.w[10][k] = __uint_as_float(leaves);
        if (kMore) st.w[kMore ? 11 : 0][k] = __uint_as_float(more);
    }
    st.n += __popc(m);
    if (st.n >= kStageFlush) stage_flush<kMore>(st, R, lane);
}

// The slab test of a TLAS leaf's box for a world-space ray (inverse direction and origin
// offsets set), as a 4-wide node applies it to the slot holding that leaf.
__device__ __forceinline__ bool leaf_overlaps(const LaneRay& r, const float4* __restrict__ leaf_box, uint32_t leaf) {
    const float4 lo = __ldg(leaf_box + 2 * (size_t)leaf), hi = __ldg(leaf_box + 2 * (size_t)leaf + 1);
    const bool sx = r.signs & 1, sy = (r.signs >> 1) & 1, sz = (r.signs >> 2) & 1;
    float tn;
    return slab_ordered(sx ? hi.x : lo.x, sx ? lo.x : hi.x, sy ? hi.y : lo.y, sy ? lo.y : hi.y, sz ? hi.z : lo.z,
                        sz ? lo.z : hi.z, r, tn);
}

// Whether a ray gets anywhere below a TLAS leaf that its slab test keeps: the traversal's
// own tests on the way in, the bounding sphere and the four boxes of the leaf's cut (its
// BLAS's root without one).
__device__ __forceinline__ bool leaf_enters(const DevInstance* __restrict__ I, const float4* __restrict__ cut, V3 wo, V3 wd,
                                            float tmin, float tmax) {
    const float4* wp = reinterpret_cast<const float4*>(I->w2o);
    const float4 q0 = __ldg(wp), q1 = __ldg(wp + 1), q2 = __ldg(wp + 2), sph = __ldg(&I->sphere);
    const float m[12] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w, q2.x, q2.y, q2.z, q2.w};
    const V3 od = xform_dir(m, wd), oo = xform_point(m, wo);
    if (sphere_misses(oo, od, tmin, tmax, sph)) return false;
    if (!cut) cut = I->nodes4;
    LaneRay r;
    r.tmin = tmin;
    r.tmax = tmax;
    r.idir = safe_inv(od);
    set_origin(r, oo);
    near_planes(r);
    const int sx = r.signs & 1, sy = (r.signs >> 1) & 1, sz = r.signs >> 2;
    const float4 nx = __ldg(cut + sx), fx = __ldg(cut + (sx ^ 1)), ny = __ldg(cut + 2 + sy), fy = __ldg(cut + 3 - sy),
                 nz = __ldg(cut + 4 + sz), fz = __ldg(cut + 5 - sz);
    float tn;
    return slab_ordered(nx.x, fx.x, ny.x, fy.x, nz.x, fz.x, r, tn) || slab_ordered(nx.y, fx.y, ny.y, fy.y, nz.y, fz.y, r, tn) ||
           slab_ordered(nx.z, fx.z, ny.z, fy.z, nz.z, fz.z, r, tn) || slab_ordered(nx.w, fx.w, ny.w, fy.w, nz.w, fz.w, r, tn);
}

// ---------------------------------------------------------------- patches and shafts
constexpr uint32_t kPatch = 32;              // lit pixels per patch: one warp of ray generation
constexpr uint32_t kGroupSamples = 4;        // samples of one light that share a group at most
// A group's start list (Entries, vis_trace.cuh): word 0 the count (kListAll: start at the
// TLAS root), then leaves, nearest first, and their cuts; or a long list's leaves alone.
constexpr uint32_t kListAll = 0xFFFFFFFFu;
// Leaves a list may hold before its group falls back to the TLAS root, and leaves up to which
// a list's leaves get cuts and ray generation tests the way into them: on longer lists a
// ray's tests end at the leaf boxes. 720p over 201 cubes: lists, generation and traversal
// 0.473 ms (15 leaves, longer ones at the root 0.479; 31 with cuts and tests 0.498), 512x512
// over 65 0.110 (0.116), 1080p over 1024 meshes of 81,920 triangles 1.736 (1.735; 1.768). Above
// 2048 instances lists of up to 31 keep both, and lists of up to 62, unsorted, go without:
// 1021x573 over 8000 2.86 ms against 3.02 with 31 at most (46: 2.95); below, the room for long
// lists in ray generation costs what they save (720p 0.454 against 0.444). The line at 2048
// was drawn between scenes of 1024 and 8000 instances. Traces of 720p frames, us, long lists
// (with super_cap's and cut_cap's larger values) and short: 1900 instances of 1280 triangles
// 403 / 388, of 81,920 400 / 373, cubes 716 / 654; 3000: 667 / 661, 802 / 791, 709 / 612; 4096:
// 861 / 858, 948 / 941, 718 / 640; 8000: 1842 / 1900, 2283 / 2376, 850 / 773. So up to 4096 the
// short ones would be faster by up to 14 %, and above it they are only where meshes are small.
constexpr uint32_t kListCap = 62, kListShort = kEntryCuts - 1, kCutCapSmall = 15, kCutCapLarge = 31;
inline uint32_t list_cap(uint32_t instances) { return instances > 2048 ? kListCap : kListShort; }
inline uint32_t cut_cap(uint32_t instances) { return instances > 2048 ? kCutCapLarge : kCutCapSmall; }
constexpr uint32_t kSuper = 8;               // patches per block: 16x16 pixels where all are lit
// Leaves a block's shaft may reach, and nodes it may have to visit; past either its groups
// start at the TLAS root. Where the lists are long as well, long shafts pay: 1021x573 over
// 8000 instances, lists and traversal: 128 leaves 0.79 + 2.42 ms, 250 0.86 + 2.24, 400
// 0.89 + 2.17, 600 0.93 + 2.13. Over a few hundred instances a block that reaches 128 has
// groups past their own lists' room: 183x97 over 375 instances 272 us with 128, 281 with 400.
constexpr uint32_t kSuperLeaves = 400, kSuperLeavesSmall = 128, kSuperStack = 128;
inline uint32_t super_cap(uint32_t instances) { return instances > 2048 ? kSuperLeaves : kSuperLeavesSmall; }
constexpr uint32_t kCutsPerPair = 3;         // room for cuts per (light, patch) of a chunk
// Triangles above which a BLAS is descended: below, the per-ray tests of ray generation
// against its root cost no more than a cut.
constexpr uint32_t kCutPrims = 16;
constexpr uint32_t kCutVisits = 16;          // 4-wide BLAS nodes expanded per cut at most

// Bounds of a patch's shadow-ray origins O = p + N * bias (lo, hi), of their offsets
// O - p, of the pixels' normals and of their positions; the mean normal n and the least
// dot(n, O) and dot(n, O - p).
struct __align__(16) PatchRec {
    float olo[3], ohi[3], flo[3], fhi[3], nlo[3], nhi[3], plo[3], phi[3];
    float n[3], on, fn;
    float pad[3];
};
static_assert(sizeof(PatchRec) == 128, "PatchRec layout");

// One instruction for the warp (a NaN lane is left out, as by fminf / fmaxf): with five
// shuffles for each of its 26 reductions patch_kernel took 22 us at 1080p, now 14.5, and 9.7 at
// 512x512, now 6.5.
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
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
    return v;
}

// p[0, n) = 0 by the whole grid (p 16-B aligned).
__device__ __forceinline__ void clear_words(uint32_t* p, size_t n) {
    const size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x, step = gridDim.x * (size_t)blockDim.x;
    uint4* p4 = reinterpret_cast<uint4*>(p);
    for (size_t i = t; i < n / 4; i += step) p4[i] = make_uint4(0u, 0u, 0u, 0u);
    if (t < n % 4) p[n - 1 - t] = 0u;
}

// One block per block of patches, one warp per patch: the patches' bounds, then the
// block's (the unions of the boxes; the mean normal with its least dot product over the
// patches' origin and offset boxes). fminf / fmaxf leave out a NaN pixel, which has no
// ray to trace.
__global__ void __launch_bounds__(kSuper * 32) patch_kernel(SceneVis S, PatchRec* __restrict__ patches,
                                                           PatchRec* __restrict__ supers,
                                                           VisCounters* __restrict__ counters, uint32_t chunks) {
    chain_wait();
    __shared__ float s_rec[kSuper][32];
    // for the chunks' launches that follow: zero counters and hit/miss planes
    if (blockIdx.x == 0)
        for (uint32_t k = threadIdx.x; k < chunks; k += blockDim.x) counters[k] = VisCounters{};
    clear_words(S.shadow_bits, (size_t)S.shadow_slots * S.words);
    clear_words(S.ao_bits, (size_t)S.ao_samples * S.words);
    const uint32_t lit = *S.lit_count, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t count = (lit + kPatch - 1) / kPatch;
    const V3 cam = V3{S.cam[0], S.cam[1], S.cam[2]};
    const float inf = __int_as_float(0x7f800000);
    for (uint32_t sb = blockIdx.x; sb * kSuper < count; sb += gridDim.x) {
        const uint32_t w = sb * kSuper + warp, n_rec = min(kSuper, count - sb * kSuper);
        if (w < count) {
            const uint32_t j = w * kPatch + lane;
            const bool in = j < lit;
            const float4* sp = S.surf + 2 * (size_t)(in ? j : w * kPatch);
            const float4 s0 = __ldg(sp), s1 = __ldg(sp + 1);
            const V3 p = V3{s0.x, s0.y, s0.z}, N = V3{s1.x, s1.y, s1.z};
            const float bias = fmax_(length(p - cam) * 0.01f, 0.05f);   // shadow_ray's origin
            const V3 f = N * bias, o = p + f;
            V3 n = normalize(V3{warp_sum(in ? N.x : 0.f), warp_sum(in ? N.y : 0.f), warp_sum(in ? N.z : 0.f)});
            if (!finite3(n)) n = V3{0.f, 0.f, 0.f};                     // no normal bound
            const float v[8][3] = {{o.x, o.y, o.z}, {o.x, o.y, o.z}, {f.x, f.y, f.z}, {f.x, f.y, f.z},
                                   {N.x, N.y, N.z}, {N.x, N.y, N.z}, {p.x, p.y, p.z}, {p.x, p.y, p.z}};
            float r[32];
#pragma unroll
            for (int k = 0; k < 8; ++k)
#pragma unroll
                for (int a = 0; a < 3; ++a) r[3 * k + a] = k & 1 ? warp_max(v[k][a]) : warp_min(v[k][a]);
            r[24] = n.x; r[25] = n.y; r[26] = n.z;
            r[27] = warp_min(dot(n, o));
            r[28] = warp_min(dot(n, f));
            r[29] = r[30] = r[31] = 0.f;
            float out = inf;
#pragma unroll
            for (int k = 0; k < 32; ++k) out = (int)lane == k ? r[k] : out;
            reinterpret_cast<float*>(patches + w)[lane] = out;
            s_rec[warp][lane] = out;
        }
        __syncthreads();
        if (warp == 0) {   // lane = word of the record
            float out = s_rec[0][lane];
            for (uint32_t k = 1; k < n_rec; ++k) {
                const float q = s_rec[k][lane];
                out = lane >= 24 ? out + q : ((lane / 3) & 1 ? fmaxf(out, q) : fminf(out, q));
            }
            V3 m = normalize(V3{__shfl_sync(0xFFFFFFFFu, out, 24), __shfl_sync(0xFFFFFFFFu, out, 25),
                                __shfl_sync(0xFFFFFFFFu, out, 26)});
            if (!finite3(m)) m = V3{0.f, 0.f, 0.f};
            // lanes 0..7: the least dot products over patch lane's boxes
            float on = inf, fn = inf;
            if (lane < n_rec) {
                const float* q = s_rec[lane];
                on = (fminf(m.x * q[0], m.x * q[3]) + fminf(m.y * q[1], m.y * q[4])) + fminf(m.z * q[2], m.z * q[5]);
                fn = (fminf(m.x * q[6], m.x * q[9]) + fminf(m.y * q[7], m.y * q[10])) + fminf(m.z * q[8], m.z * q[11]);
            }
            on = warp_min(on);
            fn = warp_min(fn);
            if (lane >= 24)
                out = lane == 24 ? m.x : lane == 25 ? m.y : lane == 26 ? m.z : lane == 27 ? on : lane == 28 ? fn : 0.f;
            reinterpret_cast<float*>(supers + sb)[lane] = out;
        }
        __syncthreads();
    }
}

// A shaft. Axis a of a box is in reach at t where the lower line L + t l is at most the
// box's upper plane and the upper line U + t u at least its lower plane; along n, where
// N + t m is at most the box's largest dot product with n. Each is a bound of t at
// (plane - value at 0) / slope, an upper or a lower one by the slope's sign: the line has
// two coefficient pairs, t = plane * i + k for the bound that it is and a constant out of
// the way for the other (4 instructions a line without a select). The rounding of the
// products is an error of 2^-23 of the coordinates in position, far inside the boxes'
// margins, as are the reciprocals' two ulps; NaN (0 x inf planes) is dropped by min / max.
struct Line {
    float ui, uk, li, lk;   // upper bound of t, lower bound of t
};
struct Shaft {
    Line lo[3], hi[3], nrm;
    V3 n;
};

__device__ __forceinline__ Line shaft_line(float at0, float at1, bool below) {
    const float d = at1 - at0, tiny = 1e-20f;
    const float inv = __fdividef(1.0f, fabsf(d) > tiny ? d : copysignf(tiny, d));
    const float k = -at0 * inv, big = 3.0e38f;
    const bool up = (inv > 0.0f) == below;
    return up ? Line{inv, k, 0.0f, -big} : Line{0.0f, big, inv, k};
}
__device__ __forceinline__ void shaft_clip(const Line& l, float plane, float& t0, float& t1) {
    t1 = fminf(t1, __fmaf_rn(plane, l.ui, l.uk));
    t0 = fmaxf(t0, __fmaf_rn(plane, l.li, l.lk));
}

__device__ __forceinline__ bool shaft_reaches(const Shaft& s, const float lo[3], const float hi[3], float& t0_out) {
    float t0 = 0.0f, t1 = 1.0f;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        shaft_clip(s.lo[a], hi[a], t0, t1);
        shaft_clip(s.hi[a], lo[a], t0, t1);
    }
    const float sup = (fmaxf(s.n.x * lo[0], s.n.x * hi[0]) + fmaxf(s.n.y * lo[1], s.n.y * hi[1])) +
                      fmaxf(s.n.z * lo[2], s.n.z * hi[2]);
    shaft_clip(s.nrm, sup, t0, t1);
    t0_out = t0;
    return t0 <= __fmaf_rn(fabsf(t1), 0x1p-12f, t1) + 0x1p-20f;
}

// Shaft from its origin box c +- h and end box e +- g, normal bound (n, least dot at the
// origins, least dot at the ends). False when a value is not finite.
__device__ __forceinline__ bool make_shaft(Shaft& s, const float c[3], const float h[3], const float e[3],
                                           const float g[3], V3 n, float on, float en) {
    bool ok = true;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const float l0 = c[a] - h[a], h0 = c[a] + h[a], l1 = e[a] - g[a], h1 = e[a] + g[a];
        ok = ok && fabsf(l0) <= 1e18f && fabsf(h0) <= 1e18f && fabsf(l1) <= 1e18f && fabsf(h1) <= 1e18f;
        s.lo[a] = shaft_line(l0, l1, true);
        s.hi[a] = shaft_line(h0, h1, false);
    }
    s.n = n;
    s.nrm = shaft_line(on, en, true);
    return ok && finite3(n) && fabsf(on) <= 1e18f && fabsf(en) <= 1e18f;
}

__device__ __forceinline__ bool box_has_nan(const float lo[3], const float hi[3]) {
    const float l = (lo[0] + lo[1]) + lo[2], h = (hi[0] + hi[1]) + hi[2];
    return l != l || h != h;
}
// Whether the boxes of an instance's BLAS nest: its bounding sphere is finite, as every vertex
// then is (blas_radius_kernel).
__device__ __forceinline__ bool blas_nests(const DevInstance* __restrict__ I) {
    return __ldg(&I->sphere.w) < __int_as_float(0x7f800000);
}

__device__ __forceinline__ float dot_max(const float* lo, const float* hi, const float a[3], const float b[3]) {
    float s = 0.f;   // the largest dot product of a vector in [lo, hi] and one in [a, b]
#pragma unroll
    for (int k = 0; k < 3; ++k) s += fmaxf(fmaxf(lo[k] * a[k], lo[k] * b[k]), fmaxf(hi[k] * a[k], hi[k] * b[k]));
    return s;
}
__device__ __forceinline__ float abs_max3(const float* lo, const float* hi) {
    return fmaxf(fmaxf(fmaxf(fabsf(lo[0]), fabsf(hi[0])), fmaxf(fabsf(lo[1]), fabsf(hi[1]))),
                 fmaxf(fabsf(lo[2]), fabsf(hi[2])));
}

// Whether ray generation will leave out every sample of this light at every pixel of the
// patch (shadow_has_no_effect): the light is behind all of them, or they lie outside a
// spot light's cone, each by more than the rounding of the per-pixel test.
__device__ __forceinline__ bool light_has_no_effect(const luz_light& lt, const PatchRec& P) {
    float a[3], b[3];   // the vectors to the light
    if (lt.type == LUZ_LIGHT_DIRECTIONAL) {
#pragma unroll
        for (int k = 0; k < 3; ++k) a[k] = b[k] = -lt.direction[k];
    } else {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            a[k] = lt.position[k] - P.phi[k];
            b[k] = lt.position[k] - P.plo[k];
        }
    }
    const float vm = abs_max3(a, b), nm = abs_max3(P.nlo, P.nhi);
    if (dot_max(P.nlo, P.nhi, a, b) < -0x1p-12f * (vm * nm)) return true;
    const V3 col = V3{lt.color[0], lt.color[1], lt.color[2]} * lt.intensity;
    if (lt.type == LUZ_LIGHT_SPOT && lt.inner_angle > lt.outer_angle && lt.outer_angle > 0x1p-9f && finite3(col)) {
        const V3 d = normalize(V3{-lt.direction[0], -lt.direction[1], -lt.direction[2]});
        const float dd[3] = {d.x, d.y, d.z};
        float near2 = 0.f;   // squared distance of the light to the box of the positions
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const float q = fmaxf(fmaxf(a[k], -b[k]), 0.0f);
            near2 += q * q;
        }
        const float num = dot_max(dd, dd, a, b);
        if (near2 > 1e-30f && num < (lt.outer_angle - 0x1p-10f) * sqrtf(near2) * (1.0f - 0x1p-12f)) return true;
    }
    return false;
}

// The world-space shaft of a patch's shadow rays to a light, boxes grown by 2^-10 of
// their extents and 2^-16 of their coordinates. The ray of a pixel at p ends at
// O + Lv (shadow_ray) moved by at most the light's radius: dir = normalize(Lv + d) with
// d across Lv, |d| <= radius, and the chord between the two ends is shorter than d.
struct ShaftBox {
    float c[3], h[3], e[3], g[3];
    V3 n;
    float on, en;
};
__device__ __forceinline__ void world_shaft(const luz_light& lt, const PatchRec& P, ShaftBox& B) {
    float elo[3], ehi[3], en;
    const float rad = fabsf(lt.radius) * (1.0f + 0x1p-10f);
    const V3 n = V3{P.n[0], P.n[1], P.n[2]};
    if (lt.type == LUZ_LIGHT_DIRECTIONAL) {
        const V3 d = V3{lt.direction[0], lt.direction[1], lt.direction[2]};
        const V3 v = d * dot(d, normalize(-d));          // Lv = v * dist
        float lo2 = 0.f, hi2 = 0.f;                      // bounds of dist = |position - p|
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const float x0 = lt.position[k] - P.phi[k], x1 = lt.position[k] - P.plo[k];
            const float q = fmaxf(fmaxf(x0, -x1), 0.0f), w = fmaxf(fabsf(x0), fabsf(x1));
            lo2 += q * q;
            hi2 += w * w;
        }
        const float d0 = sqrtf(lo2) * (1.0f - 0x1p-20f), d1 = sqrtf(hi2) * (1.0f + 0x1p-20f);
        const float vv[3] = {v.x, v.y, v.z};
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            elo[k] = P.olo[k] + fminf(vv[k] * d0, vv[k] * d1) - rad;
            ehi[k] = P.ohi[k] + fmaxf(vv[k] * d0, vv[k] * d1) + rad;
        }
        const float nv = dot(n, v);
        en = P.on + fminf(nv * d0, nv * d1) - rad;
    } else {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            elo[k] = lt.position[k] + P.flo[k] - rad;
            ehi[k] = lt.position[k] + P.fhi[k] + rad;
        }
        en = dot(n, V3{lt.position[0], lt.position[1], lt.position[2]}) + P.fn - rad;
    }
    const float mo = abs_max3(P.olo, P.ohi), me = mo + abs_max3(elo, ehi);
    const float go = 0x1p-16f * mo + 0x1p-60f, ge = 0x1p-16f * me + 0x1p-60f;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        B.c[k] = 0.5f * (P.olo[k] + P.ohi[k]);
        B.h[k] = 0.5f * (P.ohi[k] - P.olo[k]) * (1.0f + 0x1p-10f) + go;
        B.e[k] = 0.5f * (elo[k] + ehi[k]);
        B.g[k] = 0.5f * (ehi[k] - elo[k]) * (1.0f + 0x1p-10f) + ge;
    }
    B.n = n;
    B.on = P.on - 4.0f * go;
    B.en = en - 4.0f * ge;
}

// The shaft in an instance's object space: boxes carried over by w2o (centre, and half
// extents by the absolute matrix), the normal by its cofactors. Grown by 2^-18 of the
// terms of each transform.
// Bound by issue: its sums are fused (1080p 0.329 -> 0.319 ms of culling, 4K 12.4 -> 12.0).
__device__ __forceinline__ float fma3(float a, float x, float b, float y, float c, float z, float d) {
    return __fmaf_rn(a, x, __fmaf_rn(b, y, __fmaf_rn(c, z, d)));
}
__device__ __forceinline__ V3 fma_cross(V3 a, V3 b) {
    return V3{__fmaf_rn(a.y, b.z, -(a.z * b.y)), __fmaf_rn(a.z, b.x, -(a.x * b.z)), __fmaf_rn(a.x, b.y, -(a.y * b.x))};
}
__device__ __forceinline__ bool object_shaft(const ShaftBox& B, float4 q0, float4 q1, float4 q2, Shaft& s) {
    const float w[3][4] = {{q0.x, q0.y, q0.z, q0.w}, {q1.x, q1.y, q1.z, q1.w}, {q2.x, q2.y, q2.z, q2.w}};
    float c[3], h[3], e[3], g[3];
#pragma unroll
    for (int r = 0; r < 3; ++r) {
        const float a0 = fabsf(w[r][0]), a1 = fabsf(w[r][1]), a2 = fabsf(w[r][2]), at = fabsf(w[r][3]);
        c[r] = fma3(w[r][0], B.c[0], w[r][1], B.c[1], w[r][2], B.c[2], w[r][3]);
        e[r] = fma3(w[r][0], B.e[0], w[r][1], B.e[1], w[r][2], B.e[2], w[r][3]);
        const float mo = fma3(a0, fabsf(B.c[0]), a1, fabsf(B.c[1]), a2, fabsf(B.c[2]), at);
        const float me = fma3(a0, fabsf(B.e[0]), a1, fabsf(B.e[1]), a2, fabsf(B.e[2]), at);
        h[r] = __fmaf_rn(fma3(a0, B.h[0], a1, B.h[1], a2, B.h[2], 0.0f), 1.0f + 0x1p-18f, __fmaf_rn(0x1p-18f, mo, 0x1p-60f));
        g[r] = __fmaf_rn(fma3(a0, B.g[0], a1, B.g[1], a2, B.g[2], 0.0f), 1.0f + 0x1p-18f,
                         __fmaf_rn(0x1p-18f, mo + me, 0x1p-60f));
    }
    const V3 r0 = V3{w[0][0], w[0][1], w[0][2]}, r1 = V3{w[1][0], w[1][1], w[1][2]}, r2 = V3{w[2][0], w[2][1], w[2][2]};
    const V3 c0 = fma_cross(r1, r2), c1 = fma_cross(r2, r0), c2 = fma_cross(r0, r1);
    const float det = fma3(r0.x, c0.x, r0.y, c0.y, r0.z, c0.z, 0.0f), sg = det < 0.0f ? -1.0f : 1.0f, ad = fabsf(det);
    // n' . (W x + t) = |det| n . x + n' . t with n' = sign(det) cof(W) n
    const V3 n = V3{sg * fma3(c0.x, B.n.x, c0.y, B.n.y, c0.z, B.n.z, 0.0f), sg * fma3(c1.x, B.n.x, c1.y, B.n.y, c1.z, B.n.z, 0.0f),
                     sg * fma3(c2.x, B.n.x, c2.y, B.n.y, c2.z, B.n.z, 0.0f)};
    const float nt = n.x * w[0][3] + n.y * w[1][3] + n.z * w[2][3];
    // Rounding of n' and det, each against the size of its own products (wm^2, wm^3), and
    // of the sums above: at most 2^-19 x 8 x the terms, x within the object-space boxes.
    const float t = fabsf(w[0][3]) + fabsf(w[1][3]) + fabsf(w[2][3]);
    float wm = 0.f;
#pragma unroll
    for (int r = 0; r < 3; ++r) wm = fmaxf(wm, fmaxf(fabsf(w[r][0]), fmaxf(fabsf(w[r][1]), fabsf(w[r][2]))));
    const float mo = fmaxf(fabsf(c[0]) + h[0], fmaxf(fabsf(c[1]) + h[1], fabsf(c[2]) + h[2]));
    const float me = mo + fmaxf(fabsf(e[0]) + g[0], fmaxf(fabsf(e[1]) + g[1], fabsf(e[2]) + g[2]));
    const float eo = 0x1p-16f * (wm * wm) * (wm * fabsf(B.on) + mo + t) + 0x1p-60f;
    const float ee = 0x1p-16f * (wm * wm) * (wm * fabsf(B.en) + me + t) + eo;
    return make_shaft(s, c, h, e, g, n, (ad * B.on + nt) - eo, (ad * B.en + nt) - ee);
}

// The pairs [q0, q0 + cap) of a frame in one chunk, q = virtual light x patch (patch
// fastest, patches padded to whole blocks of kSuper), and what the shafts leave
// for them. A virtual light is up to kGroupSamples samples of one light: word = first
// shadow slot | samples << 16.
struct ShaftOut {
    const PatchRec* patches;
    const PatchRec* supers;
    const uint32_t* vlights;
    uint32_t vlight_count;
    unsigned long long q0;
    uint32_t cap;                // a multiple of kSuper (0: no shadow rays here)
    uint32_t list_cap, cut_cap, super_cap;
    uint32_t* lists;             // kEntryWords per pair
    float4* cuts;                // kCutsPerPair nodes of kNode4F4 per pair
    uint4* active;               // groups to trace: (pair, first slot | samples << 16, patch, -)
    uint32_t* active_count;
};

// k-th set bit (from 0) of a 4-bit mask with more than k bits set.
__device__ __forceinline__ int nth_bit4(uint32_t m, int k) {
    if (k > 0) m &= m - 1;
    if (k > 1) m &= m - 1;
    if (k > 2) m &= m - 1;
    return __ffs(m) - 1;
}

// One warp's shared memory (rows padded by a word: the groups of a warp read the same
// column).
struct ShaftShared {
    uint32_t leaf[kSuper][kEntryCuts + 1], order[kSuper][kEntryCuts + 1];
    float t[kSuper][kEntryCuts + 1];     // entry parameters, then the leaves' cuts
    ShaftBox box[kSuper];
    uint32_t super[kSuperLeaves], stack[kSuperStack];
};

// Blocks of pairs of the chunk.
__device__ __forceinline__ uint32_t shaft_blocks(const ShaftOut& A, uint32_t patches) {
    const unsigned long long n = (unsigned long long)((patches + kSuper - 1) / kSuper) * A.vlight_count, b0 = A.q0 / kSuper;
    return b0 < n ? (uint32_t)min((unsigned long long)(A.cap / kSuper), n - b0) : 0u;
}

// Block `block` of the chunk (one virtual light, kSuper patches), by a whole warp. The TLAS
// with the block's shaft: lane l tests child l % 4 of node l / 4 of the eight taken from a
// stack. Then four lanes per patch: lane c of a group tests child c of the BLAS node its
// group expands and holds slot c of the group's cut. A cut grows by expanding its node with
// the largest box while the children that the shaft reaches fit the four slots.
__device__ __forceinline__ void shaft_block(const SceneVis& S, const ShaftOut& A, uint32_t patches, uint32_t block,
                                            ShaftShared& sm) {
    const uint32_t full = 0xFFFFFFFFu, lane = threadIdx.x & 31, c = lane & 3, g4 = lane & ~3u, grp = lane >> 2;
    const uint32_t lt_mask = (1u << lane) - 1u;
    uint32_t* super = sm.super;
    uint32_t* stack = sm.stack;
    const float inf = __int_as_float(0x7f800000);
    const uint32_t supers = (patches + kSuper - 1) / kSuper;
    const unsigned long long b0 = A.q0 / kSuper;
    const uint32_t v = (uint32_t)((b0 + block) / supers), sb = (uint32_t)((b0 + block) - (unsigned long long)v * supers);
    const uint32_t word = __ldg(A.vlights + v);
    const luz_light lt = S.lights[__ldg(S.slot_table + (word & 0xFFFFu)) & 0xFFFFu];
    uint32_t sn = 0;
    bool far = true;   // the block's list ran over
    {
        const PatchRec P = A.supers[sb];
        if (S.cull && light_has_no_effect(lt, P)) return;   // uniform in the warp
        ShaftBox B;
        Shaft s;
        world_shaft(lt, P, B);
        if (make_shaft(s, B.c, B.h, B.e, B.g, B.n, B.on, B.en)) {
            far = false;
            uint32_t sp = 1;
            if (lane == 0) stack[0] = 0u;
            __syncwarp();
            while (sp > 0) {
                const uint32_t take = min(sp, 8u);
                sp -= take;
                int ch = kEmptyChild;
                bool hit = false, odd = false;
                if (grp < take) {
                    const float* f = reinterpret_cast<const float*>(S.tlas_nodes + (size_t)stack[sp + grp] * kNode4F4) + c;
                    const float lo[3] = {__ldg(f), __ldg(f + 8), __ldg(f + 16)}, hi[3] = {__ldg(f + 4), __ldg(f + 12), __ldg(f + 20)};
                    ch = __float_as_int(__ldg(f + 24));
                    float t0;
                    hit = shaft_reaches(s, lo, hi, t0) && ch != kEmptyChild;
                    odd = box_has_nan(lo, hi);
                }
                if (__any_sync(full, odd)) { far = true; break; }
                const uint32_t lb = __ballot_sync(full, hit && ch < 0), nb = __ballot_sync(full, hit && ch >= 0);
                if (sn + __popc(lb) > A.super_cap || sp + __popc(nb) > kSuperStack) { far = true; break; }
                if (hit && ch < 0) super[sn + __popc(lb & lt_mask)] = (uint32_t)~ch;
                if (hit && ch >= 0) stack[sp + __popc(nb & lt_mask)] = (uint32_t)ch;
                sn += __popc(lb);
                sp += __popc(nb);
                __syncwarp();
            }
            if (!far && sn == 0) return;   // nothing to hit
        }
    }
    __syncwarp();
    const uint32_t patch = sb * kSuper + grp, pair = block * kSuper + grp;
    uint32_t* list = A.lists + (size_t)pair * kEntryWords;
    const PatchRec P = A.patches[min(patch, patches - 1u)];
    const bool eff = patch < patches && !(S.cull && light_has_no_effect(lt, P));
    bool all;
    uint32_t cnt = 0;
    {
        ShaftBox B;
        Shaft s;
        world_shaft(lt, P, B);
        if (c == 0) sm.box[grp] = B;
        all = !make_shaft(s, B.c, B.h, B.e, B.g, B.n, B.on, B.en) || far;
        for (uint32_t base = 0; !far && base < sn; base += 4) {
            const uint32_t leaf = super[min(base + c, sn - 1u)];
            const float4 lo4 = __ldg(S.leaf_box + 2 * (size_t)leaf), hi4 = __ldg(S.leaf_box + 2 * (size_t)leaf + 1);
            const float lo[3] = {lo4.x, lo4.y, lo4.z}, hi[3] = {hi4.x, hi4.y, hi4.z};
            float t0;
            const bool in = shaft_reaches(s, lo, hi, t0) && base + c < sn && eff;
            const uint32_t sub = (__ballot_sync(full, in) >> g4) & 15u;
            const uint32_t pos = cnt + __popc(sub & ((1u << c) - 1u));
            if (in && pos < kListShort) {
                sm.leaf[grp][pos] = leaf;
                sm.t[grp][pos] = t0;
            }
            if (in && pos >= kListShort && pos < A.list_cap) list[1 + pos] = leaf;   // a long list's, in place
            cnt += __popc(sub);
        }
    }
    all = all || cnt > A.list_cap;
    if (all) cnt = 0;
    __syncwarp();
    // leaves by their entry parameter, nearest first (long lists as they came)
    const bool longer = cnt > kListShort;
    for (uint32_t i = c; i < cnt && !longer; i += 4) {
        const float t = sm.t[grp][i];
        uint32_t rank = 0;
        for (uint32_t k = 0; k < cnt; ++k) rank += sm.t[grp][k] < t || (sm.t[grp][k] == t && k < i);
        sm.order[grp][rank] = sm.leaf[grp][i];
    }
    __syncwarp();
    // The leaves of a long list are entered at their BLAS's root.
    const uint32_t descend = cnt <= A.cut_cap ? cnt : 0u;
    for (uint32_t i = descend + c; i < cnt && !longer; i += 4) sm.t[grp][i] = __uint_as_float(0u);
    // The warp's (patch, leaf) entries, eight at a time: entry e belongs to the group g with
    // first[g] <= e < first[g + 1].
    uint32_t cuts = 0;               // of the warp
    uint32_t first = 0, total = 0;   // of this lane's own group; all entries
#pragma unroll
    for (uint32_t g = 0; g < kSuper; ++g) {
        const uint32_t n = __shfl_sync(full, descend, (int)g * 4);
        first += g < grp ? n : 0u;
        total += n;
    }
    for (uint32_t e0 = 0; e0 < total; e0 += kSuper) {
        const uint32_t e = e0 + grp;
        uint32_t own = 0;   // the entry's group, and its leaf there
#pragma unroll
        for (uint32_t g = 1; g < kSuper; ++g) own += e >= __shfl_sync(full, first, (int)g * 4);
        const uint32_t i = e - __shfl_sync(full, first, (int)own * 4);
        bool use = e < total, shaft = false;
        Shaft so;
        const float4* nodes = nullptr;
        if (use) {
            const DevInstance* I = S.instances + sm.order[own][i];
            const uint4 meta = __ldg(reinterpret_cast<const uint4*>(&I->custom_index));
            use = (meta.y & 0xFFu) != 0 && meta.w > 0;   // else never hit
            const float4* wp = reinterpret_cast<const float4*>(I->w2o);
            shaft = use && meta.w > kCutPrims && blas_nests(I) && object_shaft(sm.box[own], __ldg(wp), __ldg(wp + 1), __ldg(wp + 2), so);
            nodes = I->nodes4;
        }
        float lx = inf, hx = -inf, ly = inf, hy = -inf, lz = inf, hz = -inf;   // this lane's slot
        int ch = kEmptyChild;
        bool run = shaft, whole = true;   // whole: still the BLAS root's own slots
        int node = 0, slot = -1;
        for (uint32_t it = 0; it < kCutVisits && __any_sync(full, run); ++it) {
            float nlx = 0.f, nhx = 0.f, nly = 0.f, nhy = 0.f, nlz = 0.f, nhz = 0.f;
            int nch = kEmptyChild;
            bool keep = false;
            if (run) {
                const float* f = reinterpret_cast<const float*>(nodes + (size_t)node * kNode4F4) + c;
                nlx = __ldg(f); nhx = __ldg(f + 4); nly = __ldg(f + 8); nhy = __ldg(f + 12);
                nlz = __ldg(f + 16); nhz = __ldg(f + 20);
                nch = __float_as_int(__ldg(f + 24));
                const float lo[3] = {nlx, nly, nlz}, hi[3] = {nhx, nhy, nhz};
                float t0;
                keep = shaft_reaches(so, lo, hi, t0) && nch != kEmptyChild;
            }
            const uint32_t kb = (__ballot_sync(full, keep) >> g4) & 15u;
            const uint32_t lb = (__ballot_sync(full, nch != kEmptyChild) >> g4) & 15u;
            const uint32_t ob = (__ballot_sync(full, ch != kEmptyChild) >> g4) & 15u;
            const uint32_t fr = (~ob & 15u) | (slot >= 0 ? 1u << slot : 0u);   // slots to fill
            const int m = __popc(kb);
            run = run && m <= __popc(fr);   // else the children do not fit: the node stays
            const int rank = __popc(fr & ((1u << c) - 1u));
            const bool mine = run && ((fr >> c) & 1u), take = mine && rank < m;
            const int src = (int)g4 + (take ? nth_bit4(kb, rank) : (int)c);
            nlx = __shfl_sync(full, nlx, src); nhx = __shfl_sync(full, nhx, src);
            nly = __shfl_sync(full, nly, src); nhy = __shfl_sync(full, nhy, src);
            nlz = __shfl_sync(full, nlz, src); nhz = __shfl_sync(full, nhz, src);
            nch = __shfl_sync(full, nch, src);
            if (run) whole = whole && slot < 0 && kb == lb;
            if (mine) {
                ch = take ? nch : kEmptyChild;
                lx = take ? nlx : inf; hx = take ? nhx : -inf;
                ly = take ? nly : inf; hy = take ? nhy : -inf;
                lz = take ? nlz : inf; hz = take ? nhz : -inf;
            }
            const float x = hx - lx, y = hy - ly, z = hz - lz;
            float area = ch >= 0 ? x * y + y * z + z * x : -1.0f;
            int best = (int)c;
#pragma unroll
            for (int o = 1; o <= 2; o <<= 1) {
                const float a2 = __shfl_xor_sync(full, area, o);
                const int b2 = __shfl_xor_sync(full, best, o);
                if (a2 > area || (a2 == area && b2 < best)) { area = a2; best = b2; }
            }
            const int next = __shfl_sync(full, ch, (int)g4 + best);
            if (run) {
                slot = best;
                node = next;
                run = area >= 0.0f;
            }
        }
        const uint32_t ob = (__ballot_sync(full, ch != kEmptyChild) >> g4) & 15u;
        use = use && !(shaft && !whole && ob == 0u);
        // the cuts of a block of pairs have room for kCutsPerPair each; past it, the BLAS root
        const bool want = use && shaft && !whole;
        const uint32_t wb = __ballot_sync(full, want && c == 0);
        uint32_t cut = cuts + __popc(wb & ((1u << g4) - 1u)) + 1u;
        cuts += __popc(wb);
        if (!want || cut > kCutsPerPair * kSuper) {
            cut = 0;
        } else {
            cut += block * (kCutsPerPair * kSuper);
            float* o = reinterpret_cast<float*>(A.cuts + (size_t)(cut - 1u) * kNode4F4) + c;
            o[0] = lx; o[4] = hx; o[8] = ly; o[12] = hy; o[16] = lz; o[20] = hz;
            o[24] = __int_as_float(ch);
        }
        if (e < total && c == 0) sm.t[own][i] = __uint_as_float(use ? cut : 0xFFFFFFFFu);
    }
    __syncwarp();
    const uint32_t most = min(__reduce_max_sync(full, cnt), kListShort);
    uint32_t kept = 0;
    for (uint32_t base = 0; base < most; base += 4) {
        const uint32_t cut = base + c < min(cnt, kListShort) ? (longer ? 0u : __float_as_uint(sm.t[grp][base + c])) : 0xFFFFFFFFu;
        const bool in = cut != 0xFFFFFFFFu;
        const uint32_t sub = (__ballot_sync(full, in) >> g4) & 15u;
        const uint32_t pos = kept + __popc(sub & ((1u << c) - 1u));
        if (in) {
            list[1 + pos] = longer ? sm.leaf[grp][base + c] : sm.order[grp][base + c];
            if (!longer) list[kEntryCuts + pos] = cut;
        }
        kept += __popc(sub);
    }
    if (c == 0) list[0] = all ? kListAll : (longer ? cnt : kept);
    // One entry of the active list per surviving pair, one atomic per warp.
    const bool trace = c == 0 && eff && (all || kept > 0);   // (a long list keeps all)
    const uint32_t m = __ballot_sync(full, trace);
    if (m) {
        uint32_t base = 0;
        if (lane == 0) base = atomicAdd(A.active_count, __popc(m));
        base = __shfl_sync(full, base, 0);
        if (trace) A.active[base + __popc(m & lt_mask)] = make_uint4(pair, word, patch, 0u);
    }
}

}  // namespace luz
