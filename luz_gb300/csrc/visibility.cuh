// visibility.cuh — inputs of the visibility kernels, shared with the batch driver.
#pragma once
#include "internal.cuh"

namespace luz {

// Per-scene inputs of the visibility pass (a device array in batch mode).
struct SceneVis {
    const float4* tlas_nodes;
    uint32_t tlas_node_count;
    uint32_t instance_count;
    const DevInstance* instances;
    const float4* surf;
    const uint32_t* lit_count;
    const luz_light* lights;
    const uint32_t* slot_table;
    uint32_t shadow_slots, ao_samples;
    float cam[3];
    float ao_min, ao_max;
    int sampler, frame;
    int cull;                 // leave out shadow rays that cannot change the light pass's output
    uint32_t width, words;
    uint32_t* shadow_bits;
    uint32_t* ao_bits;
    const float4* leaf_box;      // TLAS leaf boxes (lo, hi), leaf order (visibility_kernel only)
};

struct VisCommon {
    const uint8_t* blue_noise;
    uint32_t bn_size;
    unsigned long long* work_counter;
    uint32_t* status;
    uint32_t refill, steps, smem_nodes;
    uint32_t step_cap;        // traversal steps per ray before it is ended (LUZ_DEV_TRAVERSAL_CAP)
};

// The context's visibility launch shape (the library defaults until one is set), of a
// single scene's traces and of batches.
const VisTuning& vis_tuning(const luz_ctx* ctx);
const VisTuning& batch_tuning(const luz_ctx* ctx);
// Launch-independent inputs of the visibility kernels (blue noise, status word, shape).
VisCommon make_vis_common(luz_ctx* ctx, const VisTuning& tu, unsigned long long* work_counter);
SceneVis make_scene_vis(const luz_frame* f, const luz_tlas* t, int frame_index);
// Boxes of the last TLAS build's leaves (leaf order, lo / hi float4 pairs).
const float4* tlas_leaf_boxes(const luz_tlas* t);
luz_status clear_visibility(luz_ctx* ctx, luz_frame* f);
// Allocates what the traces of frame f over t need from the scratch.
luz_status reserve_visibility(luz_ctx* ctx, const luz_frame* f, const luz_tlas* t, VisScratch& scratch);
// Bytes of it where a chunk has `ray_chunk` rays at most.
size_t visibility_bytes(const luz_frame* f, const luz_tlas* t, uint32_t ray_chunk);
luz_status launch_visibility(luz_ctx* ctx, luz_frame* f, const luz_tlas* t, int frame_index, unsigned long long* d_stats,
                             VisScratch& scratch);
luz_status launch_visibility_count(luz_ctx* ctx, const SceneVis* d_scenes, uint32_t n, unsigned long long* d_offsets,
                                   unsigned long long* work_counter, unsigned long long* d_stats);

}  // namespace luz
