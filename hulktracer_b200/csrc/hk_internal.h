// hk_internal.h -- launch descriptors shared between the host API and the
// kernel translation units.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#include "../../include/hulkcuda.h"

namespace hk {

struct TriRec;

// one scene of a batched launch (device table entry)
struct SceneDesc {
    const uint2 *nodes;
    const uint32_t *refs;
    const TriRec *tris;
    const uint32_t *ropes;
    const float4 *cbox;
    float box[8];
    uint32_t nn;        // compact nodes (ropes legs bound)
    uint32_t ntris;
    uint32_t pad[2];
};

struct TraceLaunch {
    const uint2 *nodes;
    const uint32_t *refs;
    const TriRec *tris;
    const float4 *rays;
    hk_hit *hits;
    uint32_t n;                 // ray count (ignored when n_dev != nullptr)
    const uint32_t *n_dev;      // device-side ray count, or nullptr
    uint32_t ntris;
    const float *box;           // device pointer, 8 floats
    uint32_t *fetch;            // ray-batch counter
    bool fetch_clear;           // it is zero already (else launch_trace clears it)
    unsigned long long *counters;
    uint32_t *err;
    uint32_t stack_depth;
    uint32_t max_steps;
    int variant;
    bool count;
    bool occlusion;             // shadow rays: origin w = light distance, stop at the first hit closer than it
    uint32_t *leaf_out;         // ropes: per ray, the leaf its traversal ended in (a start hint), or nullptr
    uint32_t refill;            // idle lanes before a warp takes new rays (0: kRefillBatch / kRefillRays)
    int block;
    int grid;                   // blocks, or 0: one resident wave on sm_count SMs
    int sm_count;
    // ropes
    const uint32_t *ropes;      // 6 per node
    const float4 *cbox;         // 2 per node (min, max)
    uint32_t rope_nn;           // compact node count
    const uint32_t *rope_nn_dev;
    // batch mode (scenes != nullptr)
    const SceneDesc *scenes;
    const uint32_t *ray_offsets;
    uint32_t nscenes;
    uint32_t *remaining;
    unsigned long long *done_ns;
    unsigned long long *start_ns;
};

// The trace kernel is compiled for at most kTraceMaxBlock threads per block
// (its __launch_bounds__) and launched without opting in to more than the
// default 48 KB of dynamic shared memory.
constexpr uint32_t kTraceMaxBlock = 256;
constexpr size_t kTraceMaxSmem = 48 * 1024;

// Idle lanes that a warp gathers before it takes new rays. A fresh ray descends
// from the root while its neighbours follow ropes a step or two, so lanes
// refilled one by one hold the others at nearly every step; idle lanes still
// share the leaf tests meanwhile. Camera and shadow rays come in tiles that run
// alike: a warp finishes all 32 first (six-light frame 2,095 us at one, 1,974 at
// 8, 1,929 at 16, 1,883 at 32). Rays of unknown order: 8 (a million incoherent
// rays 710 us at one, 677 at 8, 683 at 16, 820 at 32); batches, whose lanes
// also wait for memory longer: 4.
constexpr uint32_t kRefillRays = 8, kRefillBatch = 4, kRefillCoherent = 32, kRefillMirror = 24;

// Whether an instantiation shares its warp's leaf tests (coop_leaf, one
// 8-byte slot per thread): every closest-hit kernel but brute force and the
// batches' shared-memory stack, whose ring may fill the shared memory alone;
// occlusion rays of the stack variants too (a 24,576-triangle frame's take 45
// us less), not of ropes, where stopping at the first hit closer than the light
// saves more (a six-light frame's would take 145 us more). Counting launches
// of occlusion rays take the closest-hit kernel. The kernel and the launcher
// both use this.
__host__ __device__ constexpr bool trace_coop_slots(int variant, bool batch, bool any) {
    if (variant == HK_TRACE_BRUTE) return false;
    return batch ? variant != HK_TRACE_SMEMSTACK : !(any && variant == HK_TRACE_ROPES);
}

// Blocks of kTraceMaxBlock threads that an instantiation is compiled to keep
// resident on an SM (its __launch_bounds__; smaller blocks in proportion).
__host__ __device__ constexpr uint32_t trace_resident_blocks(int variant, bool batch, bool any) {
    if (batch) return variant == HK_TRACE_BRUTE ? 5u : 4u;
    return trace_coop_slots(variant, batch, any) ? 5u : 6u;
}

// dynamic shared memory of one trace launch: the shared-memory ring of
// SMEMSTACK (12 bytes per thread and ring entry) plus the coop_leaf slots
__host__ __device__ constexpr size_t trace_smem_bytes(int variant, uint32_t block, uint32_t stack_depth, bool batch,
                                                      bool occlusion, bool count) {
    return (variant == HK_TRACE_SMEMSTACK ? (size_t)stack_depth * block * 12 : 0) +
           (trace_coop_slots(variant, batch, occlusion && !count) ? (size_t)block * 8 : 0);
}

cudaError_t launch_trace(const TraceLaunch &L, cudaStream_t s);
// load the closest-hit and occlusion kernels of one variant (single scene, not
// counting) into the current device's context without launching them
cudaError_t preload_trace_kernels(int variant);

// hk_shade.cu
cudaError_t launch_precompute(const float4 *verts, const uint4 *tris, uint32_t nt, TriRec *out,
                              cudaStream_t s);
cudaError_t launch_cache_to_rec(const float *cache16, const float4 *verts, const uint4 *tris, uint32_t nt,
                                TriRec *out, cudaStream_t s);
cudaError_t launch_rec_to_cache(const TriRec *rec, uint32_t nt, float *cache16, cudaStream_t s);
// box_ord: kBoxWords words, set once by launch_box_reset; box: the transformed
// scene's box, or null (the caller's own box stays)
constexpr uint32_t kBoxWords = 8;
cudaError_t launch_box_reset(uint32_t *box_ord, cudaStream_t s);
cudaError_t launch_transform(const float4 *rest, const uint32_t *part, uint32_t nv, const float *mats12, float4 *out,
                             uint32_t *box_ord, float *box, int sm_count, cudaStream_t s);
// a frame's counters, cleared by its camera-ray launch: the traces' ray-batch
// counters and the lists' lengths
enum FrameCounter : uint32_t { kFetchPrimary, kFetchMirror, kFetchShadow, kShadowCount, kMirrorCount, kFrameCounters };
// rays of rows row0 .. row0 + h - 1 of a w x full_h image (full_h 0: h);
// counters: kFrameCounters words to clear, or null
cudaError_t launch_camera_rays(const float *cam16_dev, uint32_t w, uint32_t h, float4 *rays, cudaStream_t s,
                               bool tiled = false, uint32_t row0 = 0, uint32_t full_h = 0,
                               uint32_t *counters = nullptr);
// scount: the list's length, zero before
cudaError_t launch_shadow_rays(const float4 *rays, const hk_hit *hits, const TriRec *tris, uint32_t npix,
                               const float *lights_dev, uint32_t nl, const uint32_t *leaf_hint, float4 *srays,
                               uint32_t *slot, uint32_t *scount, cudaStream_t s);
cudaError_t launch_shade_cpu(const float4 *rays, const hk_hit *hits, const TriRec *tris, uint32_t npix,
                             const float *lights_dev, uint32_t nl, const uint32_t *slot, const hk_hit *shits,
                             uint32_t *rgba, cudaStream_t s, uint32_t w = 0, bool tiled = false);
cudaError_t launch_hit4(const hk_hit *hits, const TriRec *tris, uint32_t n, float4 *hit4, cudaStream_t s);
// load the kernels of the trace + shadow + CPU-shading pipeline's shading side
cudaError_t preload_render_kernels();
cudaError_t launch_shade_picture(const float4 *rays, const float4 *hit4, uint32_t n, const float *lights_dev,
                                 uint32_t nl, uint32_t *rgba, cudaStream_t s, uint32_t w = 0, bool tiled = false);

cudaError_t launch_mirror_rays(const float4 *rays, const hk_hit *hits, const TriRec *tris, const uint8_t *mirror,
                               uint32_t npix, float4 *mrays, uint32_t *mslot, uint32_t *mcount, cudaStream_t s);
cudaError_t launch_mirror_merge(const float4 *rays, const hk_hit *hits, const uint32_t *mslot, const float4 *mrays,
                                const hk_hit *mhits, uint32_t npix, float4 *srays, hk_hit *shits, cudaStream_t s);

}  // namespace hk
