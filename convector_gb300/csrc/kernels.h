// Launchers of the device kernels (kernels.cu), used by the C-ABI (capi.cu).
#pragma once
#include <cuda_runtime.h>

#include "../../include/convector_gpu.h"
#include "layout.cuh"
#include "wavefront.cuh"

namespace cvx {

// SM count of the calling thread's current device (cached per device).
int sm_count();
// The traversal stack limit (traverse.cuh c_stack_limit) on the current
// device, for the kernels of kernels.cu and of wavefront.cu.
cudaError_t set_stack_limit(int entries);
cudaError_t set_stack_limit_wave(int entries);
cudaError_t upload_tables(const uint16_t* rcp, const uint16_t* rsqrt);
cudaError_t upload_tables_wave(const uint16_t* rcp, const uint16_t* rsqrt);
cudaError_t launch_prep_geom(const cvx_triangle* tris, uint32_t n, float4* geom, TriShade* shade, cudaStream_t st);
cudaError_t launch_prep_wide(const float4* nodes, uint32_t n_pairs, float4* wide, cudaStream_t st);
cudaError_t launch_prep_lights(const cvx_triangle* tris, const uint32_t* ds, uint32_t n, float4* lights,
                               cudaStream_t st);
// The six ray components of a nearest-hit query (origin x, y, z, direction
// x, y, z), each an array of n floats. The pointers may be device memory or,
// where the device shares the host's page tables, host memory read in place.
struct RayCols {
    const float* c[6];
};
inline RayCols soa_cols(const float* rays, uint32_t n) {  // one (6, n) device array
    RayCols r;
    for (int k = 0; k < 6; k++) r.c[k] = rays + (size_t)k * n;
    return r;
}

// Whether a query takes the direct kernels (one packet per warp, one ray per lane):
// up to kDirectRays rays (packets on a scene without wide records up to
// kDirectPairRays), unless a launch shape of the persistent kernels is set (times
// at k_intersect_warp). They store to `err`, which may then be page-locked host
// memory, and use no counter behind it; the others claim from err[1], which must be
// device memory. They have no stack in shared memory.
constexpr uint32_t kDirectRays = 262144, kDirectPairRays = 32768;
inline bool direct_query(const DeviceScene& s, uint32_t n, bool packet, uint32_t blocks_per_sm) {
    return n <= (packet && !s.wide ? kDirectPairRays : kDirectRays) && blocks_per_sm == 0;
}
// shared_stack: stack entries of each lane kept in shared memory by the
// persistent single-ray kernel at 8 blocks per SM (0, 4, 8 or 12; other launch
// shapes keep 8).
constexpr uint32_t kQueryStackDefault = 0;
cudaError_t launch_intersect(const DeviceScene& s, const RayCols& rays, uint32_t n, float far_dist, bool packet,
                             float* t_out, int32_t* tri_out, uint32_t* counters, uint32_t* err, uint32_t block,
                             uint32_t blocks_per_sm, cudaStream_t st, uint32_t shared_stack = kQueryStackDefault);
// Single-launch form of single-ray frames and waves in the per-group RNG
// order: paths per lane with ray refill (k_render_refill, k_wave_refill), or
// one octet per 8-pixel group (k_render_group, k_wave_fused). CVX_REFILL_ALL
// and CVX_REFILL_NONE choose. By default the tree's depth and the frame's size
// decide: refill keeps lanes busy where paths are long and many, the octets keep
// warps of neighbouring camera rays together, and start a frame that does not
// fill the GPU sooner. Measured, octet against refill, us per frame:
//                            320x184    640x368    900x516     1280x736    1920x1080
//   tube, 70 levels         1002/790  1409/1056  2065/1286   3492/1921   6866/3446
//   icosphere, 28 levels     243/259    448/398    748/590   1372/991    2869/1920
//   room, 19 levels          144/174    217/239    360/302    659/485    1335/937
//   open scene, 21 levels    117/137    144/179    192/219    280/306     528/535
//   open scene, 16 levels     68/85      87/105     97/122    124/150     185/228
// (480x276: icosphere 324/335.) The open scene of 21 levels loses 1-14 % by the
// line at 18 levels, a closed room gains 16-30 %; nothing in the tree tells them
// apart. For a wave, whether at least half of its groups belong to scenes of
// kRefillMinDepth levels (32 open scenes of 11 to 20 levels, 6.1/7.7 ms).
constexpr uint32_t kRefillMinDepth = 25;
inline bool path_refill_frames(uint32_t refill_mode, uint32_t depth, uint64_t pixels) {
    if (refill_mode != CVX_REFILL_AFTER_CAMERA) return refill_mode == CVX_REFILL_ALL;
    return depth > 40 || (depth >= kRefillMinDepth && pixels >= 160000) || (depth >= 18 && pixels >= 400000);
}
// deep_groups of a wave's groups belong to scenes of kRefillMinDepth levels or more.
inline bool path_refill_wave(uint32_t refill_mode, uint32_t deep_groups, uint32_t groups) {
    return refill_mode == CVX_REFILL_ALL ||
           (refill_mode == CVX_REFILL_AFTER_CAMERA && 2ull * deep_groups >= (uint64_t)groups && groups > 0);
}

// group_em: one word per 8-pixel group; given, a single-ray frame in the
// per-group RNG order takes the per-lane path refill form (k_render_refill),
// else one octet per group (k_render_group). work (3 words, zeroed by the
// caller; needs group_em): the counting form of k_render_refill adds the
// frame's boxes tested, triangles tested and light-PDF shading steps.
cudaError_t launch_render(const DeviceScene& s, const DeviceCamera& cam, uint32_t w, uint32_t h, uint32_t frame,
                          bool packet, bool patch_order, uint32_t* rgba, uint32_t* gbuf, float* color, float* accum,
                          unsigned long long* rays, uint32_t* err, uint32_t block, bool debug, cudaStream_t st, uint32_t patch = 32,
                          const uint32_t* patches = nullptr, uint32_t n_patches = 0, uint32_t* group_em = nullptr,
                          unsigned long long* work = nullptr, uint32_t samples = 1, float* sample_color = nullptr);
// Frames with the per-lane path refill (group_em set, single-ray traversal,
// per-group RNG order) may render `samples` > 1 frames, frame .. frame +
// samples - 1, in one launch, accumulating them into `accum` in frame order
// (bit-identical to one launch per frame); color and gbuf then hold the last
// frame's values, and sample_color holds 3 * w * h * (samples - 1) floats.
// Other forms take samples == 1 only.
cudaError_t launch_resolve(const float* accum, uint32_t npx, float factor, uint32_t* rgba, cudaStream_t st);
// refill_from: first bounce whose single-ray traversal uses ray refill (the
// earlier ones traverse one octet per group); packet traversal ignores it.
cudaError_t launch_wave(const Job* jobs, const WaveHeader* hdr, const DeviceScene* scenes, const WaveState& st,
                        const WaveOutputs& out, bool packet, uint32_t blocks_per_sm, uint32_t refill_from, bool deep,
                        cudaStream_t stream);
// The fused (megakernel) form of a wave: one persistent launch.
// deep: a scene of the wave is deeper than 40 levels (claim threshold 8, else 16)
cudaError_t launch_wave_fused(const Job* jobs, const WaveHeader* hdr, const DeviceScene* scenes,
                              const WaveOutputs& out, bool packet, uint32_t blocks_per_sm, bool deep, bool wide,
                              cudaStream_t stream);
cudaError_t launch_resolve_multi(const ResolveItem* items, uint32_t n_items, const float* accum, uint32_t* rgba,
                                 cudaStream_t stream);
// After a wave with sample slots (WaveOutputs::samples): adds each item's
// slots to its accumulator pixels in sample order.
cudaError_t launch_accumulate_slots(const SlotItem* items, uint32_t n_items, float* accum, const float* samples,
                                    cudaStream_t stream);

}  // namespace cvx
