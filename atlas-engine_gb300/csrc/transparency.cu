// The transparency traversal variants (include/atlas_rt.h,
// ae_rt_trace_scene_*_transparency):
//   HitClosestTransparency  data/shader/raytracer/bvh.hsh:275-357
//                           (+ CheckLeafClosestTransparency :106-138)
//   HitAnyTransparency      data/shader/raytracer/bvh.hsh:443-524
//                           (+ CheckLeafTransparency :140-170)
// over the context's two-level scene: the OPACITY instances of the traversal
// kernel (trace_kernels.cuh).
#include "atlas_rt.h"
#include "context.cuh"
#include "trace_kernels.cuh"
#include "texture.cuh"

#include <algorithm>

using namespace atlas::rt::host;
using namespace atlas::rt::dev;

namespace {

// 128 stack entries per lane, or the 32 in shared memory alone for scenes of
// fewer levels; 128 threads, 7 CTAs an SM (72 registers; at 8 CTAs the spills
// cost more: a 321 x 181 real-time frame over alpha-tested boxes takes 362
// instead of 344 us).  The same frame took 393 us with one thread per ray and
// a local-memory stack: a warp then kept its 32 rays to the end, and the
// launch waited, 12 warps an SM and half of the SMs done, for the longest.
template <bool ANY, int SPILL, bool FEW>
void* KernelFor() {
    return reinterpret_cast<void*>(
        &trace_kernel<ANY, false, MODE_SCENE, 4, 32, SPILL, 7, false, false, 0, false, false, true, FEW>);
}

template <bool FEW>
void* Pick(bool any, bool shallow) {
    return any ? (shallow ? KernelFor<true, 0, FEW>() : KernelFor<true, 96, FEW>())
               : (shallow ? KernelFor<false, 0, FEW>() : KernelFor<false, 96, FEW>());
}

}  // namespace

ae_rt_status atlas::rt::host::TraceTransparency(ae_rt_ctx* ctx, bool any, const ae_packed_ray* rays, uint32_t n,
                                                float tmin, float tmax, uint32_t cull_mask, void* out, void* stream,
                                                const uint32_t* count_dev, bool per_ray_tmax, uint32_t* counter) {
    if (!ctx) return AE_RT_INVALID_ARG;
    if (!ctx->scene_ready) return Fail(ctx, AE_RT_INVALID_ARG, "no scene has been set");
    if (n == 0) return AE_RT_OK;
    if (!rays || !out) return Fail(ctx, AE_RT_INVALID_ARG, "null ray or result buffer");
    if (n > (1u << 30)) return Fail(ctx, AE_RT_INVALID_ARG, "more than 2^30 rays in one call");
    if (count_dev && (!IsDevicePointer(rays) || !IsDevicePointer(out)))
        return Fail(ctx, AE_RT_INVALID_ARG, "queue traces take device buffers");
    for (const DeviceMesh& m : ctx->meshes)
        if (m.n_nodes > 0 && !m.shading)
            return Fail(ctx, AE_RT_INVALID_ARG, "transparency queries need the meshes' shading triangles");
    AE_CUDA(ctx, cudaSetDevice(ctx->device));
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const size_t rb = size_t(n) * sizeof(ae_packed_ray), ob = size_t(n) * (any ? sizeof(float) : sizeof(ae_hit));
    const bool rays_dev = IsDevicePointer(rays), out_dev = IsDevicePointer(out);
    const void* d_rays = rays;
    void* d_out = out;
    if (!rays_dev) {
        AE_CUDA(ctx, ctx->rays_in.ensure(rb));
        AE_CUDA(ctx, cudaMemcpyAsync(ctx->rays_in.ptr, rays, rb, cudaMemcpyHostToDevice, s));
        d_rays = ctx->rays_in.ptr;
    }
    if (!out_dev) {
        AE_CUDA(ctx, ctx->results_out.ensure(ob));
        d_out = ctx->results_out.ptr;
    }
    TraceParams p{};
    p.tlas = ctx->d_tlas;
    p.n_tlas = ctx->n_tlas;
    p.instances = ctx->d_instances;
    p.n_instances = ctx->n_instances;
    p.meshes = ctx->d_mesh_table;
    p.n_meshes = ctx->n_mesh_table;
    p.materials = ctx->d_materials;
    p.n_materials = ctx->n_materials;
    p.textures.pool = ctx->d_tex_pool;
    p.textures.desc = static_cast<const TexDesc*>(ctx->d_tex_desc);
    p.textures.n = ctx->n_textures;
    p.rays = static_cast<const float4*>(d_rays);
    p.n_rays = n;
    p.n_rays_dev = count_dev;
    p.per_ray_tmax = per_ray_tmax ? 1u : 0u;
    p.tmin = tmin;
    p.tmax = tmax;
    p.cull_mask = cull_mask;
    p.max_steps = ctx->max_steps_cfg ? ctx->max_steps_cfg : ctx->scene_steps;
    p.hits = any ? nullptr : static_cast<float4*>(d_out);
    p.transparency = any ? static_cast<float*>(d_out) : nullptr;
    p.error_word = ctx->d_counter + 1;
    p.work_counter = counter;
    p.refill_steps = ctx->refill_steps;
    p.spread_warps = SpreadWarps(ctx);
    const bool shallow = ctx->scene_depth < 32u;
    // A caller's own queries take no work counter, of which a context has only
    // a few in rotation: any number of them may be in flight, on as many
    // streams, and captured ones beside their replays.  Each warp holds its rays
    // once, in as many blocks as that takes.  (With a counter of the rotation,
    // which the seventh launch in flight cleared under the first, and its memset:
    // a ray that misses everything 7 us against 5, 58,000 random rays 58 / 55
    // against 55 / 52, two million camera rays 297 / 269 against 291 / 282, two
    // million random ones 420 / 404 against 548 / 551, closest / any.  Ranges of
    // 2 to 16 rays a lane win back a part of the last and lose up to twice the
    // time on the camera's.)
    void* fn = counter ? Pick<false>(any, shallow) : Pick<true>(any, shallow);
    uint32_t grid = GridFor(ctx, fn, n, 128);
    if (!counter) grid = std::max(grid, n / 128 + (n % 128 ? 1u : 0u));
    void* args[] = { &p };
    AE_CUDA(ctx, LaunchNext(static_cast<const void*>(fn), grid, 128, s, args));
    if (!out_dev) AE_CUDA(ctx, cudaMemcpyAsync(out, d_out, ob, cudaMemcpyDeviceToHost, s));
    if (!out_dev || !rays_dev) return ae_rt_synchronize(ctx, stream);
    return AE_RT_OK;
}

extern "C" {

ae_rt_status ae_rt_trace_scene_closest_transparency(ae_rt_ctx* ctx, const ae_packed_ray* rays, uint32_t n_rays,
                                                    float tmin, float tmax, uint32_t cull_mask, ae_hit* out,
                                                    void* stream) {
    return TraceTransparency(ctx, false, rays, n_rays, tmin, tmax, cull_mask, out, stream);
}

ae_rt_status ae_rt_trace_scene_any_transparency(ae_rt_ctx* ctx, const ae_packed_ray* rays, uint32_t n_rays,
                                                float tmin, float tmax, uint32_t cull_mask, float* transparency,
                                                void* stream) {
    return TraceTransparency(ctx, true, rays, n_rays, tmin, tmax, cull_mask, transparency, stream);
}

}  // extern "C"
