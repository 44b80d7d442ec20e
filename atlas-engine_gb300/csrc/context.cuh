// Device context of the C ABI, shared by the library's translation units.
#pragma once

#include "atlas_rt.h"
#include "trace_kernels.cuh"

#include <cuda_runtime.h>

#include <mutex>
#include <string>
#include <tuple>
#include <vector>

struct ae_rc;

namespace atlas::rt::host {

struct DeviceMesh {
    float4* nodes = nullptr;
    float4* tris = nullptr;
    float4* shading = nullptr;
    uint32_t n_nodes = 0;
    uint32_t n_tris = 0;
    bool transparent = false;   // a shading triangle's opacity (d2.w) is not 1: opacity texture or partial
    uint32_t depth = 0;         // inner-node levels on the longest root-to-leaf path (stack entries it can need)
};

// A node in the library's device order (load_node in trace_kernels.cuh) from
// the engine's layout (ae_rt_mesh_get_bvh: back).  padding0 is the node's
// `slow` word.
struct PairedNode {
    uint32_t w[16];
};
static_assert(sizeof(PairedNode) == sizeof(ae_bvh_node), "node size");

__host__ __device__ inline PairedNode PairNode(const ae_bvh_node& e) {
    PairedNode p;
    const uint32_t* src = reinterpret_cast<const uint32_t*>(&e);
    for (int k = 0; k < 16; k++) p.w[k] = src[dev::engine_node_word(k)];
    return p;
}

// Grow-only device scratch buffer.
struct Scratch {
    void* ptr = nullptr;
    size_t bytes = 0;
    cudaError_t ensure(size_t want) {
        if (want <= bytes) return cudaSuccess;
        if (ptr) cudaFree(ptr);
        ptr = nullptr;
        bytes = 0;
        cudaError_t e = cudaMalloc(&ptr, want);
        if (e == cudaSuccess) bytes = want;
        return e;
    }
    void release() {
        if (ptr) cudaFree(ptr);
        ptr = nullptr;
        bytes = 0;
    }
};


}  // namespace atlas::rt::host

struct ae_rt_ctx {
    int device = 0;
    int sm_count = 0;
    uint32_t blocks_per_sm = 0;         // 0: occupancy of each kernel
    int shape = 0;                      // index into kShapes
    uint32_t threads = 128;
    uint32_t max_steps_cfg = 0;
    uint32_t refill_steps = 0;
    bool count_fetches = false;
    bool near_ties = true;            // complete near-tie detection on closest-hit traces
    bool staged_rays = false;         // ray tiles through shared memory by bulk copy
    bool approximate = false;   // AE_RT_CFG_APPROXIMATE
    uint32_t scene_depth = 0;   // top-level depth + the deepest mesh's: stack entries a scene ray can need
    std::vector<atlas::rt::host::DeviceMesh> meshes;
    // two-level scene: TLAS nodes, instances (TLAS order), mesh table snapshot
    float4* d_tlas = nullptr;
    uint32_t n_tlas = 0;
    float4* d_instances = nullptr;
    uint32_t n_instances = 0;
    atlas::rt::dev::MeshDesc* d_mesh_table = nullptr;
    uint32_t n_mesh_table = 0;
    uint32_t scene_steps = 0;
    bool scene_ready = false;
    float4* d_inst_model = nullptr;     // object-to-world rows per instance (shading)
    float* d_materials = nullptr;       // GPUMaterial array
    uint32_t n_materials = 0;
    uint8_t* d_tex_pool = nullptr;      // level 0 of every texture (texture.cuh)
    void* d_tex_desc = nullptr;         // dev::TexDesc per texture
    uint32_t n_textures = 0;
    float4* d_lights = nullptr;         // GPULight array
    uint32_t n_lights = 0;
    float env[3] = { 0.0f, 0.0f, 0.0f };  // constant environment radiance of the path tracer's misses
    // path tracer queues
    atlas::rt::host::Scratch pt_rays[2], pt_pay[2], pt_hits, pt_shadow, pt_shadow_pay, pt_occ;
    atlas::rt::host::Scratch pt_words;  // per-bounce counters of a sample
    atlas::rt::host::Scratch pt_gb;     // real-time G-buffer matrices
    atlas::rt::host::Scratch pt_vis[2]; // shadow visibility of the transparency traversal, per shadow queue
    // a second shadow queue: a bounce's shadow trace runs beside the next bounce's trace
    atlas::rt::host::Scratch pt_shadow2, pt_shadow_pay2, pt_occ2;
    cudaEvent_t pt_events[4] = { nullptr, nullptr, nullptr, nullptr };
    // scratch of the RTAO / reflection / GI / DDGI passes (consumers.cu)
    atlas::rt::host::Scratch pass_rays, pass_key, pass_hits, pass_rad, pass_shadow, pass_shadow_pay, pass_vis,
        pass_counts;
    uint32_t* d_pt_counts = nullptr;    // radiance-cache render: [0], [1] ray queues, [2], [3] shadow queues
    uint32_t* d_counter = nullptr;     // [1] error word; [2..] work counters, two a launch (kWorkSlots in rotation)
    uint32_t next_work_slot = 0;
    unsigned long long* d_fetch = nullptr;
    atlas::rt::host::Scratch rays_in, results_out, batch_table, retest_count;
    // buffers of ae_rt_cast_pass
    atlas::rt::host::Scratch cast_primary, cast_primary_hits, cast_secondary, cast_secondary_hits, cast_shadow, cast_occluded;
    uint32_t* d_cast_counts = nullptr;
    // result copies of ae_rt_cast_pass overlap the later stages on this stream
    cudaStream_t copy_stream = nullptr;
    cudaStream_t trace_stream = nullptr;  // ae_rt_cast_pass: the shadow trace beside the bounce trace
    cudaEvent_t cast_events[4] = { nullptr, nullptr, nullptr, nullptr };
    uint32_t* h_cast_counts = nullptr;  // pinned, mapped
    uint32_t* d_cast_counts_mapped = nullptr;   // its device address
    uint32_t* h_error = nullptr;        // pinned, mapped: the error word as last published
    uint32_t* d_error_mapped = nullptr;
    std::string last_error;
    std::mutex upload_mutex;
};

namespace atlas::rt::host {

inline ae_rt_status Fail(ae_rt_ctx* ctx, ae_rt_status s, const std::string& msg) {
    if (ctx) ctx->last_error = msg;
    return s;
}

inline ae_rt_status CudaFail(ae_rt_ctx* ctx, cudaError_t e, const char* what) {
    std::string m = std::string(what) + ": " + cudaGetErrorName(e) + " (" + cudaGetErrorString(e) + ")";
    if (e == cudaErrorMemoryAllocation) return Fail(ctx, AE_RT_OUT_OF_MEMORY, m);
    return Fail(ctx, AE_RT_CUDA_ERROR, m);
}

#define AE_CUDA(ctx, call)                                         \
    do {                                                           \
        cudaError_t e_ = (call);                                   \
        if (e_ != cudaSuccess) return CudaFail((ctx), e_, #call);  \
    } while (0)

// True when the GPU can read `p` directly as device memory.
inline bool IsDevicePointer(const void* p) {
    cudaPointerAttributes a{};
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return a.type == cudaMemoryTypeDevice || a.type == cudaMemoryTypeManaged;
}


// Launches a kernel that begins with dev::wait_for_previous: it is set up while
// the kernel before it on the stream drains, instead of after it has ended
// (programmatic dependent launch).  The chains of short kernels gain most: a
// real-time frame at 321 x 181 326 -> 305 us, the four GI passes 1,046 ->
// 1,018, a path-traced sample at 1920 x 1080 1,265 -> 1,247.  No kernel lets
// the next one start before it ends: the waiting blocks then hold places that
// the shadow traces on the other stream could use (329, 1,023 and 1,290 us).
inline cudaError_t LaunchNext(const void* fn, uint32_t grid, uint32_t threads, cudaStream_t s, void** args) {
    cudaLaunchAttribute early{};
    early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    early.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c{};
    c.gridDim = dim3(grid);
    c.blockDim = dim3(threads);
    c.stream = s;
    c.attrs = &early;
    c.numAttrs = 1;
    return cudaLaunchKernelExC(&c, fn, args);
}

template <class... P, class... A>
cudaError_t LaunchNext(void (*kernel)(P...), uint32_t grid, uint32_t threads, cudaStream_t s, A&&... a) {
    std::tuple<P...> values(static_cast<P>(a)...);
    return std::apply(
        [&](P&... v) {
            void* args[] = { static_cast<void*>(&v)... };
            return LaunchNext(reinterpret_cast<const void*>(kernel), grid, threads, s, args);
        },
        values);
}

// The work counters (two words; most launches use the first alone) of the
// context's next persistent launch, zeroed on its stream: kWorkSlots in
// rotation, so that launches on different streams can overlap.
constexpr uint32_t kWorkSlots = 6;
cudaError_t NextWorkCounter(ae_rt_ctx* ctx, cudaStream_t s, uint32_t** counter);

// Persistent grid for kernel `fn`: SMs x resident CTAs (the configured count,
// or the kernel's occupancy), never more warps than rays.  threads: the block
// size when it is not the context's (then the occupancy alone counts).
uint32_t GridFor(const ae_rt_ctx* ctx, const void* fn, uint32_t n_rays, uint32_t threads = 0);

// Warps that share the rays of a launch too small to fill the GPU.
uint32_t SpreadWarps(const ae_rt_ctx* ctx);

// Queue-driven trace over the context's two-level scene (rays, out and count
// in device memory), for the other translation units.
// Closest / any-hit trace of a scene queue for the library's own consumers
// (passes, radiance cache): the near-tie detection is skipped; counter: a work
// counter that an earlier operation on the stream zeroed, or null.
ae_rt_status TraceSceneQueue(ae_rt_ctx* ctx, bool any, const ae_packed_ray* rays, uint32_t capacity, float tmin,
                             float tmax, void* out, void* stream, const uint32_t* count_dev, uint32_t cull_mask,
                             bool per_ray_tmax, uint32_t* counter = nullptr);

// The transparency traversal variants over the scene (transparency.cu); with
// count_dev, `n` is the queue capacity and the count lives on the device;
// with per_ray_tmax, ray i's tmax is its third vector's x; counter: a work
// counter that an earlier kernel on the stream zeroed, or null.
ae_rt_status TraceTransparency(ae_rt_ctx* ctx, bool any, const ae_packed_ray* rays, uint32_t n, float tmin,
                               float tmax, uint32_t cull_mask, void* out, void* stream,
                               const uint32_t* count_dev = nullptr, bool per_ray_tmax = false,
                               uint32_t* counter = nullptr);

// The bounce loop's queues for `capacity` rays: two ray/payload queues, the
// hit buffer, two shadow queues (a bounce's shadow trace runs on
// ctx->trace_stream beside the next bounce), their counts and events.
ae_rt_status EnsureBounceQueues(ae_rt_ctx* ctx, uint32_t capacity);

}  // namespace atlas::rt::host
