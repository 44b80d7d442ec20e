// Persistent wavefront BVH traversal kernels for sm_103a.
//
// Semantics: the engine's shader traversal on one BLAS --
//   HitClosest  data/shader/raytracer/bvh.hsh:191-273 (+ CheckLeafClosest :44-72)
//   HitAny      data/shader/raytracer/bvh.hsh:359-441 (+ CheckLeaf :74-104)
//   IntersectAABB / IntersectTriangle  data/shader/raytracer/intersections.hsh:18-57
// reproduced bit for bit: every multiply, add and divide is an explicitly
// rounded IEEE operation in the shader's order (no FMA contraction), GLSL
// min/max are min.f32/max.f32 (a NaN operand loses), the descent goes to the
// nearer child first (hitL <= hitR) and pushes the farther one.
//
// Execution model (not the shader's):
//  * persistent CTAs, a few per SM; each warp pulls rays from a global
//    counter.  A lane that finishes its ray takes a fresh one at the next
//    refill point: the idle lanes are found by a warp ballot and served with
//    one atomic per warp, so live rays stay packed in the warp;
//  * the traversal stack of each lane lives in shared memory, lane-interleaved
//    (entry k of lane l at [k][l], conflict-free), with a local-memory spill
//    area behind it;
//  * nodes are fetched with two 256-bit read-only loads, triangles with three
//    128-bit ones;
//  * every ray carries a step cap and a stack bound; exceeding either sets a
//    flag on the ray and in the context's error word instead of faulting.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "camera.cuh"
#include "texture.cuh"

namespace atlas::rt::dev {

constexpr uint32_t kErrStackOverflow = 0x1u;
constexpr uint32_t kErrIterationCap = 0x2u;
constexpr uint32_t kErrQueueOverflow = 0x8u;   // a wavefront queue append found the queue full

constexpr uint32_t kHitFlagHit = 0x1u;
constexpr uint32_t kHitFlagNearTie = 0x2u;
constexpr uint32_t kHitFlagOverflow = 0x4u;
constexpr uint32_t kHitFlagIterCap = 0x8u;

// One uploaded mesh (BLAS): the bindless blasNodes[mesh] / bvhTriangles[mesh]
// pair of the engine (data/shader/raytracer/buffers.hsh:45-57).
struct MeshDesc {
    const float4* nodes;
    const float4* tris;
    const float4* shading;       // GPUTriangle (6 float4), may be null
    uint32_t n_nodes;
    uint32_t n_tris;
};

struct TraceParams {
    const float4* nodes;         // 4 float4 per GPUBVHNode
    const float4* tris;          // 3 float4 per GPUBVHTriangle
    uint32_t n_nodes;
    uint32_t n_tris;
    const float4* rays;          // 3 float4 per PackedRay
    uint32_t n_rays;             // ray count, or the queue capacity when n_rays_dev is set
    const uint32_t* n_rays_dev;  // optional: ray count written by an earlier kernel
    float tmin;
    float tmax;
    float4* hits;                // 2 float4 per ae_hit (closest)
    uint8_t* occluded;           // 1 byte per ray (any)
    uint32_t* work_counter;      // rays handed out so far (zeroed before launch)
    uint32_t* error_word;        // kErr* bits
    unsigned long long* fetch_counts;  // [0] nodes, [1] triangles (optional)
    uint32_t max_steps;
    // two-level scenes (TLAS instantiation only)
    const float4* tlas;          // TLAS nodes, 4 float4 each
    uint32_t n_tlas;
    const float4* instances;     // GPUBVHInstance, 4 float4 each
    uint32_t n_instances;
    const MeshDesc* meshes;      // indexed by GPUBVHInstance::meshOffset
    uint32_t n_meshes;
    uint32_t cull_mask;
    // batched multi-mesh launches (MODE_BATCH): n_rays = total over the batches
    // of the query kind
    const struct BatchDesc* batches;
    uint32_t n_batches;
    uint32_t refill_steps;       // traversal steps between warp refills
    uint32_t spread_warps;       // warps that share the rays of a small launch (kSpreadWarps an SM)
    uint32_t per_ray_tmax;       // nonzero: a ray's tmax is its PackedRay hit.x (shadow queues)
    // transparency launches (OPACITY)
    const float* materials;      // GPUMaterial (23 words), may be null (opacity 1)
    uint32_t n_materials;
    TexTable textures;
    float* transparency;         // one float per ray (any hit)
    CameraParams cam;            // the camera variant: ray i is camera_ray(cam, i), `rays` unused
};

// One ray batch of a batched launch: its mesh, its rays and results, and its
// first index in the global ray numbering of its query kind.
struct BatchDesc {
    const float4* nodes;
    const float4* tris;
    const float4* rays;
    void* out;                   // ae_hit[] (closest) or uint8_t[] (any)
    uint32_t n_nodes;
    uint32_t n_tris;
    uint32_t n_rays;
    uint32_t reserved;
    float tmin;
    float tmax;
    uint32_t first;              // global index of the batch's first ray
    uint32_t max_steps;
};
static_assert(sizeof(BatchDesc) == 64, "batch descriptor layout");

// Default per-ray step cap of a BVH with n_nodes nodes: a valid tree visits
// each node at most once per ray, so 4 n + 64 never cuts a correct traversal
// short.  Computed in 64 bits and saturated, so that arrays of 2^30 nodes and
// more (64 GB of nodes fits in HBM) do not wrap to a small cap.
__host__ __device__ constexpr uint32_t default_step_cap(uint32_t n_nodes) {
    return 4ull * n_nodes + 64ull > 0xffffffffull ? 0xffffffffu : uint32_t(4ull * n_nodes + 64ull);
}

// ae_rt_config::refill_steps when left 0.
constexpr uint32_t kDefaultRefillSteps = 24;

// A launch with fewer rays than this many full warps on every SM spreads them
// over that many warps, which then hold only some lanes each: such a launch
// waits for its longest rays, and a warp of 32 of them takes every branch of
// every one.  1,000 rays on 65,536 triangles: 149 -> 117 us, occlusion of
// 8,000 rays 161 -> 131 us; at 16 or 32 warps 8,000 closest hits on 4,096
// triangles get slower (54 -> 57, 77 us), at 4 occlusion gains less.
constexpr uint32_t kSpreadWarps = 8;

constexpr int MODE_MESH = 0;     // one BLAS
constexpr int MODE_SCENE = 1;    // TLAS over instances
constexpr int MODE_BATCH = 2;    // many BLASes, one per batch

__device__ __forceinline__ float4 ldg4(const float4* p) { return __ldg(p); }

// Two floats in one 64-bit register pair, and the packed FP32 arithmetic of
// sm_100 and later on them: one instruction issues the operation for both
// halves, each rounded to nearest even as the scalar instruction rounds it.
using f32x2 = unsigned long long;

__host__ __device__ __forceinline__ f32x2 pack2(float lo, float hi) {
#ifdef __CUDA_ARCH__
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
#else
    return 0;
#endif
}
__device__ __forceinline__ float lo2(f32x2 v) { return __uint_as_float(uint32_t(v)); }
__device__ __forceinline__ float hi2(f32x2 v) { return __uint_as_float(uint32_t(v >> 32)); }
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// The node value that ends a traversal: the bottom of the stack, and no
// pointer of a valid tree (arrays hold fewer than 2^31 - 1 elements).
constexpr int32_t kStackEnd = INT32_MIN;

// First statement of every kernel that host::LaunchNext launches: such a
// kernel is set up while the one before it on the stream drains, and this
// waits until that has ended and its writes are visible.
__device__ __forceinline__ void wait_for_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Stack entries of a lane; meshes and scenes whose trees can need more take
// kernels with a deeper stack.
constexpr int kStackEntries = 128;

// A node as the traversal holds it: the two children's boxes in the pairs
// that the packed slab arithmetic takes, the child pointers, and `slow`, set
// when a coordinate lies outside the fast-division window (kFastLo / kFastHi).
struct NodeBoxes {
    f32x2 l_lo_xy, l_hi_xy, l_z, r_z, r_lo_xy, r_hi_xy;   // *_z: (min z, max z)
    int32_t lptr, rptr;
    int32_t slow;
};

// The library keeps its nodes in device memory in this order (64 bytes, the
// engine's fields permuted at upload and by the GPU builder):
//   l.min.xy, l.max.xy, l.min.z, l.max.z, r.min.z, r.max.z |
//   r.min.xy, r.max.xy, leftPtr, rightPtr, slow, 0
// so that every pair of coordinates arrives in a register pair without a
// move: two 32-byte read-only loads, one L1 sector each (four 16-byte loads
// would look each sector up twice, and the L1 pipeline limits incoherent
// rays).  Arrays are cudaMalloc'ed by the library, so nodes are 32-byte
// aligned.
__device__ __forceinline__ NodeBoxes load_node(const float4* p) {
    NodeBoxes n;
    f32x2 ptrs, flags;
    asm("ld.global.nc.v4.b64 {%0, %1, %2, %3}, [%4];"
        : "=l"(n.l_lo_xy), "=l"(n.l_hi_xy), "=l"(n.l_z), "=l"(n.r_z) : "l"(p));
    asm("ld.global.nc.v4.b64 {%0, %1, %2, %3}, [%4+32];"
        : "=l"(n.r_lo_xy), "=l"(n.r_hi_xy), "=l"(ptrs), "=l"(flags) : "l"(p));
    n.lptr = int32_t(uint32_t(ptrs));
    n.rptr = int32_t(uint32_t(ptrs >> 32));
    n.slow = int32_t(uint32_t(flags));
    return n;
}

// A caller-owned node in the engine's own field order, 16-byte aligned; its
// coordinates have not been looked at, so it counts as slow.  A pointer equal
// to kStackEnd becomes its neighbour, which is past any triangle array too.
__device__ __forceinline__ NodeBoxes load_engine_node(const float4* p) {
    const float4 n0 = ldg4(p), n1 = ldg4(p + 1), n2 = ldg4(p + 2), n3 = ldg4(p + 3);
    NodeBoxes n;
    n.l_lo_xy = pack2(n0.x, n0.y);
    n.l_hi_xy = pack2(n0.w, n1.x);
    n.l_z = pack2(n0.z, n1.y);
    n.r_lo_xy = pack2(n1.z, n1.w);
    n.r_hi_xy = pack2(n2.y, n2.z);
    n.r_z = pack2(n2.x, n2.w);
    n.lptr = max(__float_as_int(n3.x), kStackEnd + 1);
    n.rptr = max(__float_as_int(n3.y), kStackEnd + 1);
    n.slow = 1;
    return n;
}

// Index in the engine's node (16 words) of word k of the library's.
__host__ __device__ constexpr int engine_node_word(int k) {
    // lmin 0-2, lmax 3-5, rmin 6-8, rmax 9-11, pointers 12-13, padding 14-15
    constexpr int order[16] = { 0, 1, 3, 4, 2, 5, 8, 11, 6, 7, 9, 10, 12, 13, 14, 15 };
    return order[k];
}

// IEEE single operations with explicit rounding (no contraction into FMA).
__device__ __forceinline__ float fmul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float fadd(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float fsub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float fdiv(float a, float b) { return __fdiv_rn(a, b); }

// Correctly rounded quotients (c - o) / d of both halves from no = -o,
// nd = -d and y = RN(1/d), without a divide instruction: q0 = RN(a*y) is
// within 1.5 ulp of a/d; one residual correction q1 = RN(q0 + RN(a - d*q0)*y)
// makes it faithful; with a faithful quotient the residual a - d*q1 is exact
// (computed by FMA) and Markstein's theorem (P. Markstein, IBM J. Res. Dev.
// 34(1), 1990) gives RN(q1 + r1*y) = RN(a/d).  Valid while no intermediate
// under- or overflows, which the callers ensure by range (see kFastLo /
// kFastHi); everything else takes div.rn.
__device__ __forceinline__ f32x2 slab_quotients(f32x2 c, f32x2 no, f32x2 nd, f32x2 y) {
    const f32x2 a = add2(c, no);
    f32x2 q = mul2(a, y);
    f32x2 r = fma2(q, nd, a);
    q = fma2(r, y, q);
    r = fma2(q, nd, a);
    return fma2(r, y, q);
}

// Exponent window of the fast quotient: every |origin|, |box coordinate| is 0
// or in [2^-40, 2^40] and every |direction| in [2^-40, 2^40], so |a| = |c - o|
// is 0 or in [2^-63, 2^41] and all intermediates stay normal.
constexpr float kFastLo = 9.094947017729282e-13f;   // 2^-40
constexpr float kFastHi = 1.099511627776e12f;       // 2^40

__device__ __forceinline__ bool in_fast_range(float v, bool zero_ok) {
    const float m = fabsf(v);
    return (zero_ok && m == 0.0f) || (m >= kFastLo && m <= kFastHi);
}

// Near ties.  The nearest triangle of a closest-hit ray is decided by FP32
// rounding when a second triangle lies within 1e-6 relative t of it; such
// rays carry kHitFlagNearTie and are re-tested in double.  The flag must
// cover every ray whose two nearest double-precision hits are that close,
// including hits the FP32 traversal never sees, so it is set (a superset)
// when any of these holds:
//  * a second accepted triangle lies within kTieWindow relative t of the
//    nearest (1e-6 plus the FP32 error of the two distances);
//  * a child box rejected by the shader's test had its entry within
//    kTieWindow of the bound it was tested against (its triangles could tie
//    with the final hit, which is at most that bound);
//  * a triangle rejected by the FP32 test lies within the rounding error of
//    its barycentric tests (tri_test's nearMiss) at a distance up to
//    kTieWindow past the current nearest hit -- a shared edge, where either
//    side's FP32 test may fail;
//  * the shader's descent dropped a hit right child whose entry equals the
//    bound (bvh.hsh:234-236: a missed left child reports the bound too, and
//    hitL <= hitR then picks it).
// None of this changes which triangle the traversal returns.
constexpr float kTieWindow = 4e-6f;
constexpr float kTieWiden = 1.0f + kTieWindow;
constexpr float kNearMissScale = 9.5367431640625e-07f;   // 2^-20

// Three-input minimum / maximum (one instruction; a NaN operand loses).
__device__ __forceinline__ float min3(float a, float b, float c) {
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

// IntersectAABB(ray, aabb, tmin, tmax, out dist) -- intersections.hsh:18-34 --
// from the six slab quotients.  nearCull: the box was rejected but its entry
// lies within kTieWindow of the exit bound.
__device__ __forceinline__ bool box_decide(float t0x, float t0y, float t0z, float t1x, float t1y, float t1z,
                                           float tmin, float tmax, float& dist, bool& nearCull) {
    const float tminf = fmaxf(tmin, max3(fminf(t0x, t1x), fminf(t0y, t1y), fminf(t0z, t1z)));
    const float tmaxf = fminf(tmax, min3(fmaxf(t0x, t1x), fmaxf(t0y, t1y), fmaxf(t0z, t1z)));
    const bool hit = tminf <= tmaxf;
    dist = hit ? tminf : tmax;
    nearCull = !hit && tminf <= fmul(tmaxf, kTieWiden);
    return hit;
}

// The same with the shader's divisions, for any operands.
__device__ __forceinline__ bool box_test(float ox, float oy, float oz, float dx, float dy, float dz,
                                         float lx, float ly, float lz, float hx, float hy, float hz,
                                         float tmin, float tmax, float& dist, bool& nearCull) {
    return box_decide(fdiv(fsub(lx, ox), dx), fdiv(fsub(ly, oy), dy), fdiv(fsub(lz, oz), dz),
                      fdiv(fsub(hx, ox), dx), fdiv(fsub(hy, oy), dy), fdiv(fsub(hz, oz), dz), tmin, tmax, dist,
                      nearCull);
}

// IntersectTriangle -- intersections.hsh:36-57.  Returns the shader's accept
// test; (t, u, v) = sol.  NEAR: *nearMiss tells whether (u, v) lie within the
// rounding error of the barycentric bounds.  With the L1 norms Sd, S0, S1, Ss
// of d, e0, e1 and s = o - v0, every operation of the formula contributes at
// most a few ulps of products bounded by Sd (S0+S1) (Ss+S0+S1), so
// |error(u)|, |error(v)| < beta = m / |den| with
// m = 2^-20 Sd (S0+S1) (Ss+S0+S1) (2^-20 = 16 ulps of 1).  The tests are
// taken multiplied by |den| (u |den| + m >= 0, ...), one correctly rounded
// FMA each, so the oracle reproduces them.  slack (optional) receives |den| and m.
struct TriTerms {
    float den, nt, nu, nv;     // t = nt / den, u = nu / den, v = nv / den
    float m;                   // the slack (NEAR)
};

template <bool NEAR>
__device__ __forceinline__ TriTerms tri_terms(float ox, float oy, float oz, float dx, float dy, float dz,
                                              const float4& a, const float4& b, const float4& c) {
    TriTerms r;
    const float e0x = fsub(b.x, a.x), e0y = fsub(b.y, a.y), e0z = fsub(b.z, a.z);
    const float e1x = fsub(c.x, a.x), e1y = fsub(c.y, a.y), e1z = fsub(c.z, a.z);
    const float sx = fsub(ox, a.x), sy = fsub(oy, a.y), sz = fsub(oz, a.z);
    // the slack's scale, folded at once so that one value stays live
    r.m = 0.0f;
    if (NEAR) {
        const float s01 = fadd(fadd(fadd(fabsf(e0x), fabsf(e0y)), fabsf(e0z)),
                               fadd(fadd(fabsf(e1x), fabsf(e1y)), fabsf(e1z)));
        const float ss = fadd(fadd(fabsf(sx), fabsf(sy)), fabsf(sz));
        const float sd = fadd(fadd(fabsf(dx), fabsf(dy)), fabsf(dz));
        r.m = fmul(fmul(fmul(sd, s01), fadd(ss, s01)), kNearMissScale);
    }
    // p = cross(s, e0), q = cross(d, e1)
    const float px = fsub(fmul(sy, e0z), fmul(e0y, sz));
    const float py = fsub(fmul(sz, e0x), fmul(e0z, sx));
    const float pz = fsub(fmul(sx, e0y), fmul(e0x, sy));
    const float qx = fsub(fmul(dy, e1z), fmul(e1y, dz));
    const float qy = fsub(fmul(dz, e1x), fmul(e1z, dx));
    const float qz = fsub(fmul(dx, e1y), fmul(e1x, dy));
    r.den = fadd(fadd(fmul(qx, e0x), fmul(qy, e0y)), fmul(qz, e0z));
    r.nt = fadd(fadd(fmul(px, e1x), fmul(py, e1y)), fmul(pz, e1z));
    r.nu = fadd(fadd(fmul(qx, sx), fmul(qy, sy)), fmul(qz, sz));
    r.nv = fadd(fadd(fmul(px, dx), fmul(py, dy)), fmul(pz, dz));
    return r;
}

template <bool NEAR>
__device__ __forceinline__ bool tri_decide(const TriTerms& r, float& t, float& u, float& v, bool* nearMiss) {
    t = fdiv(r.nt, r.den);
    u = fdiv(r.nu, r.den);
    v = fdiv(r.nv, r.den);
    if (NEAR) {
        const float ad = fabsf(r.den);
        *nearMiss = __fmaf_rn(u, ad, r.m) >= 0.0f && __fmaf_rn(v, ad, r.m) >= 0.0f &&
                    __fmaf_rn(fsub(1.0f, fadd(u, v)), ad, fadd(r.m, r.m)) >= 0.0f;
    }
    return t >= 0.0f && u >= 0.0f && v >= 0.0f && fadd(u, v) <= 1.0f;
}

template <bool NEAR = false>
__device__ __forceinline__ bool tri_test(float ox, float oy, float oz, float dx, float dy, float dz,
                                         const float4& a, const float4& b, const float4& c,
                                         float& t, float& u, float& v, bool* nearMiss = nullptr,
                                         float* slack = nullptr) {
    const TriTerms r = tri_terms<NEAR>(ox, oy, oz, dx, dy, dz, a, b, c);
    if (NEAR && slack) { slack[0] = fabsf(r.den); slack[1] = r.m; }
    return tri_decide<NEAR>(r, t, u, v, nearMiss);
}

// tri_test for the traversal, which reads t, u, v only of accepted or
// near-miss triangles: the three divisions (a third of the test) are left out
// when the numerators show that it is neither.  With x = nu / den exactly
// and w = x |den|, w < -(2 m + 2^-20 |den|) puts u below -2^-20 (1 - 2^-24) and
// u |den| + m below 0; the same holds for v.  When neither holds, a negative
// one of u, v is small, so their sum keeps its relative accuracy, and
// u + v > 1 + 2^-18 + 4 m / |den| puts the rounded sum above 1 and its slack
// test below 0.  A comparison with a NaN or an infinite slack is false and
// leaves the decision to the divisions.  Most of the triangles a ray meets
// are missed by more than that.
template <bool NEAR>
__device__ __forceinline__ bool tri_test_traversal(float ox, float oy, float oz, float dx, float dy, float dz,
                                                   const float4& a, const float4& b, const float4& c, float& t,
                                                   float& u, float& v, bool& nearMiss) {
    const TriTerms r = tri_terms<NEAR>(ox, oy, oz, dx, dy, dz, a, b, c);
    const float ad = fabsf(r.den);
    const uint32_t sign = __float_as_uint(r.den) & 0x80000000u;
    const float wu = __uint_as_float(__float_as_uint(r.nu) ^ sign), wv = __uint_as_float(__float_as_uint(r.nv) ^ sign);
    const float e = NEAR ? __fmaf_rn(ad, 9.5367431640625e-07f, fadd(r.m, r.m)) : fmul(ad, 9.5367431640625e-07f);
    nearMiss = false;
    if (fminf(wu, wv) < -e || fadd(wu, wv) > __fmaf_rn(e, 4.0f, ad)) return false;
    return tri_decide<NEAR>(r, t, u, v, &nearMiss);
}

// IntersectTriangle with one reciprocal of the denominator instead of three
// divisions, for traversals whose results are statistical (the radiance
// cache, AE_RT_CFG_APPROXIMATE): the numerators and the denominator are the
// shader's, operation by operation (no contraction: the dot products of
// nearly edge-on triangles cancel), and each of t, u, v is RN(RN(n) *
// RN(1/den)), within 1.5 units of 2^-24 (relative) of the shader's RN(n / den);
// the same accept test.
__device__ __forceinline__ bool tri_test_fast(float ox, float oy, float oz, float dx, float dy, float dz,
                                              const float4& a, const float4& b, const float4& c,
                                              float& t, float& u, float& v) {
    const float e0x = fsub(b.x, a.x), e0y = fsub(b.y, a.y), e0z = fsub(b.z, a.z);
    const float e1x = fsub(c.x, a.x), e1y = fsub(c.y, a.y), e1z = fsub(c.z, a.z);
    const float sx = fsub(ox, a.x), sy = fsub(oy, a.y), sz = fsub(oz, a.z);
    const float px = fsub(fmul(sy, e0z), fmul(e0y, sz));
    const float py = fsub(fmul(sz, e0x), fmul(e0z, sx));
    const float pz = fsub(fmul(sx, e0y), fmul(e0x, sy));
    const float qx = fsub(fmul(dy, e1z), fmul(e1y, dz));
    const float qy = fsub(fmul(dz, e1x), fmul(e1z, dx));
    const float qz = fsub(fmul(dx, e1y), fmul(e1x, dy));
    const float inv = __frcp_rn(fadd(fadd(fmul(qx, e0x), fmul(qy, e0y)), fmul(qz, e0z)));
    t = fmul(fadd(fadd(fmul(px, e1x), fmul(py, e1y)), fmul(pz, e1z)), inv);
    u = fmul(fadd(fadd(fmul(qx, sx), fmul(qy, sy)), fmul(qz, sz)), inv);
    v = fmul(fadd(fadd(fmul(px, dx), fmul(py, dy)), fmul(pz, dz)), inv);
    return t >= 0.0f && u >= 0.0f && v >= 0.0f && fadd(u, v) <= 1.0f;
}

__device__ __forceinline__ uint32_t lanemask_lt() {
    uint32_t m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

// ---- staged ray queue: 1-D bulk copies (TMA) of ray tiles into shared memory ----
constexpr uint32_t kErrWaitTimeout = 0x4u;     // a bounded device wait gave up
constexpr int kStageRays = 16;                 // rays per staged tile (768 bytes)

__device__ __forceinline__ uint32_t shared_addr(const void* ptr) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(ptr));
}

__device__ __forceinline__ void stage_barrier_init(uint32_t bar) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(bar) : "memory");
}

// One bulk copy of `bytes` (a multiple of 16, both addresses 16-byte
// aligned) from global into this CTA's shared memory; the barrier's phase
// completes when the bytes have landed.  The proxy fence orders the warp's
// earlier reads of the buffer before the copy's writes.
__device__ __forceinline__ void stage_bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" :: "r"(bar), "r"(bytes) : "memory");
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 :: "r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}

__device__ __forceinline__ uint64_t stage_clock_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Waits for the completion of the barrier phase of parity `parity`; false
// after ~200 ms of the global timer, or after 2^25 polls whatever it says.
__device__ __forceinline__ bool stage_wait(uint32_t bar, uint32_t parity) {
    const uint64_t start = stage_clock_ns();
    for (uint32_t it = 0; it < (1u << 25); it++) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred q;\n\tmbarrier.try_wait.parity.shared::cta.b64 q, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, q;\n\t}"
            : "=r"(done) : "r"(bar), "r"(parity) : "memory");
        if (done) return true;
        if ((it & 63u) == 63u && stage_clock_ns() - start > 200000000ull) return false;
    }
    return false;
}

// Per-lane traversal stack: SMEM entries in shared memory (lane-interleaved),
// then SPILL entries in local memory.
// Entry 0 holds kStackEnd, so that a pop needs no test for an empty stack.
template <int SMEM, int SPILL>
struct LaneStack {
    int32_t* sh;           // &shared[warp][0][lane]; entry k at sh[k * 32]
    int32_t spill[SPILL + 1];
    __device__ __forceinline__ void put(uint32_t k, int32_t v) {
        if (k < SMEM) sh[k * 32] = v;
        else spill[k - SMEM] = v;
    }
    __device__ __forceinline__ int32_t get(uint32_t k) const {
        return k < SMEM ? sh[k * 32] : spill[k - SMEM];
    }
    static constexpr uint32_t capacity = SMEM + SPILL + 1;
};

// Trees of fewer than SMEM levels: shared memory alone.
template <int SMEM>
struct LaneStack<SMEM, 0> {
    int32_t* sh;
    __device__ __forceinline__ void put(uint32_t k, int32_t v) { sh[k * 32] = v; }
    __device__ __forceinline__ int32_t get(uint32_t k) const { return sh[k * 32]; }
    static constexpr uint32_t capacity = SMEM;
};

// One traversal ray in the space of the structure being traversed: its
// origin and direction, negated, and the correctly rounded reciprocals of the
// direction, in the pairs (x, y) and (z, z) that the node's coordinate pairs
// meet, and the fast-division window flag.  Twelve registers, three more than
// the nine values: the z pair is the price of pairing min z with max z.
struct TRay {
    f32x2 no_xy, no_zz, nd_xy, nd_zz, y_xy, y_zz;
    bool fast;
    __device__ __forceinline__ void set(float ox, float oy, float oz, float dx, float dy, float dz) {
        const float yz = __frcp_rn(dz);
        no_xy = pack2(-ox, -oy);
        no_zz = pack2(-oz, -oz);
        nd_xy = pack2(-dx, -dy);
        nd_zz = pack2(-dz, -dz);
        y_xy = pack2(__frcp_rn(dx), __frcp_rn(dy));
        y_zz = pack2(yz, yz);
        fast = in_fast_range(ox, true) && in_fast_range(oy, true) && in_fast_range(oz, true) &&
               in_fast_range(dx, false) && in_fast_range(dy, false) && in_fast_range(dz, false);
    }
    __device__ __forceinline__ float ox() const { return -lo2(no_xy); }
    __device__ __forceinline__ float oy() const { return -hi2(no_xy); }
    __device__ __forceinline__ float oz() const { return -lo2(no_zz); }
    __device__ __forceinline__ float dx() const { return -lo2(nd_xy); }
    __device__ __forceinline__ float dy() const { return -hi2(nd_xy); }
    __device__ __forceinline__ float dz() const { return -lo2(nd_zz); }
};

// Approximate IntersectAABB for the screening below: the six quotients as
// RN(RN(c - o) * RN(1/d)) instead of the shader's RN((c - o) / d).  Each
// lies within 3 units of 2^-24 (relative) of the shader's quotient and has
// its sign (zero exactly when c == o), and min / max carry that bound over
// to the entry lo and exit hi.
__device__ __forceinline__ void box_approx(const TRay& r, f32x2 lo_xy, f32x2 hi_xy, f32x2 z, float tmin, float tmax,
                                           float& lo, float& hi) {
    const f32x2 t0 = mul2(add2(lo_xy, r.no_xy), r.y_xy), t1 = mul2(add2(hi_xy, r.no_xy), r.y_xy),
                tz = mul2(add2(z, r.no_zz), r.y_zz);
    lo = fmaxf(tmin, max3(fminf(lo2(t0), lo2(t1)), fminf(hi2(t0), hi2(t1)), fminf(lo2(tz), hi2(tz))));
    hi = fminf(tmax, min3(fmaxf(lo2(t0), lo2(t1)), fmaxf(hi2(t0), hi2(t1)), fmaxf(lo2(tz), hi2(tz))));
}

// IntersectAABB with the quotients of the fast-division window, bit for bit
// those of the divisions.
__device__ __forceinline__ bool box_fast(const TRay& r, f32x2 lo_xy, f32x2 hi_xy, f32x2 z, float tmin, float tmax,
                                         float& dist, bool& nearCull) {
    const f32x2 t0 = slab_quotients(lo_xy, r.no_xy, r.nd_xy, r.y_xy),
                t1 = slab_quotients(hi_xy, r.no_xy, r.nd_xy, r.y_xy),
                tz = slab_quotients(z, r.no_zz, r.nd_zz, r.y_zz);
    return box_decide(lo2(t0), hi2(t0), lo2(tz), lo2(t1), hi2(t1), hi2(tz), tmin, tmax, dist, nearCull);
}

// x <= y decided from approximations x', y' >= 0 that are each within 8 units
// of 2^-24 (relative) of x and y: x' <= y' * kSure proves x <= y, and
// x' * kSure > y' proves x > y (kSure = 1 - 2^-20 leaves room for the rounding
// of the product); anything between is a close call.
constexpr float kSure = 0.99999904632568359375f;

// Both child boxes of a node (IntersectAABB x 2, bvh.hsh:229-232 / :253-256)
// as the traversal uses them: il / ir whether each box is hit;
// leftFirst = (distL <= distR) for the descent order (only read when
// `ordered`), with a missed box reporting the bound as the shader's does;
// nearCull (only when `ties`): a box was rejected with its entry within
// kTieWindow of the bound (see kTieWindow).
// Inside the fast-division window (the node's `slow` word is 0 when its
// coordinates are in it, set by the upload; the ray's own flag) the quotients
// are correctly rounded from the reciprocal (slab_quotients); outside it and
// for the BOUNDS variant (whose nodes did not go through the upload) they
// divide with div.rn.  The packed form issues 36 instructions for the 12
// quotients of a node instead of 72; the traversal is bound by instruction
// issue (72 % of the cycles on 65,536 random triangles), and a million closest
// hits there went from 1,342 to 1,231 us with it, 400,009 closest hits and as
// many occlusion tests over 512 instances from 2,312 to 2,084 us.  A traversal that needs only il / ir (any
// hit: neither ordered nor ties) first screens the boxes with box_approx:
// every hit decision that the approximations settle with a margin of 16
// units of 2^-24 is the shader's, and only a lane with a close call (a
// grazing ray) computes the quotients exactly.  Closest-hit traversals
// compare entry distances, which are often exactly equal (sibling boxes
// with a common face), so they take the exact quotients at once.
__device__ __forceinline__ void test_children(const TRay& r, const NodeBoxes& n, float tmin, float bound, bool ordered,
                                              bool ties, bool& il, bool& ir, bool& leftFirst, bool& nearCull) {
    const bool fast = r.fast && n.slow == 0;
    if (fast && !ordered && !ties && tmin >= 0.0f) {
        float lol, hil, lor, hir;
        box_approx(r, n.l_lo_xy, n.l_hi_xy, n.l_z, tmin, bound, lol, hil);
        box_approx(r, n.r_lo_xy, n.r_hi_xy, n.r_z, tmin, bound, lor, hir);
        // lo >= tmin >= 0, so a negative exit is a sure miss
        il = hil >= 0.0f && lol <= fmul(hil, kSure);
        ir = hir >= 0.0f && lor <= fmul(hir, kSure);
        const bool close = (!il && hil >= 0.0f && !(fmul(lol, kSure) > hil)) ||
                           (!ir && hir >= 0.0f && !(fmul(lor, kSure) > hir));
        leftFirst = true;
        nearCull = false;
        if (!close) return;
    }
    bool nl, nr;
    float hl, hr;
    if (fast) {
        il = box_fast(r, n.l_lo_xy, n.l_hi_xy, n.l_z, tmin, bound, hl, nl);
        ir = box_fast(r, n.r_lo_xy, n.r_hi_xy, n.r_z, tmin, bound, hr, nr);
    } else {
        il = box_test(r.ox(), r.oy(), r.oz(), r.dx(), r.dy(), r.dz(), lo2(n.l_lo_xy), hi2(n.l_lo_xy), lo2(n.l_z),
                      lo2(n.l_hi_xy), hi2(n.l_hi_xy), hi2(n.l_z), tmin, bound, hl, nl);
        ir = box_test(r.ox(), r.oy(), r.oz(), r.dx(), r.dy(), r.dz(), lo2(n.r_lo_xy), hi2(n.r_lo_xy), lo2(n.r_z),
                      lo2(n.r_hi_xy), hi2(n.r_hi_xy), hi2(n.r_z), tmin, bound, hr, nr);
    }
    leftFirst = hl <= hr;
    nearCull = nl || nr;
}

// Both child boxes for traversals whose results are statistical rather than
// the shader's bit for bit (the radiance cache's training paths): the
// approximate quotients of box_approx with no exact re-test.  A box counts
// as hit when its entry is at most its exit times 1 + 2^-20, so the test
// never rejects a box that the exact test accepts (it may accept a grazed
// one); the order follows the approximate entries.  Outside the
// fast-division window it is test_children.
constexpr float kLoose = 1.00000095367431640625f;   // 1 + 2^-20

__device__ __forceinline__ void test_children_loose(const TRay& r, const NodeBoxes& n, float tmin, float bound,
                                                    bool& il, bool& ir, bool& leftFirst) {
    if (r.fast && n.slow == 0 && tmin >= 0.0f) {
        float lol, hil, lor, hir;
        box_approx(r, n.l_lo_xy, n.l_hi_xy, n.l_z, tmin, bound, lol, hil);
        box_approx(r, n.r_lo_xy, n.r_hi_xy, n.r_z, tmin, bound, lor, hir);
        il = lol <= fmul(hil, kLoose);
        ir = lor <= fmul(hir, kLoose);
        leftFirst = (il ? lol : bound) <= (ir ? lor : bound);
        return;
    }
    bool unused;
    test_children(r, n, tmin, bound, true, false, il, ir, leftFirst, unused);
}

// vec4(v, w) * inverseMatrix (bvh.hsh:179-180): component i = dot(vec4(v, w),
// column i), summed left to right with separate roundings.
__device__ __forceinline__ float xform_row(float x, float y, float z, float w, const float4& c) {
    return fadd(fadd(fadd(fmul(x, c.x), fmul(y, c.y)), fmul(z, c.z)), fmul(w, c.w));
}

// CheckInstance's object-space ray (bvh.hsh:172-189).
__device__ __forceinline__ TRay transform_ray(const TRay& w, const float4& c0, const float4& c1, const float4& c2) {
    const float ox = w.ox(), oy = w.oy(), oz = w.oz(), dx = w.dx(), dy = w.dy(), dz = w.dz();
    TRay r;
    r.set(xform_row(ox, oy, oz, 1.0f, c0), xform_row(ox, oy, oz, 1.0f, c1), xform_row(ox, oy, oz, 1.0f, c2),
          xform_row(dx, dy, dz, 0.0f, c0), xform_row(dx, dy, dz, 0.0f, c1), xform_row(dx, dy, dz, 0.0f, c2));
    return r;
}

constexpr uint32_t kTlasInvalid = 0xffffffffu;

// Batch holding global ray index g: the last descriptor whose first <= g.
__device__ __forceinline__ uint32_t find_batch(const BatchDesc* b, uint32_t n, uint32_t g) {
    uint32_t lo = 0, hi = n;            // invariant: b[lo].first <= g < b[hi].first
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (__ldg(&b[mid].first) <= g) lo = mid;
        else hi = mid;
    }
    return lo;
}

// `tri.opacity < 0.0 ? GetOpacity(tri, sol.yz, materialOffset, 0) : tri.opacity`
// (out of line: the texture path is rare and would take the registers of the
// whole traversal).
static __device__ __noinline__ float texture_opacity(const float* materials, uint32_t n_materials, const uint8_t* pool,
                                              const TexDesc* desc, uint32_t n_tex, const float4* d0, int32_t matOffset,
                                              float u, float v) {
    return get_opacity(materials, n_materials, TexTable{ pool, desc, n_tex }, __ldg(d0), matOffset, u, v);
}

// ANY: HitAny instead of HitClosest.  COUNT: per-launch node / triangle fetch
// totals.  MODE_SCENE: two-level traversal over instances (CheckInstance,
// bvh.hsh:172-189, with the TLAS/BLAS switch keyed on the stack depth at which
// the instance was entered, bvh.hsh:212-223).  MODE_BATCH: every lane finds
// its ray's batch (mesh, t range, result buffer) when it takes a ray, so one
// launch serves many meshes.
// BOUNDS = true adds range checks of every node and triangle index against
// n_nodes / n_tris (for callers whose BVH did not pass the host validator);
// an out-of-range index ends the ray with the overflow flag set.
// TIES: closest-hit rays get the complete near-tie flag (kTieWindow); the
// library's own consumers that discard the flag (path tracer, passes,
// radiance cache) launch TIES = false.
//
// STAGE > 0: each warp claims its rays in tiles of STAGE consecutive rays and
// copies every tile into shared memory with one bulk copy (TMA, 1-D) on an
// mbarrier, the next tile in flight while the current one is handed out
// (double-buffered); refills then read rays from shared memory.  Single-mesh
// and scene launches only.  A copy that does not complete within the bounded
// wait sets kErrWaitTimeout and ends the warp's refills.
//
// LOOSE: the conservative approximate box test (test_children_loose) and
// tri_test_fast, for consumers whose results are Monte Carlo estimates
// (AE_RT_CFG_APPROXIMATE), not the shader's bit for bit.
//
// OPACITY: the transparency variants HitClosestTransparency (bvh.hsh:275-357,
// + CheckLeafClosestTransparency :106-138) and HitAnyTransparency
// (bvh.hsh:443-524, + CheckLeafTransparency :140-170).  Leaves read the
// 96-byte shading triangle (UnpackTriangle, common.hsh:17-44): its vertices,
// endOfNode = d1.z > 0 and opacity = d2.w or GetOpacity.  Closest: a hit counts
// only where its opacity is > 0.  Any: every accepted triangle multiplies the
// leaf's running transparency, which starts from the current value; the
// leaf's result multiplies the current value again (bvh.hsh:500), values
// below 1e-6 become 0, and the traversal ends at 0.
//
// FEW: the launch's warps hold all of its rays at once (the host has checked
// the count; the transparency queries launch as many blocks as that takes),
// each warp its own range, so there is no work counter and no memset before
// the launch (1,000 closest hits 39 -> 36 us; a test for it at run time cost
// the large launches up to 3 %).
//
// CAMERA: ray i is the camera ray of queue slot i (camera_ray), made by the
// lane that takes it, instead of a load from a ray buffer written by a
// separate ray-generation launch.
template <bool ANY, bool COUNT, int MODE, int WARPS, int SMEM_STACK, int SPILL_STACK, bool BOUNDS, bool TIES,
          int STAGE, bool LOOSE, bool CAMERA, bool OPACITY, bool FEW>
__device__ __forceinline__ void trace_rays(const TraceParams& p) {
    constexpr bool TLAS = MODE == MODE_SCENE;
    constexpr bool BATCH = MODE == MODE_BATCH;
    // Whether a push can meet a full stack.  Single-mesh and scene launches of
    // up to kStackEntries are chosen by the depth of validated trees, so it
    // cannot.  The test itself is cheap, but its way out of the loop moves the
    // point where the lanes of a warp meet again from the end of each round to
    // the end of the burst: without it 400,000 rays through 512 instances take
    // 1,470 us for both kinds against 1,840 (9.6 against 7.3 lanes at work per
    // instruction), a million random closest hits 1,063 against 1,074.
    constexpr bool CHECKED = BOUNDS || (SPILL_STACK > 0 && (OPACITY || BATCH || SMEM_STACK + SPILL_STACK > kStackEntries));
    static_assert(STAGE == 0 || (!BATCH && !BOUNDS), "staged rays: single-mesh and scene launches only");
    static_assert(!LOOSE || (!TIES && !BOUNDS), "loose traversal: no near-tie flag, uploaded nodes");
    static_assert(!OPACITY || (TLAS && !TIES && !LOOSE && !COUNT && !BOUNDS && STAGE == 0), "transparency: exact scenes");
    static_assert(!CAMERA || (MODE == MODE_MESH && STAGE == 0 && !ANY), "camera rays: single-mesh closest hits");
    // the batched launch's two loops share their stacks: dynamic shared memory
    __shared__ int32_t s_stack[BATCH ? 1 : WARPS][BATCH ? 1 : SMEM_STACK][32];
    extern __shared__ int32_t s_batch_stack[];
    // scenes: the world-space ray of each lane while it is inside an instance
    // (held in registers beside the object-space one it cost spills, and every
    // step selected between the two)
    __shared__ uint32_t s_world[TLAS ? WARPS : 1][TLAS ? 10 : 1][32];
    __shared__ __align__(128) float4 s_rays[STAGE > 0 ? WARPS : 1][2][STAGE > 0 ? STAGE * 3 : 1];
    __shared__ __align__(8) uint64_t s_rbar[STAGE > 0 ? WARPS : 1][2];
    __shared__ uint32_t s_rstate[STAGE > 0 ? WARPS : 1][3];
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t warp = threadIdx.x >> 5;
    constexpr unsigned kFull = 0xffffffffu;

    LaneStack<SMEM_STACK, SPILL_STACK> st;
    st.sh = BATCH ? s_batch_stack + warp * (SMEM_STACK * 32) + lane : &s_stack[BATCH ? 0 : warp][0][lane];
    st.put(0, kStackEnd);

    bool live = false;
    bool queueDry = false;          // warp-uniform
    uint32_t rid = 0;
    TRay r{};                       // ray in the space of the structure being traversed
    float hitDist = 0, second = 0, hu = 0, hv = 0;
    int32_t hitID = -1, hitInst = -1, curInst = -1;
    int32_t node = 0;
    uint32_t sp = 0, steps = 0, flags = 0, tlasIndex = kTlasInvalid;
    const float4* nodes = TLAS ? p.tlas : p.nodes;     // of the structure being traversed
    const float4* blasTris = p.tris;
    bool occl = false;
    bool tieSuspect = false;        // closest hit: a near tie the second distance cannot show (kTieWindow)
    float tmin = p.tmin, tmax = p.tmax;
    uint32_t maxSteps = p.max_steps;
    void* out = nullptr;            // batched: the lane's result array
    unsigned long long nodeCount = 0, triCount = 0;
    float transparency = 1.0f;      // OPACITY, any hit
    int32_t matOffset = 0;          // OPACITY: of the current instance
    const uint32_t nRays = p.n_rays_dev ? min(*p.n_rays_dev, p.n_rays) : p.n_rays;
    const uint32_t nTop = TLAS ? p.n_tlas : p.n_nodes;
    // Steps between refills.  Two refinements were measured and left out: a
    // test of the live lanes at every step, to refill as soon as few are left,
    // costs more than its earlier refills give back (a million random closest
    // hits 1,127 against 1,103 us, the camera pass 951 against 940), and
    // postponing leaf tests until several lanes of the warp are at one holds
    // back lanes whose loads would overlap (1,168 against 1,112 us at three
    // lanes, the camera pass 1,025 against 976).
    const uint32_t burst = p.refill_steps;
    // rays a warp holds at a time: all lanes, or its share of a small launch
    const uint32_t share = min(p.spread_warps, gridDim.x * uint32_t(WARPS));
    // (staged warps claim whole tiles, which a few lanes would work off one after
    // the other: 1,000 closest hits on 65,536 triangles 740 instead of 142 us)
    const bool mayHold = STAGE > 0 || lane < (FEW ? (nRays - 1) / share + 1 : (nRays + share - 1) / share);

    // a ray's traversal state from its origin and direction (tmax already set)
    auto beginRay = [&](const float4& o4, const float4& d4, uint32_t nodesHere) {
        r.set(o4.x, o4.y, o4.z, d4.x, d4.y, d4.z);
        if (TLAS) {
            uint32_t* w = &s_world[warp][0][lane];
            const float v[9] = { lo2(r.no_xy), hi2(r.no_xy), lo2(r.no_zz), lo2(r.nd_xy), hi2(r.nd_xy), lo2(r.nd_zz),
                                 lo2(r.y_xy), hi2(r.y_xy), lo2(r.y_zz) };
#pragma unroll
            for (int k = 0; k < 9; k++) w[k * 32] = __float_as_uint(v[k]);
            w[9 * 32] = r.fast ? 1u : 0u;
            nodes = p.tlas;
        }
        hitDist = tmax; second = tmax; hu = 0.0f; hv = 0.0f;
        hitID = -1; hitInst = -1; curInst = -1;
        node = 0; sp = 1; steps = 0; flags = 0; occl = false; tieSuspect = false;
        tlasIndex = kTlasInvalid;
        transparency = 1.0f;
        live = true;
        // NaN direction or an empty BVH: miss (bvh.hsh:204, BVH.cpp:107)
        if (isnan(d4.x) || isnan(d4.y) || isnan(d4.z) || nodesHere == 0) node = kStackEnd;
    };

    // scenes: back to the top level, the world-space ray again
    auto leaveInstance = [&]() {
        const uint32_t* w = &s_world[warp][0][lane];
        float v[9];
#pragma unroll
        for (int k = 0; k < 9; k++) v[k] = __uint_as_float(w[k * 32]);
        r.no_xy = pack2(v[0], v[1]);
        r.no_zz = pack2(v[2], v[2]);
        r.nd_xy = pack2(v[3], v[4]);
        r.nd_zz = pack2(v[5], v[5]);
        r.y_xy = pack2(v[6], v[7]);
        r.y_zz = pack2(v[8], v[8]);
        r.fast = w[9 * 32] != 0u;
        nodes = p.tlas;
        tlasIndex = kTlasInvalid;
    };

    // staged queue of the warp, kept in shared memory between refills (no
    // registers during traversal): word 0 the current tile's first ray,
    // word 1 the next tile's (in flight while kStPending), word 2 the rays of
    // the current tile handed out (bits 0-7) and the flags below; the current
    // tile sits in buffer kStCur's value, the next in the other one
    constexpr uint32_t kStUsed = 0xffu, kStCur = 1u << 8, kStPhase0 = 1u << 9, kStPending = 1u << 11,
                       kStDry = 1u << 12, kStFault = 1u << 13, kStEmpty = 1u << 14;
    if constexpr (STAGE > 0) {
        if (lane == 0) {
            stage_barrier_init(shared_addr(&s_rbar[warp][0]));
            stage_barrier_init(shared_addr(&s_rbar[warp][1]));
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
            s_rstate[warp][0] = 0;
            s_rstate[warp][1] = 0;
            s_rstate[warp][2] = kStEmpty;     // no current tile yet
        }
        __syncwarp();
    }

    for (;;) {
        // ---- refill idle lanes (one atomic per warp) ----
        if (!queueDry) {
            const uint32_t idle = __ballot_sync(kFull, !live && mayHold);
            if (STAGE > 0 && idle) {
                uint32_t base = s_rstate[warp][0], nxt = s_rstate[warp][1], bits = s_rstate[warp][2];
                // the rays of a tile starting at b
                auto tileRays = [&](uint32_t b) { return min(uint32_t(STAGE), nRays - b); };
                // claims the next tile and starts its copy into the free buffer
                auto issue = [&]() {
                    __syncwarp();
                    uint32_t b = 0;
                    if (lane == 0) b = atomicAdd(p.work_counter, uint32_t(STAGE));
                    b = __shfl_sync(kFull, b, 0);
                    if (b >= nRays) { bits |= kStDry; return; }
                    if (b + uint32_t(STAGE) >= nRays) bits |= kStDry;
                    const uint32_t nb = (bits & kStCur) ? 0u : 1u;
                    if (lane == 0)
                        stage_bulk_load(shared_addr(&s_rays[warp][nb][0]), p.rays + size_t(b) * 3,
                                        tileRays(b) * 48u, shared_addr(&s_rbar[warp][nb]));
                    nxt = b;
                    bits |= kStPending;
                };
                uint32_t need = idle;
                while (need && !(bits & kStFault)) {
                    if ((bits & kStEmpty) || (bits & kStUsed) == tileRays(base)) {
                        if (!(bits & kStPending)) {
                            if (bits & kStDry) break;
                            issue();
                            if (!(bits & kStPending)) break;
                        }
                        const uint32_t nb = (bits & kStCur) ? 0u : 1u;
                        const uint32_t parity = (bits >> (9 + nb)) & 1u;
                        if (!__all_sync(kFull, stage_wait(shared_addr(&s_rbar[warp][nb]), parity))) {
                            if (lane == 0) atomicOr(p.error_word, kErrWaitTimeout);
                            bits |= kStFault;      // the copy stays pending: waited for again at exit
                            break;
                        }
                        bits ^= kStPhase0 << nb;
                        bits = (bits & ~(kStUsed | kStPending | kStEmpty | kStCur)) | (nb ? kStCur : 0u);
                        base = nxt;
                        if (!(bits & kStDry)) issue();
                    }
                    const uint32_t used = bits & kStUsed;
                    const uint32_t rank = __popc(need & lanemask_lt());
                    const uint32_t k = min(uint32_t(__popc(need)), tileRays(base) - used);
                    const bool mine = ((need >> lane) & 1u) && rank < k;
                    if (mine) {
                        const float4* src = &s_rays[warp][(bits & kStCur) ? 1 : 0][(used + rank) * 3];
                        rid = base + used + rank;
                        if (p.per_ray_tmax) tmax = src[2].x;
                        beginRay(src[0], src[1], nTop);
                    }
                    need &= ~__ballot_sync(kFull, mine);
                    bits += k;
                }
                if ((bits & kStFault) ||
                    ((bits & kStDry) && !(bits & kStPending) &&
                     ((bits & kStEmpty) || (bits & kStUsed) == tileRays(base))))
                    queueDry = true;
                __syncwarp();
                if (lane == 0) {
                    s_rstate[warp][0] = base;
                    s_rstate[warp][1] = nxt;
                    s_rstate[warp][2] = bits;
                }
                __syncwarp();
            } else if (idle) {
                uint32_t base = 0;
                if constexpr (FEW) {
                    base = (blockIdx.x * uint32_t(WARPS) + warp) * __popc(idle);
                    queueDry = true;
                } else {
                    const uint32_t leader = __ffs(idle) - 1;
                    if (lane == leader) base = atomicAdd(p.work_counter, __popc(idle));
                    base = __shfl_sync(kFull, base, leader);
                    if (base + __popc(idle) >= nRays) queueDry = true;
                }
                if ((idle >> lane) & 1u) {
                    const uint32_t gi = base + __popc(idle & lanemask_lt());
                    if (gi < nRays) {
                        const float4* raySrc = p.rays;
                        uint32_t ri = gi;
                        uint32_t nodesHere = nTop;
                        if (BATCH) {
                            const BatchDesc& bd = p.batches[find_batch(p.batches, p.n_batches, gi)];
                            ri = gi - bd.first;
                            raySrc = bd.rays;
                            nodes = bd.nodes;
                            blasTris = bd.tris;
                            nodesHere = bd.n_nodes;
                            tmin = bd.tmin;
                            tmax = bd.tmax;
                            maxSteps = bd.max_steps;
                            out = bd.out;
                        }
                        rid = ri;
                        float4 o4, d4;
                        if (CAMERA) {
                            // the ray made where it is traced (no ray buffer)
                            camera_ray(p.cam, ri, o4, d4);
                        } else {
                            o4 = ldg4(raySrc + size_t(ri) * 3);
                            d4 = ldg4(raySrc + size_t(ri) * 3 + 1);
                            if (p.per_ray_tmax) tmax = ldg4(raySrc + size_t(ri) * 3 + 2).x;
                        }
                        beginRay(o4, d4, nodesHere);
                    }
                }
            }
        }
        if (!__any_sync(kFull, live)) break;

        // ---- traverse: a bounded number of steps, then refill again ----
        if (live) {
            // the burst ends after `burst` steps or at the ray's step cap
            const uint32_t lim = min(steps + burst, maxSteps);
            while (node != kStackEnd) {
                if (steps >= lim) break;
                steps++;
                if (TLAS && sp < tlasIndex) {
                    if (tlasIndex != kTlasInvalid) leaveInstance();
                    if (node < 0) {
                        // CheckInstance: object-space ray, mesh, cull mask
                        const uint32_t ii = uint32_t(~node);
                        const float4* ip = p.instances + size_t(ii) * 4;
                        const float4 c0 = ldg4(ip), c1 = ldg4(ip + 1), c2 = ldg4(ip + 2), c3 = ldg4(ip + 3);
                        curInst = int32_t(ii);
                        bool enter = (__float_as_uint(c3.w) & p.cull_mask) != 0u;
                        MeshDesc m{};
                        if (enter) {
                            m = p.meshes[__float_as_int(c3.x)];
                            // an empty BLAS has no root to visit
                            enter = m.n_nodes > 0 && (!OPACITY || m.shading);
                        }
                        if (enter) {
                            r = transform_ray(r, c0, c1, c2);
                            nodes = m.nodes;
                            blasTris = OPACITY ? m.shading : m.tris;
                            if (OPACITY) matOffset = __float_as_int(c3.y);
                            node = 0;
                            tlasIndex = sp;
                        } else {
                            node = st.get(--sp);
                        }
                        // on to the root in the same round, with the lanes
                        // that are at other nodes of a mesh
                        if (!enter || steps >= lim) continue;
                        steps++;
                    }
                }
                if (BOUNDS && (node < 0 ? uint32_t(~node) >= p.n_tris : uint32_t(node) >= p.n_nodes)) {
                    flags |= kHitFlagOverflow;
                    atomicOr(p.error_word, kErrStackOverflow);
                    node = kStackEnd;
                    break;
                }
                if (node < 0) {
                    // Leaf: contiguous triangles up to the end-of-node flag.
                    int32_t tp = ~node;
                    bool end = false;
                    float leafTransparency = transparency;
                    do {
                        if (BOUNDS && uint32_t(tp) >= p.n_tris) {
                            flags |= kHitFlagOverflow;
                            atomicOr(p.error_word, kErrStackOverflow);
                            break;
                        }
                        const float4* tri = blasTris + size_t(tp) * (OPACITY ? 6 : 3);
                        const float4 a = ldg4(tri), b = ldg4(tri + 1), c = ldg4(tri + 2);
                        float opacity = 1.0f;
                        if (OPACITY) {
                            end = ldg4(tri + 4).z > 0.0f;
                            opacity = ldg4(tri + 5).w;
                        } else {
                            end = a.w > 0.0f;
                        }
                        if (COUNT) triCount++;
                        float t, u, v;
                        bool nearMiss = false;
                        const bool hit = LOOSE ? tri_test_fast(r.ox(), r.oy(), r.oz(), r.dx(), r.dy(), r.dz(), a, b, c,
                                                               t, u, v)
                                               : tri_test_traversal<TIES && !ANY>(r.ox(), r.oy(), r.oz(), r.dx(),
                                                                                  r.dy(), r.dz(), a, b, c, t, u, v,
                                                                                  nearMiss);
                        if (OPACITY) {
                            if (hit && t > tmin && t < (ANY ? tmax : hitDist)) {
                                if (opacity < 0.0f)
                                    opacity = texture_opacity(p.materials, p.n_materials, p.textures.pool,
                                                              p.textures.desc, p.textures.n, tri + 3, matOffset, u, v);
                                if (ANY) {
                                    leafTransparency = fmul(leafTransparency, fsub(1.0f, opacity));
                                } else if (opacity > 0.0f) {
                                    hitDist = t; hitID = tp; hu = u; hv = v; hitInst = curInst;
                                }
                            }
                        } else if (ANY) {
                            if (hit && t > tmin && t < tmax) { occl = true; end = true; }
                        } else if (hit && t > tmin && t < tmax) {
                            if (t < hitDist) {
                                second = hitDist;
                                hitDist = t; hitID = tp; hu = u; hv = v; hitInst = curInst;
                            } else if (t < second) {
                                second = t;
                            }
                        } else if (TIES && nearMiss && t > tmin && t < tmax && t <= fmul(hitDist, kTieWiden)) {
                            tieSuspect = true;
                        }
                        tp++;
                    } while (!end);
                    if (OPACITY && ANY) {
                        transparency = fmul(transparency, leafTransparency);
                        if (transparency < 0.000001f) transparency = 0.0f;
                        occl = !(transparency > 0.0f);
                    }
                    if ((BOUNDS && (flags & kHitFlagOverflow)) || (ANY && occl)) node = kStackEnd;
                    else node = st.get(--sp);
                    // scenes: on to a node of the same mesh in the same round
                    // (with entering's like step a path-traced sample 1,278 ->
                    // 1,267 us, the GI passes 1,057 -> 1,047; single meshes lose
                    // by it, 64 batches 2,769 -> 2,807)
                    if (!TLAS || node < 0 || steps >= lim || sp < tlasIndex) continue;
                    steps++;
                }
                {
                    const float4* np = nodes + size_t(node) * 4;
                    const NodeBoxes n = BOUNDS ? load_engine_node(np) : load_node(np);
                    if (COUNT) nodeCount++;
                    const int32_t lptr = n.lptr, rptr = n.rptr;
                    bool il, ir, leftFirst, nearCull = false;
                    if (LOOSE)
                        test_children_loose(r, n, tmin, ANY ? tmax : hitDist, il, ir, leftFirst);
                    else
                        test_children(r, n, tmin, ANY ? tmax : hitDist, !ANY, TIES && !ANY, il, ir, leftFirst, nearCull);
                    if (TIES && !ANY) tieSuspect = tieSuspect || nearCull;
                    int32_t next, far;
                    if (ANY) {
                        next = il ? lptr : rptr;
                        far = rptr;
                    } else {
                        next = leftFirst ? lptr : rptr;
                        far = leftFirst ? rptr : lptr;
                        // bvh.hsh:234-236: with only the right box hit and its
                        // entry equal to the bound, the missed left box also
                        // reports the bound, so the shader descends left and
                        // drops the right subtree, whose triangles may tie
                        if (TIES) tieSuspect = tieSuspect || (!il && ir && leftFirst);
                    }
                    if (il && ir) {
                        if (CHECKED && sp >= st.capacity) {
                            flags |= kHitFlagOverflow;
                            atomicOr(p.error_word, kErrStackOverflow);
                            node = kStackEnd;
                            break;
                        }
                        st.put(sp++, far);
                    } else if (!il && !ir) {
                        next = st.get(--sp);
                    }
                    node = next;
                }
            }
            if (node != kStackEnd && steps >= maxSteps) {
                // one more visit would exceed the cap
                flags |= kHitFlagIterCap;
                atomicOr(p.error_word, kErrIterationCap);
                node = kStackEnd;
            }
            if (node == kStackEnd) {
                if (OPACITY && ANY) {
                    p.transparency[rid] = transparency;
                } else if (ANY) {
                    uint8_t* occOut = BATCH ? static_cast<uint8_t*>(out) : p.occluded;
                    occOut[rid] = (occl && !(flags & (kHitFlagOverflow | kHitFlagIterCap))) ? 1 : 0;
                } else {
                    const bool hit = hitID >= 0;
                    uint32_t f = flags | (hit ? kHitFlagHit : 0u);
                    if (OPACITY) second = tmax;
                    else if (TIES ? (hit && fsub(second, hitDist) <= fmul(kTieWindow, hitDist)) || tieSuspect
                             : hit && fsub(second, hitDist) <= fmul(1e-6f, hitDist))
                        f |= kHitFlagNearTie;
                    float4* hp = (BATCH ? static_cast<float4*>(out) : p.hits) + size_t(rid) * 2;
                    hp[0] = make_float4(hitDist, __int_as_float(hitID), __int_as_float(hitInst), __uint_as_float(f));
                    hp[1] = make_float4(hu, hv, second, 0.0f);
                }
                live = false;
            }
        }
    }

    if constexpr (STAGE > 0) {
        // a copy left in flight by a timed-out wait must land before the CTA exits
        const uint32_t bits = s_rstate[warp][2];
        if (bits & kStPending) {
            const uint32_t nb = (bits & kStCur) ? 0u : 1u;
            (void)__all_sync(kFull, stage_wait(shared_addr(&s_rbar[warp][nb]), (bits >> (9 + nb)) & 1u));
        }
    }

    if (COUNT) {
        unsigned long long nc = nodeCount, tc = triCount;
        for (int off = 16; off > 0; off >>= 1) {
            nc += __shfl_down_sync(kFull, nc, off);
            tc += __shfl_down_sync(kFull, tc, off);
        }
        if (lane == 0) {
            atomicAdd(p.fetch_counts, nc);
            atomicAdd(p.fetch_counts + 1, tc);
        }
    }
}

template <bool ANY, bool COUNT, int MODE, int WARPS, int SMEM_STACK, int SPILL_STACK, int MIN_BLOCKS,
          bool BOUNDS = false, bool TIES = true, int STAGE = 0, bool LOOSE = false, bool CAMERA = false,
          bool OPACITY = false, bool FEW = false>
__global__ void __launch_bounds__(WARPS * 32, MIN_BLOCKS) trace_kernel(TraceParams p) {
    wait_for_previous();
    trace_rays<ANY, COUNT, MODE, WARPS, SMEM_STACK, SPILL_STACK, BOUNDS, TIES, STAGE, LOOSE, CAMERA, OPACITY, FEW>(p);
}

// One launch over batches of both query kinds: every warp takes closest-hit
// rays until none is left, then any-hit rays, so that either loop is compiled
// for its kind alone (the any-hit one with the screened box test; with the
// kind decided per lane, 64 meshes took 3,020 instead of 2,801 us).
template <bool COUNT, int WARPS, int SMEM_STACK, int SPILL_STACK, int MIN_BLOCKS, bool TIES>
__global__ void __launch_bounds__(WARPS * 32, MIN_BLOCKS) batch_kernel(TraceParams closest, TraceParams any) {
    if (closest.n_rays)
        trace_rays<false, COUNT, MODE_BATCH, WARPS, SMEM_STACK, SPILL_STACK, false, TIES, 0, false, false, false,
                   false>(closest);
    if (any.n_rays)
        trace_rays<true, COUNT, MODE_BATCH, WARPS, SMEM_STACK, SPILL_STACK, false, false, 0, false, false, false,
                   false>(any);
}

}  // namespace atlas::rt::dev
