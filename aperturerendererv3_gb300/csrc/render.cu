// Wavefront spectral path tracer (sm_103a) and the spectral LUT builder.
//
// The reference runs one megakernel thread per pixel sample through the whole
// path (CalculateRadiance, core/render/render.cuh:460-999).  Here each bounce is
// split into kernels over compacted queues of live paths:
//   raygen  -> camera ray + hero wavelength           (core/scene.cu:146-164, render.cuh:466-473)
//   extend  -> closest-hit traversal                  (render.cuh:77-108)
//   shade   -> material sample/eval, hit offset, emitter MIS, NEE light sample,
//              Russian roulette, next ray             (render.cuh:109-163, 541-907)
//   shadow  -> any-hit traversal of the NEE segments  (render.cuh:254-263)
//   finalize/accumulate -> XYZ per sample, FP64 per-pixel sums in sample order.
// Per path, random numbers are drawn in exactly the reference's order, so the
// GPU replays the reference's paths (see ar_rng.h for the stream layout).
// Queues are compacted with warp ballots and one atomic per warp.
#include <cuda_runtime.h>

#include <algorithm>

#include "ar_internal.h"
#include "ar_rng.h"

namespace ar
{
#define AR_BLOCK 256

__device__ __forceinline__ int lane_id() { return threadIdx.x & 31; }

// warp-aggregated append: one atomic per warp, order within the warp by lane
__device__ __forceinline__ int warp_append_slot(int* counter, bool pred)
{
    const unsigned m = __ballot_sync(0xffffffffu, pred);
    int base = 0;
    if (lane_id() == 0 && m) base = atomicAdd(counter, __popc(m));
    base = __shfl_sync(0xffffffffu, base, 0);
    return base + __popc(m & ((1u << lane_id()) - 1u));
}

struct DevRand
{
    ar_pcg g;
    __device__ float operator()() { return ar_rand1(&g); }
};

// ---------------------------------------------------------------- LUT build
// RGB -> basis LUT, one lattice point per thread; MLP weights staged in shared
// memory (34 KB, read as broadcast), the same arithmetic as rgb_encode.
__global__ void __launch_bounds__(AR_BLOCK) k_build_rgb_lut(float4* __restrict__ lut, const float* __restrict__ w)
{
    __shared__ float sw[AR_RGB_MLP_FLOATS];
    for (int i = threadIdx.x; i < AR_RGB_MLP_FLOATS; i += blockDim.x) sw[i] = w[i];
    __syncthreads();
    const long long total = (long long)AR_LUT_RES * AR_LUT_RES * AR_LUT_RES;
    const float invRes = 1.0f / static_cast<float>(AR_LUT_RES);
    for (long long v = blockIdx.x * (long long)blockDim.x + threadIdx.x; v < total; v += (long long)gridDim.x * blockDim.x)
    {
        const int x = (int)(v % AR_LUT_RES);
        const int y = (int)((v / AR_LUT_RES) % AR_LUT_RES);
        const int z = (int)(v / ((long long)AR_LUT_RES * AR_LUT_RES));
        const float in3[3] = {(x + 0.5f) * invRes, (y + 0.5f) * invRes, (z + 0.5f) * invRes};
        float o[4];
        rgb_encode(in3, o, sw);
        lut[v] = make_float4(o[0], o[1], o[2], o[3]);
    }
}

cudaError_t launch_build_rgb_lut(float* lut, const float* weights_dev, cudaStream_t s)
{
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    k_build_rgb_lut<<<sms * 4, AR_BLOCK, 0, s>>>(reinterpret_cast<float4*>(lut), weights_dev);
    return cudaGetLastError();
}

// Per-material spectral colours (albedo and emission bases), computed with
// the same trilinear LUT query the reference performs per interaction.
__global__ void k_prepare_materials(Material* mats, int n, const float* __restrict__ lut)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const PlainFetch f{lut};
    mats[i].albedo_c = prepare_color(mats[i].albedo, f);
    mats[i].emissive_c = prepare_color(mats[i].emissive, f);
}

cudaError_t launch_prepare_materials(Material* mats, int n, const float* lut, cudaStream_t s)
{
    if (n <= 0) return cudaSuccess;
    k_prepare_materials<<<(n + 127) / 128, 128, 0, s>>>(mats, n, lut);
    return cudaGetLastError();
}

// ---------------------------------------------------------------- hit reconstruction
// Full hit record for primitive slot `slot` at distance t (the traversal's t);
// SDF hits (the union and SDF objects) take the normal k_extend stored in *sdf_nrm.
__device__ __forceinline__ void hit_context(const DevScene& sc, int slot, V3 o, V3 d, float t, Hit* h,
                                            const float4* sdf_nrm)
{
    if (slot == AR_SLOT_SDF)
    {
        const int id = sc.trav.sdf_id;
        h->hit = true;
        h->obj = id;
        h->light = sc.prim_light[id];
        h->material = sc.prim_material[id];
        h->dist = t;
        h->pos = o + d * t;
        const float4 n = *sdf_nrm;
        h->nrm = v3(n.x, n.y, n.z);
        h->local_pos = h->pos;
        return;
    }
    const bool sdf_obj = slot <= AR_SLOT_SDFOBJ_BASE;
    const float4 a = sdf_obj ? __ldg(&sc.sdf_trav.slots[3 * (size_t)(AR_SLOT_SDFOBJ_BASE - slot)])
                             : __ldg(&sc.trav.slots[3 * (size_t)slot + 0]);
    const uint32_t tag = __float_as_uint(a.w);
    const uint32_t kind = tag >> AR_PRIM_KIND_SHIFT;
    const int id = (int)(tag & AR_PRIM_ID_MASK);
    h->hit = true;
    h->obj = id;
    h->dist = t;
    if (kind == AR_PRIM_KIND_TRI)
    {
        // triangle slots carry their primitive's material and light index in the
        // spare w lanes (filled at upload): no dependent per-primitive table reads
        const float4 b = __ldg(&sc.trav.slots[3 * (size_t)slot + 1]);
        const float4 c = __ldg(&sc.trav.slots[3 * (size_t)slot + 2]);
        h->material = __float_as_int(b.w);
        h->light = __float_as_int(c.w);
        tri_frame(o, d, t, v3(a.x, a.y, a.z), v3(b.x, b.y, b.z), v3(c.x, c.y, c.z), &h->pos, &h->nrm);
        h->local_pos = v3(0.0f, 0.0f, 0.0f);
    }
    else if (kind == AR_PRIM_KIND_SDF)
    {
        h->material = sc.prim_material[id];
        h->light = sc.prim_light[id];
        // IntersectSDFObject's hit frame (core/object/sdf/sdf_base.cuh:140-151); slot is in sdf_trav
        const Object ob = sc.trav.objects[id];
        const V3 lo = mul(ob.w2o, o - ob.center);
        const V3 ld = normalize(mul(ob.w2o, d));
        const V3 lp = lo + ld * t;
        h->pos = mul(ob.o2w, lp) + ob.center;
        const float4 n = *sdf_nrm;
        h->nrm = v3(n.x, n.y, n.z);
        h->local_pos = lp;
    }
    else
    {
        h->material = sc.prim_material[id];
        h->light = sc.prim_light[id];
        const Object ob = sc.trav.objects[id];
        if (kind == AR_PRIM_KIND_BOX) intersect_box(o, d, ob, h, true);
        else intersect_sphere(o, d, ob, h, true);
    }
}

// Albedo texel at a triangle hit: the mesh uv interpolated with the
// barycentric weights of pos, nearest texel, clamped to the edge.  Returns the
// texel index (in RGB units) or -1 when the primitive is not a triangle.
__device__ __forceinline__ int albedo_texel(const DevScene& sc, int tex, int slot, int prim, V3 pos)
{
    if (slot < 0) return -1;
    const float4 a = __ldg(&sc.trav.slots[3 * (size_t)slot + 0]);
    if ((__float_as_uint(a.w) >> AR_PRIM_KIND_SHIFT) != AR_PRIM_KIND_TRI) return -1;
    const float4 b = __ldg(&sc.trav.slots[3 * (size_t)slot + 1]);
    const float4 c = __ldg(&sc.trav.slots[3 * (size_t)slot + 2]);
    const V3 v0 = v3(a.x, a.y, a.z);
    const V3 e1 = v3(b.x, b.y, b.z) - v0, e2 = v3(c.x, c.y, c.z) - v0, d = pos - v0;
    const float d00 = dot(e1, e1), d01 = dot(e1, e2), d11 = dot(e2, e2);
    const float d20 = dot(d, e1), d21 = dot(d, e2);
    const float den = d00 * d11 - d01 * d01;
    float b1 = 0.0f, b2 = 0.0f;
    if (den > 0.0f)
    {
        b1 = (d11 * d20 - d01 * d21) / den;
        b2 = (d00 * d21 - d01 * d20) / den;
    }
    const float b0 = 1.0f - b1 - b2;
    const float* uv = sc.prim_uv + 6 * (size_t)prim;
    float u = b0 * __ldg(uv + 0) + b1 * __ldg(uv + 2) + b2 * __ldg(uv + 4);
    float v = b0 * __ldg(uv + 1) + b1 * __ldg(uv + 3) + b2 * __ldg(uv + 5);
    if (!(u == u)) u = 0.0f;
    if (!(v == v)) v = 0.0f;
    const int4 ti = __ldg(&sc.tex_info[tex]);
    const int x = min(max((int)floorf(fminf(fmaxf(u, 0.0f), 1.0f) * (float)ti.y), 0), ti.y - 1);
    const int y = min(max((int)floorf(fminf(fmaxf(v, 0.0f), 1.0f) * (float)ti.z), 0), ti.z - 1);
    return ti.x + y * ti.y + x;
}

// counters of a render wave (c.d_counters / the allocation-free scratch)
#define AR_CNT_Q0 0          // queue 0 length
#define AR_CNT_Q1 1          // queue 1 length
#define AR_CNT_PART 2        // k_partition: hits placed from the front, misses from the back
#define AR_CNT_MLP 4
#define AR_CNT_SDF 5         // k_sdf_extend's fetch counter
// by the parity of the depth, because a depth's shadow rays may still be traced
// while the next depth is extended:
#define AR_CNT_FETCH 6       // k_extend's fetch counter
#define AR_CNT_SHADOW 8      // four each: shadow queue length, k_shadow's fetch counter, shadow rays left
                             // for the SDF passes, k_sdf_shadow's fetch counter

// ---------------------------------------------------------------- raygen
struct CamParams
{
    V3 o, d, right, up;
    float tan_x, tan_y;
};

__global__ void __launch_bounds__(AR_BLOCK) k_raygen(PathState ps, int* queue, int* counter, long long first_path, int n,
                                                   int width, int height, uint64_t seed, int first_frame, CamParams cam,
                                                   int camera_inside, int* fetch_reset, bool media_record,
                                                   bool frame_record, PathOrder po,
                                                   const ulonglong2* __restrict__ jumps)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k == 0)
    {
        *counter = n;
        *fetch_reset = 0;  // the first k_extend's fetch counter
    }
    // stream jumps per sample: the render's table, or (allocation-free renders)
    // those of the samples this block's paths can belong to (its first path's
    // block of samples and the next: 2 x po.block frames), computed once
    __shared__ uint64_t s_jump[2 * AR_SAMPLE_BLOCK][2];
    uint32_t s_base = 0u, n_jump = 0u;
    if (!jumps)  // the same for every thread of the launch
    {
        const long long g_first = first_path + (long long)blockIdx.x * blockDim.x;
        s_base = (uint32_t)(g_first / ((long long)po.npix * po.block)) * po.block;
        n_jump = 2 * po.block;
        if (threadIdx.x < n_jump)
        {
            uint64_t m, c;
            ar_pcg_jump((uint64_t)(s_base + threadIdx.x + (uint32_t)first_frame) << 32, &m, &c);
            s_jump[threadIdx.x][0] = m;
            s_jump[threadIdx.x][1] = c;
        }
        __syncthreads();
    }
    if (k >= n) return;
    const long long g = first_path + k;
    uint32_t slot, smp;
    path_slot(po, (unsigned long long)g, &slot, &smp);
    const uint32_t pixel = slot_pixel(slot, (uint32_t)width, (uint32_t)height);
    const uint32_t frame = smp + (uint32_t)first_frame;
    const int i = (int)(pixel % (uint32_t)width), j = (int)(pixel / (uint32_t)width);
    DevRand R;
    const uint32_t jf = smp - s_base;
    if (jumps)
    {
        const ulonglong2 jm = jumps[smp];
        R.g = ar_pcg_init_jumped(seed, pixel, frame, jm.x, jm.y);
    }
    else if (smp >= s_base && jf < n_jump)
        R.g = ar_pcg_init_jumped(seed, pixel, frame, s_jump[jf][0], s_jump[jf][1]);
    else
        R.g = ar_pcg_init(seed, pixel, frame);  // blocks spanning more samples (images under 256 pixels)
    const float u = (i + R()) / static_cast<float>(width);
    const float v = (j + R()) / static_cast<float>(height);
    const float nx = u * 2.f - 1.f;
    // the float nearest to 2 (1 - v) - 1, without FP64: there 1 - v is exact for
    // v >= 2^-29, and below that both round to 1
    const float ny = fmaf(-2.0f, v, 1.0f);
    const float sx = nx * cam.tan_x;
    const float sy = ny * cam.tan_y;
    V3 dir = normalize(cam.d + cam.right * sx + cam.up * sy);
    dir = normalize(dir);  // CalculateRadiance normalizes its input again
    const float r0 = R(), r1 = R(), r2 = R();
    const LambdaSample ls = sample_cie1931(r0, r1, r2);
    ps.rng[k] = R.g.state;
    ps.pixel[k] = pixel;
    if (frame_record) ps.frame[k] = frame;  // read by the guided shading only
    ps.ray_o[k] = make_float4(cam.o.x, cam.o.y, cam.o.z, ls.lambda);
    ps.ray_d[k] = make_float4(dir.x, dir.y, dir.z, ls.pdf);
    ps.radiance[k] = 0.0f;
    ps.mask[k] = 1.0f;
    ps.depths[k] = 0u;
    ps.flags[k] = camera_inside ? 1u : 0u;
    // the media record is read only by shading instantiations that track media
    // (and by k_extend for rays inside an object); prev (last vertex, pdf) is
    // read only after a vertex has written it (flag bit 1)
    if (media_record)
    {
        ps.media_v[k] = make_float4(cam.o.x, cam.o.y, cam.o.z, __int_as_float(-1));
        ps.media_depth[k] = 0;
    }
    queue[k] = k;
}

// ---------------------------------------------------------------- extend
// The traversal kernels are persistent over the queue: a warp's lanes take
// rays from a global fetch counter, step their traversals, and whenever at
// least a threshold of lanes have finished, the warp fetches that many new rays
// (one atomic per warp), so lanes do not idle behind the warp's longest ray.
#ifndef AR_EXT_REFILL_MIN
#define AR_EXT_REFILL_MIN 4      // closest hit: idle lanes that trigger a refill
#endif
#ifndef AR_EXT_STEPS
#define AR_EXT_STEPS 8           // closest hit: node visits between refill checks
#endif
#ifndef AR_SHD_REFILL_MIN
#define AR_SHD_REFILL_MIN 8      // shadow rays
#endif
#ifndef AR_SHD_STEPS
#define AR_SHD_STEPS 16
#endif
#ifndef AR_EXT_REFILL_MIN0
#define AR_EXT_REFILL_MIN0 32    // camera rays: a warp refills only when all its lanes are idle, so that it
                                 // keeps one pixel's samples together (32-sample 1920x1080 terrain:
                                 // closest hits 18.5 ms, 19.3 with a refill at 8 idle lanes)
#endif
#ifndef AR_SHD_REFILL_MIN0
#define AR_SHD_REFILL_MIN0 16    // shadow rays of the first vertices (16: 6.55 ms of the same render, 32: 6.75)
#endif
#ifndef AR_ACC_BLOCK
#define AR_ACC_BLOCK 128         // k_accumulate
#endif
#ifndef AR_ACC_SAMPLES
#define AR_ACC_SAMPLES 8         // its tile's samples per pixel: 13 KB of shared memory per block; 1920x1080x32 samples
                                 // finalised and summed in 0.85 ms (4: 0.83, 16: 0.93, 32 at blocks of 32: 1.33; samples
                                 // stored by one kernel and summed by a thread per pixel in the next: 1.35)
#endif
#ifndef AR_PASS_PATHS
#define AR_PASS_PATHS 16         // grid of the passes over a whole queue (k_partition, the guide query and the
                                 // analytic SDF objects): one thread per this many paths of the wave
#endif
#ifndef AR_TRAV_MIN_BLOCKS
#define AR_TRAV_MIN_BLOCKS 4     // blocks per SM the traversal kernels are compiled for (64 registers)
#endif

// Warp-wide fetch of rays for the idle lanes: true and *q = the lane's queue
// index when it got one; *exhausted (warp-uniform) once the queue is used up.
__device__ __forceinline__ bool warp_refill(int* fetch, int n, bool active, bool* exhausted, int* q, int min_idle)
{
    const unsigned idle = __ballot_sync(0xffffffffu, !active);
    if (*exhausted || __popc(idle) < min_idle) return false;
    const int need = __popc(idle);
    const int leader = __ffs(idle) - 1;
    int base = 0;
    if (lane_id() == leader) base = atomicAdd(fetch, need);
    base = __shfl_sync(0xffffffffu, base, leader);
    if (base + need >= n) *exhausted = true;
    if (active) return false;
    *q = base + __popc(idle & ((1u << lane_id()) - 1u));
    return *q < n;
}

// The same for groups of G lanes that hold one ray each: every lane of a group
// gets the group's queue index.
template <int G>
__device__ __forceinline__ bool group_refill(int* fetch, int n, bool active, bool* exhausted, int* q, int min_idle)
{
    unsigned leaders = 1u;
    for (int k = G; k < 32; k += G) leaders |= 1u << k;
    const unsigned idle = __ballot_sync(0xffffffffu, !active) & leaders;
    const int need = __popc(idle);
    if (*exhausted || need < min_idle) return false;
    int base = 0;
    if (lane_id() == 0) base = atomicAdd(fetch, need);
    base = __shfl_sync(0xffffffffu, base, 0);
    if (base + need >= n) *exhausted = true;
    if (active) return false;
    *q = base + __popc(idle & ((1u << (lane_id() & ~(G - 1))) - 1u));
    return *q < n;
}

// Counters a kernel zeroes for later kernels of the wave (block 0, thread 0,
// before any other work): each is one that the kernel itself does not use and
// that no kernel still running could use, so the per-depth counter resets need
// no memset launches.
struct CounterReset
{
    int* a;
    int* b;
    int* c;
    int* d;
    int* e = nullptr;
    int* f = nullptr;
    int* g = nullptr;
    int* h = nullptr;
    int* i = nullptr;
};

__device__ __forceinline__ void reset_counters(const CounterReset& r)
{
    if (blockIdx.x == 0 && threadIdx.x == 0)
    {
        if (r.a) *r.a = 0;
        if (r.b) *r.b = 0;
        if (r.c) *r.c = 0;
        if (r.d) *r.d = 0;
        if (r.e) *r.e = 0;
        if (r.f) *r.f = 0;
        if (r.g) *r.g = 0;
        if (r.h) *r.h = 0;
        if (r.i) *r.i = 0;
    }
}

// Shadow rays the traversal left unoccluded, for k_sdf_shadow (list ==
// nullptr when the scene has no SDF geometry).
struct SdfPending
{
    int* list;
    int* count;
};

// closest hit of a finished traversal of the main BVH
__device__ __forceinline__ void extend_finish(const DevScene& sc, const PathState& ps, int p, int q,
                                              const TravState<false>& st)
{
    const TravResult r = st.result();
    if (sc.stats)
    {
        atomicAdd(&sc.stats[0], (unsigned long long)st.n_visits);
        atomicAdd(&sc.stats[1], (unsigned long long)st.n_tests);
        atomicAdd(&sc.stats[4], 1ull);
    }
    ps.hit_t[p] = r.t;
    ps.hit_slot[p] = r.slot;
    ps.q_slot[q] = r.slot;
}

// What bounds the smooth union's passes is the chain of field evaluations along a
// ray: 9-12 on average, a few hundred for rays that graze the surface, each the
// blend of four to six primitives one after the other.  So an evaluation reads
// the few primitives its cell can need (sdf_cell_mask; 32 primitives before),
// two lanes share a ray and its primitives, and a warp fetches new rays as soon
// as a quarter of its lanes have none, so that grazing rays do not hold the rest.
// The last few rays of a warp, marches of hundreds of steps on an emptying chip,
// get eight lanes each: one round of distances per step instead of two or three.
// Terrain with 32 primitives in a medium, 4 samples, depth 24 (all passes and
// shading): 1280x720 61.0 -> 15.7 ms, 640x360 28.8 -> 7.2, 320x180 4.9, 160x90 14.1
// -> 2.9 (with k_finish); without the wide tails 640x360 7.9 (groups of 4 there 7.4, of
// 16 7.3).  At 640x360 groups of 1 / 2 / 4 / 8 lanes took
// 13.4 / 11.8 / 11.3 / 13.2 ms, at 1280x720 22.1 / 22.2 / 24.9 / 34.3; 4 blocks per
// SM 10.9, 3 blocks 11.3.
#define AR_SDF_GROUP 2        // lanes per ray
#define AR_SDF_MIN_BLOCKS 4   // blocks per SM the marches are compiled for
#define AR_SDF_IDLE 4         // idle groups that trigger a refill (2 and 8 measure alike)
#define AR_SDF_EVALS 4        // evaluations between refill checks (2 and 8 alike)
#define AR_SDF_TAIL_GROUP 8   // lanes per ray once a warp's last rays are few (sdf_tail_source)

// sdf_fold by a group of G lanes with the same p and mask: each lane computes one
// primitive's distance, every lane folds them in order.
template <int G>
__device__ __forceinline__ float sdf_fold_group(const SdfUnion& s, unsigned long long mask, V3 p)
{
    const int sub = lane_id() & (G - 1), lead = lane_id() & ~(G - 1);
    const unsigned gm = ((1u << G) - 1u) << lead;  // the group's lanes take the same branches
    float d = 0.0f;
    bool first = true;
    for (int base = 0; base < 64; base += 32)
    {
        uint32_t m = (uint32_t)(mask >> base);
        while (m)
        {
            uint32_t mine = m, rest = m;
#pragma unroll
            for (int j = 0; j < G; ++j)
            {
                if (j == sub) mine = rest;
                rest &= rest - 1u;
            }
            float di = 0.0f;
            if (mine)
            {
                const int i = base + __ffs((int)mine) - 1;
                di = sdf_prim_flat(s.prims[2 * i], s.prims[2 * i + 1], p);
            }
#pragma unroll
            for (int j = 0; j < G; ++j)
            {
                const float dj = __shfl_sync(gm, di, lead + j);
                if (m)
                {
                    d = first ? dj : sdf_blend(s, d, dj);
                    first = false;
                }
                m &= m - 1u;
            }
        }
    }
    return d;
}

// A ray's march through the smooth union (sdf_march, one evaluation of the
// field per step() so that a warp's lanes can be at different points of
// different rays): the sign at the origin, the march, and, for a surface hit
// that is kept, the six evaluations of its normal (sdf_normal).
struct SdfMarch
{
    V3 o, d;
    float t, t1, eps;
    int n;          // -1: at the origin; then the march's steps; then AR_SDF_STEPS + axis sample
    bool inside;
    V3 g;           // the normal's differences
    int cell = -2;  // the cell whose mask this is
    unsigned long long mask = 0ull;

    // false: the ray does not reach the union before tmax
    __device__ bool begin(const SdfUnion& s, V3 o_, V3 d_, float eps_, float tmax)
    {
        float t0;
        if (s.count <= 0 || !sdf_bounds_interval(s, o_, d_, &t0, &t1) || t0 >= tmax) return false;
        o = o_;
        d = d_;
        eps = eps_;
        t1 = fminf(t1, tmax);
        t = fmaxf(0.0f, t0);
        n = -1;
        return true;
    }
    __device__ void begin_normal()
    {
        o = o + d * t;
        n = AR_SDF_STEPS;
    }
    __device__ V3 point() const
    {
        if (n < 0) return o;
        if (n < AR_SDF_STEPS) return o + d * t;
        const int k = n - AR_SDF_STEPS;
        const float h = 1.0e-4f;
        const V3 e = v3(k < 2 ? h : 0.0f, k == 2 || k == 3 ? h : 0.0f, k >= 4 ? h : 0.0f);
        return (k & 1) ? o - e : o + e;
    }
    // the field there, by this lane or by the group of G lanes that holds this ray
    // (all of them call with the same state); the mask stays while the ray is in
    // one cell
    template <int G>
    __device__ float field(const SdfUnion& s)
    {
        const V3 p = point();
        const int c = sdf_cell(s, p);
        if (c != cell)
        {
            cell = c;
            mask = c >= 0 ? s.cells[c] : sdf_all(s);
        }
        return G > 1 ? sdf_fold_group<G>(s, mask, p) : sdf_fold(s, mask, p);
    }
    // takes the field's value at point(): 0 goes on, 1 no crossing, 2 crossing
    // at t, 3 the normal is complete in g
    __device__ int take(float f)
    {
        if (n < 0)
        {
            inside = f <= 0.0f;
            n = 0;
            return 0;
        }
        if (n < AR_SDF_STEPS)
        {
            if (inside ? (f > 0.0f && f < eps) : (f < 0.0f && -f < eps)) return 2;
            t += fmaxf(fabsf(f), eps * 0.5f);
            ++n;
            return (t > t1 || n >= AR_SDF_STEPS) ? 1 : 0;
        }
        const int k = n - AR_SDF_STEPS;
        if (k == 0) g.x = f;
        else if (k == 1) g.x = g.x - f;
        else if (k == 2) g.y = f;
        else if (k == 3) g.y = g.y - f;
        else if (k == 4) g.z = f;
        else g.z = g.z - f;
        ++n;
        return k == 5 ? 3 : 0;
    }
    // this march as lane src holds it (a whole warp calls)
    __device__ void copy_from(int src)
    {
        const unsigned all = 0xffffffffu;
        o = v3(__shfl_sync(all, o.x, src), __shfl_sync(all, o.y, src), __shfl_sync(all, o.z, src));
        d = v3(__shfl_sync(all, d.x, src), __shfl_sync(all, d.y, src), __shfl_sync(all, d.z, src));
        g = v3(__shfl_sync(all, g.x, src), __shfl_sync(all, g.y, src), __shfl_sync(all, g.z, src));
        t = __shfl_sync(all, t, src);
        t1 = __shfl_sync(all, t1, src);
        eps = __shfl_sync(all, eps, src);
        n = __shfl_sync(all, n, src);
        inside = __shfl_sync(all, (int)inside, src) != 0;
        cell = -2;
    }
};

// The end of a marching kernel: with no ray left to fetch and at most
// 32 / AR_SDF_TAIL_GROUP in the warp, those rays are spread over its idle lanes.
// Returns the lane that holds the ray of this lane's wide group (-1: none), or -2
// while there are more rays or some to fetch.
__device__ __forceinline__ int sdf_tail_source(bool active, bool exhausted)
{
    const unsigned act = __ballot_sync(0xffffffffu, active);
    unsigned leaders = 1u;
    for (int k = AR_SDF_GROUP; k < 32; k += AR_SDF_GROUP) leaders |= 1u << k;
    unsigned left = act & leaders;
    if (!exhausted || __popc(left) > 32 / AR_SDF_TAIL_GROUP) return -2;
    for (int j = lane_id() / AR_SDF_TAIL_GROUP; j > 0; --j) left &= left - 1u;
    return left ? __ffs((int)left) - 1 : -1;
}

// The object a ray is inside of, as the path's media record has it, may be any
// primitive: inside one, a path that scatters off another surface (the camera in a
// room, the union in glass) takes that one.  Rays inside an SDF object test it in
// the SDF pass.
__device__ __forceinline__ bool inside_sdf_object(const Object* objects, int object_count, int id)
{
    return id >= 0 && id < object_count && objects[id].type == AR_OBJ_SDF;
}

// Rays inside any other: the hit on it alone, its slot or -1 and t.  The union has
// no slot; its own pass marches it.
__device__ __forceinline__ int enclosing_hit(const DevScene& sc, int id, V3 o, V3 d, float tmin, float* t)
{
    const int s = sc.prim_slot[id];
    int hit_id;
    const float th = s >= 0 ? prim_hit<false>(sc.trav, s, make_shear(d), o, d, &hit_id, tmin) : -1.0f;
    *t = th >= tmin ? th : 0.0f;
    return th >= tmin ? s : -1;
}

// The SDF objects' part of a closest hit (slot, t: the main BVH's): their own
// BVH, or, for a ray inside one of them (AR_SLOT_SOLO), that object alone.  A hit
// on one replaces slot and t and leaves its normal in hit_nrm.  Returns whether
// the smooth union is still to be marched.
__device__ __forceinline__ bool sdf_objects_hit(const DevScene& sc, const PathState& ps, int p, V3 o, V3 d, float tmin,
                                                int& slot, float& t)
{
    const float seps = 0.5f * fmaxf(tmin, 1.0e-3f);
    int obj_slot = -1;  // slot in the SDF objects' BVH
    const bool solo = slot == AR_SLOT_SOLO;
    if (solo)
    {
        const int s = sc.prim_slot[__float_as_int(ps.media_v[p].w)];
        int id;
        const float th = prim_hit<true>(sc.sdf_trav, s, make_shear(d), o, d, &id, tmin, seps);
        slot = -1;
        t = 0.0f;
        if (th >= tmin)
        {
            obj_slot = s;
            t = th;
        }
    }
    else if (sc.sdf_trav.node_count > 0)
    {
        TravResult r;
        r.slot = slot;
        r.t = slot >= 0 ? t : __int_as_float(0x7f800000);
        r.id = slot >= 0 ? (int)(__float_as_uint(sc.trav.slots[3 * (size_t)slot].w) & AR_PRIM_ID_MASK) : -1;
        const TravResult r2 = sdf_bvh_trace<false>(sc.sdf_trav, o, d, tmin, __int_as_float(0x7f800000), seps, r);
        if (r2.id != r.id)
        {
            obj_slot = r2.slot;
            t = r2.t;
        }
    }
    if (obj_slot >= 0)
    {
        const int id = (int)(__float_as_uint(sc.sdf_trav.slots[3 * (size_t)obj_slot].w) & AR_PRIM_ID_MASK);
        const Object ob = sc.trav.objects[id];
        const V3 lo = mul(ob.w2o, o - ob.center);
        const V3 ld = normalize(mul(ob.w2o, d));
        const V3 nn = sdf_obj_normal(sdf_obj_field(sc.trav, ob, id), ob.extent, ob.o2w, lo + ld * t, seps);
        ps.hit_nrm[p] = make_float4(nn.x, nn.y, nn.z, 0.0f);
        slot = AR_SLOT_SDFOBJ_BASE - obj_slot;
    }
    return !solo;
}

// whether an SDF object lies on the shadow segment
__device__ __forceinline__ bool sdf_objects_occlude(const DevScene& sc, V3 o, V3 d, float tmax, float sdf_eps)
{
    if (sc.sdf_trav.node_count <= 0) return false;
    TravResult r;
    r.t = tmax;
    r.slot = -1;
    r.id = -1;
    return sdf_bvh_trace<true>(sc.sdf_trav, o, d, 0.0f, tmax, sdf_eps, r).slot >= 0;
}

// The SDF objects' pass of the closest hits (scenes with SDF objects only).
__global__ void __launch_bounds__(AR_BLOCK) k_sdf_objects(DevScene sc, PathState ps, const int* __restrict__ queue,
                                                        const int* __restrict__ counter)
{
    const int n = *counter;
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < n; q += gridDim.x * blockDim.x)
    {
        const int p = queue[q];
        const float4 ro = ps.ray_o[p], rd = ps.ray_d[p];
        int slot = ps.hit_slot[p];
        float t = ps.hit_t[p];
        sdf_objects_hit(sc, ps, p, v3(ro.x, ro.y, ro.z), v3(rd.x, rd.y, rd.z),
                        intersect_eps((int)(ps.depths[p] >> 16)), slot, t);
        ps.hit_t[p] = t;
        ps.hit_slot[p] = slot;
        ps.q_slot[q] = slot;
    }
}

// Some evaluations of a closest hit's march by its group of G lanes; false when it is done.
template <int G>
__device__ __forceinline__ bool sdf_extend_advance(const SdfUnion& un, const PathState& ps, SdfMarch& m, int p, int q, int slot,
                                                   float& t, float tmin)
{
    for (int it = 0; it < AR_SDF_EVALS; ++it)
    {
        const int r = m.take(m.field<G>(un));
        if (r == 0) continue;
        if (r == 2 && m.t >= tmin && (slot == -1 || m.t < t))
        {
            t = m.t;
            m.begin_normal();
            continue;
        }
        if (r == 3)
        {
            // every lane of the group stores the same values
            const V3 nn = normalize(m.g);
            ps.hit_nrm[p] = make_float4(nn.x, nn.y, nn.z, 0.0f);
            ps.hit_t[p] = t;
            ps.hit_slot[p] = AR_SLOT_SDF;
            ps.q_slot[q] = AR_SLOT_SDF;
        }
        return false;
    }
    return true;
}

// The smooth union's pass of the closest hits: marched up to the hit so far (it
// has the largest primitive id, so a hit at equal t wins), and the normal of a
// hit (central differences of the field), which k_shade reads from hit_nrm.
// Rays inside an SDF object test only that object (objects: null without any).
__global__ void __launch_bounds__(AR_BLOCK, AR_SDF_MIN_BLOCKS)
    k_sdf_extend(SdfUnion un, const Object* __restrict__ objects, int object_count, PathState ps, const int* __restrict__ queue,
                 const int* __restrict__ counter, int* fetch)
{
    const int n = *counter;
    SdfMarch m;
    m.n = 0;
    int p = 0, q = 0, slot = -1;
    float t = 0.0f, tmin = 0.0f;
    bool active = false, exhausted = false;
    while (true)
    {
        if (group_refill<AR_SDF_GROUP>(fetch, n, active, &exhausted, &q, AR_SDF_IDLE))
        {
            p = queue[q];
            const float4 ro = ps.ray_o[p], rd = ps.ray_d[p];
            tmin = intersect_eps((int)(ps.depths[p] >> 16));
            slot = ps.hit_slot[p];
            t = ps.hit_t[p];
            const int mobj = objects && (ps.flags[p] & 1u) ? __float_as_int(ps.media_v[p].w) : -1;
            const bool solo = inside_sdf_object(objects, object_count, mobj);
            active = !solo && m.begin(un, v3(ro.x, ro.y, ro.z), v3(rd.x, rd.y, rd.z), sdf_eps(tmin),
                                      slot != -1 ? t : 3.0e38f);
        }
        if (__ballot_sync(0xffffffffu, active) == 0)
        {
            if (exhausted) break;
            continue;
        }
        const int src = sdf_tail_source(active, exhausted);
        if (src != -2)
        {
            const int from = max(src, 0);
            m.copy_from(from);
            p = __shfl_sync(0xffffffffu, p, from);
            q = __shfl_sync(0xffffffffu, q, from);
            slot = __shfl_sync(0xffffffffu, slot, from);
            t = __shfl_sync(0xffffffffu, t, from);
            tmin = __shfl_sync(0xffffffffu, tmin, from);
            if (src >= 0)
                while (sdf_extend_advance<AR_SDF_TAIL_GROUP>(un, ps, m, p, q, slot, t, tmin)) {}
            break;
        }
        if (active) active = sdf_extend_advance<AR_SDF_GROUP>(un, ps, m, p, q, slot, t, tmin);
    }
}

__global__ void __launch_bounds__(AR_BLOCK, AR_TRAV_MIN_BLOCKS) k_extend(DevScene sc, PathState ps, const int* __restrict__ queue,
                                                   const int* __restrict__ counter, int* fetch, unsigned int* err,
                                                   int min_idle, CounterReset rs)
{
    reset_counters(rs);
    const int n = *counter;
    TravState<false> st;
    uint2 stk[AR_TRAV_STACK];
    int p = 0, q = 0;
    bool active = false, exhausted = false;
    while (true)
    {
        if (warp_refill(fetch, n, active, &exhausted, &q, min_idle))
        {
            p = queue[q];
            const float4 ro = ps.ray_o[p], rd = ps.ray_d[p];
            const V3 o = v3(ro.x, ro.y, ro.z), d = v3(rd.x, rd.y, rd.z);
            const float tmin = intersect_eps((int)(ps.depths[p] >> 16));
            // the media record is read only for rays inside an object (rare)
            const int mobj = (ps.flags[p] & 1u) ? __float_as_int(ps.media_v[p].w) : -1;
            if (mobj >= 0)
            {
                // inside a medium: intersect only the enclosing object (render.cuh:89-92);
                // an SDF object is left to the SDF pass
                if (inside_sdf_object(sc.trav.objects, sc.trav.object_count, mobj))
                {
                    ps.hit_t[p] = 0.0f;
                    ps.hit_slot[p] = AR_SLOT_SOLO;
                    ps.q_slot[q] = AR_SLOT_SOLO;
                }
                else
                {
                    float th;
                    const int s = enclosing_hit(sc, mobj, o, d, tmin, &th);
                    ps.hit_t[p] = th;
                    ps.hit_slot[p] = s;
                    ps.q_slot[q] = s;
                }
                if (sc.stats) atomicAdd(&sc.stats[4], 1ull);
            }
            else
            {
                st.init(sc.trav, o, d, tmin, __int_as_float(0x7f800000), stk);
                active = true;
            }
        }
        if (__ballot_sync(0xffffffffu, active) == 0)
        {
            if (exhausted) break;
            continue;
        }
        if (active)
        {
            for (int it = 0; it < AR_EXT_STEPS; ++it)
            {
                if (!st.step(sc.trav, err))
                {
                    extend_finish(sc, ps, p, q, st);
                    active = false;
                    break;
                }
            }
        }
    }
}

// MLP guide: the network inputs (position and reflected view direction) of
// the queued paths that hit a surface at one of their first AR_MLP_MAX_NDD
// non-delta vertices, outside media; those paths are appended to `list` (the
// inference queue) and flagged in q_pos.w, the others flagged off.
__global__ void __launch_bounds__(AR_BLOCK) k_mlp_query(DevScene sc, PathState ps, const int* __restrict__ queue,
                                                      const int* __restrict__ counter, int* list, int* list_counter)
{
    const int n = *counter;
    const int stride = gridDim.x * blockDim.x;
    for (int base = (blockIdx.x * blockDim.x + threadIdx.x) & ~31; base < n; base += stride)
    {
        const int q = base + lane_id();
        bool want = false;
        int p = 0;
        if (q < n)
        {
            p = queue[q];
            const int slot = ps.hit_slot[p];
            const int ndd = (int)(ps.depths[p] >> 16);
            want = slot != -1 && ndd < AR_MLP_MAX_NDD && (ps.flags[p] & 1u) == 0u;
            if (want)
            {
                const float4 ro = ps.ray_o[p], rd = ps.ray_d[p];
                Hit h;
                hit_context(sc, slot, v3(ro.x, ro.y, ro.z), v3(rd.x, rd.y, rd.z), ps.hit_t[p], &h, &ps.hit_nrm[p]);
                const V3 wr = reflect(v3(rd.x, rd.y, rd.z), h.nrm);
                ps.q_pos[p] = make_float4(h.pos.x, h.pos.y, h.pos.z, 1.0f);
                ps.q_wr[p] = make_float4(wr.x, wr.y, wr.z, 0.0f);
            }
            else
            {
                ps.q_pos[p] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            }
        }
        const int slot_out = warp_append_slot(list_counter, want);
        if (want) list[slot_out] = p;
    }
}

// ---------------------------------------------------------------- shade
struct ShadeParams
{
    int use_nee;
    int max_depth;
    float* grad;  // replay adjoint: float32 texel gradients (3 per texel), or null
    int mlp_ready;  // MLP guide: the network has trained long enough to replace the voxel probes
    double* grad_medium;  // replay adjoint: d loss / d (medium albedo, medium emission), or null
    float4* gbuf;         // denoiser: first-hit record per path (2 float4), or null
};

// CollectRadiance (core/render/render.cuh:353-432) on the path's collection
// slots; valid bits live in flags bits 8..12.
__device__ __forceinline__ void collect_radiance(const PathState& ps, int p, uint32_t& fl, float endpointLe, V3 nextDir,
                                                 float segContrib, float rrProb, int ndd, bool allowStart, bool advance,
                                                 V3 rayDir, V3 hitLoc, V3 hitNrm)
{
    const int cap = ps.capacity;
    if (endpointLe != 0.0f)
    {
        const int hi = min(ndd, AR_PG_COLLECT_DEPTH);
        for (int i = 0; i < hi; ++i)
        {
            const float m = ps.pg_loc[i * cap + p].w;
            if (m != 0.0f)
            {
                float4 d = ps.pg_dir[i * cap + p];
                d.w = d.w + m * endpointLe;
                ps.pg_dir[i * cap + p] = d;
                fl |= 1u << (8 + i);
            }
        }
    }
    if (allowStart && ndd < AR_PG_COLLECT_DEPTH)
    {
        const float4 l = ps.pg_loc[ndd * cap + p];
        if (l.w == 0.0f)
        {
            const float w = ps.pg_dir[ndd * cap + p].w;
            ps.pg_dir[ndd * cap + p] = make_float4(nextDir.x, nextDir.y, nextDir.z, w);
            ps.pg_loc[ndd * cap + p] = make_float4(hitLoc.x, hitLoc.y, hitLoc.z, 1.0f);
            const V3 vd = reflect(rayDir, hitNrm);
            ps.pg_vdir[ndd * cap + p] = make_float4(vd.x, vd.y, vd.z, mlp_pack_normal(hitNrm));
        }
    }
    if (advance)
    {
        const float invQ = (float)(1.0 / (double)rrProb);
        const int hi = min(ndd + (allowStart ? 1 : 0), AR_PG_COLLECT_DEPTH);
        for (int i = 0; i < hi; ++i)
        {
            float4 l = ps.pg_loc[i * cap + p];
            if (l.w != 0.0f)
            {
                l.w = l.w * (segContrib * invQ);
                ps.pg_loc[i * cap + p] = l;
            }
        }
    }
}

// Prefetch into L2 of the path state k_shade reads first (and of the hit's
// primitive slot), for a path this thread shades in its next pass.
__device__ __forceinline__ void prefetch_l2(const void* a) { asm volatile("prefetch.global.L2 [%0];" ::"l"(a)); }

__device__ __forceinline__ void prefetch_shade_inputs(const DevScene& sc, const PathState& ps, int2 e)
{
    const int p = e.x;
    prefetch_l2(&ps.ray_o[p]);
    prefetch_l2(&ps.ray_d[p]);
    prefetch_l2(&ps.rng[p]);
    prefetch_l2(&ps.pixel[p]);
    prefetch_l2(&ps.depths[p]);
    prefetch_l2(&ps.flags[p]);
    prefetch_l2(&ps.radiance[p]);
    prefetch_l2(&ps.mask[p]);
    prefetch_l2(&ps.hit_t[p]);
    if (e.y >= 0)
    {
        const float4* sl = sc.trav.slots + 3 * (size_t)e.y;
        prefetch_l2(sl);
        prefetch_l2(sl + 2);
    }
}

// The extended queue ordered for shading: hits with their slot from the front,
// misses from the back.  k_shade then gives whole warps and blocks to one kind
// of work (a hit runs the BSDF, NEE and roulette; a miss adds the sky and
// ends) without reordering inside the kernel.  One atomic per block and end.
// Which thread shades which path does not change any path's result.
__global__ void __launch_bounds__(AR_BLOCK) k_partition(const int* __restrict__ queue, const int* __restrict__ q_slot,
                                                        const int* __restrict__ counter, int2* __restrict__ out,
                                                        int* front, int* back)
{
    const int n = *counter;
    __shared__ int s_hits[AR_BLOCK / 32], s_miss[AR_BLOCK / 32], s_base[2];
    const int w = threadIdx.x >> 5;
    for (int bbase = blockIdx.x * blockDim.x; bbase < n; bbase += gridDim.x * blockDim.x)
    {
        const int q = bbase + (int)threadIdx.x;
        const bool valid = q < n;
        const int p = valid ? queue[q] : -1;
        const int slot = valid ? q_slot[q] : -1;
        const bool hit = valid && slot != -1;
        const unsigned hb = __ballot_sync(0xffffffffu, hit), mb = __ballot_sync(0xffffffffu, valid && !hit);
        if (lane_id() == 0)
        {
            s_hits[w] = __popc(hb);
            s_miss[w] = __popc(mb);
        }
        __syncthreads();
        int hbase = 0, mbase = 0, th = 0, tm = 0;
        for (int k = 0; k < AR_BLOCK / 32; ++k)
        {
            if (k < w)
            {
                hbase += s_hits[k];
                mbase += s_miss[k];
            }
            th += s_hits[k];
            tm += s_miss[k];
        }
        if (threadIdx.x == 0)
        {
            s_base[0] = th ? atomicAdd(front, th) : 0;
            s_base[1] = tm ? atomicAdd(back, tm) : 0;
        }
        __syncthreads();
        const unsigned below = (1u << lane_id()) - 1u;
        if (hit) out[s_base[0] + hbase + __popc(hb & below)] = make_int2(p, slot);
        else if (valid) out[n - 1 - (s_base[1] + mbase + __popc(mb & below))] = make_int2(p, -1);
        __syncthreads();  // the shared counts are rewritten by the next pass
    }
}

// Scene features a k_shade instantiation handles, fixed at compile time: the
// BSDF models (AR_MATS_* bits), the participating medium and albedo textures.
// Scenes of opaque surfaces only (no glass or medium, the camera outside every
// object) run an instantiation without that code, with or without textures: the
// same arithmetic for everything it keeps, less code and fewer registers
// (textured Cornell box 256 x 256, forward and replay: 24.8 ms with every
// feature compiled in, 22.8 without glass and medium; voxel guide 480 x 270
// untextured 8.9 ms with every feature, 8.2 with AR_FEAT_SURFACE).
#define AR_FEAT_MEDIUM (1 << 4)
#define AR_FEAT_TEX (1 << 5)
#define AR_FEAT_ALL (AR_MATS_ALL | AR_FEAT_MEDIUM | AR_FEAT_TEX)
#define AR_FEAT_SURFACE (AR_MATS_DIFFUSE | AR_MATS_LIGHT | AR_MATS_GGX)
#define AR_FEAT_TEXTURED (AR_FEAT_SURFACE | AR_FEAT_TEX)

// The shadow ray a vertex casts for its light sample, and what it adds to the
// path's radiance either way.
struct ShadowRay
{
    bool cast = false, valid = false;
    V3 o = v3(0, 0, 0), d = v3(0, 0, 0);
    float tmax = 0.0f, vun = 0.0f, vocc = 0.0f, sdf_eps = 0.0f;
};

// One vertex of path p: the hit (slot, -1: none) reconstructed, the BSDF sampled,
// emission and next-event estimation, roulette, the path's state for its next
// ray.  Returns whether the path goes on; sh is the shadow ray to test.  Every
// thread of the block calls it (barriers inside), those without a path with
// active = false.  next: the entry this thread shades after this one, whose
// state is prefetched once this one's loads have arrived (path -1: none).
// Without glass the path never enters an object: its media record stays
// the default and is neither read nor written.  Unguided forward renders
// read nothing of an ended path but its radiance.
template <int GUIDE, int ADJ, int FEAT, bool SYNC_NEE>
__device__ __forceinline__ bool shade_vertex(const DevScene& sc, const PathState& ps, const ShadeParams& prm,
                                             const float* s_lam, bool active, int p, int slot, int2 next, ShadowRay& sh,
                                             float& g_med_albedo, float& g_med_emission)
{
    constexpr bool TRACK_MEDIA = (FEAT & AR_MATS_GLASS) != 0;
    constexpr bool STORE_ENDED = GUIDE != 0 || ADJ == AR_ADJ_REPLAY;
    bool keep = false;
    // state of the vertex, across the phases below
    V3 rayO = v3(0, 0, 0), rayD = v3(0, 0, 0);
    float lambda = 0.0f, lambda_pdf = 0.0f, d65 = 0.0f, radiance = 0.0f, mask = 0.0f, eps = 0.0f;
    Basis lb = {{0.0f, 0.0f, 0.0f, 0.0f}};
    int depth = 0, ndd = 0, texel = -1;
    uint32_t fl = 0u;
    bool prev_did_nee = false, scatter = false, ended = true;
    Media media = media_default();
    DevRand R;
    R.g.state = 0u;
    R.g.inc = 0u;
    Hit h;
    h.hit = false;
    h.obj = -1;
    h.light = -1;
    h.dist = 0.0f;
    h.pos = v3(0, 0, 0);
    h.nrm = v3(0, 0, 0);
    h.local_pos = v3(0, 0, 0);
    BsdfSample S = bsdf_sample_default();
    // the hit's material: read where it is used (a copy would stay in registers
    // through the whole vertex); a textured one is a copy with its texel's colour
    constexpr bool TEX = (FEAT & AR_FEAT_TEX) != 0;
    const Material* mp = sc.materials;
    Material textured;
#define VERTEX_MAT (TEX ? textured : *mp)
    if (active)
    {
        const float4 ro = ps.ray_o[p], rd = ps.ray_d[p];
        rayO = v3(ro.x, ro.y, ro.z);
        rayD = v3(rd.x, rd.y, rd.z);
        lambda = ro.w;
        lambda_pdf = rd.w;
        lb = query_lambda(lambda, s_lam);
        d65 = d65_norm(lambda, sc.d65);
        const uint32_t dep = ps.depths[p];
        depth = (int)(dep & 0xffffu);
        ndd = (int)(dep >> 16);
        fl = ps.flags[p];
        if constexpr (TRACK_MEDIA)
        {
            const float4 mv = ps.media_v[p];
            media.inside = (fl & 1u) != 0u;
            media.vertex = v3(mv.x, mv.y, mv.z);
            media.obj = __float_as_int(mv.w);
            media.depth = ps.media_depth[p];
        }
        radiance = ps.radiance[p];
        mask = ps.mask[p];
        prev_did_nee = (fl & 2u) != 0u;
        R.g.state = ps.rng[p];
        R.g.inc = ar_pcg_increment(ps.pixel[p]);

        eps = intersect_eps(ndd);
        if (slot != -1) hit_context(sc, slot, rayO, rayD, ps.hit_t[p], &h, &ps.hit_nrm[p]);
        if (next.x >= 0) prefetch_shade_inputs(sc, ps, next);

        // ---- participating medium: a free flight sampled in the medium box
        // ends the segment early with probability 1 - transmittance
        if ((FEAT & AR_FEAT_MEDIUM) && sc.medium.on)
        {
            float m0, m1;
            if (medium_segment(sc.medium, rayO, rayD, 0.0f, h.hit ? h.dist : 3.0e38f, &m0, &m1))
            {
                const float ts = m0 - arm_logf(R()) / sc.medium.sigma_t;
                if (ts < m1)
                {
                    scatter = true;
                    h.hit = false;
                    h.obj = -1;
                    h.light = -1;
                    h.dist = ts;
                    h.pos = rayO + rayD * ts;
                    h.nrm = v3(0.0f, 0.0f, 0.0f);
                }
            }
        }

        // ---- Trace (render.cuh:109-155)
        if (!h.hit && !scatter && media.inside)
        {
            S.miss_thin = true;
            S.brdf = 1.0f;
            S.next_dir = rayD;
            S.pdf = 1.0f;
            h.local_pos = rayO;
            h.obj = media.obj;
            S.delta = true;
            S.emissive = v3(0, 0, 0);
            S.media.inside = false;
            S.media.vertex = h.local_pos;
        }
        if (h.hit)
        {
            mp = sc.materials + h.material;
            if constexpr (TEX)
            {
                textured = *mp;
                if (textured.albedo_tex >= 0 && sc.tex_count > 0)
                {
                    texel = albedo_texel(sc, textured.albedo_tex, slot, h.obj, h.pos);
                    if (texel >= 0)
                    {
                        const float* tx = sc.texels + 3 * (size_t)texel;
                        textured.albedo = v3(__ldg(tx), __ldg(tx + 1), __ldg(tx + 2));
                        textured.albedo_c = prepare_color(textured.albedo, PlainFetch{sc.lut_rgb});
                    }
                }
            }
            S = evaluate_material<FEAT & AR_MATS_ALL>(lambda, lb, R, VERTEX_MAT, rayD, h, media);
        }
        else if (scatter)
        {
            // Henyey-Greenstein phase sampling; throughput x albedo
            const float e0 = R();
            const float e1 = R();
            const DirSample ph = hg_sample(e0, e1, rayD, sc.medium.g);
            S.next_dir = ph.dir;
            S.pdf = ph.pdf;
            S.brdf = sc.medium.albedo * ph.pdf;
            S.delta = false;
            S.emissive = v3(0.0f, 0.0f, 0.0f);
            S.media = media;
        }
        else
        {
            S.brdf = 1.0f;
            S.delta = false;
            S.next_dir = rayD;
            S.pdf = 1.0f;
            S.emissive = sky_lighting(rayD);
            S.media.inside = false;
        }
        // denoiser G-buffer of the camera ray's hit (RecordScreenGBuffer at
        // depth 0, core/render/render.cuh:640-643): albedo (texel when
        // textured), material index (-1: no surface), normal, distance
        if constexpr (!ADJ)
        {
            if (prm.gbuf && depth == 0)
            {
                const int mid = h.hit ? h.material : -1;
                const V3 alb = h.hit ? VERTEX_MAT.albedo : v3(0.0f, 0.0f, 0.0f);
                prm.gbuf[2 * (size_t)p] = make_float4(alb.x, alb.y, alb.z, __int_as_float(mid));
                prm.gbuf[2 * (size_t)p + 1] = make_float4(h.nrm.x, h.nrm.y, h.nrm.z, h.dist);
            }
        }
        {
            const float offsetEPS = eps * fmaxf(1.0f, length(h.pos));
            h.pos = h.pos + signf(dot(h.nrm, S.next_dir)) * h.nrm * offsetEPS * (R() + 0.5f);
        }
        media = S.media;

    }
    // ---- guided mixture sampling (render.cuh:553-638)
    const Probe* probe = nullptr;
    V3 maskq = v3(1.0f, 1.0f, 1.0f);
    float pgProb = 0.0f;
    bool mlp_on = false;           // GUIDE == 2: this vertex mixes in the network's distribution
    const uint8_t* qcells = nullptr;  // its 64 quantised cell weights (the path's inference record)
    float q_total = 1.0f;
    if (active)
    {
        if constexpr (GUIDE)
        {
            const float4 mq = ps.maskq[p];
            maskq = v3(mq.x, mq.y, mq.z);
            pgProb = guide_probability((int)ps.frame[p]);  // the path's own frame (waves may hold several)
            const bool eligible = h.hit && !S.delta && !S.pure_light && !media.inside;
            if constexpr (GUIDE == 2)
            {
                if (eligible && prm.mlp_ready && ps.q_pos[p].w > 0.0f)
                {
                    const uint8_t* q = ps.q_dist + 64 * (size_t)p;
                    qcells = q;
                    q_total = mlp_total(q);
                    mlp_on = true;
                    const float pB = S.pdf;
                    const float pP = mlp_hemisphere_pdf(q, 1.0f / q_total, S.next_dir, h.nrm);
                    if (pB > 1.0e-12f && pP > 1.0e-12f)
                    {
                        if (R() < pgProb)
                        {
                            const GuideSample g = mlp_sample_hemisphere(q, q_total, R, h.nrm);
                            if (dot(g.dir, h.nrm) > 1.0e-12f)
                            {
                                const float pBs = bsdf_pdf<FEAT & AR_MATS_ALL>(lb, VERTEX_MAT, h.nrm, rayD, g.dir);
                                S.next_dir = g.dir;
                                S.brdf = eval_bsdf_cos<FEAT & AR_MATS_ALL>(lambda, lb, VERTEX_MAT, rayD, g.dir, h, media);
                                S.pdf = (1.0f - pgProb) * fmaxf(pBs, 1.0e-12f) + pgProb * g.pdf;
                            }
                            else
                            {
                                mlp_on = false;
                            }
                        }
                        else
                        {
                            S.pdf = (1.0f - pgProb) * pB + pgProb * pP;
                        }
                    }
                    else
                    {
                        mlp_on = false;
                    }
                }
            }
            if (!mlp_on && eligible && sc.guide.probe_count > 0)
            {
                const VoxelKey key = voxel_key(h.pos, reflect(rayD, h.nrm), sc.guide.inv_unit);
                const int idx = guide_lookup(sc.guide, guide_pack(key));
                if (idx >= 0)
                {
                    probe = &sc.guide.probes[idx];
                    const float pB = S.pdf;
                    const float pP = octahedron_hemisphere_pdf(*probe, S.next_dir, h.nrm, maskq);
                    if (pB > 1.0e-12f && pP > 1.0e-12f)
                    {
                        if (R() < pgProb)
                        {
                            const GuideSample g = sample_octahedron_hemisphere(*probe, R, h.nrm, maskq);
                            if (dot(g.dir, h.nrm) > 1.0e-12f)
                            {
                                const float pBs = bsdf_pdf<FEAT & AR_MATS_ALL>(lb, VERTEX_MAT, h.nrm, rayD, g.dir);
                                S.next_dir = g.dir;
                                S.brdf = eval_bsdf_cos<FEAT & AR_MATS_ALL>(lambda, lb, VERTEX_MAT, rayD, g.dir, h, media);
                                S.pdf = (1.0f - pgProb) * fmaxf(pBs, 1.0e-12f) + pgProb * g.pdf;
                            }
                            else
                            {
                                probe = nullptr;
                            }
                        }
                        else
                        {
                            S.pdf = (1.0f - pgProb) * pB + pgProb * pP;
                        }
                    }
                    else
                    {
                        probe = nullptr;
                    }
                }
            }
        }

        // ---- emission (render.cuh:647-723)
        V3 endpointLe = v3(0.0f, 0.0f, 0.0f);
        float medium_unit = 0.0f;  // emission released at this scattering point per unit emission
        if (scatter)
        {
            medium_unit = mask * (1.0f - sc.medium.albedo) * d65;
            radiance = radiance + medium_unit * sc.medium.emission;
        }
        else if (!h.hit)
        {
            if (!S.miss_thin)
            {
                endpointLe = S.emissive;
                const PlainFetch f{sc.lut_rgb};
                radiance = radiance + mask * interact_rgb(lb, S.emissive, f) * d65;
            }
        }
        else if (h.light >= 0)
        {
            float misW = 1.0f;
            if (prm.use_nee && depth > 0 && prev_did_nee)
            {
                const float4 pv = ps.prev[p];
                const float pB = fmaxf(pv.w, 0.0f);
                const Light L = sc.lights[h.light];
                float pL = 0.0f;
                const V3 lastPos = v3(pv.x, pv.y, pv.z);
                if (L.type == AR_OBJ_CUBE) pL = box_light_pdf_omega(sc.trav.objects[L.obj], L.select_prob, lastPos, h.pos, h.nrm);
                else if (L.type == AR_OBJ_SPHERE) pL = sphere_light_pdf_omega(sc.trav.objects[L.obj], L.select_prob, lastPos, h.pos, h.nrm);
                if (pL >= 0.0f && pB > 0.0f) misW = power_heuristic(pB, pL);
            }
            endpointLe = S.emissive * misW;
            radiance = radiance + mask * interact(VERTEX_MAT.emissive_c, lb) * d65 * misW;
        }
        else if (!all_zero(S.emissive))
        {
            endpointLe = S.emissive;
        }
        if constexpr (ADJ == AR_ADJ_RECORD)
        {
            // what the gradient of this vertex's texel needs once the path's total is known
            const bool albedo_hit = texel >= 0 && VERTEX_MAT.shading == AR_MAT_DIFFUSE;
            ps.adj_rec[(size_t)depth * ps.adj_stride + p] = make_int2(albedo_hit ? texel : -1, __float_as_int(radiance));
        }
        if constexpr (ADJ == AR_ADJ_REPLAY)
        {
            // replay adjoint: every contribution still to come on this path
            // (NEE here, emission and NEE further on) carries this vertex's
            // albedo once; radiance holds the contributions that do not
            if (scatter && prm.grad_medium)
            {
                // later contributions carry this albedo once; the emission here carries (1 - albedo)
                const float dlt = ps.adj_delta[p];
                const float a = sc.medium.albedo;
                const float rest = ps.adj_total[p] - radiance;
                if (a > 1.0e-8f) g_med_albedo += dlt * rest / a;
                // d/d albedo of (1 - albedo) x emission x mask, and d/d emission
                g_med_albedo -= dlt * mask * sc.medium.emission * d65;
                g_med_emission += dlt * medium_unit;
            }
            if (prm.grad && texel >= 0 && VERTEX_MAT.shading == AR_MAT_DIFFUSE)
            {
                const float rest = ps.adj_total[p] - radiance;
                const float dlt = ps.adj_delta[p];
                const float alb = interact(VERTEX_MAT.albedo_c, lb);
                if (rest != 0.0f && dlt != 0.0f && alb > 1.0e-8f)
                {
                    const V3 g = interact_rgb_grad(lb, VERTEX_MAT.albedo, PlainFetch{sc.lut_rgb}) * (dlt * rest / alb);
                    float* gp = prm.grad + 3 * (size_t)texel;
                    if (g.x != 0.0f) atomicAdd(gp + 0, g.x);
                    if (g.y != 0.0f) atomicAdd(gp + 1, g.y);
                    if (g.z != 0.0f) atomicAdd(gp + 2, g.z);
                }
            }
        }
        if constexpr (GUIDE)
        {
            const PlainFetch f{sc.lut_rgb};
            collect_radiance(ps, p, fl, interact_rgb(lb, endpointLe, f) * d65, S.next_dir, 0.0f, 1.0f, ndd, false,
                             false, rayD, h.pos, h.nrm);
        }

        ended = (!h.hit && !S.miss_thin && !scatter) || S.terminate;
    }
    if (SYNC_NEE) __syncthreads();
    if (active)
    {
        if (!ended)
        {
            // ---- NEE (render.cuh:766-827, 206-343)
            if (!S.miss_thin)
            {
                const float useNEERate = sqrtf(saturate(mask));
                bool neeValid = false;
                if (prm.use_nee && ndd < AR_NEE_MAX_NON_DELTA_DEPTH && !S.delta && !media.inside && R() < useNEERate)
                {
                    LightSample ls;
                    ls.valid = false;
                    if (sc.light_count > 0)
                    {
                        const float r = R();
                        int pick = sc.light_count - 1;
                        float pickProb = 0.0f;
                        // first light whose running CDF exceeds r (same as the sequential scan)
                        int lo = 0, hi = sc.light_count;
                        while (lo < hi)
                        {
                            const int mid = (lo + hi) >> 1;
                            if (r < sc.lights[mid].cdf) hi = mid;
                            else lo = mid + 1;
                        }
                        if (lo < sc.light_count)
                        {
                            pick = lo;
                            pickProb = sc.lights[lo].select_prob;
                        }
                        const Light L = sc.lights[pick];
                        if (L.type == AR_OBJ_CUBE) ls = sample_box_light(R, sc.trav.objects[L.obj], h.pos);
                        else if (L.type == AR_OBJ_SPHERE) ls = sample_sphere_light(R, sc.trav.objects[L.obj], h.pos);
                        if (ls.valid)
                        {
                            ls.obj = L.obj;
                            ls.material = L.material;
                            ls.p_facet = ls.p_facet * pickProb;
                        }
                    }
                    const float vZero = mask * 0.0f * d65;
                    if (!ls.valid)
                    {
                        radiance = radiance + vZero;
                    }
                    else
                    {
                        const float pATotal = fmaxf(1e-20f, ls.p_a * ls.p_facet);
                        const V3 lun = ls.point - h.pos;
                        const float dist2 = fmaxf(dot(lun, lun), (float)1.0e-12);
                        const V3 L = lun * arm_rsqrtf(dist2);
                        const float cosX = scatter ? 1.0f : fmaxf(0.0f, dot(h.nrm, L));
                        const float cosY = fmaxf(0.0f, dot(ls.normal, -L));
                        float vUn = vZero;
                        bool validUn = false;
                        if (!(cosX <= 0.0f || cosY <= 0.0f))
                        {
                            const float brdfCos =
                                scatter ? sc.medium.albedo * hg_pdf(dot(rayD, L), sc.medium.g)
                                        : eval_bsdf_cos<FEAT & AR_MATS_ALL>(lambda, lb, VERTEX_MAT, rayD, L, h, media_default());
                            const float G = (cosY / dist2);
                            const float le = interact(sc.materials[ls.material].emissive_c, lb);
                            const float contribution = brdfCos * le * (G / pATotal);
                            const float pLight = area_to_solid_angle_pdf(h.pos, ls.point, ls.normal, ls.p_facet * ls.p_a);
                            float pBsdf = scatter ? hg_pdf(dot(rayD, L), sc.medium.g)
                                                  : fmaxf(bsdf_pdf<FEAT & AR_MATS_ALL>(lb, VERTEX_MAT, h.nrm, rayD, L), 0.0f);
                            if constexpr (GUIDE)
                            {
                                if (probe)
                                    pBsdf = (1.0f - pgProb) * pBsdf +
                                            pgProb * octahedron_hemisphere_pdf(*probe, L, h.nrm, maskq);
                                if (mlp_on)
                                    pBsdf = (1.0f - pgProb) * pBsdf +
                                            pgProb * mlp_hemisphere_pdf(qcells, 1.0f / q_total, L, h.nrm);
                            }
                            const float misW = power_heuristic(pLight, pBsdf);
                            vUn = mask * (contribution * misW) * d65;
                            if ((FEAT & AR_FEAT_MEDIUM) && sc.medium.on)
                                vUn *= medium_transmittance(sc.medium, h.pos, L, sqrtf(dist2));
                            validUn = true;
                        }
                        // shadow segment (intersection.cuh:285-310)
                        V3 dirS = ls.point - h.pos;
                        const float distance = length(dirS);
                        bool traced = false;
                        if (distance > 0.0f)
                        {
                            dirS = dirS / distance;
                            const float seps = intersect_eps(depth) * fmaxf(1.0f, fmaxf(length(h.pos), length(ls.point)));
                            const float tmax = fmaxf(0.0f, distance - seps);
                            if (tmax > 0.0f)
                            {
                                traced = true;
                                sh.cast = true;
                                sh.o = h.pos;
                                sh.d = dirS;
                                sh.tmax = tmax;
                                sh.sdf_eps = 0.5f * intersect_eps(depth);  // SDF_EPS of the NEE depth
                                sh.vun = vUn;
                                sh.vocc = vZero;
                                sh.valid = validUn;
                            }
                        }
                        if (!traced)
                        {
                            radiance = radiance + vUn;
                            neeValid = validUn;
                        }
                    }
                }
                fl = (fl & ~2u) | (neeValid ? 2u : 0u);
                ps.prev[p] = make_float4(h.pos.x, h.pos.y, h.pos.z, S.pdf);
            }
            // ---- Russian roulette (render.cuh:829-859)
            const float contrib = S.brdf / fmaxf(S.pdf, 1e-12f);
            float pSurvive = 1.0f;
            bool survived = true;
            if (ndd >= AR_MIN_TRACING_DEPTH)
            {
                const float basic = clampf(mask * 0.5f + mask * 0.5f, 0.05f, 0.95f);
                pSurvive = lerpf(basic, 1.0f, media.inside ? AR_DELTA_RR_TERMINATE_REDUCE : 0.0f);
                if (R() > pSurvive) survived = false;
            }
            if (survived)
            {
                if constexpr (GUIDE)
                {
                    const bool allowStart = h.hit && !S.delta && !S.pure_light && !media.inside;
                    collect_radiance(ps, p, fl, 0.0f, S.next_dir, contrib, pSurvive, ndd, allowStart, true, rayD, h.pos,
                                     h.nrm);
                }
                mask = mask * contrib;
                mask = mask / pSurvive;
                if constexpr (GUIDE)
                {
                    const V3 xyz = lambda_to_xyz(lambda, sc.cie_cmf);
                    V3 q = vmax(mask * xyz, (float)AR_PG_QUERY_EPS);
                    const float div = (float)((double)sum3(q) + AR_PG_QUERY_EPS);
                    q = q / div;
                    ps.maskq[p] = make_float4(q.x, q.y, q.z, 0.0f);
                }
                if (!S.delta) ++ndd;
                ++depth;
                if (depth < prm.max_depth)
                {
                    keep = true;
                    ps.ray_o[p] = make_float4(h.pos.x, h.pos.y, h.pos.z, lambda);
                    ps.ray_d[p] = make_float4(S.next_dir.x, S.next_dir.y, S.next_dir.z, lambda_pdf);
                    ps.mask[p] = mask;
                    ps.depths[p] = (uint32_t)depth | ((uint32_t)ndd << 16);
                    fl = (fl & ~1u) | (media.inside ? 1u : 0u);
                    if constexpr (TRACK_MEDIA)
                    {
                        ps.media_v[p] = make_float4(media.vertex.x, media.vertex.y, media.vertex.z,
                                                    __int_as_float(media.obj));
                        ps.media_depth[p] = media.depth;
                    }
                }
            }
        }
        ps.radiance[p] = radiance;
        if (STORE_ENDED || keep)
        {
            ps.flags[p] = fl;
            ps.rng[p] = R.g.state;
        }
    }
    return keep;
}

#undef VERTEX_MAT

// the wavelength LUT into shared memory
__device__ __forceinline__ void stage_lambda_lut(const DevScene& sc, float* s_lam)
{
    for (int i = threadIdx.x; i < AR_LAMBDA_LUT_RES * 4; i += blockDim.x) s_lam[i] = sc.lut_lambda[i];
    __syncthreads();
}

// replay adjoint: the block's sums of the medium's parameter gradients
__device__ __forceinline__ void add_medium_gradient(double* grad_medium, float g_med_albedo, float g_med_emission)
{
    for (int o = 16; o > 0; o >>= 1)
    {
        g_med_albedo += __shfl_xor_sync(0xffffffffu, g_med_albedo, o);
        g_med_emission += __shfl_xor_sync(0xffffffffu, g_med_emission, o);
    }
    if (lane_id() == 0 && (g_med_albedo != 0.0f || g_med_emission != 0.0f))
    {
        atomicAdd(grad_medium, (double)g_med_albedo);
        atomicAdd(grad_medium + 1, (double)g_med_emission);
    }
}

// What bounds k_shade is instruction supply: one vertex runs some 2,800
// instructions of mostly straight-line code (45 KB), the SM holds 16 to 28 warps
// (128 to 72 registers), and when each warp is somewhere else in that code most
// stalls are instruction fetches (256x256x16 Cornell box: 3.7 of 10.4 warps per
// issue; voxel guide: 14.0 of 21.5).  A barrier at the top of each pass and one
// before next-event estimation keep a block's warps in the same part of the
// code, so that a fetch serves all of them.  Measured, shading: 256x256x16
// Cornell box 0.98 -> 0.90 ms, textured forward and backward step 27.3 -> 25.3 ms,
// voxel guide 480x270x16 6.23 -> 4.29 ms.  The opaque-surface instantiation
// keeps only the first one: its waves on large scenes wait for memory
// (1920x1080x32 terrain 9.83 ms with one barrier, 10.04 with both, 9.89 with
// none).  More barriers gain nothing further.
//
// Threads per block, two blocks on an SM: shading waits on instruction fetch and
// on scattered loads, so the leaner instantiations do better with more warps even
// where they spill: opaque untextured 80 registers with 260 / 208 bytes of spill
// stores / loads, with the voxel guide 72 with 452 / 664. On the stage's time: opaque
// untextured (1080p terrain) 10.0 ms at 256 threads, 9.2 at 320, 8.8 at 384, 8.9 at
// 448; the same with the voxel guide (480 x 270) 3.75 ms at 256, 3.5 at 320, 3.6 at
// 384, 3.3 at 448. The others keep 256: textured 256 x 256 with its replay 22.8 ms
// for a whole step, 23.1 at 320, 23.7 at 384, and the full set of materials spills
// at 128 registers already (20 / 20 bytes unguided, 56 / 84 with the voxel guide,
// 372 / 344 with the network).
template <int GUIDE, int ADJ, int FEAT>
constexpr int kShadeBlock = FEAT != AR_FEAT_SURFACE ? 256 : GUIDE ? 448 : 384;
constexpr int AR_SHADE_RESIDENT = 2;  // blocks on an SM
constexpr int AR_SHADE_PASSES = 8;    // paths per thread before the grid grows; 4 to 32 measure alike

template <int GUIDE, int ADJ, int FEAT = AR_FEAT_ALL>
__global__ void __launch_bounds__((kShadeBlock<GUIDE, ADJ, FEAT>), AR_SHADE_RESIDENT)
    k_shade(DevScene sc, PathState ps, ShadowQueue sq, const int2* __restrict__ queue,
                                                  const int* __restrict__ counter, int* next_queue, int* next_counter,
                                                  int* shadow_counter, ShadeParams prm)
{
    const int n = *counter;
    // blocks past the queue have nothing to do (the same for every thread of the
    // block): deep bounces often have few or no paths left
    if ((long long)blockIdx.x * blockDim.x >= n) return;
    __shared__ float s_lam[AR_LAMBDA_LUT_RES * 4];
    stage_lambda_lut(sc, s_lam);
    const int stride = gridDim.x * blockDim.x;
    float g_med_albedo = 0.0f, g_med_emission = 0.0f;  // replay adjoint of the medium parameters
    // the queue comes from k_partition: {path, hit slot}, hits first
    for (int bbase = blockIdx.x * blockDim.x; bbase < n; bbase += stride)
    {
        __syncthreads();  // the block's warps start the pass together
        const int qq = bbase + (int)threadIdx.x;
        const bool active = qq < n;
        // the entry this thread shades in its next pass, read now; its state is
        // prefetched once this pass's own loads have arrived
        const int qn = qq + stride;
        const int2 next = qn < n ? queue[qn] : make_int2(-1, -1);
        const int2 entry = active ? queue[qq] : make_int2(0, -1);
        const int p = entry.x;
        ShadowRay sh;
        const bool keep = shade_vertex<GUIDE, ADJ, FEAT, FEAT != AR_FEAT_SURFACE>(sc, ps, prm, s_lam, active, p, entry.y, next, sh,
                                                                               g_med_albedo, g_med_emission);
        const int nq = warp_append_slot(next_counter, keep);
        if (keep) next_queue[nq] = p;
        const int sqi = warp_append_slot(shadow_counter, sh.cast);
        if (sh.cast)
        {
            sq.path[sqi] = p;
            sq.o[sqi] = make_float4(sh.o.x, sh.o.y, sh.o.z, sh.tmax);
            sq.d[sqi] = make_float4(sh.d.x, sh.d.y, sh.d.z, sh.vun);
            sq.v_occ[sqi] = sh.vocc;
            sq.valid_unocc[sqi] = sh.valid ? 1 : 0;
            sq.sdf_eps[sqi] = sh.sdf_eps;
        }
    }
    if constexpr (ADJ == AR_ADJ_REPLAY)
    {
        if (prm.grad_medium) add_medium_gradient(prm.grad_medium, g_med_albedo, g_med_emission);
    }
}

// ---------------------------------------------------------------- shadow
__device__ __forceinline__ void shadow_apply(const PathState& ps, const ShadowQueue& sq, int i, int p, bool occluded)
{
    ps.radiance[p] = ps.radiance[p] + (occluded ? sq.v_occ[i] : sq.d[i].w);
    const bool valid = occluded ? true : (sq.valid_unocc[i] != 0);
    ps.flags[p] = (ps.flags[p] & ~2u) | (valid ? 2u : 0u);
}

__device__ __forceinline__ void shadow_finish(const DevScene& sc, const PathState& ps, const ShadowQueue& sq, int i,
                                              int p, const TravState<true>& st, const SdfPending& pend)
{
    const bool occluded = st.result().slot >= 0;
    if (sc.stats)
    {
        atomicAdd(&sc.stats[2], (unsigned long long)st.n_visits);
        atomicAdd(&sc.stats[3], (unsigned long long)st.n_tests);
        atomicAdd(&sc.stats[5], 1ull);
    }
    if (!occluded && pend.list) pend.list[atomicAdd(pend.count, 1)] = i;
    else shadow_apply(ps, sq, i, p, occluded);
}

// The SDF passes of the shadow rays the main BVH left unoccluded: the SDF
// objects (rays they block leave the list as -1), then the smooth union.
__global__ void __launch_bounds__(AR_BLOCK) k_sdf_objects_shadow(DevScene sc, PathState ps, ShadowQueue sq, SdfPending pend)
{
    const int n = *pend.count;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x)
    {
        const int i = pend.list[k];
        const float4 o4 = sq.o[i], d4 = sq.d[i];
        const bool occluded =
            sdf_objects_occlude(sc, v3(o4.x, o4.y, o4.z), v3(d4.x, d4.y, d4.z), o4.w, sq.sdf_eps[i]);
        if (occluded || sc.trav.sdf.count <= 0) shadow_apply(ps, sq, i, sq.path[i], occluded);
        if (occluded) pend.list[k] = -1;
    }
}

// Some evaluations of a shadow ray's march by its group of G lanes; false when it is done.
template <int G>
__device__ __forceinline__ bool sdf_shadow_advance(const SdfUnion& un, const PathState& ps, const ShadowQueue& sq, SdfMarch& m,
                                                   int i, float tmax, bool lead)
{
    for (int it = 0; it < AR_SDF_EVALS; ++it)
    {
        const int r = m.take(m.field<G>(un));
        if (r == 0) continue;
        if (lead) shadow_apply(ps, sq, i, sq.path[i], r == 2 && m.t >= 0.0f && m.t < tmax);
        return false;
    }
    return true;
}

__global__ void __launch_bounds__(AR_BLOCK, AR_SDF_MIN_BLOCKS)
    k_sdf_shadow(SdfUnion un, PathState ps, ShadowQueue sq, SdfPending pend, int* fetch)
{
    const int n = *pend.count;
    const bool lead = (lane_id() & (AR_SDF_GROUP - 1)) == 0;  // the group's lane that stores
    SdfMarch m;
    m.n = 0;
    int i = 0, q = 0;
    float tmax = 0.0f;
    bool active = false, exhausted = false;
    while (true)
    {
        if (group_refill<AR_SDF_GROUP>(fetch, n, active, &exhausted, &q, AR_SDF_IDLE))
        {
            i = pend.list[q];
            if (i >= 0)
            {
                const float4 o4 = sq.o[i], d4 = sq.d[i];
                tmax = o4.w;
                active = m.begin(un, v3(o4.x, o4.y, o4.z), v3(d4.x, d4.y, d4.z), sdf_eps(0.0f), tmax);
                if (!active && lead) shadow_apply(ps, sq, i, sq.path[i], false);
            }
        }
        if (__ballot_sync(0xffffffffu, active) == 0)
        {
            if (exhausted) break;
            continue;
        }
        const int src = sdf_tail_source(active, exhausted);
        if (src != -2)
        {
            const int from = max(src, 0);
            m.copy_from(from);
            i = __shfl_sync(0xffffffffu, i, from);
            tmax = __shfl_sync(0xffffffffu, tmax, from);
            const bool tail_lead = (lane_id() & (AR_SDF_TAIL_GROUP - 1)) == 0;
            if (src >= 0)
                while (sdf_shadow_advance<AR_SDF_TAIL_GROUP>(un, ps, sq, m, i, tmax, tail_lead)) {}
            break;
        }
        if (active) active = sdf_shadow_advance<AR_SDF_GROUP>(un, ps, sq, m, i, tmax, lead);
    }
}

__global__ void __launch_bounds__(AR_BLOCK, AR_TRAV_MIN_BLOCKS) k_shadow(DevScene sc, PathState ps, ShadowQueue sq, const int* __restrict__ counter,
                                                   int* fetch, SdfPending pend, unsigned int* err, int min_idle)
{
    const int n = *counter;
    TravState<true> st;
    uint2 stk[AR_TRAV_STACK];
    int i = 0, p = 0;
    bool active = false, exhausted = false;
    while (true)
    {
        int q;
        if (warp_refill(fetch, n, active, &exhausted, &q, min_idle))
        {
            i = q;
            p = sq.path[i];
            const float4 o = sq.o[i], d = sq.d[i];
            st.init(sc.trav, v3(o.x, o.y, o.z), v3(d.x, d.y, d.z), 0.0f, o.w, stk);
            active = true;
        }
        if (__ballot_sync(0xffffffffu, active) == 0)
        {
            if (exhausted) break;
            continue;
        }
        if (active)
        {
            for (int it = 0; it < AR_SHD_STEPS; ++it)
            {
                if (!st.step(sc.trav, err))
                {
                    shadow_finish(sc, ps, sq, i, p, st, pend);
                    active = false;
                    break;
                }
            }
        }
    }
}

// ---------------------------------------------------------------- whole paths
// Small waves, and the last paths of large ones, go to their end in one launch
// (k_finish): the four launches of a depth cost 60-70 us however few paths are
// left, most of it launch and ramp-up, while a block that keeps its paths pays
// only for their own rays and vertices.  The block's barriers keep its warps in
// the same phase (k_shade's comment).  The line lies at 1024 paths per SM, two
// resident sets: the launches per depth win above it, where a warp's early-ended
// lanes stay empty in k_finish but are refilled by the queues.  One frame of the
// Cornell box, depth 8, launches per depth against k_finish: 256x256 632 -> 332
// us, 320x320 697 -> 488, 400x400 739 -> 718, 512x512 884 -> 1002; with shadow rays
// beside the next depth 320x320 539 -> 478, 384x384 592 -> 590.  Glass at depth 1000
// with the switch at 1024 per SM: 413x307x8 3.56 -> 1.07 ms, 256x256 1.91 -> 0.36 ms.
// Blocks of 256 (32 / 64 / 128: 388 / 361 / 348 us for the 256x256 frame, 328 here).
#define AR_FINISH_BLOCK 256
#define AR_FINISH_MIN_BLOCKS 2
// With SDF geometry the line is the same: 320x180x4 (terrain, SDF, medium) 6.9 ms in
// k_finish and 4.9 by depth, 160x90x4 2.9 and 4.1; 640x360x4 takes 7.2 ms with the
// switch anywhere from 64 to 1024 paths per SM.  There the warps run apart: a
// barrier would make each block wait for its longest march.
#define AR_FINISH_PATHS_PER_SM 1024

// The closest hit of path p's ray: the slot, -1 for none; the distance into
// hit_t, an SDF hit's normal into hit_nrm.
template <bool SDF>
__device__ __forceinline__ int trace_path(const DevScene& sc, const PathState& ps, int p, unsigned int* err)
{
    const float4 ro = ps.ray_o[p], rd = ps.ray_d[p];
    const V3 o = v3(ro.x, ro.y, ro.z), d = v3(rd.x, rd.y, rd.z);
    const float tmin = intersect_eps((int)(ps.depths[p] >> 16));
    const int mobj = (ps.flags[p] & 1u) ? __float_as_int(ps.media_v[p].w) : -1;
    int slot;
    float t;
    if (mobj >= 0)
    {
        // inside a medium: only the enclosing object (as in k_extend)
        if (SDF && inside_sdf_object(sc.trav.objects, sc.trav.object_count, mobj))
        {
            slot = AR_SLOT_SOLO;
            t = 0.0f;
        }
        else slot = enclosing_hit(sc, mobj, o, d, tmin, &t);
    }
    else
    {
        const TravResult r = traverse<false>(sc.trav, o, d, tmin, __int_as_float(0x7f800000), err);
        t = r.t;
        slot = r.slot;
    }
    if (SDF && sdf_objects_hit(sc, ps, p, o, d, tmin, slot, t))
    {
        SdfMarch m;
        if (m.begin(sc.trav.sdf, o, d, sdf_eps(tmin), slot != -1 ? t : 3.0e38f))
        {
            int r;
            while ((r = m.take(m.field<1>(sc.trav.sdf))) == 0 || (r == 2 && m.t >= tmin && (slot == -1 || m.t < t)))
                if (r == 2)
                {
                    t = m.t;
                    m.begin_normal();
                }
            if (r == 3)
            {
                const V3 nn = normalize(m.g);
                ps.hit_nrm[p] = make_float4(nn.x, nn.y, nn.z, 0.0f);
                slot = AR_SLOT_SDF;
            }
        }
    }
    ps.hit_t[p] = t;
    return slot;
}

// whether a vertex's shadow ray is blocked
template <bool SDF>
__device__ __forceinline__ bool shadow_path(const DevScene& sc, const ShadowRay& sh, unsigned int* err)
{
    if (traverse<true>(sc.trav, sh.o, sh.d, 0.0f, sh.tmax, err).slot >= 0) return true;
    if (!SDF) return false;
    if (sdf_objects_occlude(sc, sh.o, sh.d, sh.tmax, sh.sdf_eps)) return true;
    SdfMarch m;
    if (!m.begin(sc.trav.sdf, sh.o, sh.d, sdf_eps(0.0f), sh.tmax)) return false;
    int r;
    while ((r = m.take(m.field<1>(sc.trav.sdf))) == 0) {}
    return r == 2 && m.t >= 0.0f && m.t < sh.tmax;
}

// Every queued path to its end: the arithmetic of k_extend, k_shade and k_shadow
// per path, in the same order.
template <int ADJ, int FEAT, bool SDF>
__global__ void __launch_bounds__(AR_FINISH_BLOCK, AR_FINISH_MIN_BLOCKS)
    k_finish(DevScene sc, PathState ps, const int* __restrict__ queue, const int* __restrict__ counter, ShadeParams prm,
             unsigned int* err)
{
    const int n = *counter;
    if ((long long)blockIdx.x * blockDim.x >= n) return;
    __shared__ float s_lam[AR_LAMBDA_LUT_RES * 4];
    stage_lambda_lut(sc, s_lam);
    float g_med_albedo = 0.0f, g_med_emission = 0.0f;
    for (int bbase = blockIdx.x * blockDim.x; bbase < n; bbase += gridDim.x * blockDim.x)
    {
        const int q = bbase + (int)threadIdx.x;
        bool active = q < n;
        const int p = active ? queue[q] : 0;
        while (SDF ? __any_sync(0xffffffffu, active) : __syncthreads_or(active))
        {
            const int slot = active ? trace_path<SDF>(sc, ps, p, err) : -1;
            ShadowRay sh;
            const bool keep = shade_vertex<0, ADJ, FEAT, !SDF && FEAT != AR_FEAT_SURFACE>(
                sc, ps, prm, s_lam, active, p, slot, make_int2(-1, -1), sh, g_med_albedo, g_med_emission);
            if (sh.cast)
            {
                const bool occluded = shadow_path<SDF>(sc, sh, err);
                ps.radiance[p] = ps.radiance[p] + (occluded ? sh.vocc : sh.vun);
                if (keep) ps.flags[p] = (ps.flags[p] & ~2u) | ((occluded || sh.valid) ? 2u : 0u);
            }
            active = keep;
        }
    }
    if constexpr (ADJ == AR_ADJ_REPLAY)
    {
        if (prm.grad_medium) add_medium_gradient(prm.grad_medium, g_med_albedo, g_med_emission);
    }
}

// ---------------------------------------------------------------- finalize / accumulate
__device__ __forceinline__ float nan_inf_to_zero(float x)
{
    if (x != x) return 0.0f;
    if (fabsf(x) == __int_as_float(0x7f800000)) return x > 0.0f ? 0.0f : -0.0f;
    return x;
}

// a path's clamped XYZ sample
__device__ __forceinline__ V3 path_sample(const DevScene& sc, const PathState& ps, int k)
{
    const float lambda = ps.ray_o[k].w;
    const float pdf = ps.ray_d[k].w;
    const V3 xyz = lambda_to_xyz(lambda, sc.cie_cmf);
    const float r = nan_inf_to_zero(ps.radiance[k]);
    return v3(fmaxf(0.0f, clampf(xyz.x * r / pdf, 0.0f, AR_RADIANCE_CLAMP)),
              fmaxf(0.0f, clampf(xyz.y * r / pdf, 0.0f, AR_RADIANCE_CLAMP)),
              fmaxf(0.0f, clampf(xyz.z * r / pdf, 0.0f, AR_RADIANCE_CLAMP)));
}

// the samples themselves, where the caller or the denoiser's records want them
__global__ void k_finalize(DevScene sc, PathState ps, int n, float* __restrict__ extra_out)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const V3 v = path_sample(sc, ps, k);
    ps.out_xyz[3 * k + 0] = v.x;
    ps.out_xyz[3 * k + 1] = v.y;
    ps.out_xyz[3 * k + 2] = v.z;
    if (extra_out)
    {
        extra_out[3 * k + 0] = v.x;
        extra_out[3 * k + 1] = v.y;
        extra_out[3 * k + 2] = v.z;
    }
}

// guided rendering: clear the collection slots and set the probe query
__global__ void k_guide_init(PathState ps, int n)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    ps.maskq[k] = make_float4(1.0f, 1.0f, 1.0f, 0.0f);
    for (int i = 0; i < AR_PG_COLLECT_DEPTH; ++i)
    {
        ps.pg_dir[i * ps.capacity + k] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        ps.pg_loc[i * ps.capacity + k] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        ps.pg_vdir[i * ps.capacity + k] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
}

// radiance records of finished paths (core/render/render.cuh:909-963)
__global__ void k_guide_emit(DevScene sc, PathState ps, int n, GuideSamples gs)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const uint32_t fl = ps.flags[k];
    if (((fl >> 8) & 31u) == 0u) return;
    const float lambda = ps.ray_o[k].w;
    const float pdf = ps.ray_d[k].w;
    const V3 lxyz = lambda_to_xyz(lambda, sc.cie_cmf);
    for (int i = 0; i < AR_PG_COLLECT_DEPTH; ++i)
    {
        if (!((fl >> (8 + i)) & 1u)) continue;
        const float4 d = ps.pg_dir[i * ps.capacity + k];
        const V3 xyz = lxyz * d.w / pdf;
        const float strength = fminf(max3(xyz), AR_PG_COLLECT_MAX);
        if (strength < AR_PG_COLLECT_MIN) continue;
        const float4 l = ps.pg_loc[i * ps.capacity + k];
        const float4 vd = ps.pg_vdir[i * ps.capacity + k];
        const VoxelKey key = voxel_key(v3(l.x, l.y, l.z), v3(vd.x, vd.y, vd.z), sc.guide.inv_unit);
        const unsigned long long packed = guide_pack(key);
        const int slot = atomicAdd(gs.count, 1);
        if (slot >= gs.capacity) continue;
        const V3 rad = vmax(xyz, 0.0f);
        gs.radiance[slot] = make_float4(rad.x, rad.y, rad.z, 0.0f);
        gs.dir[slot] = make_float4(d.x, d.y, d.z, 0.0f);
        gs.key[slot] = packed;
        if (gs.pos)
        {
            gs.pos[slot] = make_float4(l.x, l.y, l.z, 1.0f);
            gs.wr[slot] = make_float4(vd.x, vd.y, vd.z, vd.w);  // w: the packed surface normal
        }
    }
}

// Per pixel, adds the wave's samples in increasing sample order (deterministic).
// A warp takes 32 consecutive pixel slots and AR_ACC_SAMPLES samples of each at a
// time: it computes them with consecutive lanes on consecutive paths, passes them
// through shared memory, and each lane adds its own pixel's.  Bound by the path
// state's bytes (36 per path) and the FP64 adds.  FINAL: samples straight from the
// path state; otherwise those k_finalize stored.
template <bool FINAL>
__global__ void __launch_bounds__(AR_ACC_BLOCK)
    k_accumulate(DevScene sc, PathState ps, long long first_path, int n, int width, int height, PathOrder po,
                 double* __restrict__ accum)
{
    static_assert(AR_PATH_GROUP_PX == 1u, "a slot's samples of a block are consecutive paths");
    constexpr int H = AR_ACC_SAMPLES;
    static_assert(32 % H == 0, "a pass of the warp covers whole pixels");
    // one lane's samples start an odd number of words after the last one's: no bank is shared
    __shared__ float s_xyz[AR_ACC_BLOCK / 32][3][32 * (H + 1)];
    float(*tile)[32 * (H + 1)] = s_xyz[threadIdx.x >> 5];
    const int lane = (int)lane_id();
    const long long npix = (long long)width * height;
    const long long u0 = (blockIdx.x * (long long)blockDim.x + threadIdx.x) - lane;
    if (u0 >= npix) return;
    const int px = (int)min(32ll, npix - u0);
    const long long per = npix * po.block, last_path = first_path + n;
    bool any = false;
    double sx = 0.0, sy = 0.0, sz = 0.0;
    double* out = nullptr;
    const uint32_t fb1 = (uint32_t)((last_path - 1) / per);
    for (uint32_t fb = (uint32_t)(first_path / per); fb <= fb1; ++fb)
    {
        const int sb = (int)path_block_samples(po, fb);
        // path (u0 + x, sample s of the block) is base + x * sb + s; the wave holds [lo, hi) of them
        const long long base = (long long)fb * per + u0 * sb;
        const int lo = (int)min(max(first_path - base, 0ll), (long long)(px * sb));
        const int hi = (int)min(max(last_path - base, 0ll), (long long)(px * sb));
        if (lo >= hi) continue;
        const int k0 = (int)(base - first_path);
        const int a = max(lo, lane * sb), b = min(hi, (lane + 1) * sb);  // this lane's pixel
        if (!any && a < b)
        {
            out = accum + 3 * (size_t)slot_pixel((uint32_t)(u0 + lane), (uint32_t)width, (uint32_t)height);
            sx = out[0];
            sy = out[1];
            sz = out[2];
            any = true;
        }
        for (int h0 = 0; h0 < sb; h0 += H)
        {
            __syncwarp();
#pragma unroll 2
            for (int j = 0; j < H; ++j)
            {
                const int x = (j * 32 + lane) / H, s = (j * 32 + lane) % H, i = x * sb + h0 + s;
                if (h0 + s >= sb || i < lo || i >= hi) continue;
                const int k = k0 + i;
                V3 v;
                if (FINAL) v = path_sample(sc, ps, k);
                else v = v3(ps.out_xyz[3 * (size_t)k], ps.out_xyz[3 * (size_t)k + 1], ps.out_xyz[3 * (size_t)k + 2]);
                const int c = x * (H + 1) + s;
                tile[0][c] = v.x;
                tile[1][c] = v.y;
                tile[2][c] = v.z;
            }
            __syncwarp();
            for (int s = max(a - lane * sb, h0); s < min(b - lane * sb, h0 + H); ++s)
            {
                const int c = lane * (H + 1) + s - h0;
                sx += (double)tile[0][c];
                sy += (double)tile[1][c];
                sz += (double)tile[2][c];
            }
        }
    }
    if (any)
    {
        out[0] = sx;
        out[1] = sy;
        out[2] = sz;
    }
}

static void launch_accumulate_wave(const DevScene& sc, const PathState& ps, const RenderLaunch& rl, long long first_path, int n,
                                   bool stored, double* accum, cudaStream_t s)
{
    const long long npix = (long long)rl.width * rl.height;
    const int grid = (int)((npix + AR_ACC_BLOCK - 1) / AR_ACC_BLOCK);
    const auto k = stored ? k_accumulate<false> : k_accumulate<true>;
    k<<<grid, AR_ACC_BLOCK, 0, s>>>(sc, ps, first_path, n, rl.width, rl.height, path_order(rl), accum);
}

static CamParams make_camera(const RenderLaunch& rl)
{
    CamParams c;
    c.o = v3(rl.cam_o[0], rl.cam_o[1], rl.cam_o[2]);
    c.d = v3(rl.cam_d[0], rl.cam_d[1], rl.cam_d[2]);
    const float FOV = rl.fov_deg * 3.1415926f / 180.0f;
    const float aspect = static_cast<float>(rl.width) / fmaxf(1.0f, static_cast<float>(rl.height));
    c.tan_y = arm_tanf(0.5f * FOV);
    c.tan_x = c.tan_y * aspect;
    c.right = normalize(cross(c.d, v3(0.0f, 1.0f, 0.0f)));
    c.up = normalize(cross(c.d, c.right));
    return c;
}

// the SDF passes after k_extend and after k_shadow: objects, then the union
static void launch_sdf_extend(const DevScene& sc, const PathState& ps, const int* queue, const int* qn, int* cnt,
                              int grid_s, int grid_m, cudaStream_t s)
{
    if (sc.sdf_trav.node_count > 0) k_sdf_objects<<<grid_s, AR_BLOCK, 0, s>>>(sc, ps, queue, qn);
    if (sc.trav.sdf.count > 0)
        k_sdf_extend<<<grid_m, AR_BLOCK, 0, s>>>(sc.trav.sdf, sc.sdf_trav.node_count > 0 ? sc.trav.objects : nullptr,
                                                 sc.trav.object_count, ps, queue, qn, &cnt[AR_CNT_SDF]);
}

static void launch_sdf_shadow(const DevScene& sc, const PathState& ps, const ShadowQueue& sq, const SdfPending& pend,
                              int* fetch, int grid_s, int grid_m, cudaStream_t s)
{
    if (sc.sdf_trav.node_count > 0) k_sdf_objects_shadow<<<grid_s, AR_BLOCK, 0, s>>>(sc, ps, sq, pend);
    if (sc.trav.sdf.count > 0) k_sdf_shadow<<<grid_m, AR_BLOCK, 0, s>>>(sc.trav.sdf, ps, sq, pend, fetch);
}

struct ShadeArgs
{
    const DevScene& sc;
    const PathState& ps;
    const ShadowQueue& sq;
    const int2* queue;
    const int* counter;
    int* next_queue;
    int* next_counter;
    int* shadow_counter;
    const ShadeParams& prm;
    long long bound;  // paths at most
    int sms;
    cudaStream_t stream;
};

template <int GUIDE, int ADJ, int FEAT>
static void launch_shade(const ShadeArgs& a)
{
    constexpr int B = kShadeBlock<GUIDE, ADJ, FEAT>;
    const long long resident = (long long)AR_SHADE_RESIDENT * a.sms;
    const int grid = (int)(resident * std::max<long long>(1, a.bound / (resident * B * AR_SHADE_PASSES)));
    k_shade<GUIDE, ADJ, FEAT><<<grid, B, 0, a.stream>>>(a.sc, a.ps, a.sq, a.queue, a.counter, a.next_queue, a.next_counter,
                                                        a.shadow_counter, a.prm);
}

// what k_extend zeroes at depth b: the counters of this depth's later kernels and
// the next depth's own fetch counter
static CounterReset depth_resets(int* cnt, int b)
{
    const int odd = b & 1;
    int* sh = &cnt[AR_CNT_SHADOW + 4 * odd];
    return CounterReset{&cnt[AR_CNT_Q0 + (odd ^ 1)], &cnt[AR_CNT_FETCH + (odd ^ 1)], sh, sh + 1, sh + 2, sh + 3,
                        &cnt[AR_CNT_PART], &cnt[AR_CNT_PART + 1], &cnt[AR_CNT_SDF]};
}

// records a stage interval when profiling
struct StageScope
{
    Ctx& c;
    int stage;
    cudaEvent_t a = nullptr;
    StageScope(Ctx& cc, int st) : c(cc), stage(st)
    {
        if (c.profile & 1)
        {
            cudaEventCreate(&a);
            cudaEventRecord(a, c.stream);
        }
    }
    ~StageScope()
    {
        if (c.profile & 1)
        {
            cudaEvent_t b;
            cudaEventCreate(&b);
            cudaEventRecord(b, c.stream);
            c.stage_events.push_back(StageEvent{stage, a, b});
            c.stage_launches[stage] += 1;
        }
    }
};

cudaError_t launch_render_wave(Ctx& c, const RenderLaunch& rl, long long first_path, int n, float* per_sample_out,
                               long long* launches)
{
    const DevScene sc = dev_scene(c);
    cudaStream_t s = c.stream;
    int sms = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c.device);
    const int grid_n = (n + AR_BLOCK - 1) / AR_BLOCK;
    // the persistent traversal kernels launch as many blocks as stay
    // resident: they fetch rays from a counter, so extra blocks would only add
    // launch cost (most deep bounces have few or no paths left)
    const int grid_t = sms * AR_TRAV_MIN_BLOCKS, grid_m = sms * AR_SDF_MIN_BLOCKS;
    int* cnt = c.d_counters;  // AR_CNT_* layout
    const CamParams cam = make_camera(rl);
    // SDF geometry: its work leaves the traversal kernels for k_sdf_extend / k_sdf_shadow
    const bool has_sdf = c.sdf_object_count > 0 || c.sdf.count > 0;
    // opaque surfaces only: the shading instantiations without glass and medium
    // code (and without textures, where the scene has none); the MLP guide has one only
    bool opaque_tex = !c.medium.on && !c.camera_inside && rl.guide != 2;
    for (const Material& m : c.materials) opaque_tex = opaque_tex && m.shading != AR_MAT_GLASS;
    const bool opaque = opaque_tex && c.tex_count == 0;
    {
        StageScope st(c, ST_RAYGEN);
        k_raygen<<<grid_n, AR_BLOCK, 0, s>>>(c.ps, c.d_queue[0], &cnt[AR_CNT_Q0], first_path, n, rl.width, rl.height,
                                             rl.seed, rl.first_frame, cam, c.camera_inside, &cnt[AR_CNT_FETCH],
                                             !opaque || has_sdf || rl.adjoint, rl.guide != 0, path_order(rl), rl.jumps);
        if (rl.guide) k_guide_init<<<grid_n, AR_BLOCK, 0, s>>>(c.ps, n);
    }
    long long L = rl.guide ? 2 : 1;
    ShadeParams prm;
    prm.use_nee = rl.use_nee;
    prm.max_depth = rl.max_depth;
    prm.grad = rl.grad;
    prm.grad_medium = rl.grad_medium;
    prm.mlp_ready = rl.mlp_ready;
    prm.gbuf = rl.denoise ? c.d_dn_rec : nullptr;
    MlpDev net;
    net.wbf = c.d_mlp_wbf;
    net.w32 = c.d_mlp_w32;
    net.box = c.mlp_box;
    const int n_sdf = (sc.sdf_trav.node_count > 0 ? 1 : 0) + (sc.trav.sdf.count > 0 ? 1 : 0);  // launches of each pass
    // A depth's shadow rays run on a stream of their own, beside the next depth's
    // closest hits: neither reads what the other writes (shadow rays add to the
    // radiance and set flag bit 1; closest hits read flag bit 0), and the next
    // shading waits for both.  What it hides is the end of each kernel, when few
    // rays are left (640x360x4 combined scene, marches of up to 512 steps: 9.53 -> 7.9
    // ms; 256x256x16 Cornell box 2.21 -> 2.08 ms; 1080p terrain 36.1 -> 35.5 ms).
    // Profiled renders keep the stages apart
    const bool overlap = c.profile == 0;
    const cudaStream_t hs = overlap ? c.shadow_stream : s;
    auto join_shadows = [&](int b) {
        if (overlap && b > 0) cudaStreamWaitEvent(s, c.shadow_done, 0);
    };
    int depths_run = 0;
    // Each depth's next-queue length is copied to pinned host memory behind
    // the depth's launches.  The host stays AR_BOUNCE_LOOKAHEAD depths ahead of
    // the GPU: before it queues depth b it reads the length left by depth
    // b - AR_BOUNCE_LOOKAHEAD, which bounds every later queue.  A zero ends the
    // wave's depth loop (every later depth would find an empty queue), and the
    // bound sizes the grids of the queue-sized kernels, so deep bounces with
    // few paths left (or none, at depth limits like 1000) cost launches of a
    // few blocks instead of a wave-sized grid.
    // k_finish covers renders without a guide; profiled ones keep the stages apart
    const bool finish_ok = !rl.guide && c.profile == 0;
    const long long finish_paths = (long long)sms * AR_FINISH_PATHS_PER_SM;
    constexpr int K = AR_BOUNCE_LOOKAHEAD;
    long long bound = n;  // upper bound of the current depth's queue length
    for (int b = 0; b < rl.max_depth; ++b)
    {
        if (b >= K)
        {
            const int slot = (b - K) % (K + 1);
            const cudaError_t we = cudaEventSynchronize(c.bounce_ev[slot]);
            if (we != cudaSuccess) return we;
            const int known = c.h_bounce_cnt[slot];  // queue length of depth b - K + 1
            if (known <= 0) break;
            bound = std::min<long long>(bound, known);
        }
        if (finish_ok && bound <= finish_paths)
        {
            // few enough paths: all of them to their end in one launch
            join_shadows(b);
            depths_run = 0;
            const int grid_f = (int)std::min<long long>((bound + AR_FINISH_BLOCK - 1) / AR_FINISH_BLOCK,
                                                        (long long)sms * AR_FINISH_MIN_BLOCKS);
            const int* fq = c.d_queue[b & 1];
            const int* fn = &cnt[AR_CNT_Q0 + (b & 1)];
            const bool replay = rl.adjoint == AR_ADJ_REPLAY;
            const auto finish = rl.adjoint && has_sdf ? (replay ? k_finish<AR_ADJ_REPLAY, AR_FEAT_ALL, true>
                                                                : k_finish<AR_ADJ_RECORD, AR_FEAT_ALL, true>)
                                : rl.adjoint          ? (replay ? k_finish<AR_ADJ_REPLAY, AR_FEAT_ALL, false>
                                                                : k_finish<AR_ADJ_RECORD, AR_FEAT_ALL, false>)
                                : has_sdf             ? k_finish<0, AR_FEAT_ALL, true>
                                : opaque              ? k_finish<0, AR_FEAT_SURFACE, false>
                                                      : k_finish<0, AR_FEAT_ALL, false>;
            finish<<<grid_f, AR_FINISH_BLOCK, 0, s>>>(sc, c.ps, fq, fn, prm, c.d_err);
            ++L;
            break;
        }
        const int grid_s = std::max(2 * sms, (int)((bound + AR_BLOCK * AR_PASS_PATHS - 1) /
                                                   (AR_BLOCK * AR_PASS_PATHS)));
        const int cur = b & 1, nxt = cur ^ 1;
        int* qn = &cnt[AR_CNT_Q0 + cur];
        int* sh = &cnt[AR_CNT_SHADOW + 4 * cur];
        const SdfPending pend_shd{has_sdf ? c.d_pend_list : nullptr, sh + 2};
        {
            StageScope st(c, ST_EXTEND);
            k_extend<<<grid_t, AR_BLOCK, 0, s>>>(sc, c.ps, c.d_queue[cur], qn, &cnt[AR_CNT_FETCH + cur], c.d_err,
                                                 b == 0 ? AR_EXT_REFILL_MIN0 : AR_EXT_REFILL_MIN, depth_resets(cnt, b));
            if (has_sdf)
            {
                launch_sdf_extend(sc, c.ps, c.d_queue[cur], qn, cnt, grid_s, grid_m, s);
                L += n_sdf;
            }
        }
        join_shadows(b);
        {
            StageScope st(c, ST_SHADE);
            k_partition<<<grid_s, AR_BLOCK, 0, s>>>(c.d_queue[cur], c.ps.q_slot, qn, c.d_pq, &cnt[AR_CNT_PART],
                                                    &cnt[AR_CNT_PART + 1]);
            ++L;
            if (rl.guide == 2 && rl.mlp_ready)
            {
                // network inference for every queued hit (tensor cores), before shading
                cudaMemsetAsync(&cnt[AR_CNT_MLP], 0, sizeof(int), s);
                k_mlp_query<<<grid_s, AR_BLOCK, 0, s>>>(sc, c.ps, c.d_queue[cur], qn, c.d_mlp_list, &cnt[AR_CNT_MLP]);
                launch_mlp_infer(net, c.ps.q_pos, c.ps.q_wr, c.d_mlp_list, &cnt[AR_CNT_MLP], 0, c.ps.q_dist, nullptr, c.d_err,
                                 sms, s);
                L += 2;
            }
            int* nq = c.d_queue[nxt];
            int* nn = &cnt[AR_CNT_Q0 + nxt];
            const int2* pq = c.d_pq;
            const ShadeArgs sa{sc, c.ps, c.sq, pq, qn, nq, nn, sh, prm, bound, sms, s};
            if (rl.guide == 2) launch_shade<2, 0, AR_FEAT_ALL>(sa);
            else if (rl.guide) opaque ? launch_shade<1, 0, AR_FEAT_SURFACE>(sa) : launch_shade<1, 0, AR_FEAT_ALL>(sa);
            else if (rl.adjoint == AR_ADJ_REPLAY) launch_shade<0, AR_ADJ_REPLAY, AR_FEAT_ALL>(sa);
            else if (rl.adjoint)
                opaque_tex ? launch_shade<0, AR_ADJ_RECORD, AR_FEAT_TEXTURED>(sa) : launch_shade<0, AR_ADJ_RECORD, AR_FEAT_ALL>(sa);
            else if (opaque) launch_shade<0, 0, AR_FEAT_SURFACE>(sa);
            else if (opaque_tex) launch_shade<0, 0, AR_FEAT_TEXTURED>(sa);
            else launch_shade<0, 0, AR_FEAT_ALL>(sa);
        }
        {
            StageScope st(c, ST_SHADOW);
            if (overlap)
            {
                cudaEventRecord(c.shade_done, s);
                cudaStreamWaitEvent(hs, c.shade_done, 0);
            }
            k_shadow<<<grid_t, AR_BLOCK, 0, hs>>>(sc, c.ps, c.sq, sh, sh + 1, pend_shd, c.d_err,
                                                  b == 0 ? AR_SHD_REFILL_MIN0 : AR_SHD_REFILL_MIN);
            if (has_sdf)
            {
                launch_sdf_shadow(sc, c.ps, c.sq, pend_shd, sh + 3, grid_s, grid_m, hs);
                L += n_sdf;
            }
            if (overlap) cudaEventRecord(c.shadow_done, hs);
            depths_run = b + 1;
        }
        L += 3;
        {
            const int slot = b % (K + 1);
            cudaMemcpyAsync(&c.h_bounce_cnt[slot], &cnt[AR_CNT_Q0 + nxt], sizeof(int), cudaMemcpyDeviceToHost, s);
            cudaEventRecord(c.bounce_ev[slot], s);
        }
    }
    join_shadows(depths_run);
    if (rl.adjoint)
    {
        if (launches) *launches += L;
        return cudaGetLastError();
    }
    {
        StageScope st(c, ST_FINAL);
        if (per_sample_out || rl.denoise)
        {
            k_finalize<<<grid_n, AR_BLOCK, 0, s>>>(sc, c.ps, n, per_sample_out);
            ++L;
        }
        if (rl.guide)
        {
            k_guide_emit<<<grid_n, AR_BLOCK, 0, s>>>(sc, c.ps, n, c.gs);
            ++L;
        }
    }
    if (launches) *launches += L;
    return cudaGetLastError();
}

// Wave launch over caller-provided buffers (used by the allocation-free entry
// point): every depth by its launches, all on the caller's stream.
cudaError_t launch_render_wave_buffers(const DevScene& sc, const WaveBuffers& wb, int device, const RenderLaunch& rl,
                                       int camera_inside, long long first_path, int n, unsigned int* err)
{
    cudaStream_t s = wb.stream;
    int sms = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    const int grid_n = (n + AR_BLOCK - 1) / AR_BLOCK;
    const int grid_t = sms * AR_TRAV_MIN_BLOCKS, grid_m = sms * AR_SDF_MIN_BLOCKS;
    const int grid_s = std::max(2 * sms, (n + AR_BLOCK * AR_PASS_PATHS - 1) / (AR_BLOCK * AR_PASS_PATHS));
    int* cnt = wb.counters;  // AR_CNT_* layout
    const CamParams cam = make_camera(rl);
    k_raygen<<<grid_n, AR_BLOCK, 0, s>>>(wb.ps, wb.queue[0], &cnt[AR_CNT_Q0], first_path, n, rl.width, rl.height, rl.seed,
                                         rl.first_frame, cam, camera_inside, &cnt[AR_CNT_FETCH], true, false,
                                         path_order(rl), nullptr);
    ShadeParams prm;
    prm.use_nee = rl.use_nee;
    prm.max_depth = rl.max_depth;
    prm.grad = nullptr;
    prm.grad_medium = nullptr;
    prm.mlp_ready = 0;
    prm.gbuf = nullptr;
    const bool has_sdf = sc.sdf_trav.node_count > 0 || sc.trav.sdf.count > 0;
    for (int b = 0; b < rl.max_depth; ++b)
    {
        const int cur = b & 1, nxt = cur ^ 1;
        int* sh = &cnt[AR_CNT_SHADOW + 4 * cur];
        const SdfPending pend_shd{has_sdf ? wb.pend_list : nullptr, sh + 2};
        k_extend<<<grid_t, AR_BLOCK, 0, s>>>(sc, wb.ps, wb.queue[cur], &cnt[AR_CNT_Q0 + cur], &cnt[AR_CNT_FETCH + cur], err,
                                             b == 0 ? AR_EXT_REFILL_MIN0 : AR_EXT_REFILL_MIN, depth_resets(cnt, b));
        if (has_sdf)
            launch_sdf_extend(sc, wb.ps, wb.queue[cur], &cnt[AR_CNT_Q0 + cur], cnt, grid_s, grid_m, s);
        k_partition<<<grid_s, AR_BLOCK, 0, s>>>(wb.queue[cur], wb.ps.q_slot, &cnt[AR_CNT_Q0 + cur], wb.pq,
                                                &cnt[AR_CNT_PART], &cnt[AR_CNT_PART + 1]);
        launch_shade<0, 0, AR_FEAT_ALL>(ShadeArgs{sc, wb.ps, wb.sq, wb.pq, &cnt[AR_CNT_Q0 + cur], wb.queue[nxt],
                                                      &cnt[AR_CNT_Q0 + nxt], sh, prm, n, sms, s});
        k_shadow<<<grid_t, AR_BLOCK, 0, s>>>(sc, wb.ps, wb.sq, sh, sh + 1, pend_shd, err,
                                             b == 0 ? AR_SHD_REFILL_MIN0 : AR_SHD_REFILL_MIN);
        if (has_sdf) launch_sdf_shadow(sc, wb.ps, wb.sq, pend_shd, sh + 3, grid_s, grid_m, s);
    }
    launch_accumulate_wave(sc, wb.ps, rl, first_path, n, false, wb.accum, s);
    return cudaGetLastError();
}

// per-pixel sums -> means (one double multiply each, as the host would do it)
__global__ void k_scale_means(double* v, long long n, double inv)
{
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i < n) v[i] *= inv;
}

cudaError_t launch_scale_means(double* v, long long n, double inv, cudaStream_t s)
{
    if (n <= 0) return cudaSuccess;
    k_scale_means<<<(int)((n + 255) / 256), 256, 0, s>>>(v, n, inv);
    return cudaGetLastError();
}

cudaError_t launch_accumulate(Ctx& c, const RenderLaunch& rl, long long first_path, int n, bool stored, double* accum,
                              long long* launches)
{
    StageScope st(c, ST_FINAL);
    launch_accumulate_wave(dev_scene(c), c.ps, rl, first_path, n, stored, accum, c.stream);
    if (launches) *launches += 1;
    return cudaGetLastError();
}
} // namespace ar
