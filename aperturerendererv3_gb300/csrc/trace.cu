// Raw ray queries against the scene BVH (closest hit / any hit), the kernels
// behind ar_trace_closest / ar_trace_any.  Rays are read as two float4 (origin +
// tmin, direction + tmax).
#include <cuda_runtime.h>

#include <algorithm>

#include "ar_internal.h"
#include "ar_ray_share.h"

namespace ar
{
#define TR_BLOCK 128
#define TR_BLOCKS (1024 / TR_BLOCK)  // per SM: 64 registers
#define TR_IDLE 4                    // idle lanes that trigger a refill
#define TR_STEPS 8                   // node visits between refill checks

// Scenes without SDF geometry.  Bound by instruction issue under divergence
// (TravState's comment), so the warps are persistent: a lane whose ray is done
// takes the warp's next one as soon as four are idle, from a share of the rays
// fixed beforehand (chunks dealt round robin), so concurrent calls on other
// streams share no counter.  2.07M rays against 1M triangles: 2.86 ms with one ray
// per thread (and the SDF code's registers), 1.77 ms; refills at 8 / 16 / 32 idle
// lanes 1.85 / 1.95 / 2.38 ms.  Batches that do not fill the chip are bound by the
// longest ray's chain of node loads instead: they are spread out, down to one ray
// per warp, as far as half the resident warps go (1000 rays 22.7 -> 14.5 us, 100
// rays 39.7 -> 18.6; 20,000 rays as 8 per warp took 34.9, as 16 per warp 29.8).  Eight
// lanes per ray gained 15 % there and lost 25 % at 65,536 rays.
template <bool AnyHit>
__global__ void __launch_bounds__(TR_BLOCK, TR_BLOCKS) k_trace_rays(TravScene sc, const float4* __restrict__ rays, int n,
                                                                   int chunk_log2, int* __restrict__ out,
                                                                   float* __restrict__ tout, unsigned int* err)
{
    const int lane = threadIdx.x & 31;
    const int w = blockIdx.x * (TR_BLOCK / 32) + (threadIdx.x >> 5);
    const RayShare share{n, chunk_log2, (int)gridDim.x * (TR_BLOCK / 32)};
    const int limit = share.limit(w);
    int next = 0;
    TravState<AnyHit> st;
    uint2 stk[AR_TRAV_STACK];
    int i = 0;
    bool active = false;
    while (true)
    {
        const unsigned idle = __ballot_sync(0xffffffffu, !active);
        if (next < limit && __popc(idle) >= TR_IDLE)
        {
            if (!active)
            {
                const int j = next + __popc(idle & ((1u << lane) - 1u));
                const long long r = share.ray(w, j);
                if (j < limit && r < n)
                {
                    i = (int)r;
                    const float4 a = __ldg(&rays[2 * (size_t)i]);
                    const float4 b = __ldg(&rays[2 * (size_t)i + 1]);
                    st.init(sc, v3(a.x, a.y, a.z), v3(b.x, b.y, b.z), a.w, b.w, stk);
                    active = true;
                }
            }
            next += __popc(idle);
        }
        if (__ballot_sync(0xffffffffu, active) == 0)
        {
            if (next >= limit) break;
            continue;
        }
        if (active)
        {
            for (int it = 0; it < TR_STEPS; ++it)
            {
                if (!st.step(sc, err))
                {
                    const TravResult r = st.result();
                    if (AnyHit) out[i] = r.slot != -1 ? 1 : 0;
                    else
                    {
                        out[i] = r.id;
                        if (tout) tout[i] = r.slot != -1 ? r.t : -1.0f;
                    }
                    active = false;
                    break;
                }
            }
        }
    }
}

// Scenes with SDF geometry: one ray per thread, the marches after the traversal.
template <bool AnyHit>
__global__ void __launch_bounds__(256) k_trace(TravScene sc, TravScene sdf_objects, const float4* __restrict__ rays, int n,
                                             int* __restrict__ out, float* __restrict__ tout, unsigned int* err)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    {
        const float4 a = __ldg(&rays[2 * (size_t)i]);
        const float4 b = __ldg(&rays[2 * (size_t)i + 1]);
        const V3 o = v3(a.x, a.y, a.z), d = v3(b.x, b.y, b.z);
        TravResult r = traverse<AnyHit>(sc, o, d, a.w, b.w, err);
        if (sdf_objects.node_count > 0 && (!AnyHit || r.slot < 0))
        {
            // SDF objects (their own BVH), marched with half of max(tmin, 1e-3)
            const TravResult r2 = sdf_bvh_trace<AnyHit>(sdf_objects, o, d, a.w, b.w, 0.5f * fmaxf(a.w, 1.0e-3f), r);
            if (r2.id != r.id)
            {
                r = r2;
                r.slot = AR_SLOT_SDFOBJ_BASE - r2.slot;
            }
        }
        const bool hit = r.id >= 0;
        if (sc.sdf.count > 0 && (!AnyHit || !hit))
        {
            // the smooth-union SDF object (largest primitive id: a BVH hit at equal t wins)
            const float ts = sdf_march(sc.sdf, o, d, sdf_eps(a.w), hit ? r.t : b.w);
            if (ts >= a.w && ts < b.w && (!hit || ts < r.t))
            {
                r.t = ts;
                r.slot = AR_SLOT_SDF;
                r.id = sc.sdf_id;
            }
        }
        if (AnyHit)
        {
            out[i] = r.slot != -1 ? 1 : 0;
        }
        else
        {
            out[i] = r.id;
            if (tout) tout[i] = r.slot != -1 ? r.t : -1.0f;
        }
    }
}

cudaError_t launch_trace(const DevScene& sc, const float* rays, int n, int any, int* prim_id, float* t, unsigned int* err,
                         cudaStream_t s, long long* launches)
{
    if (n <= 0) return cudaSuccess;
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const float4* r4 = reinterpret_cast<const float4*>(rays);
    if (sc.sdf_trav.node_count <= 0 && sc.trav.sdf.count <= 0)
    {
        const long long resident = (long long)sms * (1024 / 32);  // warps
        int chunk_log2 = 0;
        while (chunk_log2 < 5 && ((long long)n >> chunk_log2) > resident / 2) ++chunk_log2;
        const long long chunks = RayShare{n, chunk_log2, 1}.chunks();
        const int grid = (int)((std::min(chunks, resident) + TR_BLOCK / 32 - 1) / (TR_BLOCK / 32));
        if (any) k_trace_rays<true><<<grid, TR_BLOCK, 0, s>>>(sc.trav, r4, n, chunk_log2, prim_id, nullptr, err);
        else k_trace_rays<false><<<grid, TR_BLOCK, 0, s>>>(sc.trav, r4, n, chunk_log2, prim_id, t, err);
        if (launches) *launches += 1;
        return cudaGetLastError();
    }
    const int blocks = (int)std::min<long long>((n + 255) / 256, (long long)sms * 16);
    if (any) k_trace<true><<<blocks, 256, 0, s>>>(sc.trav, sc.sdf_trav, r4, n, prim_id, nullptr, err);
    else k_trace<false><<<blocks, 256, 0, s>>>(sc.trav, sc.sdf_trav, r4, n, prim_id, t, err);
    if (launches) *launches += 1;
    return cudaGetLastError();
}
} // namespace ar
