// Path adjoint of the albedo textures (no counterpart in the reference).
//
// ar_adjoint renders every wave once, with shading (k_shade<0, AR_ADJ_RECORD, *>)
// leaving per vertex the texel whose colour it used and the radiance of the path
// so far.  k_adjoint_scatter then knows each path's total radiance L, turns
// d(loss)/d(image) into the path's scalar adjoint
// delta = sum_c dl/dXYZ_c * dXYZ_c/dL / spp and adds
// delta * (L - radiance so far) * d(albedo)/d(rgb) / albedo into a float32
// gradient buffer for every textured diffuse vertex.  After each wave the
// float32 buffer is folded into the caller's float64 gradient and cleared, so
// float32 sums only ever span one wave.
//
// Depth limits whose records would pass AR_ADJ_RECORDS_MAX, and the medium's
// parameters (ar_adjoint_medium), render every wave twice over the same random
// streams instead: an ordinary pass for L, k_adjoint_seed for delta, and a
// replay (k_shade<0, AR_ADJ_REPLAY, *>) that scatters as it goes.
#include <algorithm>

#include <cuda_runtime.h>

#include "ar_internal.h"

namespace ar
{
#define AR_SCATTER_BLOCK 256
#define AR_SCATTER_MIN_BLOCKS 4

// A path's total radiance and d(loss)/d(radiance).
__device__ __forceinline__ float2 path_adjoint(const DevScene& sc, const PathState& ps, int k, float lambda,
                                               const float* __restrict__ dl_dxyz, float inv_spp)
{
    const float pdf = ps.ray_d[k].w;
    float r = ps.radiance[k];
    if (!(r == r) || fabsf(r) == __int_as_float(0x7f800000)) r = 0.0f;
    const V3 xyz = lambda_to_xyz(lambda, sc.cie_cmf);
    const uint32_t pix = ps.pixel[k];
    const float* g = dl_dxyz + 3 * (size_t)pix;
    // the image is clamp(xyz * L / pdf, 0, AR_RADIANCE_CLAMP) per channel
    const float cx = xyz.x * r / pdf, cy = xyz.y * r / pdf, cz = xyz.z * r / pdf;
    float d = 0.0f;
    if (cx > 0.0f && cx < AR_RADIANCE_CLAMP) d += g[0] * (xyz.x / pdf);
    if (cy > 0.0f && cy < AR_RADIANCE_CLAMP) d += g[1] * (xyz.y / pdf);
    if (cz > 0.0f && cz < AR_RADIANCE_CLAMP) d += g[2] * (xyz.z / pdf);
    return make_float2(r, d * inv_spp);
}

__global__ void k_adjoint_seed(DevScene sc, PathState ps, int n, const float* __restrict__ dl_dxyz, float inv_spp)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const float2 a = path_adjoint(sc, ps, k, ps.ray_o[k].w, dl_dxyz, inv_spp);
    ps.adj_total[k] = a.x;
    ps.adj_delta[k] = a.y;
}

// One thread per path, over its records.  Bound by the gathers from the spectral
// table (eight corners of 16 bytes per record, each its own sector: the texels
// of a texture name cells all over the 2 GB) and by the atomics; 4.2 million
// paths of depth 8 over 512 x 512 textures took 2.45 ms with the corners read as
// 4-byte loads.  With 16-byte loads the whole 256 x 256 x 64 step takes 16.3 ms at
// 4 blocks per SM (64 registers), 16.6 / 16.5 / 17.4 at 5 / 6 / 8, and 16.7 with
// one thread per record, which repeats the path's part for each.
__global__ void __launch_bounds__(AR_SCATTER_BLOCK, AR_SCATTER_MIN_BLOCKS)
    k_adjoint_scatter(DevScene sc, PathState ps, int n, int max_depth, const float* __restrict__ dl_dxyz, float inv_spp,
                      float* __restrict__ grad)
{
    __shared__ float s_lam[AR_LAMBDA_LUT_RES * 4];
    for (int i = threadIdx.x; i < AR_LAMBDA_LUT_RES * 4; i += blockDim.x) s_lam[i] = sc.lut_lambda[i];
    __syncthreads();
    const int stride = gridDim.x * blockDim.x;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += stride)
    {
        const float lambda = ps.ray_o[k].w;
        const float2 a = path_adjoint(sc, ps, k, lambda, dl_dxyz, inv_spp);
        if (a.y == 0.0f) continue;
        const Basis lb = query_lambda(lambda, s_lam);
        const PlainFetch f{sc.lut_rgb};
        // the state keeps the depth of the path's last vertex
        const int vertices = min((int)(ps.depths[k] & 0xffffu) + 1, max_depth);
        for (int v = 0; v < vertices; ++v)
        {
            const int2 rec = ps.adj_rec[(size_t)v * ps.adj_stride + k];
            const float rest = a.x - __int_as_float(rec.y);
            if (rec.x < 0 || rest == 0.0f) continue;
            const float* tx = sc.texels + 3 * (size_t)rec.x;
            const V3 rgb = v3(__ldg(tx), __ldg(tx + 1), __ldg(tx + 2));
            const float alb = interact(prepare_color(rgb, f), lb);
            if (!(alb > 1.0e-8f)) continue;
            const V3 g = interact_rgb_grad(lb, rgb, f) * (a.y * rest / alb);
            float* gp = grad + 3 * (size_t)rec.x;
            if (g.x != 0.0f) atomicAdd(gp + 0, g.x);
            if (g.y != 0.0f) atomicAdd(gp + 1, g.y);
            if (g.z != 0.0f) atomicAdd(gp + 2, g.z);
        }
    }
}

__global__ void k_grad_fold(float* __restrict__ g32, double* __restrict__ g64, long long n)
{
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += stride)
    {
        const float v = g32[i];
        if (v != 0.0f)
        {
            g64[i] += (double)v;
            g32[i] = 0.0f;
        }
    }
}

cudaError_t launch_adjoint_seed(Ctx& c, const RenderLaunch& rl, int n, const float* dl_dxyz, long long* launches)
{
    const DevScene sc = dev_scene(c);
    k_adjoint_seed<<<(n + 255) / 256, 256, 0, c.stream>>>(sc, c.ps, n, dl_dxyz, 1.0f / (float)rl.spp);
    if (launches) *launches += 1;
    return cudaGetLastError();
}

cudaError_t launch_adjoint_scatter(Ctx& c, const RenderLaunch& rl, int n, const float* dl_dxyz, float* grad,
                                   long long* launches)
{
    const DevScene sc = dev_scene(c);
    int sms = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c.device);
    const int grid = std::min((n + AR_SCATTER_BLOCK - 1) / AR_SCATTER_BLOCK, sms * AR_SCATTER_MIN_BLOCKS * 2);
    k_adjoint_scatter<<<grid, AR_SCATTER_BLOCK, 0, c.stream>>>(sc, c.ps, n, rl.max_depth, dl_dxyz, 1.0f / (float)rl.spp,
                                                               grad);
    if (launches) *launches += 1;
    return cudaGetLastError();
}

cudaError_t launch_grad_fold(Ctx& c, double* grad64, long long n, long long* launches)
{
    int sms = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c.device);
    const long long want = (n + 255) / 256;
    const int grid = (int)std::min<long long>(want, (long long)sms * 16);
    if (grid > 0) k_grad_fold<<<grid, 256, 0, c.stream>>>(c.d_grad32, grad64, n);
    if (launches) *launches += 1;
    return cudaGetLastError();
}
} // namespace ar
