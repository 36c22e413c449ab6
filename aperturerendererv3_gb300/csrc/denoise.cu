// Denoiser of the accumulated image (SceneRenderer::Render with bDenoise_,
// core/scene.cu:324-348, and core/denoise/*).
//
// Recording: k_shade writes the camera ray's first-hit record per path; after
// each wave, k_denoise_record walks every pixel's samples of that wave in
// sample order and folds them into the pixel's G-buffer means and sample
// moments (the reference updates them inside its megakernel, one sample per
// thread per frame).
//
// Filtering: k_bilateral is the reference's Bilateral16x16<7>
// (core/denoise/denoise.cuh:360-443) restructured for the SM: one block per tile
// of 32 x 32 output pixels (32 x 8 for small images) stages the pixels it reads
// as per-pixel keys (dn_make_key, 96 B each, 203 KB per large tile) in shared
// memory, planar, so a warp reads 32 consecutive words per field.  What bounds it
// is instruction issue (83 % of the slots): 225 pairs per pixel.  Most pairs'
// t-tests are decided without divisions and the square root (dn_channel_quick, 6
// words of shared memory per pair; dn_channel_nu where the degrees of freedom
// matter; the reference's arithmetic for the rest, hardly any), and the G-buffer
// weight is evaluated only for pairs that pass (a failing pair contributes weight
// 0 in the reference as well).  1920x1080, 8 samples: 6.22 ms with the reference's
// arithmetic for every pair, 5.3 with dn_channel_quick alone, 3.4 now; 64 samples
// 2.75.  Two or four output rows per thread (shared loads, fewer warps) were
// slower: 4.6 and over 10 ms.  Every output equals the reference arithmetic's.
#include <cuda_runtime.h>

#include <algorithm>

#include "../../include/aperture/ar.h"
#include "ar_denoise.h"
#include "ar_internal.h"
#include "ar_t_quantile.h"

namespace ar
{
namespace
{
constexpr int TX = 32;                               // output tile: 32 x TY pixels, one per thread
constexpr int TY_LARGE = 32, TY_SMALL = 8;           // (k_bilateral's comment says when which)
constexpr int SX = TX + 2 * AR_DN_RADIUS;            // 46 pixels staged per row
template <int TY>
constexpr int kSpan = SX * (TY + 2 * AR_DN_RADIUS);  // staged pixels per tile
constexpr int TAPS = (2 * AR_DN_RADIUS + 1) * (2 * AR_DN_RADIUS + 1);
// planes of the staged keys (one float or one 32-bit word per pixel each)
enum
{
    P_COL = 0,
    P_NRM = 3,
    P_DEP = 6,
    P_H = 7,      // 5 words of half pairs: (albedo x, y), (albedo z, metallic), (roughness, model 0),
                  // (model 1, model 2), (model 3, model 4)
    P_TH = 12,
    P_VTH = 15,
    P_UP = 18,
    P_LO = 21,
    P_COUNT = 24
};
template <int TY>
constexpr size_t kSmemBytes = ((size_t)P_COUNT * kSpan<TY> + 2 * AR_DN_TQ_SIZE + TAPS) * sizeof(float);
} // namespace

__global__ void k_denoise_record(const float4* __restrict__ rec, const float* __restrict__ out_xyz,
                                 const Material* __restrict__ mats, long long first_path, int n, int width, int height,
                                 PathOrder po, DnGBuf* __restrict__ gb, DnStat* __restrict__ st)
{
    // one thread per pixel slot (slot_pixel maps it to its pixel): this wave's
    // samples of the slot, in sample order
    const long long npix = (long long)width * height;
    const long long u = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (u >= npix) return;
    uint32_t smp = path_first_sample(po, (uint32_t)u, (unsigned long long)first_path);
    if (smp >= po.spp || (long long)path_index(po, (uint32_t)u, smp) >= first_path + n) return;
    const long long p = slot_pixel((uint32_t)u, (uint32_t)width, (uint32_t)height);
    DnGBuf b = gb[p];
    DnStat s = st[p];
    for (long long g; smp < po.spp && (g = (long long)path_index(po, (uint32_t)u, smp)) < first_path + n; ++smp)
    {
        const long long k = g - first_path;
        const float4 r0 = rec[2 * k], r1 = rec[2 * k + 1];
        const int mid = __float_as_int(r0.w);
        if (mid >= 0)
        {
            const Material& m = mats[mid];
            dn_record_gbuffer(b, true, v3(r0.x, r0.y, r0.z), v3(r1.x, r1.y, r1.z), m.metallic, m.roughness, r1.w,
                              m.shading);
        }
        else
        {
            dn_record_gbuffer(b, false, v3(0, 0, 0), v3(0, 0, 0), 0.0f, 0.0f, 0.0f, AR_DN_NO_HIT);
        }
        const float xyz[3] = {out_xyz[3 * k], out_xyz[3 * k + 1], out_xyz[3 * k + 2]};
        dn_record_stat(s, xyz);
    }
    gb[p] = b;
    st[p] = s;
}

__device__ __forceinline__ uint32_t half2_bits(__half a, __half b)
{
    return (uint32_t)__half_as_ushort(a) | ((uint32_t)__half_as_ushort(b) << 16);
}
__device__ __forceinline__ __half half_lo(uint32_t w) { return __ushort_as_half((unsigned short)(w & 0xffffu)); }
__device__ __forceinline__ __half half_hi(uint32_t w) { return __ushort_as_half((unsigned short)(w >> 16)); }

// the differences of two pairs of halves as the reference's device code computes
// them: half subtractions (rounded to half)
__device__ __forceinline__ __half2 half_words(uint32_t a, uint32_t b)
{
    return __hsub2(*reinterpret_cast<const __half2*>(&a), *reinterpret_cast<const __half2*>(&b));
}
// whether one half of the pair is infinite or not a number
__device__ __forceinline__ bool half_extreme(uint32_t w)
{
    return (w & 0x7c00u) == 0x7c00u || (w & 0x7c000000u) == 0x7c000000u;
}

// arm_expf for x in (-87, 0], where none of its special cases applies; the same
// operations
__device__ __forceinline__ float exp_weight(float x)
{
    if (!(x > -87.0f && x <= 0.0f)) return arm_expf(x);
    const float k = rintf(x * 1.44269504088896340736f);
    float r = fmaf(-k, 6.93145751953125e-1f, x);
    r = fmaf(-k, 1.42860682030941723212e-6f, r);
    float p = ARM_INV_FACT_9;
    p = fmaf(p, r, ARM_INV_FACT_8);
    p = fmaf(p, r, ARM_INV_FACT_7);
    p = fmaf(p, r, ARM_INV_FACT_6);
    p = fmaf(p, r, ARM_INV_FACT_5);
    p = fmaf(p, r, ARM_INV_FACT_4);
    p = fmaf(p, r, ARM_INV_FACT_3);
    p = fmaf(p, r, ARM_INV_FACT_2);
    p = fmaf(p, r, 1.0f);
    p = fmaf(p, r, 1.0f);
    return p * arm_detail::pow2i((int)k);
}

// the t-test of the pair (centre ce, neighbour e) by the reference's operations
template <int SPAN>
__device__ __noinline__ bool pair_passes(const float* sm, const float* s_tq, int ce, int e)
{
    for (int ch = 0; ch < 3; ++ch)
    {
        const float t = sm[(P_TH + ch) * SPAN + ce] - sm[(P_TH + ch) * SPAN + e];
        const float u = sm[(P_UP + ch) * SPAN + ce] + sm[(P_UP + ch) * SPAN + e];
        const float lo = sm[(P_LO + ch) * SPAN + ce] + sm[(P_LO + ch) * SPAN + e];
        if (!dn_channel_passes(t, sm[(P_VTH + ch) * SPAN + ce], sm[(P_VTH + ch) * SPAN + e], u, lo, s_tq)) return false;
    }
    return true;
}

// what the output pixel contributes to its pairs, in registers
struct CentreKey
{
    float th[3], vth[3], inv_vth[3], lo[3];
    float nrm[3], dep;
    uint32_t h[5];
};

// ComputeSVGFWeight (core/denoise/denoise.cuh:178-242): the G-buffer terms of the
// pair (c, e).  same_ok: no half of the tile is infinite or not a number
template <int SPAN>
__device__ __forceinline__ float gbuffer_term(const float* sm, const uint32_t* smu, const CentreKey& c, int e, bool same_ok)
{
    float wTerm = 0.0f;
    const uint32_t b0 = smu[P_H * SPAN + e], b1 = smu[(P_H + 1) * SPAN + e];
    {
        const float d0 = __half2float(half_lo(c.h[0])) - __half2float(half_lo(b0));
        const float d1 = __half2float(half_hi(c.h[0])) - __half2float(half_hi(b0));
        const float d2 = __half2float(half_lo(c.h[1])) - __half2float(half_lo(b1));
        wTerm += (d0 * d0 + d1 * d1 + d2 * d2) * DnSigma::kAlbedo;
    }
    {
        const float dv = c.nrm[0] * sm[P_NRM * SPAN + e] + c.nrm[1] * sm[(P_NRM + 1) * SPAN + e] +
                         c.nrm[2] * sm[(P_NRM + 2) * SPAN + e];
        const float d = 1.0f - dv;
        wTerm += d * d * DnSigma::kNormal;
    }
    {
        const float b = sm[P_DEP * SPAN + e];
        const float denom = fmaxf(fmaxf(c.dep, b), 1.0e-6f);
        const float d = (c.dep - b) / denom;
        wTerm += d * d * DnSigma::kDepth;
    }
    // metallic, roughness and the shading-model histogram: equal words differ by
    // nothing (unless they are not numbers: same_ok), and neighbours on one
    // surface mostly have equal ones
    const uint32_t b2 = smu[(P_H + 2) * SPAN + e], b3 = smu[(P_H + 3) * SPAN + e], b4 = smu[(P_H + 4) * SPAN + e];
    const bool same = same_ok && ((c.h[1] ^ b1) >> 16) == 0u && c.h[2] == b2 && c.h[3] == b3 && c.h[4] == b4;
    if (!same)
    {
        const __half2 d1 = half_words(c.h[1], b1), d2 = half_words(c.h[2], b2), d3 = half_words(c.h[3], b3),
                      d4 = half_words(c.h[4], b4);
        const float dm = __high2float(d1);
        wTerm += dm * dm * DnSigma::kMetallic;
        const float dr = __low2float(d2);
        wTerm += dr * dr * DnSigma::kRough;
        float l1 = 0.0f;
        l1 += fabsf(__high2float(d2));
        l1 += fabsf(__low2float(d3));
        l1 += fabsf(__high2float(d3));
        l1 += fabsf(__low2float(d4));
        l1 += fabsf(__high2float(d4));
        const float tv = 0.5f * l1;
        wTerm += tv * tv * DnSigma::kModel;
    }
    return wTerm;
}

template <int TY>
__global__ void __launch_bounds__(TX * TY, TY == TY_LARGE ? 1 : 2)
    k_bilateral(const double* __restrict__ in_xyz, double* __restrict__ out_xyz, const DnGBuf* __restrict__ gb,
                const DnStat* __restrict__ st, const float* __restrict__ tq_global, int W, int H)
{
    constexpr int SPAN = kSpan<TY>;
    extern __shared__ float sm[];
    uint32_t* smu = reinterpret_cast<uint32_t*>(sm);
    float* s_tq = sm + (size_t)P_COUNT * SPAN;
    float* s_k2 = s_tq + AR_DN_TQ_SIZE;  // 2 (1 + q^2)
    float* s_sp = s_k2 + AR_DN_TQ_SIZE;
    __shared__ int s_odd;         // a colour of the tile is not finite: even zero weights count
    __shared__ int s_half;        // a half of the tile is infinite or not a number
    __shared__ int s_extreme;     // moments the quick test's limits do not hold for
    __shared__ uint32_t s_min_f, s_max_f;  // the tile's degrees of freedom
    constexpr int THREADS = TX * TY;
    const int tid = threadIdx.y * TX + threadIdx.x;
    if (tid == 0)
    {
        s_odd = s_half = s_extreme = 0;
        s_min_f = 0xffffffffu;
        s_max_f = 1u;
    }
    for (int i = tid; i < AR_DN_TQ_SIZE; i += THREADS)
    {
        const float q = tq_global[i];
        s_tq[i] = q;
        s_k2[i] = 2.0f * (1.0f + q * q);
    }
    for (int i = tid; i < TAPS; i += THREADS)
    {
        const int dj = i / (2 * AR_DN_RADIUS + 1) - AR_DN_RADIUS, di = i % (2 * AR_DN_RADIUS + 1) - AR_DN_RADIUS;
        s_sp[i] = arm_expf((float)(-(di * di + dj * dj)) * DnSigma::kSpatial);
    }
    __syncthreads();
    // stage the tile's keys (clamped to the image, as the reference's tile load)
    const int gx0 = blockIdx.x * TX - AR_DN_RADIUS, gy0 = blockIdx.y * TY - AR_DN_RADIUS;
    uint32_t min_f = 0xffffffffu, max_f = 1u;
    for (int e = tid; e < SPAN; e += THREADS)
    {
        const int sy = e / SX, sx = e % SX;
        const int gy = min(max(gy0 + sy, 0), H - 1), gx = min(max(gx0 + sx, 0), W - 1);
        const long long q = (long long)gy * W + gx;
        const V3 c = v3((float)in_xyz[3 * q], (float)in_xyz[3 * q + 1], (float)in_xyz[3 * q + 2]);
        const DnStat stat = st[q];
        const DnKey k = dn_make_key(gb[q], stat, c);
        const uint32_t f = stat.num > 2u ? stat.num - 1u : 1u;
        min_f = min(min_f, f);
        max_f = max(max_f, f);
        for (int ch = 0; ch < 3; ++ch)
        {
            sm[(P_COL + ch) * SPAN + e] = k.col[ch];
            sm[(P_NRM + ch) * SPAN + e] = k.nrm[ch];
            sm[(P_TH + ch) * SPAN + e] = k.theta[ch];
            sm[(P_VTH + ch) * SPAN + e] = k.vth[ch];
            sm[(P_UP + ch) * SPAN + e] = k.up[ch];
            sm[(P_LO + ch) * SPAN + e] = k.lo[ch];
            if (!(fabsf(k.col[ch]) < 3.0e38f)) s_odd = 1;
            if (!dn_ordinary(k.vth[ch], k.up[ch])) s_extreme = 1;
        }
        sm[P_DEP * SPAN + e] = k.depth;
        const uint32_t hw[5] = {half2_bits(__float2half_rn(k.alb[0]), __float2half_rn(k.alb[1])),
                                half2_bits(__float2half_rn(k.alb[2]), k.mr[0]), half2_bits(k.mr[1], k.model[0]),
                                half2_bits(k.model[1], k.model[2]), half2_bits(k.model[3], k.model[4])};
        for (int i = 0; i < 5; ++i)
        {
            smu[(P_H + i) * SPAN + e] = hw[i];
            if (half_extreme(hw[i])) s_half = 1;
        }
    }
    min_f = __reduce_min_sync(0xffffffffu, min_f);
    max_f = __reduce_max_sync(0xffffffffu, max_f);
    if ((tid & 31) == 0)
    {
        atomicMin(&s_min_f, min_f);
        atomicMax(&s_max_f, max_f);
    }
    __syncthreads();
    const bool odd = s_odd != 0, extreme = s_extreme != 0, nan_half = s_half != 0;
    const DnRho lim = dn_rho_limits(s_min_f, s_max_f, s_tq);
    const int ox = blockIdx.x * TX + threadIdx.x, oy = blockIdx.y * TY + threadIdx.y;
    if (ox >= W || oy >= H) return;

    constexpr float CENTER_EPS = 1.0e-6f;
    constexpr int D = 2 * AR_DN_RADIUS;
    const int ce = (threadIdx.y + AR_DN_RADIUS) * SX + threadIdx.x + AR_DN_RADIUS;
    CentreKey c;
    float acc[3], accW = CENTER_EPS;
    for (int ch = 0; ch < 3; ++ch)
    {
        c.th[ch] = sm[(P_TH + ch) * SPAN + ce];
        c.vth[ch] = sm[(P_VTH + ch) * SPAN + ce];
        c.inv_vth[ch] = 1.0f / c.vth[ch];
        c.lo[ch] = sm[(P_LO + ch) * SPAN + ce];
        c.nrm[ch] = sm[(P_NRM + ch) * SPAN + ce];
        acc[ch] = sm[(P_COL + ch) * SPAN + ce] * CENTER_EPS;
    }
    c.dep = sm[P_DEP * SPAN + ce];
    for (int k = 0; k < 5; ++k) c.h[k] = smu[(P_H + k) * SPAN + ce];
    for (int jj = 0; jj <= D; ++jj)
    {
        const int row = (threadIdx.y + jj) * SX + threadIdx.x;
#pragma unroll 3
        for (int ii = 0; ii <= D; ++ii)
        {
            const int e = row + ii;
            float t[3], vB[3];
#pragma unroll
            for (int ch = 0; ch < 3; ++ch)
            {
                t[ch] = c.th[ch] - sm[(P_TH + ch) * SPAN + e];
                vB[ch] = sm[(P_VTH + ch) * SPAN + e];
            }
            // all three channels below their threshold; one that fails decides the pair
            bool pass = true, fail = false;
#pragma unroll
            for (int ch = 0; ch < 3; ++ch)
            {
                bool p, f;
                dn_channel_quick(t[ch], c.vth[ch], c.inv_vth[ch], vB[ch], lim, &p, &f);
                pass = pass && p;
                fail = fail || f;
            }
            if (!pass && !fail)
            {
                pass = true;
#pragma unroll
                for (int ch = 0; ch < 3; ++ch)
                {
                    bool p, f;
                    dn_channel_nu(t[ch], c.vth[ch], c.inv_vth[ch], vB[ch], c.lo[ch] + sm[(P_LO + ch) * SPAN + e], s_k2, &p,
                                  &f);
                    pass = pass && p;
                    fail = fail || f;
                }
            }
            if ((!pass && !fail) || extreme) pass = pair_passes<SPAN>(sm, s_tq, ce, e);
            float weight = 0.0f;
            if (pass) weight = exp_weight(-gbuffer_term<SPAN>(sm, smu, c, e, !nan_half)) * s_sp[jj * (D + 1) + ii];
            // a failed pair adds zero times its colour, which only matters if that is not finite
            if (pass || odd)
            {
                acc[0] = acc[0] + sm[P_COL * SPAN + e] * weight;
                acc[1] = acc[1] + sm[(P_COL + 1) * SPAN + e] * weight;
                acc[2] = acc[2] + sm[(P_COL + 2) * SPAN + e] * weight;
                accW = accW + weight;
            }
        }
    }
    // CompositeSample (core/denoise/denoise.cuh:211-220)
    const long long o = (long long)oy * W + ox;
    for (int ch = 0; ch < 3; ++ch) out_xyz[3 * o + ch] = (double)fmaxf(arm_expf(acc[ch] / accW) - 1.0f, 0.0f);
}

// Tiles of 8 rows while those of 32 would leave SMs without one: 200x150 210 us
// against 340; at 640x360 (240 large tiles) the two are level, and at 1920x1080
// the small ones' wider margins cost 20 %.
static bool small_tiles(int W, int H, int sms)
{
    return (long long)((W + TX - 1) / TX) * ((H + TY_LARGE - 1) / TY_LARGE) < (long long)sms;
}

template <int TY>
static cudaError_t launch_bilateral(const double* src, double* dst, const DnGBuf* gb, const DnStat* st, const float* tq,
                                    int W, int H, cudaStream_t s)
{
    k_bilateral<TY><<<dim3((W + TX - 1) / TX, (H + TY - 1) / TY), dim3(TX, TY), kSmemBytes<TY>, s>>>(src, dst, gb, st, tq,
                                                                                                     W, H);
    return cudaGetLastError();
}

cudaError_t launch_denoise_record(Ctx& c, const RenderLaunch& rl, long long first_path, int n, long long* launches)
{
    const long long npix = (long long)rl.width * rl.height;
    const int grid = (int)((npix + 255) / 256);
    k_denoise_record<<<grid, 256, 0, c.stream>>>(c.d_dn_rec, c.ps.out_xyz, c.d_materials, first_path, n, rl.width,
                                                 rl.height, path_order(rl), c.d_dn_gb, c.d_dn_st);
    if (launches) *launches += 1;
    return cudaGetLastError();
}
} // namespace ar

struct ar_ctx
{
    ar::Ctx c;
};

namespace
{
float* g_tq_dev[64] = {};  // t-quantile table per device

cudaError_t tq_table(int device, const float** out)
{
    if (device < 0 || device >= 64) return cudaErrorInvalidDevice;
    if (!g_tq_dev[device])
    {
        float* p = nullptr;
        cudaError_t e = cudaMalloc((void**)&p, sizeof(ar_t_quantile_0025));
        if (e == cudaSuccess) e = cudaMemcpy(p, ar_t_quantile_0025, sizeof(ar_t_quantile_0025), cudaMemcpyHostToDevice);
        if (e != cudaSuccess)
        {
            if (p) cudaFree(p);
            return e;
        }
        e = cudaFuncSetAttribute(ar::k_bilateral<ar::TY_LARGE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)ar::kSmemBytes<ar::TY_LARGE>);
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(ar::k_bilateral<ar::TY_SMALL>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)ar::kSmemBytes<ar::TY_SMALL>);
        if (e != cudaSuccess)
        {
            cudaFree(p);
            return e;
        }
        g_tq_dev[device] = p;
    }
    *out = g_tq_dev[device];
    return cudaSuccess;
}
} // namespace

namespace ar
{
// Allocates the per-pixel records for a width x height image (zeroed when the
// image changes or a render starts at frame 0) and the per-path first-hit
// records for the wave capacity.
cudaError_t ensure_denoise(Ctx& c, int width, int height, int first_frame)
{
    cudaError_t e = cudaSuccess;
    const long long npix = (long long)width * height;
    if (c.dn_rec_cap < c.ps.capacity)
    {
        if (c.d_dn_rec) cudaFree(c.d_dn_rec);
        c.d_dn_rec = nullptr;
        c.dn_rec_cap = 0;
        e = cudaMalloc((void**)&c.d_dn_rec, 2 * (size_t)c.ps.capacity * sizeof(float4));
        if (e != cudaSuccess) return e;
        c.dn_rec_cap = c.ps.capacity;
    }
    const bool resize = c.dn_w != width || c.dn_h != height;
    if (resize)
    {
        if (c.d_dn_gb) cudaFree(c.d_dn_gb);
        if (c.d_dn_st) cudaFree(c.d_dn_st);
        c.d_dn_gb = nullptr;
        c.d_dn_st = nullptr;
        c.dn_w = c.dn_h = 0;
        e = cudaMalloc((void**)&c.d_dn_gb, (size_t)npix * sizeof(DnGBuf));
        if (e == cudaSuccess) e = cudaMalloc((void**)&c.d_dn_st, (size_t)npix * sizeof(DnStat));
        if (e != cudaSuccess) return e;
        c.dn_w = width;
        c.dn_h = height;
    }
    if (resize || first_frame == 0)
    {
        e = cudaMemsetAsync(c.d_dn_gb, 0, (size_t)npix * sizeof(DnGBuf), c.stream);
        if (e == cudaSuccess) e = cudaMemsetAsync(c.d_dn_st, 0, (size_t)npix * sizeof(DnStat), c.stream);
    }
    return e;
}

void free_denoise(Ctx& c)
{
    if (c.d_dn_gb) cudaFree(c.d_dn_gb);
    if (c.d_dn_st) cudaFree(c.d_dn_st);
    if (c.d_dn_rec) cudaFree(c.d_dn_rec);
    if (c.d_dn_io) cudaFree(c.d_dn_io);
    c.d_dn_gb = nullptr;
    c.d_dn_st = nullptr;
    c.d_dn_rec = nullptr;
    c.d_dn_io = nullptr;
    c.dn_w = c.dn_h = 0;
    c.dn_rec_cap = 0;
    c.dn_img_cap = 0;
}
} // namespace ar

extern "C" {

ar_status ar_denoise(ar_ctx* ctx, const double* xyz_in, int in_is_device, double* xyz_out, int out_is_device,
                     void* stream)
{
    using namespace ar;
    if (!ctx || !xyz_in || !xyz_out) return AR_ERR_INVALID;
    Ctx& c = ctx->c;
    if (c.dn_w <= 0 || c.dn_h <= 0) return AR_ERR_STATE;
    if (cudaSetDevice(c.device) != cudaSuccess) return AR_ERR_CUDA;
    cudaStream_t s = stream ? (cudaStream_t)stream : c.stream;
    const long long npix = (long long)c.dn_w * c.dn_h;
    const size_t bytes = (size_t)npix * 3 * sizeof(double);
    const float* tq = nullptr;
    cudaError_t e = tq_table(c.device, &tq);
    // device staging for host images: input and output halves of one buffer
    if (e == cudaSuccess && (!in_is_device || !out_is_device) && c.dn_img_cap < npix)
    {
        if (c.d_dn_io) cudaFree(c.d_dn_io);
        c.d_dn_io = nullptr;
        c.dn_img_cap = 0;
        e = cudaMalloc((void**)&c.d_dn_io, 2 * bytes);
        if (e == cudaSuccess) c.dn_img_cap = npix;
    }
    const double* src = xyz_in;
    double* dst = xyz_out;
    if (e == cudaSuccess && !in_is_device)
    {
        e = cudaMemcpyAsync(c.d_dn_io, xyz_in, bytes, cudaMemcpyHostToDevice, s);
        src = c.d_dn_io;
    }
    if (!out_is_device) dst = c.d_dn_io + 3 * npix;
    if (e == cudaSuccess)
    {
        int sms = 0;
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c.device);
        e = small_tiles(c.dn_w, c.dn_h, sms)
                ? launch_bilateral<TY_SMALL>(src, dst, c.d_dn_gb, c.d_dn_st, tq, c.dn_w, c.dn_h, s)
                : launch_bilateral<TY_LARGE>(src, dst, c.d_dn_gb, c.d_dn_st, tq, c.dn_w, c.dn_h, s);
    }
    if (e == cudaSuccess && !out_is_device) e = cudaMemcpyAsync(xyz_out, dst, bytes, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    return e == cudaSuccess ? AR_OK : AR_ERR_CUDA;
}

ar_status ar_denoise_read(ar_ctx* ctx, int32_t* width, int32_t* height, void* gbuffer, void* moments)
{
    using namespace ar;
    if (!ctx) return AR_ERR_INVALID;
    Ctx& c = ctx->c;
    if (width) *width = c.dn_w;
    if (height) *height = c.dn_h;
    if (!gbuffer && !moments) return AR_OK;
    if (c.dn_w <= 0) return AR_ERR_STATE;
    if (cudaSetDevice(c.device) != cudaSuccess) return AR_ERR_CUDA;
    const size_t npix = (size_t)c.dn_w * c.dn_h;
    cudaError_t e = cudaStreamSynchronize(c.stream);
    if (e == cudaSuccess && gbuffer) e = cudaMemcpy(gbuffer, c.d_dn_gb, npix * sizeof(DnGBuf), cudaMemcpyDeviceToHost);
    if (e == cudaSuccess && moments) e = cudaMemcpy(moments, c.d_dn_st, npix * sizeof(DnStat), cudaMemcpyDeviceToHost);
    return e == cudaSuccess ? AR_OK : AR_ERR_CUDA;
}

ar_status ar_denoise_write(ar_ctx* ctx, int32_t width, int32_t height, const void* gbuffer, const void* moments)
{
    using namespace ar;
    if (!ctx || width <= 0 || height <= 0 || !gbuffer || !moments) return AR_ERR_INVALID;
    Ctx& c = ctx->c;
    if (cudaSetDevice(c.device) != cudaSuccess) return AR_ERR_CUDA;
    const size_t npix = (size_t)width * height;
    if (c.dn_w != width || c.dn_h != height)
    {
        if (c.d_dn_gb) cudaFree(c.d_dn_gb);
        if (c.d_dn_st) cudaFree(c.d_dn_st);
        c.d_dn_gb = nullptr;
        c.d_dn_st = nullptr;
        c.dn_w = c.dn_h = 0;
        if (cudaMalloc((void**)&c.d_dn_gb, npix * sizeof(DnGBuf)) != cudaSuccess) return AR_ERR_NOMEM;
        if (cudaMalloc((void**)&c.d_dn_st, npix * sizeof(DnStat)) != cudaSuccess) return AR_ERR_NOMEM;
        c.dn_w = width;
        c.dn_h = height;
    }
    cudaError_t e = cudaStreamSynchronize(c.stream);
    if (e == cudaSuccess) e = cudaMemcpy(c.d_dn_gb, gbuffer, npix * sizeof(DnGBuf), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(c.d_dn_st, moments, npix * sizeof(DnStat), cudaMemcpyHostToDevice);
    return e == cudaSuccess ? AR_OK : AR_ERR_CUDA;
}

} // extern "C"
