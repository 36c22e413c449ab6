// Smooth-union signed-distance object: up to AR_SDF_MAX_PRIMS spheres, boxes
// and tori (torus axis +y) combined with a polynomial smooth minimum of width
// k, marched like the reference's RaymarchLocal (core/object/sdf/sdf_base.cuh:
// 53-105): the start point's sign decides which crossing ends the march, the
// step is the distance (at least eps / 2), and the hit is the last point before
// the crossing.  The reference's own shapes are the torus
// (core/object/sdf/sdf_torus.cuh:14-18) and others; the union is new.
// Host + device.
#pragma once
#include "ar_vec.h"

#define AR_SDF_MAX_PRIMS 64
#define AR_SDF_SPHERE 0
#define AR_SDF_BOX 1
#define AR_SDF_TORUS 2
#define AR_SDF_STEPS 512  // SDF_STEPS (core/config.cuh:75)

namespace ar
{
// primitives: two float4 each, (kind, centre xyz), (size xyz, bounding
// radius: sdf_bounding_radius, filled when the union is uploaded)
struct SdfUnion
{
    const float4* prims;
    int count;
    float k;
    V3 lo, hi;  // bounds of the zero set
    // a grid of res cells over [lo, hi]: per cell the primitives that can change
    // the union's value at any of its points (sdf_cell_mask); null: no grid
    const unsigned long long* cells = nullptr;
    int res[3] = {0, 0, 0};
    V3 inv_cell = {0.0f, 0.0f, 0.0f};
    float rk = 0.0f;  // sdf_reciprocal_k(k)
};

AR_HD float sdf_prim(float4 a, float4 b, V3 p)
{
    const V3 q = p - v3(a.y, a.z, a.w);
    const int kind = (int)a.x;
    if (kind == AR_SDF_SPHERE) return length(q) - b.x;
    if (kind == AR_SDF_BOX)
    {
        const V3 d = v3(fabsf(q.x) - b.x, fabsf(q.y) - b.y, fabsf(q.z) - b.z);
        const V3 dp = vmax(d, 0.0f);
        return length(dp) + fminf(fmaxf(d.x, fmaxf(d.y, d.z)), 0.0f);
    }
    // torus in the xz plane: (|q.xz| - R, q.y) at distance r
    const float rxz = sqrtf(q.x * q.x + q.z * q.z) - b.x;
    return sqrtf(rxz * rxz + q.y * q.y) - b.y;
}

// polynomial smooth minimum (width k > 0)
AR_HD float smin_poly(float a, float b, float k)
{
    const float h = fmaxf(k - fabsf(a - b), 0.0f) / k;
    return fminf(a, b) - h * h * k * 0.25f;
}

// radius of a sphere about the primitive's centre that holds it
AR_HD float sdf_bounding_radius(float kind, float sx, float sy, float sz)
{
    const int k = (int)kind;
    if (k == AR_SDF_SPHERE) return sx;
    if (k == AR_SDF_BOX) return sqrtf(sx * sx + sy * sy + sz * sz);
    return sx + sy;  // torus: major + minor radius
}

AR_HD unsigned long long sdf_all(const SdfUnion& s) { return s.count >= 64 ? ~0ull : (1ull << s.count) - 1ull; }

// x / k for 0 <= x <= k: two corrections of x rk with rk = 1 / k rounded give the
// correctly rounded quotient (P. Markstein, IBM J. Res. Dev. 34(1), 1990: a
// faithful quotient corrected once with the rounded reciprocal, unless k's
// significand is all ones); rk = 0 asks for the division.
AR_HD float sdf_over_k(float x, float k, float rk)
{
    if (rk == 0.0f) return x / k;
    float q = x * rk;
    q = fmaf(fmaf(-q, k, x), rk, q);
    return fmaf(fmaf(-q, k, x), rk, q);
}

// the reciprocal sdf_over_k takes for width k
inline float sdf_reciprocal_k(float k)
{
    uint32_t u;
    memcpy(&u, &k, 4);
    return ((u & 0x7fffffu) == 0x7fffffu || !(k > 0x1p-60f && k < 0x1p60f)) ? 0.0f : 1.0f / k;
}

// one primitive's distance with the kinds' arithmetic side by side: each is the
// length of a vector plus a number, with the operations of sdf_prim in its order
AR_HD float sdf_prim_flat(float4 a, float4 b, V3 p)
{
    const V3 q = p - v3(a.y, a.z, a.w);
    V3 v = q;
    float tail = -b.x;
    if ((int)a.x == AR_SDF_BOX)
    {
        const V3 d = v3(fabsf(q.x) - b.x, fabsf(q.y) - b.y, fabsf(q.z) - b.z);
        v = vmax(d, 0.0f);
        tail = fminf(fmaxf(d.x, fmaxf(d.y, d.z)), 0.0f);
    }
    else if ((int)a.x == AR_SDF_TORUS)
    {
        v = v3(sqrtf(q.x * q.x + q.z * q.z) - b.x, q.y, 0.0f);
        tail = -b.y;
    }
    return length(v) + tail;
}

// smin_poly(d, di, s.k)
AR_HD float sdf_blend(const SdfUnion& s, float d, float di)
{
    const float x = s.k - fabsf(d - di);
    d = fminf(d, di);
    if (x > 0.0f)
    {
        const float h = sdf_over_k(x, s.k, s.rk);
        d = d - h * h * s.k * 0.25f;
    }
    return d;
}

// The smooth union folded left to right over the primitives of mask m, which
// starts with the fold's first.  Where the blend weight is zero (the distances
// differ by the width or more) smin_poly is the smaller of the two exactly, so
// every primitive that a mask leaves out by that rule leaves the same bits.
// Four distances are computed side by side and then folded: a march is a chain
// of these evaluations, and a chain of one primitive after the other is twice
// as long.
AR_HD float sdf_fold(const SdfUnion& s, unsigned long long mask, V3 p)
{
    float d = 0.0f;
    bool first = true;
    for (int base = 0; base < 64; base += 32)
    {
        uint32_t m = (uint32_t)(mask >> base);
        while (m)
        {
            float di[4];
            bool on[4];
#pragma unroll
            for (int j = 0; j < 4; ++j)
            {
                on[j] = m != 0u;
                int i = 0;
#if defined(__CUDA_ARCH__)
                if (m) i = base + __ffs((int)m) - 1;
#else
                if (m) i = base + __builtin_ctz(m);
#endif
                m &= m - 1u;
                di[j] = on[j] ? sdf_prim_flat(s.prims[2 * i], s.prims[2 * i + 1], p) : 0.0f;
            }
#pragma unroll
            for (int j = 0; j < 4; ++j)
            {
                if (!on[j]) continue;
                d = first ? di[j] : sdf_blend(s, d, di[j]);
                first = false;
            }
        }
    }
    return d;
}

// The primitives that can change the union's value within distance r of c.
// Distances change by at most r over the ball (every primitive's field is
// 1-Lipschitz), so with [L, U] around each distance at c:
//  * primitive i is left out when L_i is k above an upper bound of the running
//    value (the smallest U so far): the fold leaves the value alone there;
//  * everything before i is dropped when a lower bound of the running value is
//    k above U_i: smin_poly then returns the new distance exactly.
// The bounds are widened by more than the rounding of any evaluation inside;
// a primitive with values that are not finite keeps the whole fold.
AR_HD unsigned long long sdf_cell_mask(const SdfUnion& s, V3 c, float r)
{
    unsigned long long m = 0ull;
    float lb = 0.0f, ub = 0.0f;
    for (int i = 0; i < s.count; ++i)
    {
        const float4 a = s.prims[2 * i], b = s.prims[2 * i + 1];
        const float di = sdf_prim(a, b, c);
        const float size = fabsf(a.y) + fabsf(a.z) + fabsf(a.w) + fabsf(c.x) + fabsf(c.y) + fabsf(c.z) + fabsf(b.x) +
                           fabsf(b.y) + fabsf(b.z) + s.k;
        const float w = r + 0x1p-18f * (size + r);
        const float L = di - w, U = di + w;
        if (!(fabsf(L) < 1.0e30f && fabsf(U) < 1.0e30f)) return sdf_all(s);
        if (i == 0 || lb - U >= s.k)
        {
            m = 1ull << i;
            lb = L;
            ub = U;
        }
        else if (!(L - ub >= s.k))
        {
            m |= 1ull << i;
            ub = fminf(ub, U);
            lb = fminf(lb, L) - 0.25f * s.k;  // a blend lowers the smaller value by at most k / 4
        }
    }
    return m;
}

// the cell p lies in, -1 outside the grid
AR_HD int sdf_cell(const SdfUnion& s, V3 p)
{
    const V3 f = (p - s.lo) * s.inv_cell;
    if (s.cells && f.x >= 0.0f && f.y >= 0.0f && f.z >= 0.0f && f.x < (float)s.res[0] && f.y < (float)s.res[1] &&
        f.z < (float)s.res[2])
        return ((int)f.z * s.res[1] + (int)f.y) * s.res[0] + (int)f.x;
    return -1;
}

// the fold's primitives at p: those of its cell, all of them outside the grid
AR_HD unsigned long long sdf_mask(const SdfUnion& s, V3 p)
{
    const int c = sdf_cell(s, p);
    return c >= 0 ? s.cells[c] : sdf_all(s);
}

AR_HD float sdf_union(const SdfUnion& s, V3 p) { return sdf_fold(s, sdf_mask(s, p), p); }

// entry / exit distances of the ray through the union's bounds
AR_HD bool sdf_bounds_interval(const SdfUnion& s, V3 o, V3 d, float* t0, float* t1)
{
    const V3 inv = v3(inv_safe(d.x), inv_safe(d.y), inv_safe(d.z));
    const V3 a = (s.lo - o) * inv, b = (s.hi - o) * inv;
    const V3 tn = vmin(a, b), tf = vmax(a, b);
    *t0 = fmaxf(fmaxf(tn.x, tn.y), tn.z);
    *t1 = fminf(fminf(tf.x, tf.y), tf.z);
    return *t0 <= *t1 && *t1 > 0.0f;
}

// The march and the normal are called out of line: inlined into the BVH
// traversal loop they would raise its register count for every ray.
#if defined(__CUDACC__)
#define AR_SDF_CALL static __host__ __device__ __noinline__
#else
#define AR_SDF_CALL inline
#endif

// distance to the first surface crossing in the bounds before tmax, or -1
AR_SDF_CALL float sdf_march(const SdfUnion& s, V3 o, V3 d, float eps, float tmax)
{
    float t0, t1;
    if (s.count <= 0 || !sdf_bounds_interval(s, o, d, &t0, &t1) || t0 >= tmax) return -1.0f;
    t1 = fminf(t1, tmax);
    const bool start_inside = sdf_union(s, o) <= 0.0f;
    const float min_step = eps * 0.5f;
    float t = fmaxf(0.0f, t0);
    for (int i = 0; i < AR_SDF_STEPS; ++i)
    {
        const float t_last = t;
        const float dist = sdf_union(s, o + d * t);
        if (start_inside ? (dist > 0.0f && dist < eps) : (dist < 0.0f && -dist < eps)) return t_last;
        t += fmaxf(fabsf(dist), min_step);
        if (t > t1) break;
    }
    return -1.0f;
}

// outward normal by central differences (sdfNormalUnit, core/object/sdf/sdf_base.cuh:40-51)
AR_SDF_CALL V3 sdf_normal(const SdfUnion& s, V3 p, float h)
{
    const float dx = sdf_union(s, p + v3(h, 0, 0)) - sdf_union(s, p - v3(h, 0, 0));
    const float dy = sdf_union(s, p + v3(0, h, 0)) - sdf_union(s, p - v3(0, h, 0));
    const float dz = sdf_union(s, p + v3(0, 0, h)) - sdf_union(s, p - v3(0, 0, h));
    return normalize(v3(dx, dy, dz));
}
} // namespace ar
