// GPU build of the 8-wide compressed BVH (the same node and slot format as the
// host builder, ar_bvh.h), and its refit after mesh vertices move (the tree is
// kept; slots take the new vertices, boxes are recomputed from the leaves up).  The reference
// builds its BVH on the host (BuildBVH, core/bvh/bvh.cuh:142-422); for meshes of
// millions of triangles the build dominates scene setup, so this path runs it
// on the GPU:
//   1. Morton codes of primitive centroids (63 bits) in the centroid bounds,
//      scaled by the largest extent on every axis (cells stay cubes);
//   2. a stable LSD radix sort of (code, primitive) pairs, 8-bit digits;
//   3. the binary radix tree over the sorted codes (Karras, "Maximizing
//      parallelism in the construction of BVHs, octrees, and k-d trees", HPG
//      2012), equal codes ordered by position;
//   4. node boxes bottom-up (the second child to arrive at a node merges);
//   5. collapse to width 8, one level of wide nodes per launch: a wide node
//      opens its largest-area child until it has 8 children; a binary node
//      covering at most 3 primitives is a leaf; children take octant slots by
//      the greedy alignment rule of the host builder; boxes are quantized
//      conservatively against the node's box, as on the host.
// Hit results do not depend on the tree (closest hits are the smallest t, equal
// t the smallest id), so a GPU-built BVH answers exactly as the host-built one.
#include <cuda_runtime.h>

#include <algorithm>
#include <cfloat>
#include <cmath>
#include <string>
#include <vector>

#include "../../include/aperture/ar.h"
#include "ar_bvh_build.h"
#include "ar_bvh_lanes.h"
#include "ar_internal.h"

namespace ar
{
namespace lbvh
{
constexpr int kMaxLeaf = 3;
constexpr int kSortBlock = 256;
// Tiles of kSortBlock keys per block and pass.  Few tiles spread a small build over
// the chip, many keep the scan short (256 counters per block, one block scans):
// 200,000 keys, eight passes of histogram, scan and scatter 514 us at 16 tiles with
// the scan by doubling steps, 264 at 4, of which the scan 135; rebuild of 200,000
// triangles 3.01 ms at 16 tiles, 2.95 at 8, 2.97 at 4, 2.99 at 2.
constexpr int kSortTiles = 8;

__device__ __forceinline__ unsigned int fmin_bits(float f)  // order-preserving float -> uint
{
    const unsigned int u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float bits_fmin(unsigned int u)
{
    return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u);
}

// The build's primitives: the objects as given, then the mesh triangles.
__global__ void k_prims(const arbvh::PrimInput* __restrict__ objects, int nobj, const float* __restrict__ mesh_v, int n,
                        int first_mesh_id, arbvh::PrimInput* prims)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    if (i < nobj)
    {
        prims[i] = objects[i];
        return;
    }
    arbvh::PrimInput p;
    p.id = (uint32_t)(first_mesh_id + (i - nobj));
    p.kind = AR_PRIM_KIND_TRI;
    for (int k = 0; k < 9; ++k) p.v[k] = mesh_v[9 * (size_t)(i - nobj) + k];
    for (int k = 0; k < 3; ++k)
    {
        // the host builder's std::min / std::max, comparison by comparison
        const float a = p.v[k], b = p.v[3 + k], c = p.v[6 + k];
        const float lo = c < b ? c : b, hi = b < c ? c : b;
        p.lo[k] = lo < a ? lo : a;
        p.hi[k] = a < hi ? hi : a;
    }
    prims[i] = p;
}

__global__ void k_slot_tables(ar_prim_slot* slots, int n, const int* __restrict__ prim_material,
                              const int* __restrict__ prim_light, int* prim_slot)
{
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n) return;
    const uint32_t tag = __float_as_uint(slots[s].a[3]);
    const uint32_t id = tag & AR_PRIM_ID_MASK;
    prim_slot[id] = s;
    if (!prim_material || (tag >> AR_PRIM_KIND_SHIFT) != AR_PRIM_KIND_TRI) return;
    slots[s].b[3] = __int_as_float(prim_material[id]);
    slots[s].c[3] = __int_as_float(prim_light[id]);
}

__global__ void k_light_ids(const Light* __restrict__ lights, int n, int* prim_light)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < n) prim_light[lights[k].obj] = k;
}

__global__ void k_iota(int* v, int n)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) v[i] = i;
}

// centroid bounds: bounds[0..2] min, [3..5] max, as ordered uints
__global__ void k_centroid_bounds(const arbvh::PrimInput* __restrict__ prims, int n, unsigned int* bounds)
{
    float lo[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, hi[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        for (int k = 0; k < 3; ++k)
        {
            const float c = 0.5f * (prims[i].lo[k] + prims[i].hi[k]);
            lo[k] = fminf(lo[k], c);
            hi[k] = fmaxf(hi[k], c);
        }
    for (int k = 0; k < 3; ++k)
    {
        for (int o = 16; o > 0; o >>= 1)
        {
            lo[k] = fminf(lo[k], __shfl_xor_sync(0xffffffffu, lo[k], o));
            hi[k] = fmaxf(hi[k], __shfl_xor_sync(0xffffffffu, hi[k], o));
        }
        if ((threadIdx.x & 31) == 0)
        {
            atomicMin(&bounds[k], fmin_bits(lo[k]));
            atomicMax(&bounds[3 + k], fmin_bits(hi[k]));
        }
    }
}

// spreads the low 21 bits of v to every third bit
__device__ __forceinline__ unsigned long long expand_bits21(unsigned long long v)
{
    v &= 0x1fffffull;
    v = (v | (v << 32)) & 0x1f00000000ffffull;
    v = (v | (v << 16)) & 0x1f0000ff0000ffull;
    v = (v | (v << 8)) & 0x100f00f00f00f00full;
    v = (v | (v << 4)) & 0x10c30c30c30c30c3ull;
    v = (v | (v << 2)) & 0x1249249249249249ull;
    return v;
}

__global__ void k_morton(const arbvh::PrimInput* __restrict__ prims, int n, const unsigned int* bounds,
                         unsigned long long* keys, unsigned int* vals)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float lo[3], ext = 0.0f;
    for (int k = 0; k < 3; ++k)
    {
        lo[k] = bits_fmin(bounds[k]);
        ext = fmaxf(ext, bits_fmin(bounds[3 + k]) - lo[k]);
    }
    unsigned long long code = 0;
    for (int k = 0; k < 3; ++k)
    {
        const float c = 0.5f * (prims[i].lo[k] + prims[i].hi[k]);
        float u = ext > 0.0f ? (c - lo[k]) / ext : 0.0f;
        u = fminf(fmaxf(u, 0.0f), 1.0f);
        const unsigned long long q = min((unsigned long long)(u * 2097152.0f), 2097151ull);
        code |= expand_bits21(q) << (2 - k);
    }
    keys[i] = code;
    vals[i] = (unsigned int)i;
}

// ---- stable LSD radix sort, 8-bit digits.  A block owns kSortTiles
// consecutive tiles of kSortBlock keys; pass: histogram per block, exclusive
// scan over (digit, block), stable scatter (rank within a tile from warp
// matches and per-warp digit counts, tiles in order).
__global__ void k_sort_hist(const unsigned long long* __restrict__ keys, int n, int shift, unsigned int* hist, int nblocks)
{
    __shared__ unsigned int h[256];
    for (int i = threadIdx.x; i < 256; i += blockDim.x) h[i] = 0;
    __syncthreads();
    const long long base = (long long)blockIdx.x * kSortBlock * kSortTiles;
    for (int t = 0; t < kSortTiles; ++t)
    {
        const long long i = base + (long long)t * kSortBlock + threadIdx.x;
        if (i < n) atomicAdd(&h[(unsigned int)(keys[i] >> shift) & 0xffu], 1u);
    }
    __syncthreads();
    for (int d = threadIdx.x; d < 256; d += blockDim.x) hist[(size_t)d * nblocks + blockIdx.x] = h[d];
}

// Exclusive scan of hist (256 x nblocks, digit-major; a multiple of 256 entries) in
// place by one block, four entries per thread and pass: sums by shuffles, one
// barrier pair per 4096 entries (50,176 entries: 17 us; with a barrier pair per
// doubling step 12,544 entries took 22).
__global__ void __launch_bounds__(1024) k_sort_scan(unsigned int* hist, int total)
{
    __shared__ unsigned int warp_sum[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned int carry = 0;
    for (int base = 0; base < total; base += 4096)
    {
        const int i = base + 4 * (int)threadIdx.x;
        uint4 v = make_uint4(0u, 0u, 0u, 0u);
        if (i < total) v = *reinterpret_cast<const uint4*>(hist + i);
        const unsigned int own = v.x + v.y + v.z + v.w;
        unsigned int run = own;  // inclusive over the warp
        for (int o = 1; o < 32; o <<= 1)
        {
            const unsigned int a = __shfl_up_sync(0xffffffffu, run, o);
            if (lane >= o) run += a;
        }
        if (lane == 31) warp_sum[warp] = run;
        __syncthreads();
        unsigned int w = warp_sum[lane];  // every warp scans the warps' sums
        for (int o = 1; o < 32; o <<= 1)
        {
            const unsigned int a = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += a;
        }
        const unsigned int all = __shfl_sync(0xffffffffu, w, 31);
        const unsigned int before = __shfl_sync(0xffffffffu, w, warp == 0 ? 0 : warp - 1);
        unsigned int x = carry + (warp ? before : 0u) + run - own;
        uint4 out;
        out.x = x;
        out.y = x += v.x;
        out.z = x += v.y;
        out.w = x += v.z;
        if (i < total) *reinterpret_cast<uint4*>(hist + i) = out;
        carry += all;
        __syncthreads();  // warp_sum is rewritten by the next pass
    }
}

__global__ void __launch_bounds__(kSortBlock) k_sort_scatter(const unsigned long long* __restrict__ keys,
                                                           const unsigned int* __restrict__ vals, int n, int shift,
                                                           const unsigned int* __restrict__ hist, int nblocks,
                                                           unsigned long long* __restrict__ okeys,
                                                           unsigned int* __restrict__ ovals)
{
    constexpr int W = kSortBlock / 32;
    __shared__ unsigned int run[256];         // next output position per digit
    __shared__ unsigned int wcnt[W][256];     // per-warp digit counts of the tile
    for (int d = threadIdx.x; d < 256; d += blockDim.x) run[d] = hist[(size_t)d * nblocks + blockIdx.x];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long base = (long long)blockIdx.x * kSortBlock * kSortTiles;
    for (int t = 0; t < kSortTiles; ++t)
    {
        for (int k = threadIdx.x; k < W * 256; k += blockDim.x) (&wcnt[0][0])[k] = 0;
        __syncthreads();
        const long long i = base + (long long)t * kSortBlock + threadIdx.x;
        const bool valid = i < n;
        const unsigned long long key = valid ? keys[i] : 0ull;
        const unsigned int dig = valid ? ((unsigned int)(key >> shift) & 0xffu) : 256u;
        const unsigned int peers = __match_any_sync(0xffffffffu, dig);
        const unsigned int rank_in_warp = __popc(peers & ((1u << lane) - 1u));
        if (valid && rank_in_warp == 0) wcnt[warp][dig] = __popc(peers);
        __syncthreads();
        unsigned int pos = 0;
        if (valid)
        {
            unsigned int before = 0;
            for (int w = 0; w < warp; ++w) before += wcnt[w][dig];
            pos = run[dig] + before + rank_in_warp;
            okeys[pos] = key;
            ovals[pos] = vals[i];
        }
        __syncthreads();
        // advance the running offsets by this tile's digit counts
        for (int d = threadIdx.x; d < 256; d += blockDim.x)
        {
            unsigned int c = 0;
            for (int w = 0; w < W; ++w) c += wcnt[w][d];
            run[d] += c;
        }
        __syncthreads();
    }
}

// ---- radix tree (Karras 2012).  Internal nodes 0..n-2, leaves n-1+k for sorted
// position k.  first/last: the sorted range a node covers.
__device__ __forceinline__ int delta(const unsigned long long* keys, int n, int i, int j)
{
    if (j < 0 || j >= n) return -1;
    const unsigned long long a = keys[i], b = keys[j];
    if (a != b) return __clzll(a ^ b);
    return 64 + __clz((unsigned int)i ^ (unsigned int)j);
}

__global__ void k_radix_tree(const unsigned long long* __restrict__ keys, int n, int2* child, int* parent, int2* range)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n - 1) return;
    const int d = (delta(keys, n, i, i + 1) - delta(keys, n, i, i - 1)) >= 0 ? 1 : -1;
    const int dmin = delta(keys, n, i, i - d);
    int lmax = 2;
    while (delta(keys, n, i, i + lmax * d) > dmin) lmax <<= 1;
    int l = 0;
    for (int t = lmax >> 1; t >= 1; t >>= 1)
        if (delta(keys, n, i, i + (l + t) * d) > dmin) l += t;
    const int j = i + l * d;
    const int dnode = delta(keys, n, i, j);
    int s = 0;
    int t = l;
    do
    {
        t = (t + 1) >> 1;
        if (delta(keys, n, i, i + (s + t) * d) > dnode) s += t;
    } while (t > 1);
    const int split = i + s * d + min(d, 0);
    const int first = min(i, j), last = max(i, j);
    const int left = (first == split) ? (n - 1 + split) : split;
    const int right = (last == split + 1) ? (n - 1 + split + 1) : split + 1;
    child[i] = make_int2(left, right);
    parent[left] = i;
    parent[right] = i;
    range[i] = make_int2(first, last);
}

struct Box6
{
    float lo[3], hi[3];
};

__global__ void k_boxes(const arbvh::PrimInput* __restrict__ prims, const unsigned int* __restrict__ order, int n,
                        const int2* __restrict__ child, const int* __restrict__ parent, Box6* box, int* flag)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    int node = n - 1 + k;
    const arbvh::PrimInput& p = prims[order[k]];
    for (int a = 0; a < 3; ++a)
    {
        box[node].lo[a] = p.lo[a];
        box[node].hi[a] = p.hi[a];
    }
    if (n == 1) return;
    node = parent[node];
    while (true)
    {
        __threadfence();
        if (atomicAdd(&flag[node], 1) == 0) return;  // the other child is not done yet
        __threadfence();
        const int2 c = child[node];
        // the other child's box was written by another SM: read it from L2
        const float* bx = reinterpret_cast<const float*>(&box[c.x]);
        const float* by = reinterpret_cast<const float*>(&box[c.y]);
        Box6 b;
        for (int a = 0; a < 3; ++a)
        {
            b.lo[a] = fminf(__ldcg(bx + a), __ldcg(by + a));
            b.hi[a] = fmaxf(__ldcg(bx + 3 + a), __ldcg(by + 3 + a));
        }
        box[node] = b;
        if (node == 0) return;
        node = parent[node];
        if (node < 0 || node >= n - 1) return;  // malformed tree: the build reports a count mismatch
    }
}

// number of sorted primitives under binary node b
__device__ __forceinline__ int node_count(int b, int n, const int2* range)
{
    if (b >= n - 1) return 1;
    const int2 r = range[b];
    return r.y - r.x + 1;
}
__device__ __forceinline__ int node_first(int b, int n, const int2* range)
{
    return b >= n - 1 ? b - (n - 1) : range[b].x;
}

struct CollapseArgs
{
    const arbvh::PrimInput* prims;
    const unsigned int* order;
    int n;
    const int2* child;
    const int2* range;
    const Box6* box;
    ar_wide_node* nodes;
    ar_prim_slot* slots;
    int* node_counter;
    int* slot_counter;
    int node_cap;
};

// Exponent e (biased by 127 in a node) of the smallest power of two with
// 255 2^e >= hi - lo, at least AR_BVH_MIN_EXP: the difference rounded up is m 2^k with m in
// [1, 2), and 255 is 1.9921875 2^7.
__device__ __forceinline__ int quant_exponent(float lo, float hi)
{
    const float ext = __fsub_ru(hi, lo);
    if (!(ext > 0.0f)) return AR_BVH_MIN_EXP;
    const uint32_t u = __float_as_uint(ext);
    const int k = (int)(u >> 23) - 127;
    const int e = k - 7 + ((u & 0x7fffffu) > 0x7f0000u || k == 128 ? 1 : 0);
    return e < AR_BVH_MIN_EXP ? AR_BVH_MIN_EXP : e;
}

// A child plane in steps of 2^e above the node's low plane, moved outwards: the
// difference is rounded away from the box, the scaling is exact.
__device__ __forceinline__ uint8_t quant_low(float lo, float node_lo, float inv_step)
{
    return (uint8_t)fminf(fmaxf(floorf(__fsub_rd(lo, node_lo) * inv_step), 0.0f), 255.0f);
}
__device__ __forceinline__ uint8_t quant_high(float hi, float node_lo, float inv_step)
{
    return (uint8_t)fminf(fmaxf(ceilf(__fsub_ru(hi, node_lo) * inv_step), 0.0f), 255.0f);
}

// One wide node per 8 lanes, one lane per child (lane k of a group: child k, then
// slot k).  A node by a single thread is a serial chain of some 1,500 double
// precision operations and its local arrays; by a group it is a few rounds of
// shuffles (200,000 triangles, 7 levels: 1068 -> 256 us).  All lanes of a group have
// to end each round with the same winner (ar_bvh_lanes.h).  queue: (wide index,
// binary index); internal children are appended to the next level's queue.
__global__ void __launch_bounds__(128) k_collapse(CollapseArgs a, const int2* __restrict__ queue, int nq, int2* next,
                                                int* next_count, unsigned int* err)
{
    const int lane = threadIdx.x & 31, sub = lane & 7, lead = lane & 24;
    const unsigned gm = 0xffu << lead;
    const int qi = (blockIdx.x * blockDim.x + threadIdx.x) >> 3;
    if (qi >= nq) return;  // whole groups
    const int wi = queue[qi].x, b = queue[qi].y;
    const int n = a.n;
    // children: the largest-area one that is no leaf is opened until there are 8
    int ch = -1, nch;
    if (node_count(b, n, a.range) <= kMaxLeaf)
    {
        if (sub == 0) ch = b;
        nch = 1;
    }
    else
    {
        const int2 c = a.child[b];
        if (sub < 2) ch = sub == 0 ? c.x : c.y;
        nch = 2;
    }
    int cnt = ch >= 0 ? node_count(ch, n, a.range) : 0;
    Box6 cb{};
    double area = -1.0;
    if (ch >= 0)
    {
        cb = a.box[ch];
        if (cnt > kMaxLeaf) area = open_area(cb.lo, cb.hi);
    }
    while (nch < 8)
    {
        double best = area;
        int pick = sub;
        for (int k = 4; k > 0; k >>= 1)
        {
            const double o = __shfl_xor_sync(gm, best, k);
            const int p = __shfl_xor_sync(gm, pick, k);
            if (opens_before(o, p, best, pick))
            {
                best = o;
                pick = p;
            }
        }
        if (best < 0.0) break;
        const int c = __shfl_sync(gm, ch, lead + pick);
        if (sub == pick || sub == nch)
        {
            const int2 cc = a.child[c];
            ch = sub == pick ? cc.x : cc.y;
            cnt = node_count(ch, n, a.range);
            cb = a.box[ch];
            area = cnt > kMaxLeaf ? open_area(cb.lo, cb.hi) : -1.0;
        }
        ++nch;
    }
    const bool real = sub < nch;
    float lo[3], hi[3];
    for (int k = 0; k < 3; ++k)
    {
        lo[k] = real ? cb.lo[k] : FLT_MAX;
        hi[k] = real ? cb.hi[k] : -FLT_MAX;
        for (int j = 4; j > 0; j >>= 1)
        {
            lo[k] = fminf(lo[k], __shfl_xor_sync(gm, lo[k], j));
            hi[k] = fmaxf(hi[k], __shfl_xor_sync(gm, hi[k], j));
        }
    }
    // octant slots: greedy over (child, slot) by decreasing alignment, ties to
    // the earlier candidate (the host builder's stable sort)
    double off[3];
    for (int k = 0; k < 3; ++k)
        off[k] = 0.5 * ((double)cb.lo[k] + cb.hi[k]) - 0.5 * ((double)lo[k] + hi[k]);
    unsigned taken = 0u;
    int slot = -1;
    for (int round = 0; round < nch; ++round)
    {
        double bc = -DBL_MAX;
        int bs = 8;
        if (real && slot < 0)
            for (int s = 0; s < 8; ++s)
            {
                if ((taken >> s) & 1u) continue;
                const double c = slot_cost(off, s);
                if (bs == 8 || c > bc)
                {
                    bc = c;
                    bs = s;
                }
            }
        int who = bs < 8 ? sub : 8 + sub;
        for (int k = 4; k > 0; k >>= 1)
        {
            const double o = __shfl_xor_sync(gm, bc, k);
            const int w = __shfl_xor_sync(gm, who, k);
            const int s = __shfl_xor_sync(gm, bs, k);
            if (placed_before(o, w, bc, who))
            {
                bc = o;
                who = w;
                bs = s;
            }
        }
        taken |= 1u << bs;
        if (sub == who) slot = bs;
    }
    // from here lane k holds the child of slot k (or none)
    int from = -1;
    for (int s = 0; s < 8; ++s)
    {
        const unsigned m = __ballot_sync(gm, real && slot == s);
        if (s == sub && m) from = __ffs((int)m) - 1;
    }
    const bool used = from >= 0;
    const int src = used ? from : lane;
    ch = __shfl_sync(gm, ch, src);
    cnt = __shfl_sync(gm, cnt, src);
    for (int k = 0; k < 3; ++k)
    {
        cb.lo[k] = __shfl_sync(gm, cb.lo[k], src);
        cb.hi[k] = __shfl_sync(gm, cb.hi[k], src);
    }
    const bool inner = used && cnt > kMaxLeaf, leaf = used && !inner;
    const unsigned imask = (__ballot_sync(gm, inner) >> lead) & 0xffu;
    const int n_int = __popc(imask), rank = __popc(imask & ((1u << sub) - 1u));
    int poff = leaf ? cnt : 0;  // exclusive sum of the leaves' primitives over the slots
    for (int k = 1; k < 8; k <<= 1)
    {
        const int o = __shfl_up_sync(gm, poff, k, 8);
        if (sub >= k) poff += o;
    }
    const int n_prims = __shfl_sync(gm, poff, lead + 7);
    poff -= leaf ? cnt : 0;
    int child_base = 0, prim_base = 0, q0 = 0;
    if (sub == 0)
    {
        if (n_int)
        {
            child_base = atomicAdd(a.node_counter, n_int);
            q0 = atomicAdd(next_count, n_int);
        }
        if (n_prims) prim_base = atomicAdd(a.slot_counter, n_prims);
    }
    child_base = __shfl_sync(gm, child_base, lead);
    prim_base = __shfl_sync(gm, prim_base, lead);
    q0 = __shfl_sync(gm, q0, lead);
    if (child_base + n_int > a.node_cap || prim_base + n_prims > n || q0 + n_int > a.node_cap)
    {
        if (sub == 0) atomicOr(err, AR_DEVERR_QUEUE);
        return;
    }
    ar_wide_node* node = &a.nodes[wi];
    const uint8_t meta = inner ? (uint8_t)(0x80u | (uint32_t)rank) : leaf ? (uint8_t)(((uint32_t)cnt << 5) | (uint32_t)poff) : 0;
    node->meta[sub] = meta;
    int e[3];
    for (int k = 0; k < 3; ++k)
    {
        e[k] = quant_exponent(lo[k], hi[k]);
        const float inv = ldexpf(1.0f, -e[k]);
        // empty slots: an inverted box that no ray meets
        node->qlo[k][sub] = used ? quant_low(cb.lo[k], lo[k], inv) : 0xff;
        node->qhi[k][sub] = used ? quant_high(cb.hi[k], lo[k], inv) : 0;
    }
    if (sub == 0)
    {
        node->px = lo[0];
        node->py = lo[1];
        node->pz = lo[2];
        for (int k = 0; k < 3; ++k) node->e[k] = (uint8_t)(e[k] + 127);
        node->imask = (uint8_t)imask;
        node->child_base = (uint32_t)child_base;
        node->prim_base = (uint32_t)prim_base;
    }
    if (inner) next[q0 + rank] = make_int2(child_base + rank, ch);
    if (leaf)
    {
        const int first = node_first(ch, n, a.range);
        for (int j = 0; j < cnt; ++j)
        {
            const arbvh::PrimInput& pi = a.prims[a.order[first + j]];
            ar_prim_slot sl;
            memset(&sl, 0, sizeof(sl));
            const uint32_t tag = pi.id | (pi.kind << AR_PRIM_KIND_SHIFT);
            if (pi.kind == AR_PRIM_KIND_TRI)
                for (int k = 0; k < 3; ++k)
                {
                    sl.a[k] = pi.v[k];
                    sl.b[k] = pi.v[3 + k];
                    sl.c[k] = pi.v[6 + k];
                }
            sl.a[3] = __uint_as_float(tag);
            a.slots[prim_base + poff + j] = sl;
        }
    }
}
} // namespace lbvh

// ---- refit
// triangle slots take the moved vertices (slot tag -> triangle id - n_objects)
__global__ void k_refit_slots(float4* slots, int nslots, const float* __restrict__ verts, const uint32_t* __restrict__ idx,
                              int nobj)
{
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= nslots) return;
    const uint32_t tag = __float_as_uint(slots[3 * (size_t)s].w);
    if ((tag >> AR_PRIM_KIND_SHIFT) != AR_PRIM_KIND_TRI) return;
    const int id = (int)(tag & AR_PRIM_ID_MASK);
    if (id < nobj) return;  // a triangle object: not part of the mesh
    const size_t t = (size_t)(id - nobj);
    for (int j = 0; j < 3; ++j)
    {
        const float* v = verts + 3 * (size_t)idx[3 * t + j];
        float4 w = slots[3 * (size_t)s + j];
        w.x = v[0];
        w.y = v[1];
        w.z = v[2];
        slots[3 * (size_t)s + j] = w;
    }
}

// One depth of wide nodes, 8 lanes per node and one per child: child boxes from
// the leaves' primitives or the deeper level's node boxes, then the node
// re-quantized as the builders do.  A level near the root has few nodes and costs
// the chain of one of them: by a single thread (8 children in turn, divisions and
// logarithms in double precision) 40-60 us, by a group 5 (all 7 levels of a
// 524,000-triangle sheet: 389 -> 39 us).
__global__ void __launch_bounds__(128) k_refit_level(ar_wide_node* nodes, const int* __restrict__ list, int nlist,
                                                   const float4* __restrict__ slots, const float* __restrict__ prim_box,
                                                   float* node_box)
{
    const int lane = threadIdx.x & 31, sub = lane & 7, lead = lane & 24;
    const unsigned gm = 0xffu << lead;
    const int li = (blockIdx.x * blockDim.x + threadIdx.x) >> 3;
    if (li >= nlist) return;  // whole groups
    const int ni = list[li];
    ar_wide_node* node = &nodes[ni];
    const uint32_t meta = node->meta[sub], child_base = node->child_base, prim_base = node->prim_base;
    const unsigned inner = (__ballot_sync(gm, (meta & 0x80u) != 0u) >> lead) & 0xffu;
    float b[6] = {FLT_MAX, FLT_MAX, FLT_MAX, -FLT_MAX, -FLT_MAX, -FLT_MAX};
    if (meta & 0x80u)
    {
        const float* src = node_box + 6 * (size_t)(child_base + __popc(inner & ((1u << sub) - 1u)));
        for (int k = 0; k < 6; ++k) b[k] = src[k];
    }
    else if (meta)
    {
        const int cnt = (int)(meta >> 5), first = (int)(prim_base + (meta & 31u));
        for (int j = 0; j < cnt; ++j)
        {
            const float4 a = slots[3 * (size_t)(first + j)];
            const uint32_t tag = __float_as_uint(a.w);
            if ((tag >> AR_PRIM_KIND_SHIFT) == AR_PRIM_KIND_TRI)
            {
                const float4 bb = slots[3 * (size_t)(first + j) + 1], cc = slots[3 * (size_t)(first + j) + 2];
                b[0] = fminf(b[0], fminf(a.x, fminf(bb.x, cc.x)));
                b[1] = fminf(b[1], fminf(a.y, fminf(bb.y, cc.y)));
                b[2] = fminf(b[2], fminf(a.z, fminf(bb.z, cc.z)));
                b[3] = fmaxf(b[3], fmaxf(a.x, fmaxf(bb.x, cc.x)));
                b[4] = fmaxf(b[4], fmaxf(a.y, fmaxf(bb.y, cc.y)));
                b[5] = fmaxf(b[5], fmaxf(a.z, fmaxf(bb.z, cc.z)));
            }
            else
            {
                const float* pb = prim_box + 6 * (size_t)(tag & AR_PRIM_ID_MASK);
                for (int k = 0; k < 3; ++k)
                {
                    b[k] = fminf(b[k], pb[k]);
                    b[3 + k] = fmaxf(b[3 + k], pb[3 + k]);
                }
            }
        }
    }
    for (int k = 0; k < 3; ++k)
    {
        float lo = b[k], hi = b[3 + k];
        for (int j = 4; j > 0; j >>= 1)
        {
            lo = fminf(lo, __shfl_xor_sync(gm, lo, j));
            hi = fmaxf(hi, __shfl_xor_sync(gm, hi, j));
        }
        const int e = lbvh::quant_exponent(lo, hi);
        const float inv = ldexpf(1.0f, -e);
        if (meta)
        {
            node->qlo[k][sub] = lbvh::quant_low(b[k], lo, inv);
            node->qhi[k][sub] = lbvh::quant_high(b[3 + k], lo, inv);
        }
        if (sub == 0)
        {
            if (k == 0) node->px = lo;
            else if (k == 1) node->py = lo;
            else node->pz = lo;
            node->e[k] = (uint8_t)(e + 127);
            node_box[6 * (size_t)ni + k] = lo;
            node_box[6 * (size_t)ni + 3 + k] = hi;
        }
    }
}

cudaError_t refit_wide_bvh(Ctx& c, const float* verts_dev, cudaStream_t s)
{
    const int nslots = c.slot_count;
    if (nslots == 0) return cudaSuccess;
    k_refit_slots<<<(nslots + 255) / 256, 256, 0, s>>>(reinterpret_cast<float4*>(c.d_slots), nslots, verts_dev,
                                                        c.d_mesh_idx, (int)c.objects.size());
    cudaError_t e = cudaGetLastError();
    for (int d = (int)c.refit_level_off.size() - 2; d >= 0 && e == cudaSuccess; --d)
    {
        const int a = c.refit_level_off[d], b = c.refit_level_off[d + 1];
        if (b <= a) continue;
        k_refit_level<<<(b - a + 15) / 16, 128, 0, s>>>(reinterpret_cast<ar_wide_node*>(c.d_nodes), c.d_refit_nodes + a,
                                                         b - a, reinterpret_cast<const float4*>(c.d_slots), c.d_prim_box,
                                                         c.d_node_box);
        e = cudaGetLastError();
    }
    return e;
}

cudaError_t launch_slot_tables(void* slots, int n, const int* prim_material, const int* prim_light, int* prim_slot,
                               cudaStream_t s)
{
    if (n > 0)
        lbvh::k_slot_tables<<<(n + 255) / 256, 256, 0, s>>>((ar_prim_slot*)slots, n, prim_material, prim_light, prim_slot);
    return cudaGetLastError();
}

cudaError_t launch_light_ids(const Light* lights, int n, int* prim_light, cudaStream_t s)
{
    if (n > 0) lbvh::k_light_ids<<<(n + 255) / 256, 256, 0, s>>>(lights, n, prim_light);
    return cudaGetLastError();
}

cudaError_t launch_iota(int* v, int n, cudaStream_t s)
{
    if (n > 0) lbvh::k_iota<<<(n + 255) / 256, 256, 0, s>>>(v, n);
    return cudaGetLastError();
}

// The primitives' boxes are made on the device and the tree stays there: a
// rebuild moves the vertices in, one queue length per level and the root box out.
// Building the primitive records on the host, bringing nodes and slots back to
// tag and regroup them there and 17 allocations were 5.9 of the 8.0 ms of a
// 200,000-triangle rebuild.
std::string build_wide_bvh_gpu(const std::vector<arbvh::PrimInput>& objects, const float* mesh_v, int nmesh, int first_mesh_id,
                               GpuBvh& out, cudaStream_t s)
{
    using namespace lbvh;
    out.level_off.assign(1, 0);
    const int nobj = (int)objects.size();
    const int n = nobj + nmesh;
    if (n == 0) return "";
    const int nblocks = (n + kSortBlock * kSortTiles - 1) / (kSortBlock * kSortTiles);
    const int node_cap = n;  // wide nodes never outnumber primitives
    // one allocation, carved twice: sizes first, then addresses
    char* base = nullptr;
    size_t used = 0;
    auto carve = [&](size_t bytes) -> void* {
        void* p = base ? base + used : nullptr;
        used += (bytes + 255) & ~(size_t)255;
        return p;
    };
    arbvh::PrimInput *dobjs = nullptr, *dprims = nullptr;
    float* dverts = nullptr;
    unsigned int *bounds = nullptr, *v0 = nullptr, *v1 = nullptr, *hist = nullptr;
    unsigned long long *k0 = nullptr, *k1 = nullptr;
    int2 *child = nullptr, *range = nullptr, *qa = nullptr, *qb = nullptr;
    int *parent = nullptr, *flag = nullptr, *counters = nullptr;
    Box6* box = nullptr;
    ar_wide_node* nodes = nullptr;
    ar_prim_slot* slots = nullptr;
    for (int pass = 0; pass < 2; ++pass)
    {
        used = 0;
        dobjs = (arbvh::PrimInput*)carve(sizeof(arbvh::PrimInput) * (size_t)nobj);
        dverts = (float*)carve(9 * sizeof(float) * (size_t)nmesh);
        dprims = (arbvh::PrimInput*)carve(sizeof(arbvh::PrimInput) * (size_t)n);
        bounds = (unsigned int*)carve(6 * sizeof(unsigned int));
        k0 = (unsigned long long*)carve(8ull * n);
        v0 = (unsigned int*)carve(4ull * n);
        k1 = (unsigned long long*)carve(8ull * n);
        v1 = (unsigned int*)carve(4ull * n);
        hist = (unsigned int*)carve(4ull * 256 * nblocks);
        child = (int2*)carve(sizeof(int2) * (size_t)std::max(1, n - 1));
        range = (int2*)carve(sizeof(int2) * (size_t)std::max(1, n - 1));
        parent = (int*)carve(sizeof(int) * (size_t)(2 * (size_t)n));
        flag = (int*)carve(sizeof(int) * (size_t)std::max(1, n - 1));
        box = (Box6*)carve(sizeof(Box6) * (size_t)(2 * (size_t)n));
        nodes = (ar_wide_node*)carve(sizeof(ar_wide_node) * (size_t)node_cap);
        slots = (ar_prim_slot*)carve(sizeof(ar_prim_slot) * (size_t)n);
        qa = (int2*)carve(sizeof(int2) * (size_t)node_cap);
        qb = (int2*)carve(sizeof(int2) * (size_t)node_cap);
        counters = (int*)carve(4 * sizeof(int));  // nodes, slots, next queue, error word
        if (pass == 0)
        {
            if (cudaMalloc(&out.arena, used) != cudaSuccess)
            {
                out.arena = nullptr;
                cudaGetLastError();
                return "GPU BVH build: out of device memory";
            }
            base = (char*)out.arena;
        }
    }
    cudaError_t e = cudaSuccess;
    if (nobj > 0)
        e = cudaMemcpyAsync(dobjs, objects.data(), sizeof(arbvh::PrimInput) * (size_t)nobj, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess && nmesh > 0)
        e = cudaMemcpyAsync(dverts, mesh_v, 9 * sizeof(float) * (size_t)nmesh, cudaMemcpyHostToDevice, s);
    const unsigned int init_bounds[6] = {0xffffffffu, 0xffffffffu, 0xffffffffu, 0u, 0u, 0u};
    if (e == cudaSuccess) e = cudaMemcpyAsync(bounds, init_bounds, sizeof(init_bounds), cudaMemcpyHostToDevice, s);
    const int grid = (n + 255) / 256;
    if (e == cudaSuccess)
    {
        k_prims<<<grid, 256, 0, s>>>(dobjs, nobj, dverts, n, first_mesh_id, dprims);
        k_centroid_bounds<<<std::min(grid, 1024), 256, 0, s>>>(dprims, n, bounds);
        k_morton<<<grid, 256, 0, s>>>(dprims, n, bounds, k0, v0);
        e = cudaGetLastError();
    }
    // 63-bit codes: eight 8-bit passes (the last one sees 7 bits)
    unsigned long long *ka = k0, *kb = k1;
    unsigned int *va = v0, *vb = v1;
    for (int pass = 0; pass < 8 && e == cudaSuccess; ++pass)
    {
        const int shift = 8 * pass;
        k_sort_hist<<<nblocks, kSortBlock, 0, s>>>(ka, n, shift, hist, nblocks);
        k_sort_scan<<<1, 1024, 0, s>>>(hist, 256 * nblocks);
        k_sort_scatter<<<nblocks, kSortBlock, 0, s>>>(ka, va, n, shift, hist, nblocks, kb, vb);
        e = cudaGetLastError();
        std::swap(ka, kb);
        std::swap(va, vb);
    }
    if (e == cudaSuccess) e = cudaMemsetAsync(flag, 0, sizeof(int) * (size_t)std::max(1, n - 1), s);
    if (e == cudaSuccess && n > 1)
    {
        k_radix_tree<<<(n - 1 + 255) / 256, 256, 0, s>>>(ka, n, child, parent, range);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess)
    {
        k_boxes<<<grid, 256, 0, s>>>(dprims, va, n, child, parent, box, flag);
        e = cudaGetLastError();
    }
    // collapse, level by level; the root is wide node 0 over binary node 0
    // (or the single leaf when n == 1)
    // the root: internal node 0, or leaf n - 1 = 0 when n == 1
    const int2 q0 = make_int2(0, 0);
    const int init_counters[4] = {1, 0, 0, 0};
    if (e == cudaSuccess) e = cudaMemcpyAsync(qa, &q0, sizeof(int2), cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(counters, init_counters, sizeof(init_counters), cudaMemcpyHostToDevice, s);
    CollapseArgs ca{dprims, va, n, child, range, box, nodes, slots, &counters[0], &counters[1], node_cap};
    int nq = 1, depth = 0;
    while (e == cudaSuccess && nq > 0)
    {
        ++depth;
        const int level = nq;
        e = cudaMemsetAsync(&counters[2], 0, sizeof(int), s);
        if (e != cudaSuccess) break;
        k_collapse<<<(nq + 15) / 16, 128, 0, s>>>(ca, qa, nq, qb, &counters[2], (unsigned int*)&counters[3]);
        e = cudaGetLastError();
        if (e == cudaSuccess) e = cudaMemcpyAsync(&nq, &counters[2], sizeof(int), cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        std::swap(qa, qb);
        // children are placed level by level, so a level's nodes are consecutive
        if (e == cudaSuccess) out.level_off.push_back(out.level_off.back() + level);
        if (depth > 4096) break;
    }
    int host_counters[4] = {0, 0, 0, 0};
    Box6 rb{};
    if (e == cudaSuccess) e = cudaMemcpyAsync(host_counters, counters, sizeof(host_counters), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(&rb, &box[0], sizeof(Box6), cudaMemcpyDeviceToHost, s);  // n == 1: the leaf
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return std::string("GPU BVH build: ") + cudaGetErrorString(e);
    if (host_counters[3] != 0) return "GPU BVH build: node capacity exceeded";
    if (host_counters[1] != n) return "GPU BVH build: primitive count mismatch";
    if (host_counters[0] != out.level_off.back()) return "GPU BVH build: node count mismatch";
    out.nodes = nodes;
    out.slots = slots;
    out.node_count = host_counters[0];
    out.slot_count = n;
    out.depth = depth;
    for (int k = 0; k < 3; ++k)
    {
        out.root_lo[k] = rb.lo[k];
        out.root_hi[k] = rb.hi[k];
    }
    return "";
}
} // namespace ar
