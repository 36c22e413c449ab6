// How a batch of n rays is divided among the warps of k_trace_rays: chunks of
// 2^chunk_log2 rays dealt to the warps round robin.  Host + device; n may be any
// int, so counts that round n up are formed in 64 bits.
#pragma once
#include "ar_vec.h"

namespace ar
{
struct RayShare
{
    int n, chunk_log2, warps;

    AR_HD int chunks() const { return (int)(((long long)n + (1 << chunk_log2) - 1) >> chunk_log2); }
    // rays of warp w, the last chunk counted whole
    AR_HD int limit(int w) const
    {
        const int c = chunks();
        return w < c ? ((c - w - 1) / warps + 1) << chunk_log2 : 0;
    }
    // warp w's ray number j; there is none when it is n or more
    AR_HD long long ray(int w, int j) const
    {
        return ((((long long)(j >> chunk_log2) * warps + w) << chunk_log2)) + (j & ((1 << chunk_log2) - 1));
    }
};
} // namespace ar
