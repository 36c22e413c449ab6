// The choices that the eight lanes of a wide node make together when the GPU
// build collapses the binary tree (k_collapse): which child to open and which
// child takes which octant slot.  The lanes exchange their candidates pairwise, so
// all of them end with the same winner only if the candidates are totally ordered.
// Areas and costs are therefore never NaN, whatever the boxes hold (a mesh with
// an infinite vertex has infinite boxes, flat ones among them: 0 x infinity).
// Host + device.
#pragma once
#include <cfloat>

#include "ar_vec.h"

namespace ar
{
namespace lbvh
{
// Surface area of a child's box, -1 where it is not a number: such a child is not opened.
AR_HD double open_area(const float* lo, const float* hi)
{
    const double dx = fmax(0.0, (double)hi[0] - lo[0]);
    const double dy = fmax(0.0, (double)hi[1] - lo[1]);
    const double dz = fmax(0.0, (double)hi[2] - lo[2]);
    const double a = 2.0 * (dx * dy + dy * dz + dz * dx);
    return a >= 0.0 ? a : -1.0;
}

// whether child p of area o is opened rather than child `pick` of area `best`
AR_HD bool opens_before(double o, int p, double best, int pick) { return o > best || (o == best && p < pick); }

// Alignment of a child with octant slot s, off: its centre against the node's;
// the lowest value where that is not a number.
AR_HD double slot_cost(const double* off, int s)
{
    double c = 0.0;
    for (int k = 0; k < 3; ++k) c += ((s >> k) & 1) ? off[k] : -off[k];
    return c >= -DBL_MAX ? c : -DBL_MAX;
}

// whether child w with alignment o takes its slot before child `who` with bc (8 and up: no child)
AR_HD bool placed_before(double o, int w, double bc, int who)
{
    return w < 8 && (who >= 8 || o > bc || (o == bc && w < who));
}
} // namespace lbvh
} // namespace ar
