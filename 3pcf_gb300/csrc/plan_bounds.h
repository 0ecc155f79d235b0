// plan_bounds.h -- the planner's tests of tile boxes (kernels.cu, plan_rows).
//
// Two passes of the planner evaluate them, compiled apart: the first counts the
// units of a row, the second writes each to the place that the counts give it.
// One unit on which the passes differ would shift all that follow, so both must
// round alike whatever the compiler contracts around them: a product here is an
// operand of an explicit fmaf, of another product, of min and max or of a
// comparison, and never of a sum or a difference, which leaves nothing to
// contract.  (Host code as well, so that this can be tested without a device.)
#ifndef TPCF_PLAN_BOUNDS_H
#define TPCF_PLAN_BOUNDS_H

#include <math.h>
#include <cuda_runtime.h>

#include "engine.h"

namespace tpcf {

#define PLAN_FN __host__ __device__ __forceinline__

// Lower and upper bounds of the squared side between two tile boxes; the
// margins cover the rounding of the bounds and of the reference's sides.  A
// lower bound that overflows stays below an infinite limit.
PLAN_FN float2 box_bounds2(float4 al, float4 ah, float4 bl, float4 bh) {
    const float gx = fmaxf(0.f, fmaxf(al.x - bh.x, bl.x - ah.x)), ux = fmaxf(ah.x - bl.x, bh.x - al.x);
    const float gy = fmaxf(0.f, fmaxf(al.y - bh.y, bl.y - ah.y)), uy = fmaxf(ah.y - bl.y, bh.y - al.y);
    const float gz = fmaxf(0.f, fmaxf(al.z - bh.z, bl.z - ah.z)), uz = fmaxf(ah.z - bl.z, bh.z - al.z);
    const float lo2 = fmaf(gz, gz, fmaf(gy, gy, gx * gx)), up2 = fmaf(uz, uz, fmaf(uy, uy, ux * ux));
    return make_float2(fminf(lo2 * (1.0f - 4e-5f), 3.4028235e38f), fmaf(up2, 1.0f + 4e-5f, 1e-37f));
}

// Whether a tile triple can hold a counted triangle-parametrization triangle:
// with the three pair bounds sorted (L1<=L2<=L3 lower, U1<=U2<=U3 upper) the
// shortest side lies in [L1,U1], the middle in [L2,U2], the longest in
// [L3,U3]; permutations 0/2 need s_lo <= shortest < s_hi and
// middle < q_hi*shortest, permutation 1 needs s_lo <= middle < s_hi and
// longest < q_hi*middle.  All squared.
PLAN_FN bool tri_possible(float2 x, float2 y, float2 z, const PlanParams& pp) {
    const float l0 = fminf(fminf(x.x, y.x), z.x), l2 = fmaxf(fmaxf(x.x, y.x), z.x);
    const float l1 = fmaxf(fminf(x.x, y.x), fminf(fmaxf(x.x, y.x), z.x));
    const float u0 = fminf(fminf(x.y, y.y), z.y);
    const float u1 = fmaxf(fminf(x.y, y.y), fminf(fmaxf(x.y, y.y), z.y));
    return (l0 < pp.s_hi2 && u0 >= pp.s_lo2 && l1 < pp.q_hi2 * u0) ||
           (l1 < pp.s_hi2 && u1 >= pp.s_lo2 && l2 < pp.q_hi2 * u1);
}

// Rough share of the pairs of two tiles that are within r of one another.
PLAN_FN float near_share(float2 b, float r) {
    const float lo = sqrtf(b.x), hi = sqrtf(fminf(b.y, 3e38f));
    if (hi <= r) return 1.f;
    const float f = fmaxf(r - lo, 0.f) / fmaxf(hi - lo, 1e-30f);
    return f * f;
}

// est plus the work of a tile triple of na, nb and nc points: its triangles
// within reach, and what walking the points i and the j's in their reach costs
// in the same unit.
PLAN_FN float add_estimate(float est, float na, float nb, float nc, float2 ab, float2 ac, float2 bc, float r) {
    const float near = nc * near_share(ac, r);
    return fmaf(na, fmaf(nb * near_share(ab, r), fmaf(near, near_share(bc, r), 2.5f), 25.f), est);
}

}  // namespace tpcf
#endif
