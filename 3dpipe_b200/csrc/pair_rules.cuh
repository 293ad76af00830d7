// pair_rules.cuh -- bounds shared by the join's pair kernels.
#pragma once
#include <float.h>

#include "common.cuh"
#include "join_kernels.cuh"

namespace tdp {

// The preset of a within item at the last LOD (LOD 100): its query's
// distance plus twice the largest FP32 error of a triangle pair that could
// be within it.  Such a pair's coordinates, taken from a vertex of the A
// voxel, stay below tau + both voxel extents (R), so its FP32 distance is
// below tau + err_bound(R): an item with nothing below the preset has no
// pair within tau.  kNN items get FLT_MAX (no preset).
__device__ __forceinline__ float within_preset(const JoinDev& d, int p, int a, int b, float tau_all) {
    float tau = tau_all;
    if (d.qk) {
        const int q = d.pq[p];
        if (d.qk[q] > 0) return FLT_MAX;
        tau = d.qtau[q];
    }
    const float4* va = d.vox1 + 3 * (size_t)a;
    const float4* vb = d.vox2 + 3 * (size_t)b;
    const float4 alo = va[0], ahi = va[1], blo = vb[0], bhi = vb[1];
    const float da = (ahi.x - alo.x) + (ahi.y - alo.y) + (ahi.z - alo.z);
    const float db = (bhi.x - blo.x) + (bhi.y - blo.y) + (bhi.z - blo.z);
    const float R = (tau + da + db) * 1.001f + 1.f;
    return tau + 2.f * err_bound(R) + 1e-6f;
}

// A voxel pair whose refine found nothing below its preset is out of its
// query's reach: both its bounds go to kFar, so it never lowers the pair's
// minimum, never reports it, and adds no error term.
constexpr float kFar = 3.0e38f;

}  // namespace tdp
