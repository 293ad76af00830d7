// result.h -- the join result behind the opaque tdp_result of the C ABI
// (rows sorted by query id, then result id).
#pragma once
#include <cstddef>
#include <vector>

struct tdp_result {
    std::vector<int> q, t;
    std::vector<float> d;
    std::vector<double> d64;  // exact LOD-100 distances (params.exact_distances)

    void take(const void* x64, const void* xq, const void* xt, const void* xd, size_t n, bool exact) {
        q.assign((const int*)xq, (const int*)xq + n);
        t.assign((const int*)xt, (const int*)xt + n);
        d.assign((const float*)xd, (const float*)xd + n);
        if (exact) d64.assign((const double*)x64, (const double*)x64 + n);
    }
};
