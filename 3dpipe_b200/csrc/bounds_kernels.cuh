// bounds_kernels.cuh -- launchers of bounds_kernels.cu used by host code.
#pragma once
#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

#include "ctx.cuh"

namespace tdp {
// (proxy, hausdorff) of n triangle records -> out[2i], out[2i+1]
cudaError_t launch_gather_bounds(const float4* tri, size_t n, float* out, cudaStream_t s);

// Triangle records of a set of objects on the device, each LOD's in voxel order.
struct BoundRecords {
    float4* tri[kNumLods];          // 3 float4 a triangle; .w of the first two receives (proxy, hausdorff)
    const uint32_t* vtri[kNumLods]; // n_vox + 1: a voxel's first record
    size_t n_tris[kNumLods];
    const uint32_t* obj_vox;        // n_obj + 1: an object's first voxel
    long n_vox, n_obj;
    float *obj_hd, *obj_phd;        // kNumLods values an object
};
// The scratch of launch_bounds for r (TDP_OK or an error, with the message set).
int bounds_scratch(tdp_ctx* ctx, const BoundRecords& r);
void bounds_scratch_free(tdp_ctx* ctx);  // nothing queued may still use it
// Queues the bounds of every record and object of r on the context's stream,
// into the records and r.obj_hd / r.obj_phd; counters() are the work done.
cudaError_t launch_bounds(tdp_ctx* ctx, const BoundRecords& r);
const unsigned long long* bounds_counters(const tdp_ctx* ctx);
}  // namespace tdp
