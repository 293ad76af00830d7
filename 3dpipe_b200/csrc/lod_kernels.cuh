// lod_kernels.cuh -- one LOD of the tuned join as a chain of task kernels
// (csrc/lod_kernels.cu).  All state stays in device memory; no kernel needs a
// count on the host.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "common.cuh"
#include "join_kernels.cuh"

namespace tdp {

constexpr int kLodCtrWords = 8;   // counters of one pass over the items
constexpr int kMaxPasses = 10;    // up to 8 LODs, the redo pass, one spare

// A queued cluster pair of item w: z and y are its gap widened for the upper
// and the lower bound, so that a later look at the running caps can drop it
// without its clusters.
struct alignas(16) LodTask {
    uint32_t w, ij;
    float z, y;
};

// A queued triangle pair: item, triangles, gap widened for the upper bound;
// -inf where its lower bound matters too.
struct alignas(16) LodEval {
    uint32_t w, a, b;
    float z;
};

struct LodDev {
    JoinDev d;
    const float* box1;  // 6 floats per object (low, high)
    const float* box2;
    int self;      // tile 2 is tile 1: one set of cluster records
    int level;     // Hausdorff level
    int nl;        // LODs of the join
    const uint32_t* vt1[8];
    const uint32_t* vt2[8];
    const float4* tri1[8];
    const float4* tri2[8];
    int li[8];
    // items of the current pass
    RefineItem* items;
    int4* ext;     // per item: voxel pair, object pair, first A cluster, first B cluster
    int2* vox;     // per item: A voxel, B voxel
    float4* mg;    // per item: FP32 margin of its bounds, slack, preset, 1 once it is in `over`
    // caps
    unsigned long long* pbest;  // per pair: (core distance, item) of the first LOD's closest cores
    float* pcap;   // per pair: smallest upper bound so far
    float* pd;     // per pair: the last LOD's running distance
    uint8_t* pown; // per pair: 1 = caps per voxel pair (vmx) instead of pcap
    uint8_t* pmiss;  // per pair: 1 = nothing of its last LOD came below its cap: done again without it
    float4* dir;   // per pair: about the direction of its closest points (any vector, or 0)
    float* vres;   // per voxel pair: distance minimum (last LOD; levels 0 and 1)
    // cluster records of the voxels in use at the current LOD
    float4* cl1;
    float4* cl2;
    float4* vb1;   // 2 float4 per voxel: exact box of its triangles at this LOD
    float4* vb2;
    int* flag1;    // per voxel: LOD stamp of its cluster records
    int* flag2;
    int* list1;    // voxels whose records are built at this LOD
    int* list2;
    long nvox1, nvox2;
    LodTask* tasks;  // cluster pairs that survive the cull
    unsigned task_cap;
    LodEval* evals;  // triangle pairs that survive their tests
    unsigned eval_cap;
    unsigned* over;  // items whose tasks or triangle pairs did not fit
    unsigned* ctr;   // kLodCtrWords words per pass, zeroed
    unsigned* n_items;         // per LOD item counts (zeroed)
    unsigned long long* tri_pairs;
    unsigned long long* n_full;
    unsigned* n_over;  // items that found a queue full (statistic)
    int use_preset;  // last LOD of a join with within queries: no distance above the query's
    float tau;
    int num_sms;
};

// mg.w of an item beyond 1: evaluated in FP64; a triangle pair was queued
constexpr int kExactFlag = 2, kEvalFlag = 4;

// words of a pass's counters
enum LodCtr { cList1, cList2, cTasks, cOver, cWork, cWorkOver, cRedo, cEvals };

#ifdef __CUDACC__
__device__ __forceinline__ size_t cluster_base(uint32_t first_tri, int voxel) {
    // sum over earlier voxels of ceil(n / 8) <= first_tri / 8 + voxel
    return (size_t)(first_tri >> 3) + (size_t)voxel;
}

// a whole warp: the lanes' voxels that are not stamped yet join the list
__device__ __forceinline__ void lod_claim(bool want, int voxel, int stamp, int* flag, int* list, unsigned* n, int lane) {
    bool mine = false;
    if (want && __ldcg(flag + voxel) != stamp) mine = atomicExch(flag + voxel, stamp) != stamp;
    const unsigned m = __ballot_sync(0xffffffffu, mine);
    if (!m) return;
    unsigned base = 0;
    if (lane == 0) base = atomicAdd(n, (unsigned)__popc(m));
    base = __shfl_sync(0xffffffffu, base, 0);
    if (mine) list[base + __popc(m & ((1u << lane) - 1u))] = voxel;
}
#endif

// the loop's state before its first LOD, in one launch instead of seven memsets
// (n_words counters and dstats 0; caps far, seeds and stamps ~0, the rest of L 0;
// every size a multiple of 4 bytes or rounded up to one within its buffer)
cudaError_t launch_lod_init(const LodDev& L, unsigned* words, int n_words, unsigned long long* dstats, size_t caps_bytes,
                            size_t best_bytes, size_t flags_bytes, size_t zero_bytes, cudaStream_t s);
cudaError_t launch_lod_items(const LodDev& L, int k, cudaStream_t s);
// clusters, (first LOD) seeds, cull, tests and evaluation of LOD k's items
cudaError_t launch_lod_refine(const LodDev& L, int k, int highest, cudaStream_t s);
// the pairs' bounds, evictions and the within decision; at the last LOD also
// the items of the pairs that have to be done again without their caps
cudaError_t launch_lod_update(const LodDev& L, int k, int highest, int decide, cudaStream_t s);
// the last LOD again for those pairs (normally none)
cudaError_t launch_lod_redo(const LodDev& L, int k, int decide, cudaStream_t s);

// The last LOD's rules over items that the caller wrote (L has that one LOD),
// in chunks that the queues hold.  First the clusters of the voxels in use and
// the chunks' counters (kLodCtrWords words each; the claims are in the first's):
cudaError_t launch_lod_exact_begin(const LodDev& L, int64_t chunk, int n_chunks, cudaStream_t s);
// then chunk by chunk, L's item arrays and counters moved to the chunk's and V
// its items: each pair's smallest FP32 distance below its cap so far in pd,
cudaError_t launch_lod_exact(const LodDev& L, cudaStream_t s);
// and the FP64 minimum of the queued triangle pairs that can hold it, per pair
// into exact (bits); the items they belong to are counted in n_f64
cudaError_t launch_lod_f64(const LodDev& L, unsigned long long* exact, unsigned* n_f64, cudaStream_t s);
// last: items without a queued triangle pair, items with a distance below the cap
cudaError_t launch_lod_exact_count(const LodDev& L, unsigned* counts, cudaStream_t s);

}  // namespace tdp
