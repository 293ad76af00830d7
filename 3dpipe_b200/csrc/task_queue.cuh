// task_queue.cuh -- places in a bounded queue that many warps fill.
#pragma once

namespace tdp {

// One warp's claims on a queue of `cap` entries with one 32-bit counter of what
// was asked for; the entries there are at the end are min(counter, cap).  What
// does not fit goes elsewhere, and a warp that has found the queue full asks no
// more: a kernel of w warps that claim up to n entries at a time leaves the
// counter below cap + (w + 1) n.  Counting on would wrap at 2^32 entries, which
// a LOD of large voxels or many voxel pairs reaches, and give used places anew.
struct QueueClaims {
    bool full = false;
    // the first place for the next n entries (entries at or beyond cap have none);
    // add(n) adds to the counter and returns what it was
    template <typename Add>
#ifdef __CUDACC__
    __device__ __forceinline__
#endif
    unsigned claim(unsigned n, unsigned cap, Add add) {
        if (full) return cap;
        const unsigned at = add(n);
        full = at >= cap;
        return at;
    }
};

}  // namespace tdp
