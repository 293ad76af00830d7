// prep_kernels.cu -- GPU LOD preparation (tdp_raw_from_meshes): LOD-100 meshes
// in, a RAW tile out, with every step of the preparation on the device.
//
// Replaces the reference's CGAL preparation of its tiles: progressive
// decimation into LODs (src/spatial/himesh_comp.cpp:28-190), skeleton voxels
// (src/spatial/himesh_skeleton.cpp:17-168), LOD triangles to voxels
// (src/spatial/himesh_retrieve.cpp:183-200), the per-triangle Hausdorff bounds
// (src/spatial/himesh_hausdorff.cpp:197-296, done here with the kernels of
// tdp_tile_compute_bounds) and the RAW writer (src/storage/tile_IO.cpp:79-172).
// The rule, per object with vertices P (float, evaluated in double) and
// LOD-100 facets F[0..m):
//  1. LODs 80, 60, 40, 20 by half-edge collapse, shortest edge first, keyed
//     (|P_a - P_b|^2, a, b) with a < b.  The smallest key among the candidate
//     edges is tried: a into b, else b into a, each refused unless exactly two
//     live facets hold both (third vertices w1 != w2), the common neighbours of
//     the two are exactly {w1, w2}, w1 and w2 have more than 3 neighbours each,
//     and no facet of the removed vertex turns (normal n0 -> n1:
//     |n1| >= 1e-12 (|n0| + 1e-300) and n0.n1 >= 0.3 |n0||n1|).  A refused edge
//     stops being a candidate until a collapse changes one of its ends; every
//     edge of the kept vertex becomes a candidate again after a collapse.  A LOD
//     is the live facets in index order once their count is <= floor(m l / 100)
//     (or no candidate is left).  This is the sequential priority-queue
//     decimation with versioned entries restated without the queue: the
//     candidate set is exactly the queue's set of current entries.
//  2. nseed = m / voxel_size + 1 farthest-point seeds from vertex 0, two Lloyd
//     steps (sums in vertex order), each facet to the seed nearest its
//     barycentre, a seed's core = vertex 0 of its nearest facet.
//  3. LOD-100 triangles to the voxel with the nearest core by first vertex;
//     voxels left without a LOD-100 triangle are dropped; then every LOD is
//     assigned the same way to the voxels kept, triangles keeping LOD order.
//  4. Transform = the vertex nearest the centre of the float bounding box.
// Ties go to the lowest index everywhere.  Work layout: one CTA per object.
// Decimation keeps the object's facets (16- or 32-bit vertex ids), flags, four
// vertex bitmasks and the smallest key of every 32 facets in shared memory
// (global memory for objects too large for it), every facet's smallest key and
// every vertex's facets in global memory.  Collapses only ever join two
// vertices' facets, so a vertex's live facets are those of the vertices merged
// into it, a chain of the first lists.  A round is a block argmin over the
// groups of 32, the facets around the edge (a warp for each end: links,
// neighbour masks, normals), those around the two third vertices, the change
// itself, and the groups that it touched; it costs what the neighbourhood
// costs, not the mesh.  The rounds of one object are a serial chain of FP64
// and memory latencies, which bounds it: vessels of 20,160 facets and 8,068
// rounds took 23.7 us a round with three scans over all facets, 4.2 here (6
// vessels 191 -> 34 ms, 1,000 nuclei of 1,280 facets 7.7 -> 4.6 ms).  This file
// is built with -fmad=false: every product and sum is rounded on its own, as on
// the host.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <cub/device/device_scan.cuh>

#include <algorithm>
#include <cfloat>
#include <chrono>
#include <climits>
#include <cmath>
#include <cstring>
#include <string>
#include <type_traits>
#include <vector>

#include "bounds_kernels.cuh"
#include "ctx.cuh"
#include "storage/dt_format.h"

namespace tdp {
namespace {

constexpr int kDecLods = kNumLods - 1;  // LODs made by decimation (20..80)
constexpr int kPrepThreads = 256;       // voxel and writer kernels
constexpr size_t kSmemSmall = 40 << 10;  // decimation in shared memory, 128 threads
constexpr size_t kSmemLarge = 220 << 10; // decimation in shared memory, 256 threads

struct Meshes {  // one batch on the device; object o: vertices V[3 voff[o]..), facets F[3 foff[o]..)
    const float* V;
    const int64_t* voff;
    const uint32_t* F;
    const int64_t* foff;
    int n;
};

struct VoxScratch {
    double* dmin;      // per vertex
    uint32_t* asg;     // per vertex
    double* seed;      // 3 per seed
    unsigned long long* bestd;  // per seed
    uint32_t* bestf;   // per seed
    uint32_t* core;    // per seed (kept voxels first)
    uint32_t* nvox;    // per object
    uint32_t* tvox;    // kNumLods planes of Ftot: voxel of each LOD triangle
    uint32_t* ord;     // kNumLods planes of Ftot: LOD triangles grouped by voxel
    uint32_t* vcnt;    // kNumLods planes of Stot: triangles per voxel
    uint32_t* vst;     // kNumLods planes of Stot: first grouped index per voxel
    const int64_t* soff;  // per object: first seed
    int64_t Ftot, Stot;
};

__host__ __device__ inline size_t round16(size_t x) { return (x + 15) & ~(size_t)15; }

__device__ __forceinline__ double3 vtx(const float* P, uint32_t i) {
    return make_double3((double)P[3 * (size_t)i], (double)P[3 * (size_t)i + 1], (double)P[3 * (size_t)i + 2]);
}
__device__ __forceinline__ double dist2(double3 a, double3 b) {
    const double dx = a.x - b.x, dy = a.y - b.y, dz = a.z - b.z;
    return dx * dx + dy * dy + dz * dz;
}
__device__ __forceinline__ double3 sub3(double3 a, double3 b) { return make_double3(a.x - b.x, a.y - b.y, a.z - b.z); }
__device__ __forceinline__ double dot3(double3 a, double3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ double3 cross3(double3 a, double3 b) {
    return make_double3(a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x);
}

// true when moving corner u of facet (x, y, z) (corners p0, p1, p2) to point q turns it
__device__ bool turns(uint32_t x, uint32_t y, double3 p0, double3 p1, double3 p2, uint32_t u, double3 q) {
    const bool at0 = x == u, at1 = !at0 && y == u;
    const double3 q0 = at0 ? q : p0, q1 = at1 ? q : p1, q2 = at0 || at1 ? p2 : q;
    const double3 n0 = cross3(sub3(p1, p0), sub3(p2, p0)), n1 = cross3(sub3(q1, q0), sub3(q2, q0));
    const double a0 = sqrt(dot3(n0, n0)), a1 = sqrt(dot3(n1, n1));
    return a1 < 1e-12 * (a0 + 1e-300) || dot3(n0, n1) < 0.3 * a0 * a1;
}

__device__ __forceinline__ void mark(uint32_t* M, uint32_t x, uint32_t y, uint32_t z, uint32_t c) {
    if (x != c) atomicOr(M + (x >> 5), 1u << (x & 31));
    if (y != c) atomicOr(M + (y >> 5), 1u << (y & 31));
    if (z != c) atomicOr(M + (z >> 5), 1u << (z & 31));
}

// An edge's key: the bits of |P_a - P_b|^2 (lengths are not negative, so the
// bits order like the values, without the latency of FP64 compares), then
// a << 32 | b (a < b).
struct alignas(16) Key {
    uint64_t l, ab;
};
constexpr uint64_t kNoLength = 0x7ff0000000000000ull;  // +inf: no candidate
__device__ __forceinline__ bool key_less(const Key& x, const Key& y) { return x.l != y.l ? x.l < y.l : x.ab < y.ab; }
__device__ __forceinline__ Key no_key() { return Key{kNoLength, ~0ull}; }
// the warp's least key: a word at a time among the lanes that still tie
__device__ __forceinline__ Key warp_least(Key k) {
    const uint32_t word[4] = {(uint32_t)(k.l >> 32), (uint32_t)k.l, (uint32_t)(k.ab >> 32), (uint32_t)k.ab};
    unsigned tie = 0xffffffffu;
#pragma unroll
    for (int w = 0; w < 4; ++w) {
        const bool in = (tie >> (threadIdx.x & 31)) & 1u;
        const uint32_t least = __reduce_min_sync(0xffffffffu, in ? word[w] : UINT_MAX);
        tie = __ballot_sync(0xffffffffu, in && word[w] == least);
        if (!(tie & (tie - 1))) break;
    }
    const int src = __ffs(tie) - 1;
    return Key{__shfl_sync(0xffffffffu, k.l, src), __shfl_sync(0xffffffffu, k.ab, src)};
}

// smallest key over the candidate edges of facet (x, y, z) with corners p, q, r
// and flags fla
__device__ __forceinline__ Key facet_key(double3 p, double3 q, double3 r, uint32_t x, uint32_t y, uint32_t z,
                                         uint32_t fla) {
    const uint32_t t[3] = {x, y, z};
    const double len[3] = {dist2(p, q), dist2(q, r), dist2(r, p)};
    Key k = no_key();
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        const uint32_t c = t[j], d = t[j == 2 ? 0 : j + 1];
        const Key e{(uint64_t)__double_as_longlong(len[j]), (uint64_t)min(c, d) << 32 | max(c, d)};
        if (!(fla & (2u << j)) && key_less(e, k)) k = e;
    }
    return k;
}

constexpr int kGroup = 32;     // facets whose smallest key is kept
constexpr int kTouched = 128;  // touched groups listed a round (more: all are redone)
// A chain is rewritten without its dead facets once, past its first rows of 32, it
// holds more than twice its live ones.  A tube whose short edges are all at one
// end merges thousands of vertices into one: 1,720 ms for 18,000 facets where every
// round went through all that its chain had ever held, 42 with this (123 with
// scans over all facets); a flat sheet of 20,000: 232, 78 (286).
constexpr int kFewRows = 2;

// bytes of an object's own storage: facets, flags, 4 masks, merge chains, group
// keys
__host__ __device__ inline size_t dec_bytes(int64_t n, int64_t m, size_t vi) {
    const size_t g = ((size_t)m + kGroup - 1) / kGroup;
    return round16(3 * (size_t)m * vi) + round16((size_t)m) + round16(16 * (size_t)((n + 31) / 32)) +
           2 * round16((size_t)n * vi) + sizeof(Key) * g;
}

// Per batch in global memory: every facet's smallest key, every vertex's facets
// (vertex v's are csr[lists[v].x .. lists[v].y), with room up to lists[v + 1].x:
// lists has one entry more per object).
struct DecLists {
    Key* keys;
    uint32_t* csr;
    uint2* lists;
};

// ------------------------------------------------------------------ validation
// first object (lowest index) without vertices or facets, with a vertex index
// out of range, a facet repeating a vertex, or a non-finite coordinate
__global__ void k_validate(Meshes M, int* first_bad) {
    for (int o = blockIdx.x; o < M.n; o += gridDim.x) {
        const int64_t v0 = M.voff[o], v1 = M.voff[o + 1], f0 = M.foff[o], f1 = M.foff[o + 1];
        bool bad = v1 <= v0 || f1 <= f0 || v1 - v0 > 0xffffffffLL;
        const uint64_t n = (uint64_t)(v1 - v0);
        for (int64_t f = f0 + threadIdx.x; !bad && f < f1; f += blockDim.x) {
            const uint32_t a = M.F[3 * f], b = M.F[3 * f + 1], c = M.F[3 * f + 2];
            bad = a >= n || b >= n || c >= n || a == b || b == c || a == c;
        }
        for (int64_t i = 3 * v0 + threadIdx.x; !bad && i < 3 * v1; i += blockDim.x) bad = !isfinite(M.V[i]);
        if (__syncthreads_or(bad) && threadIdx.x == 0) atomicMin(first_bad, o);
    }
}

// ------------------------------------------------------------------ block helpers
template <int T>
__device__ __forceinline__ uint32_t block_count_before(bool flag, uint32_t* red, uint32_t& total) {
    constexpr int NW = T / 32;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const unsigned bal = __ballot_sync(0xffffffffu, flag);
    if (lane == 0) red[wid] = __popc(bal);
    __syncthreads();
    uint32_t before = 0;
    total = 0;
    for (int w = 0; w < NW; ++w) {
        const uint32_t x = red[w];
        total += x;
        if (w < wid) before += x;
    }
    __syncthreads();
    return before + __popc(bal & ((1u << lane) - 1u));
}

// exclusive scan of x over the block's threads (in thread order)
template <int T>
__device__ __forceinline__ uint32_t block_excl_sum(uint32_t x, uint32_t* red, uint32_t& total) {
    constexpr int NW = T / 32;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    uint32_t incl = x;
#pragma unroll
    for (int s = 1; s < 32; s <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, s);
        if (lane >= s) incl += y;
    }
    if (lane == 31) red[wid] = incl;
    __syncthreads();
    uint32_t before = 0;
    total = 0;
    for (int w = 0; w < NW; ++w) {
        const uint32_t y = red[w];
        total += y;
        if (w < wid) before += y;
    }
    __syncthreads();
    return before + incl - x;
}

// ------------------------------------------------------------------ decimation
// The live facets of vertex x, 32 at a time, one a lane: fn(facet, valid) is
// called by the whole warp (where it returns a bool, until that is false).  The
// chain of vertices merged into x is followed 32 at a time, their lists taken as
// one row.  Returns the rows' number; `last` is the lane's facet in the last one
// (UINT_MAX: none).
template <typename VI, typename Fn>
__device__ __forceinline__ int each_facet(uint32_t x, const VI* next, const uint2* lists, const uint32_t* csr,
                                          const uint8_t* fl, int lane, uint32_t& last, Fn fn) {
    constexpr uint32_t kEnd = (uint32_t)(VI)~0u;
    uint32_t s = x;
    int rows = 0;
    while (s != kEnd) {
        uint32_t mine = kEnd;
        int k = 0;
        for (; k < 32 && s != kEnd; ++k) {
            if (lane == k) mine = s;
            s = next[s];
        }
        const uint2 at_to = lane < k ? lists[mine] : make_uint2(0u, 0u);
        const uint32_t b = at_to.x, c = at_to.y - b;
        uint32_t end = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            if (o >= k) break;
            const uint32_t y = __shfl_up_sync(0xffffffffu, end, o);
            if (lane >= o) end += y;
        }
        const uint32_t total = __shfl_sync(0xffffffffu, end, k - 1);
        for (uint32_t e0 = 0; e0 < total; e0 += 32) {
            const uint32_t at = min(e0 + lane, total - 1);
            int src = 0;  // the first list that ends after `at`
            if (k > 1) {
#pragma unroll
                for (int step = 16; step > 0; step >>= 1)
                    if (__shfl_sync(0xffffffffu, end, src + step - 1) <= at && src + step < k) src += step;
            }
            const uint32_t lb = __shfl_sync(0xffffffffu, b, src), lc = __shfl_sync(0xffffffffu, c, src),
                           le = __shfl_sync(0xffffffffu, end, src);
            const uint32_t f = csr[lb + (at - (le - lc))];
            const bool on = e0 + lane < total && (fl[f] & 1);
            last = on ? f : UINT_MAX;
            ++rows;
            if constexpr (std::is_void<decltype(fn(f, on))>::value) fn(f, on);
            else if (!fn(f, on)) return rows;
        }
    }
    return rows;
}

// The live facets of x to the front of its chain, in the same order, and what is
// left of the chain dropped; a vertex's list has the room it had in the mesh.
// (Up to any place in the chain no more are written than were read before it.)
template <typename VI>
__device__ __noinline__ void compact_facets(uint32_t x, VI* next, VI* tail, uint2* lists, uint32_t* csr, const uint8_t* fl,
                                            int lane) {
    uint32_t w = x, at = lists[x].x, unused;  // where the next one goes, the same on every lane
    each_facet<VI>(x, next, lists, csr, fl, lane, unused, [&](uint32_t f, bool on) {
        const unsigned live = __ballot_sync(0xffffffffu, on);
        const uint32_t rank = __popc(live & ((1u << lane) - 1u)), n = __popc(live);
        for (uint32_t done = 0; done < n;) {
            const uint32_t room = lists[w + 1].x - at, take = min(room, n - done);
            if (on && rank >= done && rank < done + take) csr[at + (rank - done)] = f;
            at += take;
            done += take;
            if (done < n) {  // that list is full
                __syncwarp();
                if (lane == 0) lists[w].y = at;
                w = next[w];
                at = lists[w].x;
            }
        }
        __syncwarp();
    });
    if (lane == 0) {
        lists[w].y = at;
        next[w] = (VI)~0u;
        tail[x] = (VI)w;
    }
    __syncwarp();
}

template <typename VI, int T>
__global__ void __launch_bounds__(T) k_decimate(Meshes M, const int* __restrict__ objs, int n_objs, DecLists D,
                                                uint8_t* gstore, const int64_t* __restrict__ gstore_off,
                                                uint32_t* __restrict__ lodF, int64_t Ftot, uint32_t* __restrict__ lodCnt) {
    constexpr int NW = T / 32;
    static_assert(NW >= 4, "a round uses four warps beside each other");
    extern __shared__ __align__(16) uint8_t dsm[];
    __shared__ Key s_key[NW];
    __shared__ uint32_t s_red[NW], s_third[2], s_cnt[3], s_list[kTouched];
    __shared__ int s_nsh, s_turn[2], s_alive, s_ng, s_long;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    for (int i = blockIdx.x; i < n_objs; i += gridDim.x) {
        const int o = objs[i];
        const int64_t v0 = M.voff[o], f0 = M.foff[o];
        const uint32_t n = (uint32_t)(M.voff[o + 1] - v0), m = (uint32_t)(M.foff[o + 1] - f0);
        const float* P = M.V + 3 * v0;
        uint8_t* base = gstore ? gstore + gstore_off[i] : dsm;
        const uint32_t W = (n + 31) / 32, G = (m + kGroup - 1) / kGroup;
        VI* fv = reinterpret_cast<VI*>(base);
        uint8_t* fl = base + round16(3 * (size_t)m * sizeof(VI));
        uint32_t* Mu = reinterpret_cast<uint32_t*>(fl + round16(m));
        uint32_t *Mv = Mu + W, *M1 = Mu + 2 * W, *M2 = Mu + 3 * W;
        VI* next = reinterpret_cast<VI*>(reinterpret_cast<uint8_t*>(Mu) + round16(16 * (size_t)W));
        VI* tail = reinterpret_cast<VI*>(reinterpret_cast<uint8_t*>(next) + round16((size_t)n * sizeof(VI)));
        Key* gk = reinterpret_cast<Key*>(reinterpret_cast<uint8_t*>(tail) + round16((size_t)n * sizeof(VI)));
        Key* keys = D.keys + f0;
        uint32_t* csr = D.csr + 3 * f0;
        uint2* lists = D.lists + v0 + o;
        for (uint32_t f = tid; f < m; f += T) {
            uint32_t t[3];
            for (int k = 0; k < 3; ++k) {
                t[k] = M.F[3 * (f0 + f) + k];
                fv[3 * f + k] = (VI)t[k];
            }
            fl[f] = 1;  // bit 0 live, bit 1 + j: edge (j, j + 1) refused
            keys[f] = facet_key(vtx(P, t[0]), vtx(P, t[1]), vtx(P, t[2]), t[0], t[1], t[2], 1);
        }
        for (uint32_t w = tid; w < 4 * W; w += T) Mu[w] = 0;
        for (uint32_t v = tid; v < n; v += T) {
            next[v] = (VI)~0u;
            tail[v] = (VI)v;
            lists[v].y = 0;
        }
        if (tid == 0) {
            s_alive = (int)m;
            s_nsh = s_turn[0] = s_turn[1] = s_ng = s_long = 0;
        }
        __syncthreads();
        // every vertex's facets
        for (uint32_t c = tid; c < 3 * m; c += T) atomicAdd(&lists[fv[c]].y, 1u);
        __syncthreads();
        uint32_t run = 0;
        for (uint32_t c0 = 0; c0 < n; c0 += T) {
            const uint32_t v = c0 + tid, x = v < n ? lists[v].y : 0u;
            uint32_t total;
            const uint32_t at = run + block_excl_sum<T>(x, s_red, total);
            if (v < n) {
                lists[v] = make_uint2(at, at);
            }
            run += total;
        }
        if (tid == 0) lists[n] = make_uint2(run, run);
        __syncthreads();
        for (uint32_t c = tid; c < 3 * m; c += T) csr[atomicAdd(&lists[fv[c]].y, 1u)] = c / 3;
        auto redo_group = [&](uint32_t g) {
            const uint32_t f = g * kGroup + lane;
            const Key k = warp_least(f < m ? keys[f] : no_key());
            if (lane == 0) gk[g] = k;
        };
        for (uint32_t g = wid; g < G; g += NW) redo_group(g);
        __syncthreads();
        // the whole warp: the groups of its changed facets f to the list, each once
        auto touched = [&](uint32_t f, bool changed) {
            const uint32_t g = changed ? f / kGroup : UINT_MAX - lane;
            const unsigned same = __match_any_sync(0xffffffffu, g);
            const bool first = changed && lane == __ffs(same) - 1;
            const unsigned all = __ballot_sync(0xffffffffu, first);
            if (!all) return;
            int at = 0;
            if (lane == 0) at = atomicAdd(&s_ng, __popc(all));
            at = __shfl_sync(0xffffffffu, at, 0) + __popc(all & ((1u << lane) - 1u));
            if (first && at < kTouched) s_list[at] = g;
        };
        int li = kDecLods - 1;
        auto target_of = [&](int l) { return (uint32_t)((uint64_t)m * (uint64_t)(20 * (l + 1)) / 100); };  // LOD 20 (l + 1)
        uint32_t target = target_of(li);
        while (li >= 0) {
            bool snap = (uint32_t)s_alive <= target;
            uint32_t u = 0, v = 0;
            if (!snap) {
                Key k = no_key();
                for (uint32_t g = tid; g < G; g += 4 * T) {  // the loads of four at a time beside each other
                    Key x[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) x[j] = g + j * T < G ? gk[g + j * T] : no_key();
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        if (key_less(x[j], k)) k = x[j];
                }
                k = warp_least(k);
                if (lane == 0) s_key[wid] = k;
                __syncthreads();
                k = warp_least(lane < NW ? s_key[lane] : no_key());
                snap = k.l >= kNoLength;  // no candidate edge left
                u = (uint32_t)(k.ab >> 32);
                v = (uint32_t)k.ab;
            }
            if (snap) {  // LOD li: the live facets in index order
                __syncthreads();
                uint32_t pos = 0;
                uint32_t* out = lodF + (size_t)li * 3 * Ftot + 3 * f0;
                for (uint32_t c = 0; c < m; c += T) {
                    const uint32_t f = c + tid;
                    const bool al = f < m && (fl[f] & 1);
                    uint32_t total;
                    const uint32_t at = pos + block_count_before<T>(al, s_red, total);
                    if (al)
                        for (int k = 0; k < 3; ++k) out[3 * (size_t)at + k] = fv[3 * f + k];
                    pos += total;
                }
                if (tid == 0) lodCnt[(size_t)o * kDecLods + li] = pos;
                target = target_of(--li);
                continue;
            }
            // the facets around u (warp 0) and v (warp 1): shared ones, neighbours
            const uint32_t own = wid ? v : u, other = wid ? u : v;  // of warps 0 and 1
            uint32_t row = UINT_MAX;  // the lane's facet around its warp's end of the edge
            int rows = 0, nsh = 0;
            if (wid < 2) {
                uint32_t* mask = wid ? Mv : Mu;
                rows = each_facet<VI>(own, next, lists, csr, fl, lane, row, [&](uint32_t f, bool on) {
                    uint32_t a = 0, b = 0, c = 0;
                    if (on) {
                        a = fv[3 * f];
                        b = fv[3 * f + 1];
                        c = fv[3 * f + 2];
                        mark(mask, a, b, c, own);
                    }
                    if (wid) return;
                    const bool both = on && (a == v || b == v || c == v);
                    const unsigned sh = __ballot_sync(0xffffffffu, both);
                    const int at = nsh + __popc(sh & ((1u << lane) - 1u));
                    if (both && at < 2) s_third[at] = (a != u && a != v) ? a : (b != u && b != v) ? b : c;
                    nsh += __popc(sh);
                });
                if (tid == 0) s_nsh = nsh;
                if (rows > kFewRows) {
                    int live = 0;
                    uint32_t unused;
                    each_facet<VI>(own, next, lists, csr, fl, lane, unused, [&](uint32_t, bool on) {
                        live += __popc(__ballot_sync(0xffffffffu, on));
                    });
                    if (lane == 0 && 32 * (rows - kFewRows) > 2 * live) atomicOr(&s_long, 1 << wid);
                }
            }
            __syncthreads();
            const bool cand = s_nsh == 2 && s_third[0] != s_third[1];
            // A facet around the edge with its corners' points: kept from the normals
            // to the change where the row is one.
            struct Facet {
                uint32_t f, a, b, c;
                double3 p, q, r;
            };
            Facet held;
            auto load = [&](uint32_t f) {
                const uint32_t a = fv[3 * f], b = fv[3 * f + 1], c = fv[3 * f + 2];
                return Facet{f, a, b, c, vtx(P, a), vtx(P, b), vtx(P, c)};
            };
            auto around = [&](auto fn) {  // fn(facet, on) by the whole warp
                uint32_t unused;
                if (rows == 1) fn(held, row != UINT_MAX);
                else
                    each_facet<VI>(own, next, lists, csr, fl, lane, unused, [&](uint32_t f, bool on) {
                        Facet t{};
                        if (on) t = load(f);
                        fn(t, on);
                    });
            };
            double3 to = make_double3(0.0, 0.0, 0.0);  // the other end
            if (wid < 2) {
                to = vtx(P, other);
                if (rows == 1 && row != UINT_MAX) held = load(row);
            }
            if (cand) {
                if (wid < 2) {  // does a facet turn when its end moves to the other?
                    bool turn = false;
                    around([&](const Facet& t, bool on) {
                        if (on && t.a != other && t.b != other && t.c != other && turns(t.a, t.b, t.p, t.q, t.r, own, to)) turn = true;
                    });
                    if (turn) s_turn[wid] = 1;
                } else if (wid < 4) {  // neighbours of the two third vertices
                    const uint32_t x = s_third[wid - 2];
                    uint32_t* mask = wid == 2 ? M1 : M2;
                    uint32_t cnt = 0, all = 0, unused;
                    auto add = [&](uint32_t a) {
                        if (a != x && !(atomicOr(mask + (a >> 5), 1u << (a & 31)) & (1u << (a & 31)))) ++cnt;
                    };
                    // (more than three is all that is asked: the apex of a fan of 10,000
                    // facets, the third vertex of every edge around it, is not gone round)
                    each_facet<VI>(x, next, lists, csr, fl, lane, unused, [&](uint32_t f, bool on) {
                        if (on) {
                            add(fv[3 * f]);
                            add(fv[3 * f + 1]);
                            add(fv[3 * f + 2]);
                        }
                        all = __reduce_add_sync(0xffffffffu, cnt);
                        return all <= 3;
                    });
                    if (lane == 0) s_cnt[wid - 2] = all;
                }
                if (wid == (NW > 4 ? 4 : 3)) {  // neighbours that u and v share
                    uint32_t cnt = 0;
                    for (uint32_t w = lane; w < W; w += 32) cnt += __popc(Mu[w] & Mv[w]);
                    cnt = __reduce_add_sync(0xffffffffu, cnt);
                    if (lane == 0) s_cnt[2] = cnt;
                }
            }
            __syncthreads();
            const bool link = cand && s_cnt[2] == 2 && s_cnt[0] > 3 && s_cnt[1] > 3;
            // collapse r into k, or refuse the edge
            const bool uv = link && !s_turn[0], vu = link && !uv && !s_turn[1], go = uv || vu;
            const uint32_t r = uv ? u : v, k = uv ? v : u;
            if (go && wid < 2) {
                const bool moves = own == r;  // this warp's end goes to the other
                around([&](const Facet& t, bool on) {
                    const bool both = on && (t.a == other || t.b == other || t.c == other);
                    const bool dies = both && moves, stays = on && !both;  // (a shared one is in both rows)
                    if (dies) {
                        fl[t.f] = 0;
                        keys[t.f] = no_key();
                    }
                    if (stays) {
                        const uint32_t a = t.a == r ? k : t.a, b = t.b == r ? k : t.b, c = t.c == r ? k : t.c;
                        if (moves) {
                            VI* w = fv + 3 * t.f;
                            w[0] = (VI)a;
                            w[1] = (VI)b;
                            w[2] = (VI)c;
                        }
                        uint32_t nf = fl[t.f];  // every edge at k is a candidate again
                        if (a == k || b == k) nf &= ~2u;
                        if (b == k || c == k) nf &= ~4u;
                        if (c == k || a == k) nf &= ~8u;
                        fl[t.f] = (uint8_t)nf;
                        keys[t.f] = facet_key(t.a == r ? to : t.p, t.b == r ? to : t.q, t.c == r ? to : t.r, a, b, c, nf);
                    }
                    const unsigned dead = __ballot_sync(0xffffffffu, dies);
                    if (dead && lane == 0) atomicSub(&s_alive, __popc(dead));
                    touched(t.f, dies || stays);
                });
            } else if (!go && wid == 0) {
                around([&](const Facet& t, bool on) {
                    const bool both = on && (t.a == v || t.b == v || t.c == v);
                    if (both) {
                        uint32_t nf = fl[t.f];
                        if ((t.a == u && t.b == v) || (t.a == v && t.b == u)) nf |= 2u;
                        if ((t.b == u && t.c == v) || (t.b == v && t.c == u)) nf |= 4u;
                        if ((t.c == u && t.a == v) || (t.c == v && t.a == u)) nf |= 8u;
                        fl[t.f] = (uint8_t)nf;
                        keys[t.f] = facet_key(t.p, t.q, t.r, t.a, t.b, t.c, nf);
                    }
                    touched(t.f, both);
                });
            } else {
                for (uint32_t w = tid - 64; w < 4 * W; w += T - 64) Mu[w] = 0;
            }
            __syncthreads();
            // the touched groups; k's chain goes on with r's
            const int ng = s_ng, is_long = s_long;
            if (ng <= kTouched)
                for (int q = wid; q < ng; q += NW) redo_group(s_list[q]);
            else
                for (uint32_t g = wid; g < G; g += NW) redo_group(g);
            if (tid == 0 && go) {
                next[tail[k]] = (VI)r;
                tail[k] = tail[r];
            }
            if (is_long && wid < 2) {  // (both chains are one where the edge went)
                __syncwarp();
                if (go ? wid == 0 : is_long >> wid & 1) compact_facets<VI>(go ? k : own, next, tail, lists, csr, fl, lane);
            }
            __syncthreads();
            if (tid == 0) s_turn[0] = s_turn[1] = s_ng = s_long = 0;  // read again after the next barrier
        }
        __syncthreads();  // the next object reuses the storage
    }
}

// nearest of the points c[0..k) (double triples) to p; ties to the lowest index
__device__ __forceinline__ uint32_t nearest(double3 p, const double* c, uint32_t k, double& best) {
    uint32_t g = 0;
    best = INFINITY;
    for (uint32_t s = 0; s < k; ++s) {
        const double d = dist2(p, make_double3(c[3 * s], c[3 * s + 1], c[3 * s + 2]));
        if (d < best) { best = d; g = s; }
    }
    return g;
}

// nearest core (vertex ids) to p; ties to the lowest voxel
__device__ __forceinline__ uint32_t nearest_core(double3 p, const float* P, const uint32_t* core, uint32_t k) {
    uint32_t g = 0;
    double best = INFINITY;
    for (uint32_t s = 0; s < k; ++s) {
        const double d = dist2(p, vtx(P, core[s]));
        if (d < best) { best = d; g = s; }
    }
    return g;
}

// ------------------------------------------------------------------ voxels
// A cluster of C blocks per object (1 for many objects, so that the chip is
// full either way): the FP64 nearest-seed and nearest-core searches, which bound
// it, are spread over all its threads, the small prefix sums are its first
// block's.  6 vessels of 20,160 facets: 14.1 ms with one block of 256 threads
// each, 8.9 with 1,024, 3.3 with eight blocks of 1,024.
template <int T>
__global__ void __launch_bounds__(T) k_voxels(Meshes M, int voxel_size, const uint32_t* __restrict__ lodF,
                                              const uint32_t* __restrict__ lodCnt, VoxScratch S,
                                              unsigned long long* __restrict__ obj_bytes) {
    constexpr int NW = T / 32;
    __shared__ double s_v[NW];
    __shared__ uint32_t s_i[NW], s_red[NW];
    __shared__ double best_v[2];    // the block's farthest vertex, by the round's parity
    __shared__ uint32_t best_i[2];
    const cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
    const int C = (int)cl.num_blocks(), rank = (int)cl.block_rank();
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const uint32_t tid = rank * T + threadIdx.x, TT = C * T;  // within the cluster
    auto sync = [&] {
        if (C == 1) __syncthreads();
        else cl.sync();
    };
    for (int o = blockIdx.x / C; o < M.n; o += gridDim.x / C) {
        const int64_t v0 = M.voff[o], f0 = M.foff[o], s0 = S.soff[o];
        const uint32_t n = (uint32_t)(M.voff[o + 1] - v0), m = (uint32_t)(M.foff[o + 1] - f0);
        const uint32_t ns = m / (uint32_t)voxel_size + 1;
        const float* P = M.V + 3 * v0;
        const uint32_t* F100 = M.F + 3 * f0;
        double* sd = S.seed + 3 * s0;
        double* dmin = S.dmin + v0;
        uint32_t* asg = S.asg + v0;
        volatile uint32_t* nvox_at = S.nvox + o;
        // 2a. farthest-point seeds from vertex 0
        uint32_t cur = 0;
        for (uint32_t s = 0; s < ns; ++s) {
            const double3 c = vtx(P, cur);
            if (tid == 0) { sd[3 * s] = c.x; sd[3 * s + 1] = c.y; sd[3 * s + 2] = c.z; }
            double bv = -1.0;
            uint32_t bi = UINT_MAX;
            auto better = [&](double v2, uint32_t i2) {
                if (v2 > bv || (v2 == bv && i2 < bi)) { bv = v2; bi = i2; }
            };
            for (uint32_t i = tid; i < n; i += TT) {
                const double d = sqrt(dist2(vtx(P, i), c));
                const double dm = s == 0 ? d : fmin(dmin[i], d);
                dmin[i] = dm;
                if (dm > bv) { bv = dm; bi = i; }
            }
#pragma unroll
            for (int k = 16; k > 0; k >>= 1)
                better(__shfl_xor_sync(0xffffffffu, bv, k), __shfl_xor_sync(0xffffffffu, bi, k));
            if (lane == 0) { s_v[wid] = bv; s_i[wid] = bi; }
            __syncthreads();
            if (wid == 0) {
                bv = lane < NW ? s_v[lane] : -1.0;
                bi = lane < NW ? s_i[lane] : UINT_MAX;
#pragma unroll
                for (int k = 16; k > 0; k >>= 1)
                    better(__shfl_xor_sync(0xffffffffu, bv, k), __shfl_xor_sync(0xffffffffu, bi, k));
                if (lane == 0) { best_v[s & 1] = bv; best_i[s & 1] = bi; }
            }
            sync();  // (the other parity's values are read until the next round's)
            bv = best_v[s & 1];
            bi = best_i[s & 1];
            for (int k = 0; k < C; ++k)
                if (k != rank) better(*cl.map_shared_rank(&best_v[s & 1], k), *cl.map_shared_rank(&best_i[s & 1], k));
            cur = bi;
        }
        sync();
        // 2b. two Lloyd steps
        for (int it = 0; it < 2; ++it) {
            for (uint32_t i = tid; i < n; i += TT) {
                double d;
                asg[i] = nearest(vtx(P, i), sd, ns, d);
            }
            sync();
            for (uint32_t s = tid; s < ns; s += TT) {  // sums in vertex order
                double ax = 0.0, ay = 0.0, az = 0.0;
                uint32_t cnt = 0;
                for (uint32_t i = 0; i < n; ++i)
                    if (asg[i] == s) {
                        const double3 p = vtx(P, i);
                        ax = ax + p.x; ay = ay + p.y; az = az + p.z;
                        ++cnt;
                    }
                if (cnt) {
                    const double r = 1.0 / (double)cnt;
                    sd[3 * s] = ax * r; sd[3 * s + 1] = ay * r; sd[3 * s + 2] = az * r;
                }
            }
            sync();
        }
        // 2c. facets to seeds by barycentre; a seed's nearest facet gives its core
        unsigned long long* bestd = S.bestd + s0;
        uint32_t* bestf = S.bestf + s0;
        for (uint32_t s = tid; s < ns; s += TT) { bestd[s] = ~0ull; bestf[s] = UINT_MAX; }
        sync();
        for (int pass = 0; pass < 2; ++pass) {
            for (uint32_t f = tid; f < m; f += TT) {
                const double3 a = vtx(P, F100[3 * f]), b = vtx(P, F100[3 * f + 1]), c = vtx(P, F100[3 * f + 2]);
                const double k3 = 1.0 / 3.0;
                const double3 q = make_double3(((a.x + b.x) + c.x) * k3, ((a.y + b.y) + c.y) * k3, ((a.z + b.z) + c.z) * k3);
                double d;
                const uint32_t g = nearest(q, sd, ns, d);
                const unsigned long long bits = (unsigned long long)__double_as_longlong(d);
                if (pass == 0) atomicMin(bestd + g, bits);
                else if (bestd[g] == bits) atomicMin(bestf + g, f);
            }
            sync();
        }
        uint32_t* core = S.core + s0;
        uint32_t* cnt100 = S.vcnt + (size_t)(kNumLods - 1) * S.Stot + s0;
        if (rank == 0) {
            uint32_t found = 0;
            for (uint32_t c0 = 0; c0 < ns; c0 += T) {  // cores of the seeds with a facet, in seed order
                const uint32_t s = c0 + threadIdx.x;
                const bool has = s < ns && bestf[s] != UINT_MAX;
                const uint32_t fb = has ? bestf[s] : 0;
                uint32_t total;
                const uint32_t at = block_count_before<T>(has, s_red, total);
                if (has) core[found + at] = F100[3 * fb];
                found += total;
            }
            for (uint32_t v = threadIdx.x; v < found; v += T) cnt100[v] = 0;
            if (threadIdx.x == 0) *nvox_at = found;
        }
        sync();
        // 3. LOD-100 triangles to cores; keep the cores that receive one
        uint32_t nvox = *nvox_at;
        for (uint32_t f = tid; f < m; f += TT) atomicAdd(cnt100 + nearest_core(vtx(P, F100[3 * f]), P, core, nvox), 1u);
        sync();
        if (rank == 0) {
            uint32_t kept = 0;
            for (uint32_t c0 = 0; c0 < nvox; c0 += T) {  // in place: kept cores move down
                const uint32_t v = c0 + threadIdx.x;
                const bool has = v < nvox && cnt100[v] > 0;
                const uint32_t cv = has ? core[v] : 0;
                uint32_t total;
                const uint32_t at = block_count_before<T>(has, s_red, total);
                if (has) core[kept + at] = cv;
                kept += total;
                __syncthreads();
            }
            if (threadIdx.x == 0) *nvox_at = kept;
        }
        sync();
        nvox = *nvox_at;
        // every LOD: triangles to the kept voxels, grouped by voxel in LOD order
        uint32_t ntri = 0;
        for (int l = 0; l < kNumLods; ++l) {
            const uint32_t* LF = l < kNumLods - 1 ? lodF + (size_t)l * 3 * S.Ftot + 3 * f0 : F100;
            const uint32_t cl_n = l < kNumLods - 1 ? lodCnt[(size_t)o * kDecLods + l] : m;
            uint32_t* tv = S.tvox + (size_t)l * S.Ftot + f0;
            uint32_t* od = S.ord + (size_t)l * S.Ftot + f0;
            uint32_t* vc = S.vcnt + (size_t)l * S.Stot + s0;
            uint32_t* vs = S.vst + (size_t)l * S.Stot + s0;
            for (uint32_t v = tid; v < nvox; v += TT) vc[v] = 0;
            sync();
            for (uint32_t t = tid; t < cl_n; t += TT) {
                const uint32_t g = nearest_core(vtx(P, LF[3 * t]), P, core, nvox);
                tv[t] = g;
                atomicAdd(vc + g, 1u);
            }
            sync();
            if (rank == 0) {
                uint32_t run = 0;
                for (uint32_t c0 = 0; c0 < nvox; c0 += T) {
                    const uint32_t v = c0 + threadIdx.x;
                    const uint32_t x = v < nvox ? vc[v] : 0;
                    uint32_t total;
                    const uint32_t at = block_excl_sum<T>(x, s_red, total);
                    if (v < nvox) vs[v] = run + at;
                    run += total;
                }
            }
            sync();
            for (uint32_t v = tid >> 5; v < nvox; v += TT >> 5) {  // stable: a warp per voxel walks the LOD in order
                uint32_t c = vs[v];
                for (uint32_t t0 = 0; t0 < cl_n; t0 += 32) {
                    const bool mine = t0 + lane < cl_n && tv[t0 + lane] == v;
                    const unsigned ms = __ballot_sync(0xffffffffu, mine);
                    if (mine) od[c + __popc(ms & ((1u << lane) - 1u))] = t0 + lane;
                    c += __popc(ms);
                }
            }
            ntri += cl_n;
        }
        if (tid == 0) obj_bytes[o] = 68ull + 44ull * ntri + 116ull * nvox;
        sync();
    }
}

// ------------------------------------------------------------------ records
// The batch's triangle records for the bound preparation, as a resident tile of
// its RAW bytes would hold them: block (o, l) places LOD l of object o, grouped
// by voxel, from record t0[l][o] on.  (Through the host, that tile took 30 of
// the 48 ms of bounds of 1,000 nuclei: 169 MB down, parsed, up and unpacked.)
struct RecordsDev {
    float4* tri[kNumLods];
    uint32_t* vtri[kNumLods];
    const uint32_t* t0[kNumLods];  // n + 1: an object's first record at the LOD
    const uint32_t* vox0;          // n + 1: an object's first voxel
    const float *hd, *phd;         // kNumLods object-level values an object, once computed
};

__global__ void __launch_bounds__(kPrepThreads) k_records(Meshes M, const uint32_t* __restrict__ lodF, VoxScratch S, RecordsDev R) {
    const int l = blockIdx.y;
    for (int o = blockIdx.x; o < M.n; o += gridDim.x) {
        const int64_t f0 = M.foff[o], s0 = S.soff[o];
        const float* P = M.V + 3 * M.voff[o];
        const uint32_t* LF = l < kNumLods - 1 ? lodF + (size_t)l * 3 * S.Ftot + 3 * f0 : M.F + 3 * f0;
        const uint32_t* od = S.ord + (size_t)l * S.Ftot + f0;
        const uint32_t t0 = R.t0[l][o], n = R.t0[l][o + 1] - t0, v0 = R.vox0[o], nv = R.vox0[o + 1] - v0;
        for (uint32_t i = threadIdx.x; i < 3 * n; i += blockDim.x) {
            const float* q = P + 3 * (size_t)LF[3 * od[i / 3] + i % 3];
            R.tri[l][3 * (size_t)t0 + i] = make_float4(q[0], q[1], q[2], 0.f);
        }
        for (uint32_t v = threadIdx.x; v < nv; v += blockDim.x) R.vtri[l][v0 + v] = t0 + S.vst[(size_t)l * S.Stot + s0 + v];
        if (threadIdx.x == 0 && o == M.n - 1) R.vtri[l][v0 + nv] = t0 + n;
    }
}

// ------------------------------------------------------------------ RAW writer
// Object o's bytes start at word pos[o] / 4 of `out` (every object is a
// multiple of 4 bytes long and the batch starts on an object).  The bounds are
// those of R's records, 0 without records.
template <int T>
__global__ void __launch_bounds__(T) k_write(Meshes M, const uint32_t* __restrict__ lodF, const uint32_t* __restrict__ lodCnt,
                                             VoxScratch S, const unsigned long long* __restrict__ pos, RecordsDev R,
                                             uint32_t* __restrict__ out) {
    constexpr int NW = T / 32;
    __shared__ float s_f[6][NW];
    __shared__ float s_d[NW];
    __shared__ uint32_t s_i[NW];
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    for (int o = blockIdx.x; o < M.n; o += gridDim.x) {
        const int64_t v0 = M.voff[o], f0 = M.foff[o], s0 = S.soff[o];
        const uint32_t n = (uint32_t)(M.voff[o + 1] - v0), m = (uint32_t)(M.foff[o + 1] - f0);
        const float* P = M.V + 3 * v0;
        const uint32_t nvox = S.nvox[o];
        const uint32_t* core = S.core + s0;
        uint32_t* W = out + pos[o] / 4;
        uint32_t cl[kNumLods], lstart[kNumLods], ntri = 0;
        for (int l = 0; l < kNumLods; ++l) {
            cl[l] = l < kNumLods - 1 ? lodCnt[(size_t)o * kDecLods + l] : m;
            lstart[l] = ntri;
            ntri += cl[l];
        }
        const uint64_t data = 44ull * ntri;
        if (tid == 0) { W[0] = (uint32_t)data; W[1] = (uint32_t)(data >> 32); }
        uint32_t* D = W + 2;
        for (int l = 0; l < kNumLods; ++l) {
            const uint32_t* LF = l < kNumLods - 1 ? lodF + (size_t)l * 3 * S.Ftot + 3 * f0 : M.F + 3 * f0;
            const uint32_t* tv = S.tvox + (size_t)l * S.Ftot + f0;
            const uint32_t* od = S.ord + (size_t)l * S.Ftot + f0;
            const uint32_t* vc = S.vcnt + (size_t)l * S.Stot + s0;
            const uint32_t* vs = S.vst + (size_t)l * S.Stot + s0;
            for (uint32_t g = tid; g < cl[l]; g += T) {
                const uint32_t t = od[g], v = tv[t], sv = vs[v], cv = vc[v], j = g - sv;
                uint32_t* grp = D + 11 * (size_t)(lstart[l] + sv);
                uint32_t* c = grp + 9 * j;
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    const float* q = P + 3 * (size_t)LF[3 * t + k];
                    c[3 * k] = __float_as_uint(q[0]);
                    c[3 * k + 1] = __float_as_uint(q[1]);
                    c[3 * k + 2] = __float_as_uint(q[2]);
                }
                const float4* r = R.tri[l] ? R.tri[l] + 3 * ((size_t)R.t0[l][o] + g) : nullptr;
                grp[9 * cv + 2 * j] = r ? __float_as_uint(r[0].w) : 0u;
                grp[9 * cv + 2 * j + 1] = r ? __float_as_uint(r[1].w) : 0u;
            }
        }
        uint32_t* H = D + 11 * (size_t)ntri;
        if (tid == 0) { H[0] = nvox; H[1] = 0u; }
        if (tid < 2 * kNumLods)  // object-level bounds: (hausdorff, proxy) of every LOD
            H[2 + tid] = R.hd ? __float_as_uint((tid & 1 ? R.phd : R.hd)[(size_t)o * kNumLods + tid / 2]) : 0u;
        for (uint32_t v = tid; v < nvox; v += T) {
            float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
            for (int l = 0; l < kNumLods; ++l) {
                const uint32_t* LF = l < kNumLods - 1 ? lodF + (size_t)l * 3 * S.Ftot + 3 * f0 : M.F + 3 * f0;
                const uint32_t* od = S.ord + (size_t)l * S.Ftot + f0;
                const uint32_t sv = S.vst[(size_t)l * S.Stot + s0 + v], cv = S.vcnt[(size_t)l * S.Stot + s0 + v];
                for (uint32_t g = sv; g < sv + cv; ++g)
                    for (int k = 0; k < 3; ++k) {
                        const float* q = P + 3 * (size_t)LF[3 * od[g] + k];
                        for (int d = 0; d < 3; ++d) {  // a tie keeps the value held (-0 vs +0)
                            lo[d] = q[d] < lo[d] ? q[d] : lo[d];
                            hi[d] = hi[d] < q[d] ? q[d] : hi[d];
                        }
                    }
            }
            uint32_t* X = H + 12 + 29 * (size_t)v;
            for (int d = 0; d < 3; ++d) { X[d] = __float_as_uint(lo[d]); X[3 + d] = __float_as_uint(hi[d]); }
            for (int d = 0; d < 3; ++d) X[6 + d] = __float_as_uint(P[3 * (size_t)core[v] + d]);
            for (int l = 0; l < kNumLods; ++l) {
                const uint64_t off = 44ull * (lstart[l] + S.vst[(size_t)l * S.Stot + s0 + v]);
                const uint32_t cv = S.vcnt[(size_t)l * S.Stot + s0 + v];
                X[9 + 4 * l] = (uint32_t)off;
                X[10 + 4 * l] = (uint32_t)(off >> 32);
                X[11 + 4 * l] = cv;
                X[12 + 4 * l] = 0u;
            }
        }
        // 4. transform: the vertex nearest the centre of the float bounding box
        float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
        for (uint32_t i = tid; i < n; i += T)
            for (int d = 0; d < 3; ++d) {
                lo[d] = fminf(lo[d], P[3 * (size_t)i + d]);
                hi[d] = fmaxf(hi[d], P[3 * (size_t)i + d]);
            }
#pragma unroll
        for (int k = 16; k > 0; k >>= 1)
            for (int d = 0; d < 3; ++d) {
                lo[d] = fminf(lo[d], __shfl_xor_sync(0xffffffffu, lo[d], k));
                hi[d] = fmaxf(hi[d], __shfl_xor_sync(0xffffffffu, hi[d], k));
            }
        if (lane == 0)
            for (int d = 0; d < 3; ++d) { s_f[d][wid] = lo[d]; s_f[3 + d][wid] = hi[d]; }
        __syncthreads();
        for (int w = 0; w < NW; ++w)
            for (int d = 0; d < 3; ++d) { lo[d] = fminf(lo[d], s_f[d][w]); hi[d] = fmaxf(hi[d], s_f[3 + d][w]); }
        const float cx = 0.5f * (lo[0] + hi[0]), cy = 0.5f * (lo[1] + hi[1]), cz = 0.5f * (lo[2] + hi[2]);
        float bd = INFINITY;
        uint32_t bi = UINT_MAX;
        for (uint32_t i = tid; i < n; i += T) {
            const float dx = P[3 * (size_t)i] - cx, dy = P[3 * (size_t)i + 1] - cy, dz = P[3 * (size_t)i + 2] - cz;
            const float d = dx * dx + dy * dy + dz * dz;
            // (FP32 squares overflow on meshes of 1e19 units: all infinite, the lowest index)
            if (d < bd || bi == UINT_MAX) { bd = d; bi = i; }
        }
#pragma unroll
        for (int k = 16; k > 0; k >>= 1) {
            const float d2 = __shfl_xor_sync(0xffffffffu, bd, k);
            const uint32_t i2 = __shfl_xor_sync(0xffffffffu, bi, k);
            if (d2 < bd || (d2 == bd && i2 < bi)) { bd = d2; bi = i2; }
        }
        if (lane == 0) { s_d[wid] = bd; s_i[wid] = bi; }
        __syncthreads();
        if (tid == 0) {
            for (int w = 1; w < NW; ++w)
                if (s_d[w] < bd || (s_d[w] == bd && s_i[w] < bi)) { bd = s_d[w]; bi = s_i[w]; }
            uint32_t* X = H + 12 + 29 * (size_t)nvox;
            for (int d = 0; d < 3; ++d) X[d] = __float_as_uint(P[3 * (size_t)bi + d]);
        }
        __syncthreads();
    }
}

}  // namespace
}  // namespace tdp

// ------------------------------------------------------------------ host driver
using namespace tdp;

namespace {

struct DevMem {  // allocations of one batch, back to the context's block cache on every return
    tdp_ctx* ctx;
    std::vector<void*> ps;
    ~DevMem() { release(); }
    void release() {
        if (ps.empty()) return;
        cudaStreamSynchronize(ctx->stream);  // nothing queued may still use a block
        hand_on();
    }
    void hand_on() {  // to what is queued on the context's stream after this
        for (void* p : ps) block_release(ctx, p);
        ps.clear();
    }
    template <typename X>
    cudaError_t get(X** p, size_t count) {
        void* q = nullptr;
        const cudaError_t e = block_alloc(ctx, &q, std::max<size_t>(count, 1) * sizeof(X));
        if (e == cudaSuccess) ps.push_back(q);
        *p = (X*)q;
        return e;
    }
};

inline size_t upper_bytes(int64_t m, int voxel_size) {  // RAW bytes of an object, at most
    return 68 + 44 * (size_t)kNumLods * (size_t)m + 116 * ((size_t)m / (size_t)voxel_size + 1);
}

}  // namespace

extern "C" int tdp_raw_prep_bound(const int64_t* face_off, long n_objects, int voxel_size, size_t* max_len) {
    if (!max_len || n_objects < 0 || voxel_size <= 0 || (n_objects > 0 && !face_off)) return TDP_ERR_ARG;
    size_t s = 1;
    for (long o = 0; o < n_objects; ++o) {
        const int64_t m = face_off[o + 1] - face_off[o];
        if (m < 0) return TDP_ERR_ARG;
        s += upper_bytes(m, voxel_size);
    }
    *max_len = s;
    return TDP_OK;
}

extern "C" int tdp_raw_from_meshes(tdp_ctx* ctx, const float* vertices, const int64_t* vert_off, const uint32_t* faces,
                                   const int64_t* face_off, long n_objects, int voxel_size, void* out, size_t cap,
                                   size_t* len, tdp_prep_info* info) {
    if (!ctx) return TDP_ERR_ARG;
    if (n_objects < 0 || n_objects > INT_MAX || voxel_size <= 0 || (n_objects > 0 && (!vertices || !vert_off || !faces || !face_off)))
        return fail(ctx, TDP_ERR_ARG, "tdp_raw_from_meshes: bad arguments");
    for (long o = 0; o < n_objects; ++o)
        if (vert_off[o + 1] < vert_off[o] || face_off[o + 1] < face_off[o] || vert_off[o] < 0 || face_off[o] < 0)
            return fail(ctx, TDP_ERR_ARG, "tdp_raw_from_meshes: offsets must be non-decreasing");
    const auto t_start = std::chrono::steady_clock::now();
    tdp_prep_info inf{};
    inf.n_objects = n_objects;
    cudaStream_t s = ctx->stream;
#define CU(x) do { cudaError_t _e = (x); if (_e != cudaSuccess) return fail(ctx, TDP_ERR_CUDA, std::string("tdp_raw_from_meshes: " #x ": ") + cudaGetErrorString(_e)); } while (0)
    // batches of consecutive objects within a device-memory budget
    size_t free_b = 0, total_b = 0;
    CU(cudaMemGetInfo(&free_b, &total_b));
    // a batch holds at most min(6 GiB, a quarter of the free memory, an eighth of the context's cap)
    size_t budget = std::min<size_t>((size_t)6 << 30, free_b / 4);
    if (ctx->budget) budget = std::min(budget, ctx->budget / 8);
    budget = std::max<size_t>(budget, (size_t)16 << 20);
    std::vector<long> cuts{0};
    {
        size_t acc = 0;
        for (long o = 0; o < n_objects; ++o) {
            const int64_t n = vert_off[o + 1] - vert_off[o], m = face_off[o + 1] - face_off[o];
            const size_t need = 32 * (size_t)n + (12 + 48 + 40 + 28) * (size_t)m + 80 * ((size_t)m / voxel_size + 1) +
                                upper_bytes(m, voxel_size) + dec_bytes(n, m, 4) + 64;
            if (acc > 0 && acc + need > budget) {
                cuts.push_back(o);
                acc = 0;
            }
            acc += need;
        }
        cuts.push_back(n_objects);
    }
    size_t pos_out = 1;  // the tile's type byte
    // bounds batch by batch; an object beyond the limits of a resident tile is
    // left to the upload of the finished tile, which names the limit
    bool dev_bounds = true;
    for (long o = 0; o < n_objects; ++o) dev_bounds = dev_bounds && face_off[o + 1] - face_off[o] <= (1 << 24);
    std::vector<unsigned long long> bytes;
    cudaEvent_t ev[4];
    for (auto& e : ev) CU(cudaEventCreate(&e));
    struct EvFree {
        cudaEvent_t* e;
        ~EvFree() { for (int k = 0; k < 4; ++k) cudaEventDestroy(e[k]); }
    } evfree{ev};
    for (size_t b = 0; b + 1 < cuts.size(); ++b) {
        const long o0 = cuts[b], o1 = cuts[b + 1], nb = o1 - o0;
        if (nb <= 0) continue;
        DevMem dm{ctx, {}};
        const int64_t vb = vert_off[o0], fb = face_off[o0];
        const int64_t Vtot = vert_off[o1] - vb, Ftot = face_off[o1] - fb;
        std::vector<int64_t> voff(nb + 1), foff(nb + 1), soff(nb + 1);
        soff[0] = 0;
        for (long i = 0; i <= nb; ++i) {
            voff[i] = vert_off[o0 + i] - vb;
            foff[i] = face_off[o0 + i] - fb;
            if (i < nb) soff[i + 1] = soff[i] + (face_off[o0 + i + 1] - face_off[o0 + i]) / voxel_size + 1;
        }
        const int64_t Stot = soff[nb];
        float* dV;
        uint32_t* dF;
        int64_t *dvoff, *dfoff, *dsoff;
        int* dbad;
        CU(dm.get(&dV, 3 * (size_t)Vtot));
        CU(dm.get(&dF, 3 * (size_t)Ftot));
        CU(dm.get(&dvoff, nb + 1));
        CU(dm.get(&dfoff, nb + 1));
        CU(dm.get(&dsoff, nb + 1));
        CU(dm.get(&dbad, 1));
        CU(cudaMemcpyAsync(dV, vertices + 3 * vb, 12 * (size_t)Vtot, cudaMemcpyHostToDevice, s));
        CU(cudaMemcpyAsync(dF, faces + 3 * fb, 12 * (size_t)Ftot, cudaMemcpyHostToDevice, s));
        CU(cudaMemcpyAsync(dvoff, voff.data(), 8 * (nb + 1), cudaMemcpyHostToDevice, s));
        CU(cudaMemcpyAsync(dfoff, foff.data(), 8 * (nb + 1), cudaMemcpyHostToDevice, s));
        CU(cudaMemcpyAsync(dsoff, soff.data(), 8 * (nb + 1), cudaMemcpyHostToDevice, s));
        const int big = INT_MAX;
        CU(cudaMemcpyAsync(dbad, &big, 4, cudaMemcpyHostToDevice, s));
        Meshes Mh{dV, dvoff, dF, dfoff, (int)nb};
        k_validate<<<(int)std::min<long>(nb, 65535), 256, 0, s>>>(Mh, dbad);
        CU(cudaGetLastError());
        int bad = INT_MAX;
        CU(cudaMemcpyAsync(&bad, dbad, 4, cudaMemcpyDeviceToHost, s));
        CU(cudaStreamSynchronize(s));
        if (bad != INT_MAX)
            return fail(ctx, TDP_ERR_ARG, "tdp_raw_from_meshes: object " + std::to_string(o0 + bad) +
                                              " has no vertex or facet, a vertex index out of range, a facet repeating "
                                              "a vertex or a non-finite coordinate");
        CU(cudaEventRecord(ev[0], s));
        // 1. decimation, three launch shapes by the object's storage
        uint32_t *lodF, *lodCnt;
        CU(dm.get(&lodF, (size_t)kDecLods * 3 * Ftot));
        CU(dm.get(&lodCnt, (size_t)kDecLods * nb));
        std::vector<int> small, large, huge;
        std::vector<int64_t> hoff{0};
        size_t s_small = 0, s_large = 0;
        for (long i = 0; i < nb; ++i) {
            const int64_t n = voff[i + 1] - voff[i], m = foff[i + 1] - foff[i];
            const size_t b16 = dec_bytes(n, m, 2);
            if (n <= 65535 && b16 <= kSmemSmall) { small.push_back((int)i); s_small = std::max(s_small, b16); }
            else if (n <= 65535 && b16 <= kSmemLarge) { large.push_back((int)i); s_large = std::max(s_large, b16); }
            else { huge.push_back((int)i); hoff.push_back(hoff.back() + (int64_t)dec_bytes(n, m, 4)); }
        }
        DevMem dec{ctx, {}};  // what only the decimation needs
        DecLists dls{};
        CU(dec.get(&dls.keys, (size_t)Ftot));
        CU(dec.get(&dls.csr, 3 * (size_t)Ftot));
        CU(dec.get(&dls.lists, (size_t)(Vtot + nb)));
        int* dl;
        CU(dec.get(&dl, small.size() + large.size() + huge.size()));
        std::vector<int> all(small);
        all.insert(all.end(), large.begin(), large.end());
        all.insert(all.end(), huge.begin(), huge.end());
        if (!all.empty()) CU(cudaMemcpyAsync(dl, all.data(), 4 * all.size(), cudaMemcpyHostToDevice, s));
        if (!small.empty()) {
            auto kern = k_decimate<uint16_t, 128>;
            CU(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemSmall));  // (one limit for every thread)
            kern<<<(int)std::min<size_t>(small.size(), 1u << 30), 128, s_small, s>>>(Mh, dl, (int)small.size(), dls,
                                                                                    nullptr, nullptr, lodF, Ftot, lodCnt);
            CU(cudaGetLastError());
        }
        if (!large.empty()) {
            auto kern = k_decimate<uint16_t, 256>;
            CU(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemLarge));
            kern<<<(int)large.size(), 256, s_large, s>>>(Mh, dl + small.size(), (int)large.size(), dls, nullptr, nullptr,
                                                        lodF, Ftot, lodCnt);
            CU(cudaGetLastError());
        }
        if (!huge.empty()) {
            uint8_t* gst;
            int64_t* dho;
            CU(dec.get(&gst, (size_t)hoff.back()));
            CU(dec.get(&dho, hoff.size()));
            CU(cudaMemcpyAsync(dho, hoff.data(), 8 * hoff.size(), cudaMemcpyHostToDevice, s));
            k_decimate<uint32_t, 1024><<<(int)huge.size(), 1024, 0, s>>>(Mh, dl + small.size() + large.size(),
                                                                      (int)huge.size(), dls, gst, dho, lodF, Ftot,
                                                                      lodCnt);
            CU(cudaGetLastError());
        }
        CU(cudaEventRecord(ev[1], s));
        if (ctx->budget) dec.hand_on();  // under a memory cap its room is the next steps'
        // 2-3. voxels
        VoxScratch S{};
        CU(dm.get(&S.dmin, (size_t)Vtot));
        CU(dm.get(&S.asg, (size_t)Vtot));
        CU(dm.get(&S.seed, 3 * (size_t)Stot));
        CU(dm.get(&S.bestd, (size_t)Stot));
        CU(dm.get(&S.bestf, (size_t)Stot));
        CU(dm.get(&S.core, (size_t)Stot));
        CU(dm.get(&S.nvox, (size_t)nb));
        CU(dm.get(&S.tvox, (size_t)kNumLods * Ftot));
        CU(dm.get(&S.ord, (size_t)kNumLods * Ftot));
        CU(dm.get(&S.vcnt, (size_t)kNumLods * Stot));
        CU(dm.get(&S.vst, (size_t)kNumLods * Stot));
        S.soff = dsoff;
        S.Ftot = Ftot;
        S.Stot = Stot;
        unsigned long long *dbytes, *dpos;
        CU(dm.get(&dbytes, (size_t)nb));
        CU(dm.get(&dpos, (size_t)nb));
        // fewer objects than SMs: more threads for each, and as many blocks as fit
        if (nb < ctx->num_sms) {
            int C = 1;
            while (C < 8 && 2 * C * nb <= ctx->num_sms) C *= 2;
            cudaLaunchAttribute at{};
            at.id = cudaLaunchAttributeClusterDimension;
            at.val.clusterDim.x = (unsigned)C;
            at.val.clusterDim.y = at.val.clusterDim.z = 1;
            cudaLaunchConfig_t cfg{};
            cfg.gridDim = dim3((unsigned)(nb * C));
            cfg.blockDim = dim3(1024);
            cfg.stream = s;
            cfg.attrs = &at;
            cfg.numAttrs = 1;
            CU(cudaLaunchKernelEx(&cfg, k_voxels<1024>, Mh, voxel_size, (const uint32_t*)lodF, (const uint32_t*)lodCnt, S, dbytes));
        } else {
            k_voxels<kPrepThreads><<<(int)nb, kPrepThreads, 0, s>>>(Mh, voxel_size, lodF, lodCnt, S, dbytes);
        }
        CU(cudaGetLastError());
        CU(cudaEventRecord(ev[2], s));
        bytes.assign(nb, 0);
        float ms_vox[2] = {0, 0};
        std::vector<uint32_t> hcnt((size_t)kDecLods * nb), hnvox(nb);
        CU(cudaMemcpyAsync(bytes.data(), dbytes, 8 * nb, cudaMemcpyDeviceToHost, s));
        CU(cudaMemcpyAsync(hcnt.data(), lodCnt, 4 * hcnt.size(), cudaMemcpyDeviceToHost, s));
        CU(cudaMemcpyAsync(hnvox.data(), S.nvox, 4 * nb, cudaMemcpyDeviceToHost, s));
        CU(cudaStreamSynchronize(s));
        cudaEventElapsedTime(&ms_vox[0], ev[0], ev[1]);
        cudaEventElapsedTime(&ms_vox[1], ev[1], ev[2]);
        inf.decimate_ms += ms_vox[0];
        inf.voxel_ms += ms_vox[1];
        std::vector<unsigned long long> hpos(nb);
        unsigned long long run = 0;
        for (long i = 0; i < nb; ++i) {
            hpos[i] = run;
            run += bytes[i];
            for (int l = 0; l < kDecLods; ++l) inf.n_triangles[l] += hcnt[(size_t)i * kDecLods + l];
            inf.n_triangles[kNumLods - 1] += foff[i + 1] - foff[i];
            inf.n_voxels += hnvox[i];
        }
        if (out && pos_out + run <= cap) {
            uint32_t* dout;
            CU(dm.get(&dout, (size_t)(run / 4)));
            // 4. the bounds of the batch's triangles and objects
            DevMem bm{ctx, {}};
            RecordsDev R{};
            BoundRecords br{};
            std::vector<uint32_t> at((size_t)(kNumLods + 1) * (nb + 1));  // t0 of every LOD, then vox0
            if (dev_bounds) {
                for (int l = 0; l <= kNumLods; ++l) {
                    uint64_t sum = 0;
                    for (long i = 0; i <= nb; ++i) {
                        at[(size_t)l * (nb + 1) + i] = (uint32_t)sum;
                        if (i < nb) sum += l == kNumLods ? hnvox[i] : l == kNumLods - 1 ? (uint64_t)(foff[i + 1] - foff[i]) : hcnt[(size_t)i * kDecLods + l];
                    }
                    if (l < kNumLods) br.n_tris[l] = (size_t)sum;
                    else br.n_vox = (long)sum;
                    if (sum >= UINT_MAX) dev_bounds = false;
                }
                br.n_obj = nb;
            }
            if (dev_bounds) {
                uint32_t* dat;
                float* obj;
                bool ok = bm.get(&dat, at.size()) == cudaSuccess && bm.get(&obj, 2 * (size_t)kNumLods * nb) == cudaSuccess;
                for (int l = 0; ok && l < kNumLods; ++l) {
                    uint32_t* vt;
                    ok = bm.get(&br.tri[l], 3 * br.n_tris[l]) == cudaSuccess && bm.get(&vt, (size_t)br.n_vox + 1) == cudaSuccess;
                    R.tri[l] = br.tri[l];
                    R.vtri[l] = vt;
                    br.vtri[l] = vt;
                    R.t0[l] = dat + (size_t)l * (nb + 1);
                }
                ok = ok && bounds_scratch(ctx, br) == TDP_OK;
                if (ok) {
                    R.vox0 = br.obj_vox = dat + (size_t)kNumLods * (nb + 1);
                    R.hd = br.obj_hd = obj;
                    R.phd = br.obj_phd = obj + (size_t)kNumLods * nb;
                    CU(cudaMemcpyAsync(dat, at.data(), 4 * at.size(), cudaMemcpyHostToDevice, s));
                    CU(cudaEventRecord(ev[0], s));
                    k_records<<<dim3((unsigned)nb, kNumLods), kPrepThreads, 0, s>>>(Mh, lodF, S, R);
                    CU(cudaGetLastError());
                    CU(launch_bounds(ctx, br));
                    CU(cudaEventRecord(ev[1], s));
                } else {  // no room beside the batch: the finished tile's bounds, below
                    cudaGetLastError();
                    bm.release();
                    bounds_scratch_free(ctx);
                    R = RecordsDev{};
                    dev_bounds = false;
                }
            }
            // 5. RAW bytes of the batch, then to the caller's buffer
            CU(cudaMemcpyAsync(dpos, hpos.data(), 8 * nb, cudaMemcpyHostToDevice, s));
            CU(cudaEventRecord(ev[2], s));  // the writer alone (the host's allocation above is not timed)
            k_write<kPrepThreads><<<(int)nb, kPrepThreads, 0, s>>>(Mh, lodF, lodCnt, S, dpos, R, dout);
            CU(cudaGetLastError());
            CU(cudaEventRecord(ev[3], s));
            CU(cudaMemcpyAsync((uint8_t*)out + pos_out, dout, (size_t)run, cudaMemcpyDeviceToHost, s));
            CU(cudaStreamSynchronize(s));
            float ms = 0;
            cudaEventElapsedTime(&ms, ev[2], ev[3]);
            inf.write_ms += ms;
            if (R.hd) {
                cudaEventElapsedTime(&ms, ev[0], ev[1]);
                inf.bounds_ms += ms;
                if (ctx->budget) bounds_scratch_free(ctx);  // the next batch's room is what it was
            }
        }
        pos_out += (size_t)run;
        inf.batches += 1;
    }
#undef CU
    if (len) *len = pos_out;
    if (!out) {
        if (info) *info = inf;
        return TDP_OK;
    }
    if (cap < pos_out) return fail(ctx, TDP_ERR_ARG, "tdp_raw_from_meshes: output buffer too small");
    ((uint8_t*)out)[0] = kRawType;
    const auto t_b = std::chrono::steady_clock::now();
    if (n_objects > 0 && !dev_bounds) {
        if (ctx->budget) cache_trim(ctx);  // blocks of just the sizes asked for
        tdp_bounds_info bi{};
        if (const int rc = tdp_raw_compute_bounds(ctx, out, pos_out, out, &bi)) return rc;
    }
    const auto t_end = std::chrono::steady_clock::now();
    if (!dev_bounds) inf.bounds_ms = std::chrono::duration<double, std::milli>(t_end - t_b).count();
    inf.total_ms = std::chrono::duration<double, std::milli>(t_end - t_start).count();
    if (info) *info = inf;
    return TDP_OK;
}
