// bounds_kernels.cu -- GPU preparation of the per-triangle Hausdorff bounds of a
// resident tile (tdp_tile_compute_bounds).
//
// Replaces the reference's CGAL preparation of the bounds that the join reads
// (sampling in src/spatial/himesh_hausdorff.cpp:197-270; stored per triangle as
// (proxy, hausdorff) at src/spatial/himesh_retrieve.cpp:131-151 and consumed by
// the refine at src/geometry/computing_gpu.cu:1115-1117) with a conservative
// rule evaluated in FP64 from each object's own LOD-100 surface S:
//   ph(t): each LOD-100 facet s is assigned to the LOD-l triangle t nearest its
//          barycentre (ties to the lower index); ph(t) = max over assigned s
//          and the vertices q of s of dist(q, t).  dist(., t) is convex, so
//          every point of s lies within ph(t) of t: d(t1, t2) - ph1 - ph2 is a
//          lower bound of the LOD-100 distance.
//   h(t):  t is cut by d midpoint subdivisions (d = least of 0..3 with
//          longest edge / 2^d <= 1.5 x the mean LOD-100 edge of the object) and
//          h(t) = max over pieces of min over s of max over the piece's corners
//          of dist(corner, s).  By convexity of dist(., s) every point of t lies
//          within h(t) of S: d(t1, t2) + h1 + h2 is an upper bound.
// Both round up to float; the object-level values are the per-LOD maxima.
//
// Layout of the work: one warp per (LOD, voxel) item, 32 queries (facets, or
// pieces of triangles) at a time, one a lane.  A query starts from the nearest
// triangle of its own voxel by FP32 centres, then goes through the voxels of the
// object whose box is within the best distance so far.  A voxel's triangles are
// staged as FP32 bounding spheres; a (query, triangle) pair whose sphere gap,
// less a margin far above the rounding, is above the query's best distance so far
// cannot be its nearest, and the others collect in a queue from which they are
// evaluated in FP64, 32 at a time and one a lane.  Every triangle that could be
// nearest or tie is evaluated, so both searches return exactly what a scan of
// every triangle returns.  Distances are compared squared and rooted once per
// result (sqrt is monotone and correctly rounded, so this changes no bound); the
// nearest-triangle assignment breaks ties on the squared distance, then on the
// index.  This file is built with -fmad=false: each product and sum is rounded
// on its own, so the FP64 values equal a host evaluation of the same expressions.
//
// A warp per query with every triangle of a visited voxel in FP64 was bound by
// the divergent FP64 point-triangle distance (about 300 evaluations a query).
#include <cuda_runtime.h>

#include <algorithm>
#include <cfloat>
#include <climits>
#include <cstring>
#include <string>

#include "ctx.cuh"
#include "bounds_kernels.cuh"
#include "fetch_kernels.cuh"
#include "ptdist.cuh"
#include "storage/dev_tile.h"

namespace tdp {
namespace {

using pd::D3;

constexpr int kBoundsThreads = 256;
constexpr int kBoundsBlocksPerSm = 2;
enum BoundSlot { kBoxes = 84, kVobj, kMeanEdge, kBoundCounters };

struct BoundsDev {
    const float4* tri[kNumLods];
    const uint32_t* vtri[kNumLods];
    const float4* box[kNumLods];  // per voxel: (lo, 0), (hi, 0) of its triangles at that LOD
    const uint32_t* obj_vox;
    const int* vobj;
    const double* e0;
    long n_vox, n_obj;
    int share;              // log2 of the warps that share a (LOD, voxel) item's batches
    unsigned long long* counters;  // [0] distance evaluations, [1] facet queries, [2] pieces
};

__device__ inline D3 vert(const float4* tri, size_t t, int k) {
    const float4 v = tri[3 * t + k];
    return D3{(double)v.x, (double)v.y, (double)v.z};
}

__device__ inline unsigned long long warp_sum(unsigned long long v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// zero the (proxy, hausdorff) fields of every triangle record of one LOD
__global__ void k_zero_bounds(float4* tri, size_t n) {
    for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < n; t += (size_t)gridDim.x * blockDim.x) {
        tri[3 * t].w = 0.f;
        tri[3 * t + 1].w = 0.f;
    }
}

// box of every voxel's triangles at one LOD (+inf/-inf for an empty voxel)
__global__ void k_voxel_boxes(const float4* __restrict__ tri, const uint32_t* __restrict__ vtri, long n_vox,
                              float4* __restrict__ box) {
    const int lane = threadIdx.x & 31;
    const long warps = ((long)gridDim.x * blockDim.x) >> 5;
    for (long v = ((long)blockIdx.x * blockDim.x + threadIdx.x) >> 5; v < n_vox; v += warps) {
        float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
        for (size_t i = 3 * (size_t)vtri[v] + lane; i < 3 * (size_t)vtri[v + 1]; i += 32) {
            const float4 p = tri[i];
            lo[0] = fminf(lo[0], p.x); lo[1] = fminf(lo[1], p.y); lo[2] = fminf(lo[2], p.z);
            hi[0] = fmaxf(hi[0], p.x); hi[1] = fmaxf(hi[1], p.y); hi[2] = fmaxf(hi[2], p.z);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
            for (int k = 0; k < 3; ++k) {
                lo[k] = fminf(lo[k], __shfl_xor_sync(0xffffffffu, lo[k], o));
                hi[k] = fmaxf(hi[k], __shfl_xor_sync(0xffffffffu, hi[k], o));
            }
        if (lane == 0) {
            box[2 * v] = make_float4(lo[0], lo[1], lo[2], 0.f);
            box[2 * v + 1] = make_float4(hi[0], hi[1], hi[2], 0.f);
        }
    }
}

// object of every voxel; mean LOD-100 edge length of every object (its facets
// and their edges (0,1), (1,2), (2,0) summed in stored order).  One warp per
// object: the lanes root 32 facets' edges, lane 0 adds them up in order.
__global__ void k_objects(BoundsDev b, int* vobj, double* e0) {
    __shared__ double len[4][96];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const long warps = ((long)gridDim.x * blockDim.x) >> 5;
    for (long o = ((long)blockIdx.x * blockDim.x + threadIdx.x) >> 5; o < b.n_obj; o += warps) {
        const uint32_t vb = b.obj_vox[o], ve = b.obj_vox[o + 1];
        for (uint32_t v = vb + lane; v < ve; v += 32) vobj[v] = (int)o;
        const uint32_t s0 = b.vtri[4][vb], s1 = b.vtri[4][ve];
        double sum = 0;
        for (uint32_t base = s0; base < s1; base += 32) {
            __syncwarp();
            if (base + lane < s1) {
                const D3 p = vert(b.tri[4], base + lane, 0), q = vert(b.tri[4], base + lane, 1), r = vert(b.tri[4], base + lane, 2);
                len[w][3 * lane] = pd::dist(p, q);
                len[w][3 * lane + 1] = pd::dist(q, r);
                len[w][3 * lane + 2] = pd::dist(r, p);
            }
            __syncwarp();
            if (lane == 0) {
                const int n = 3 * (int)min(32u, s1 - base);
                for (int i = 0; i < n; i += 3) {
                    sum = sum + len[w][i];
                    sum = sum + len[w][i + 1];
                    sum = sum + len[w][i + 2];
                }
            }
        }
        if (lane == 0) e0[o] = s1 > s0 ? sum / (3.0 * (double)(s1 - s0)) : 0.0;
    }
}

constexpr int kStage = 64;  // spheres staged at a time

// A warp's shared memory: K points a query (1: a barycentre, 3: a piece's corners).
template <int K>
struct Search {
    double q[K][3][32];                // the queries' points
    unsigned long long best[32];       // squared distance of each one's best triangle so far (bits)
    unsigned best_i[32];               // that triangle
    float4 sph[kStage];
    uint2 queue[64];                   // (query, triangle)
};

__device__ inline float rmin32(float v) {
    float r;
    asm("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}
__device__ inline float rmax32(float v) {
    float r;
    asm("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}

// no more than the length of (x, y, z >= 0), also where its square overflows
__device__ inline float length_down(float x, float y, float z) {
    const float s = x * x + y * y + z * z;
    return (s < INFINITY ? sqrtf(s) : fmaxf(x, fmaxf(y, z))) * 0.999999f;
}

// one copy of the FP64 distance in a kernel
__device__ __noinline__ double point_tri2(D3 p, D3 a, D3 b, D3 c) { return pd::tri2_dev(p, a, b, c); }

// largest squared distance of query j's points to triangle t; with K > 1 cut
// short (and then not below `limit`) once a point is at `limit` or beyond
template <int K>
__device__ inline double query_dist(const Search<K>& S, int j, const float4* T, unsigned t, double limit, unsigned& evals) {
    const D3 a = vert(T, t, 0), b = vert(T, t, 1), c = vert(T, t, 2);
    double acc = 0;
#pragma unroll 1
    for (int k = 0; k < K; ++k) {
        acc = pd::dmax(acc, point_tri2(D3{S.q[k][0][j], S.q[k][1][j], S.q[k][2][j]}, a, b, c));
        ++evals;
        if (K > 1 && acc >= limit) break;
    }
    return acc;
}

// The first `take` queued pairs, one a lane: their queries' best squared
// distance, ties to the lowest triangle.  (Not inlined, nor is the FP64
// distance: several copies of it in a kernel made instruction fetches its
// largest stall, 27 ms against 19 for 1,000 nuclei.)
template <int K>
__device__ __noinline__ void drain(Search<K>& S, const float4* T, int& qn, int take, int lane, unsigned& evals) {
    __syncwarp();
    const bool on = lane < take;
    const uint2 e = on ? S.queue[lane] : make_uint2(0, 0);
    const unsigned long long was = S.best[e.x];
    __syncwarp();
    unsigned long long d = ~0ull;
    if (on) {
        d = (unsigned long long)__double_as_longlong(
            query_dist<K>(S, (int)e.x, T, e.y, __longlong_as_double((long long)was), evals));
        if (d < was) atomicMin(&S.best[e.x], d);
    }
    __syncwarp();
    const bool hit = on && d == S.best[e.x];
    if (hit && d < was) S.best_i[e.x] = UINT_MAX;  // a nearer one: earlier triangles no longer tie
    __syncwarp();
    if (hit) atomicMin(&S.best_i[e.x], e.y);
    const uint2 moved = lane + take < qn ? S.queue[lane + take] : make_uint2(0, 0);
    __syncwarp();
    qn -= take;
    if (lane < qn) S.queue[lane] = moved;
    __syncwarp();
}

// FP32 stand-in of a lane's query: its points relative to an origin near them
// all, and their middle (no farther from a centre than the farthest point).
template <int K>
struct Query32 {
    float x[K], y[K], z[K], gx, gy, gz;
};

// nearest triangles of up to 32 queries (lane < n; points in S.q) among the
// triangles of the object's voxels [vb, ve), starting with voxel v0.
// Leaves S.best / S.best_i (UINT_MAX: the object has no triangle here).
template <int K>
__device__ inline void search(Search<K>& S, int n, const float4* T, const uint32_t* VT, const float4* box, uint32_t vb,
                              uint32_t ve, uint32_t v0, int lane, unsigned& evals) {
    const bool on = lane < n;
    const int j = on ? lane : 0;
    // the origin: the first query's first point; every lane's box of its points
    const float ox = (float)S.q[0][0][0], oy = (float)S.q[0][1][0], oz = (float)S.q[0][2][0];
    Query32<K> Q;
    float scale = 0.f;
    float lx = INFINITY, ly = INFINITY, lz = INFINITY, hx = -INFINITY, hy = -INFINITY, hz = -INFINITY;
#pragma unroll
    for (int k = 0; k < K; ++k) {
        Q.x[k] = (float)(S.q[k][0][j] - (double)ox);
        Q.y[k] = (float)(S.q[k][1][j] - (double)oy);
        Q.z[k] = (float)(S.q[k][2][j] - (double)oz);
        scale = fmaxf(scale, fmaxf(fabsf(Q.x[k]), fmaxf(fabsf(Q.y[k]), fabsf(Q.z[k]))));
        lx = fminf(lx, Q.x[k]); ly = fminf(ly, Q.y[k]); lz = fminf(lz, Q.z[k]);
        hx = fmaxf(hx, Q.x[k]); hy = fmaxf(hy, Q.y[k]); hz = fmaxf(hz, Q.z[k]);
    }
    if (K == 1) {
        Q.gx = Q.x[0]; Q.gy = Q.y[0]; Q.gz = Q.z[0];
    } else {
        Q.gx = (Q.x[0] + Q.x[K / 2] + Q.x[K - 1]) * (1.f / 3.f);
        Q.gy = (Q.y[0] + Q.y[K / 2] + Q.y[K - 1]) * (1.f / 3.f);
        Q.gz = (Q.z[0] + Q.z[K / 2] + Q.z[K - 1]) * (1.f / 3.f);
    }
    scale = rmax32(scale);
    const float blx = rmin32(lx), bly = rmin32(ly), blz = rmin32(lz), bhx = rmax32(hx), bhy = rmax32(hy), bhz = rmax32(hz);
    S.best[lane] = (unsigned long long)__double_as_longlong(INFINITY);
    S.best_i[lane] = UINT_MAX;
    int qn = 0;
    float bf = INFINITY;  // the lane's best distance so far, rounded up
    auto refresh = [&] { bf = __double2float_ru(sqrt(__longlong_as_double((long long)S.best[lane]))) * 1.000001f; };
    // stage spheres of triangles [t0, t0 + m): centre relative to the origin,
    // radius with the margin of the FP32 tests
    auto stage = [&](uint32_t t0, int m) {
        __syncwarp();
        for (int i = lane; i < m; i += 32) {
            const float4 a = T[3 * (size_t)(t0 + i)], b = T[3 * (size_t)(t0 + i) + 1], c = T[3 * (size_t)(t0 + i) + 2];
            const float ax = a.x - ox, ay = a.y - oy, az = a.z - oz, bx = b.x - ox, by = b.y - oy, bz = b.z - oz;
            const float cx = c.x - ox, cy = c.y - oy, cz = c.z - oz;
            const float mx = (ax + bx + cx) * (1.f / 3.f), my = (ay + by + cy) * (1.f / 3.f), mz = (az + bz + cz) * (1.f / 3.f);
            float r2 = (ax - mx) * (ax - mx) + (ay - my) * (ay - my) + (az - mz) * (az - mz);
            r2 = fmaxf(r2, (bx - mx) * (bx - mx) + (by - my) * (by - my) + (bz - mz) * (bz - mz));
            r2 = fmaxf(r2, (cx - mx) * (cx - mx) + (cy - my) * (cy - my) + (cz - mz) * (cz - mz));
            S.sph[i] = make_float4(mx, my, mz, sqrtf(r2) * 1.00001f + 2e-6f * (fabsf(mx) + fabsf(my) + fabsf(mz) + scale) + 1e-6f);
        }
        __syncwarp();
    };
    // seeds: the nearest centre of the first voxel with triangles
    uint32_t first = v0;
    if (VT[v0] == VT[v0 + 1])
        for (first = vb; first < ve && VT[first] == VT[first + 1]; ++first) {}
    if (first >= ve) return;
    {
        float best = INFINITY;
        unsigned bi = VT[first];
        for (uint32_t t0 = VT[first]; t0 < VT[first + 1]; t0 += kStage) {
            const int m = (int)min((uint32_t)kStage, VT[first + 1] - t0);
            stage(t0, m);
            for (int i = 0; i < m; ++i) {
                const float4 c = S.sph[i];
                const float x = Q.gx - c.x, y = Q.gy - c.y, z = Q.gz - c.z;
                const float d = x * x + y * y + z * z;
                if (d < best) {
                    best = d;
                    bi = t0 + i;
                }
            }
        }
        __syncwarp();
        if (on) S.queue[lane] = make_uint2((unsigned)lane, bi);
        qn = n;
        drain<K>(S, T, qn, n, lane, evals);
        refresh();
    }
    // the first voxel, then the object's others, 32 at a time: their box against
    // the box of all the points, then against each point.  (One loop, so that
    // the scan of a voxel is in the kernel once.)
    uint32_t u = first, base = vb;
    unsigned mask = 0;
    // The lane's own query is near enough to voxel u.  (Where spheres say little, as
    // those of a double cone's 20,000 needles, a voxel scanned for all 32 queries
    // when one was near took 279 M distances, 37.8 ms; this way 141 M, 20.6 ms.)
    bool near = on;
    float ulx = 0.f, uly = 0.f, ulz = 0.f, uhx = 0.f, uhy = 0.f, uhz = 0.f;  // voxel base - 32 + lane
    for (;;) {
        for (uint32_t t0 = VT[u]; t0 < VT[u + 1]; t0 += kStage) {
            const int m = (int)min((uint32_t)kStage, VT[u + 1] - t0);
            stage(t0, m);
            for (int i = 0; i < m; ++i) {
                const float4 c = S.sph[i];
                const float reach = (bf + c.w) * 1.000001f;
                const float gx = Q.gx - c.x, gy = Q.gy - c.y, gz = Q.gz - c.z;
                bool keep = near && !(gx * gx + gy * gy + gz * gz > reach * reach);
                unsigned mk = __ballot_sync(0xffffffffu, keep);
                if (!mk) continue;
                if (K > 1) {
#pragma unroll
                    for (int k = 0; k < K; ++k) {
                        const float x = Q.x[k] - c.x, y = Q.y[k] - c.y, z = Q.z[k] - c.z;
                        keep = keep && !(x * x + y * y + z * z > reach * reach);
                    }
                    mk = __ballot_sync(0xffffffffu, keep);
                    if (!mk) continue;
                }
                if (keep) S.queue[qn + __popc(mk & ((1u << lane) - 1u))] = make_uint2((unsigned)lane, t0 + i);
                qn += __popc(mk);
                if (qn >= 32) {
                    drain<K>(S, T, qn, 32, lane, evals);
                    refresh();
                }
            }
        }
        if (qn > 0) {
            drain<K>(S, T, qn, qn, lane, evals);
            refresh();
        }
        for (;;) {  // the next voxel with a point near enough
            if (!mask) {
                if (base >= ve) return;
                const uint32_t w = base + lane;
                const bool other = w < ve && w != first && VT[w] != VT[w + 1];
                float gap = 0.f;
                if (other) {
                    const float4 lo = box[2 * (size_t)w], hi = box[2 * (size_t)w + 1];
                    ulx = lo.x - ox; uly = lo.y - oy; ulz = lo.z - oz;
                    uhx = hi.x - ox; uhy = hi.y - oy; uhz = hi.z - oz;
                    const float x = fmaxf(fmaxf(ulx - bhx, blx - uhx), 0.f), y = fmaxf(fmaxf(uly - bhy, bly - uhy), 0.f),
                                z = fmaxf(fmaxf(ulz - bhz, blz - uhz), 0.f);
                    const float mg = 4e-6f * (fmaxf(fabsf(ulx), fabsf(uhx)) + fmaxf(fabsf(uly), fabsf(uhy)) +
                                              fmaxf(fabsf(ulz), fabsf(uhz)) + scale) + 1e-6f;
                    gap = length_down(x, y, z) - mg;
                }
                const float most = rmax32(on ? bf : 0.f);
                mask = __ballot_sync(0xffffffffu, other && !(gap > most));  // (what is not a number is looked at)
                base += 32;
                continue;
            }
            const int k = __ffs(mask) - 1;
            mask &= mask - 1;
            const float ax = __shfl_sync(0xffffffffu, ulx, k), ay = __shfl_sync(0xffffffffu, uly, k), az = __shfl_sync(0xffffffffu, ulz, k);
            const float ex = __shfl_sync(0xffffffffu, uhx, k), ey = __shfl_sync(0xffffffffu, uhy, k), ez = __shfl_sync(0xffffffffu, uhz, k);
            const float mg = 4e-6f * (fmaxf(fabsf(ax), fabsf(ex)) + fmaxf(fabsf(ay), fabsf(ey)) + fmaxf(fabsf(az), fabsf(ez)) + scale) + 1e-6f;
            near = on;
#pragma unroll
            for (int c = 0; c < K; ++c) {
                const float x = fmaxf(fmaxf(ax - Q.x[c], Q.x[c] - ex), 0.f), y = fmaxf(fmaxf(ay - Q.y[c], Q.y[c] - ey), 0.f),
                            z = fmaxf(fmaxf(az - Q.z[c], Q.z[c] - ez), 0.f);
                near = near && !(length_down(x, y, z) - mg > bf);
            }
            if (!__any_sync(0xffffffffu, near)) continue;
            u = base - 32 + k;
            break;
        }
    }
}

// ph: every LOD-100 facet of voxel v -> nearest LOD-l triangle; raise that
// triangle's proxy bound to the facet's farthest vertex distance
__global__ void __launch_bounds__(kBoundsThreads, kBoundsBlocksPerSm) k_proxy(BoundsDev b) {
    __shared__ Search<1> warps_s[kBoundsThreads / 32];
    Search<1>& Q = warps_s[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    const long warps = ((long)gridDim.x * blockDim.x) >> 5;
    unsigned long long all = 0, queries = 0;
    for (long w = ((long)blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < (4 * b.n_vox) << b.share; w += warps) {
        const long it = w >> b.share;
        const int part = (int)(w - (it << b.share));
        const int l = (int)(it / b.n_vox);
        const long v = it - (long)l * b.n_vox;
        const int o = b.vobj[v];
        const uint32_t vb = b.obj_vox[o], ve = b.obj_vox[o + 1];
        const float4* T = b.tri[l];
        const uint32_t* VT = b.vtri[l];
        if (VT[vb] == VT[ve]) continue;  // the object has no triangle at this LOD
        const float4* S = b.tri[4];
        const uint32_t s0 = b.vtri[4][v], s1 = b.vtri[4][v + 1];
        for (uint32_t base = s0 + 32 * part; base < s1; base += 32u << b.share) {
            const int n = (int)min(32u, s1 - base);
            unsigned evals = 0;
            __syncwarp();
            if (lane < n) {
                const D3 a = vert(S, base + lane, 0), c1 = vert(S, base + lane, 1), c2 = vert(S, base + lane, 2);
                Q.q[0][0][lane] = (a.x + c1.x + c2.x) * (1.0 / 3.0);
                Q.q[0][1][lane] = (a.y + c1.y + c2.y) * (1.0 / 3.0);
                Q.q[0][2][lane] = (a.z + c1.z + c2.z) * (1.0 / 3.0);
            }
            __syncwarp();
            search<1>(Q, n, T, VT, b.box[l], vb, ve, (uint32_t)v, lane, evals);
            __syncwarp();
            if (lane < n) {
                const unsigned bi = Q.best_i[lane];
                ++queries;
                if (bi != UINT_MAX) {
                    const D3 a = vert(T, bi, 0), c1 = vert(T, bi, 1), c2 = vert(T, bi, 2);
                    double m = 0;
#pragma unroll 1
                    for (int k = 0; k < 3; ++k) m = pd::dmax(m, point_tri2(vert(S, base + lane, k), a, c1, c2));
                    evals += 3;
                    atomicMax(reinterpret_cast<unsigned*>(const_cast<float*>(&T[3 * (size_t)bi].w)),
                              __float_as_uint(__double2float_ru(sqrt(m))));
                }
            }
            all += evals;
        }
    }
    all = warp_sum(all);
    queries = warp_sum(queries);
    if (lane == 0) {
        atomicAdd(&b.counters[0], all);
        atomicAdd(&b.counters[1], queries);
    }
}

// h: every LOD-l triangle of voxel v, cut into pieces, each piece's nearest
// LOD-100 facet by the largest corner distance
__global__ void __launch_bounds__(kBoundsThreads, kBoundsBlocksPerSm) k_hausdorff(BoundsDev b) {
    __shared__ Search<3> warps_s[kBoundsThreads / 32];
    Search<3>& Q = warps_s[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    const long warps = ((long)gridDim.x * blockDim.x) >> 5;
    unsigned long long all = 0, npieces = 0;
    for (long w = ((long)blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < (4 * b.n_vox) << b.share; w += warps) {
        const long it = w >> b.share;
        const int part = (int)(w - (it << b.share));
        const int l = (int)(it / b.n_vox);
        const long v = it - (long)l * b.n_vox;
        const int o = b.vobj[v];
        const uint32_t vb = b.obj_vox[o], ve = b.obj_vox[o + 1];
        const float4* T = b.tri[l];
        const float4* S = b.tri[4];
        const uint32_t* VS = b.vtri[4];
        if (VS[vb] == VS[ve]) continue;  // no surface: the bounds stay 0
        const double e0 = b.e0[o];
        const uint32_t t1 = b.vtri[l][v + 1];
        for (uint32_t tb = b.vtri[l][v]; tb < t1; tb += 32) {
            // 32 triangles: their subdivision depths, and their pieces in one row
            int dep = 0;
            if (tb + lane < t1) {
                const D3 a = vert(T, tb + lane, 0), c1 = vert(T, tb + lane, 1), c2 = vert(T, tb + lane, 2);
                const double L = pd::dmax(pd::dist(a, c1), pd::dmax(pd::dist(c1, c2), pd::dist(c2, a)));
                while (dep < 3 && L / (double)(1 << dep) > 1.5 * e0) ++dep;
            }
            const int np = tb + lane < t1 ? 1 << (2 * dep) : 0;
            int end = np;
#pragma unroll
            for (int o2 = 1; o2 < 32; o2 <<= 1) {
                const int x = __shfl_up_sync(0xffffffffu, end, o2);
                if (lane >= o2) end += x;
            }
            const int total = __shfl_sync(0xffffffffu, end, 31);
            for (int p0 = 32 * part; p0 < total; p0 += 32 << b.share) {
                const int n = min(32, total - p0);
                const int at = min(p0 + lane, total - 1);
                int src = 0;  // the triangle of piece `at`: the first whose pieces end after it
#pragma unroll
                for (int step = 16; step > 0; step >>= 1)
                    if (__shfl_sync(0xffffffffu, end, src + step - 1) <= at) src += step;
                const int dp = __shfl_sync(0xffffffffu, dep, src);
                const int p = at - (__shfl_sync(0xffffffffu, end, src) - (1 << (2 * dp)));
                const uint32_t t = tb + src;
                __syncwarp();
                if (lane < n) {
                    const D3 a = vert(T, t, 0), c1 = vert(T, t, 1), c2 = vert(T, t, 2);
                    D3 w0{1, 0, 0}, w1{0, 1, 0}, w2{0, 0, 1};
                    for (int lvl = 0; lvl < dp; ++lvl) {
                        const int ch = (p >> (2 * (dp - 1 - lvl))) & 3;
                        const D3 m01{(w0.x + w1.x) * 0.5, (w0.y + w1.y) * 0.5, (w0.z + w1.z) * 0.5};
                        const D3 m12{(w1.x + w2.x) * 0.5, (w1.y + w2.y) * 0.5, (w1.z + w2.z) * 0.5};
                        const D3 m20{(w2.x + w0.x) * 0.5, (w2.y + w0.y) * 0.5, (w2.z + w0.z) * 0.5};
                        if (ch == 0) { w1 = m01; w2 = m20; }
                        else if (ch == 1) { w0 = w1; w1 = m12; w2 = m01; }
                        else if (ch == 2) { w0 = w2; w1 = m20; w2 = m12; }
                        else { w0 = m01; w1 = m12; w2 = m20; }
                    }
                    const D3 W[3] = {w0, w1, w2};
#pragma unroll
                    for (int k = 0; k < 3; ++k) {
                        Q.q[k][0][lane] = a.x * W[k].x + c1.x * W[k].y + c2.x * W[k].z;
                        Q.q[k][1][lane] = a.y * W[k].x + c1.y * W[k].y + c2.y * W[k].z;
                        Q.q[k][2][lane] = a.z * W[k].x + c1.z * W[k].y + c2.z * W[k].z;
                    }
                }
                __syncwarp();
                unsigned evals = 0;
                search<3>(Q, n, S, VS, b.box[4], vb, ve, (uint32_t)v, lane, evals);
                __syncwarp();
                // the largest over the triangle's pieces: the root and the rounding up are monotone
                if (lane < n)
                    atomicMax(reinterpret_cast<unsigned*>(const_cast<float*>(&T[3 * (size_t)t + 1].w)),
                              __float_as_uint(__double2float_ru(sqrt(__longlong_as_double((long long)Q.best[lane])))));
                all += evals;
            }
            if (lane == 0 && part == 0) npieces += total;
        }
    }
    all = warp_sum(all);
    if (lane == 0) {
        atomicAdd(&b.counters[0], all);
        atomicAdd(&b.counters[2], npieces);
    }
}

// object-level values: per LOD the largest hausdorff and proxy bound (0 at LOD 100)
__global__ void k_object_bounds(BoundsDev b, float* obj_hd, float* obj_phd) {
    const int lane = threadIdx.x & 31;
    const long warps = ((long)gridDim.x * blockDim.x) >> 5;
    for (long it = ((long)blockIdx.x * blockDim.x + threadIdx.x) >> 5; it < kNumLods * b.n_obj; it += warps) {
        const long o = it / kNumLods;
        const int l = (int)(it - o * kNumLods);
        float mh = 0.f, mp = 0.f;
        if (l < kNumLods - 1) {
            const uint32_t t0 = b.vtri[l][b.obj_vox[o]], t1 = b.vtri[l][b.obj_vox[o + 1]];
            for (uint32_t t = t0 + lane; t < t1; t += 32) {
                mp = fmaxf(mp, b.tri[l][3 * (size_t)t].w);
                mh = fmaxf(mh, b.tri[l][3 * (size_t)t + 1].w);
            }
#pragma unroll
            for (int k = 16; k > 0; k >>= 1) {
                mp = fmaxf(mp, __shfl_xor_sync(0xffffffffu, mp, k));
                mh = fmaxf(mh, __shfl_xor_sync(0xffffffffu, mh, k));
            }
        }
        if (lane == 0) {
            obj_hd[o * kNumLods + l] = mh;
            obj_phd[o * kNumLods + l] = mp;
        }
    }
}

__global__ void k_gather_bounds(const float4* __restrict__ tri, size_t n, float2* __restrict__ out) {
    for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < n; t += (size_t)gridDim.x * blockDim.x)
        out[t] = make_float2(tri[3 * t].w, tri[3 * t + 1].w);
}

}  // namespace

cudaError_t launch_gather_bounds(const float4* tri, size_t n, float* out, cudaStream_t s) {
    if (!n) return cudaSuccess;
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    k_gather_bounds<<<sms * 8, 256, 0, s>>>(tri, n, reinterpret_cast<float2*>(out));
    return cudaGetLastError();
}

int bounds_scratch(tdp_ctx* ctx, const BoundRecords& r) {
    int rc;
    if ((rc = ensure(ctx, ctx->scratch[kBoxes], (size_t)kNumLods * r.n_vox * 2 * sizeof(float4)))) return rc;
    if ((rc = ensure(ctx, ctx->scratch[kVobj], (size_t)r.n_vox * sizeof(int)))) return rc;
    if ((rc = ensure(ctx, ctx->scratch[kMeanEdge], (size_t)r.n_obj * sizeof(double)))) return rc;
    return ensure(ctx, ctx->scratch[kBoundCounters], 4 * sizeof(unsigned long long));
}

void bounds_scratch_free(tdp_ctx* ctx) {
    for (int k = kBoxes; k <= kBoundCounters; ++k) {
        Buf& b = ctx->scratch[k];
        if (b.p) dfree(ctx, b.p);
        b = Buf{};
    }
}

const unsigned long long* bounds_counters(const tdp_ctx* ctx) {
    return (const unsigned long long*)ctx->scratch[kBoundCounters].p;
}

cudaError_t launch_bounds(tdp_ctx* ctx, const BoundRecords& r) {
    cudaStream_t s = ctx->stream;
    BoundsDev b{};
    float4* boxes = (float4*)ctx->scratch[kBoxes].p;
    for (int l = 0; l < kNumLods; ++l) {
        b.tri[l] = r.tri[l];
        b.vtri[l] = r.vtri[l];
        b.box[l] = boxes + (size_t)l * r.n_vox * 2;
    }
    b.obj_vox = r.obj_vox;
    b.vobj = (const int*)ctx->scratch[kVobj].p;
    b.e0 = (const double*)ctx->scratch[kMeanEdge].p;
    b.n_vox = r.n_vox;
    b.n_obj = r.n_obj;
    b.counters = (unsigned long long*)ctx->scratch[kBoundCounters].p;
    cudaError_t e = cudaMemsetAsync(b.counters, 0, 4 * sizeof(unsigned long long), s);
    if (e != cudaSuccess) return e;
    const int small_grid = ctx->num_sms * 8;
    for (int l = 0; l < kNumLods; ++l) {
        if (r.n_tris[l]) k_zero_bounds<<<small_grid, 256, 0, s>>>(r.tri[l], r.n_tris[l]);
        k_voxel_boxes<<<small_grid, 128, 0, s>>>(r.tri[l], r.vtri[l], r.n_vox, boxes + (size_t)l * r.n_vox * 2);
    }
    k_objects<<<(int)std::min<long>((r.n_obj + 3) / 4, (long)ctx->num_sms * 16), 128, 0, s>>>(
        b, (int*)ctx->scratch[kVobj].p, (double*)ctx->scratch[kMeanEdge].p);
    const int grid = ctx->num_sms * kBoundsBlocksPerSm;
    // Few voxels: several warps an item (every batch of 32 queries stands alone),
    // so that a warp has four to eight parts and the last ones end together (6
    // vessels, 4,844 items for 2,368 warps: 9.1 ms with a warp an item,
    // 6.3 with two).
    const long warps = (long)grid * kBoundsThreads / 32;
    while (b.share < 3 && (4 * r.n_vox) << b.share < 4 * warps) ++b.share;
    k_proxy<<<grid, kBoundsThreads, 0, s>>>(b);
    k_hausdorff<<<grid, kBoundsThreads, 0, s>>>(b);
    k_object_bounds<<<small_grid, 256, 0, s>>>(b, r.obj_hd, r.obj_phd);
    return cudaGetLastError();
}

}  // namespace tdp

using namespace tdp;

extern "C" int tdp_tile_compute_bounds(tdp_ctx* ctx, tdp_tile* tile, tdp_bounds_info* info) {
    if (!ctx || !tile) return TDP_ERR_ARG;
    if (tile->device != ctx->device) return fail(ctx, TDP_ERR_ARG, "tile lives on another device");
    if (info) std::memset(info, 0, sizeof(*info));
    cudaSetDevice(ctx->device);
    cudaStream_t s = ctx->stream;
    const long nv = tile->n_vox, no = tile->n_obj;
    if (no == 0 || nv == 0) return TDP_OK;
    BoundRecords r{};
    for (int l = 0; l < kNumLods; ++l) {
        r.tri[l] = tile->tri[l];
        r.vtri[l] = tile->vtri[l];
        r.n_tris[l] = tile->host.n_tris[l];
    }
    r.obj_vox = tile->obj_vox;
    r.n_vox = nv;
    r.n_obj = no;
    r.obj_hd = tile->obj_hd;
    r.obj_phd = tile->obj_phd;
    if (const int rc = bounds_scratch(ctx, r)) return rc;
#define CU(x) do { cudaError_t _e = (x); if (_e != cudaSuccess) return fail(ctx, TDP_ERR_CUDA, std::string(#x) + ": " + cudaGetErrorString(_e)); } while (0)
    // an attached tile first fetches every voxel: the bounds are written into
    // the device records, which later fetches must not overwrite
    CU(launch_fetch_all(lazy_view(tile), ctx->num_sms, s));
    CU(cudaEventRecord(ctx->ev[0], s));
    CU(launch_bounds(ctx, r));
    CU(cudaEventRecord(ctx->ev[1], s));
    unsigned long long cnt[4] = {0, 0, 0, 0};
    CU(cudaMemcpyAsync(cnt, bounds_counters(ctx), sizeof(cnt), cudaMemcpyDeviceToHost, s));
    tile->host.obj_hd.resize((size_t)no * kNumLods);
    tile->host.obj_phd.resize((size_t)no * kNumLods);
    CU(cudaMemcpyAsync(tile->host.obj_hd.data(), tile->obj_hd, (size_t)no * kNumLods * 4, cudaMemcpyDeviceToHost, s));
    CU(cudaMemcpyAsync(tile->host.obj_phd.data(), tile->obj_phd, (size_t)no * kNumLods * 4, cudaMemcpyDeviceToHost, s));
    CU(cudaStreamSynchronize(s));
#undef CU
    if (info) {
        float ms = 0;
        cudaEventElapsedTime(&ms, ctx->ev[0], ctx->ev[1]);
        info->ms = ms;
        info->objects = no;
        long tris = 0;
        for (int l = 0; l < kNumLods - 1; ++l) tris += (long)tile->host.n_tris[l];
        info->triangles = tris;
        info->dist_evals = (double)cnt[0];
        info->facet_queries = (long)cnt[1];
        info->pieces = (long)cnt[2];
    }
    return TDP_OK;
}
