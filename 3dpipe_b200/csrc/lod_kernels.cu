// lod_kernels.cu -- one LOD of the tuned join as a chain of task kernels.
//
// The same decisions as the one-warp-per-voxel-pair refine (refine.cu) with
// k_apply_results and k_pair_update behind it: every bound and distance that a
// decision reads has the same bits; a voxel pair's error term is another sound
// one (k_lod_cull).  What differs is which triangle pairs are looked at.
//
// A decision reads, of a pair's voxel pairs, only the smallest upper bound
// (d + h1 + h2) of the pair and each voxel pair's own lower bound
// (max(d - ph1 - ph2, 0)) where it falls below the one it had.  So a triangle
// pair matters only if its upper bound can come below the pair's running one
// (the cap, shared by all voxel pairs of the object pair in device memory) or
// its lower bound below the voxel pair's.  At the last LOD only the pair's
// smallest distance matters, and every voxel pair within the FP32 error band
// of it (those are kept for the FP64 recheck).
//
//   k_lod_items     the LOD's items (voxel pairs still alive), the caps'
//                   first values, the voxels in use
//   k_lod_clusters  per voxel in use: its triangles in clusters of 8, each a
//                   flat disc (centre, radius across its normal, half
//                   thickness along it) with the largest ph and smallest h,
//                   and the exact box of the voxel's triangles
//   k_lod_seed      first LOD only: the most promising cluster pair of each
//                   item lowers its pair's cap to near its final value
//   k_lod_cull      the cluster pairs that can matter go to a queue in device
//                   memory
//   k_lod_test      half a warp tests a queued cluster pair's 64 triangle pairs
//                   by their exact extents along the line of the two centres
//   k_lod_eval      what is left is evaluated 32 at a time, one triangle pair a
//                   lane, whichever items they belong to
//   k_lod_update    the pair's bounds, evictions, the within decision
//
// One warp per voxel pair spent half of its issue slots on staging bounds and
// culling against loose per-item minima, and a LOD of few voxel pairs took as
// long as its slowest one.  Here most items end after one pass over cluster
// pairs and the rest of the work is spread over the chip.  The loop's refine on
// one B200 (kernels between a LOD's items and its update, five LODs), with one
// warp per voxel pair (configuration 0 of it) and with this file:
//   10-NN, 20,000 nuclei x 100 vessels   30.5 -> 2.9 ms (137 M full evaluations -> 1.9 M)
//   10-NN self-join, 3,000 nuclei        35.7 -> 3.7 ms (158 M -> 2.4 M)
//   within 60 self-join, 4,181 nuclei    2.87 -> 0.52 ms
//   within 150, 2,000 x 100              1.28 -> 0.22 ms
//   within 400, 20,000 x 100             0.51 -> 0.17 ms
// Evaluating inside the kernel that tests the triangle pairs (128 registers,
// 16 warps per SM) took 2.4 times the two kernels' time: the tests wait for
// loads and want many warps, the evaluations want registers.

#include <float.h>

#include <algorithm>

#include "cull.cuh"
#include "lod_kernels.cuh"
#include "pair_rules.cuh"
#include "task_queue.cuh"
#include "tridist.cuh"

namespace tdp {
namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kClF4 = 3;  // float4 records of a cluster: (c, r) (n, t) (ph, h, -, -)

// how the bounds of a pass are formed
enum Mode {
    kTriH,    // level 2: each triangle's own Hausdorff values
    kObjH,    // levels 0 and 1: the objects' values (0 at level 0)
    kLast,    // the last LOD: the distance itself
};


__device__ __forceinline__ float sqrt_up(float x) { return radius_sqrt(fmaxf(x, 0.f)); }

// ---------------------------------------------------------------- init
__global__ void __launch_bounds__(256) k_lod_init(LodDev L, unsigned* words, int n_words, unsigned long long* dstats,
                                                  size_t caps, size_t best, size_t flags, size_t zero) {
    const size_t i0 = blockIdx.x * (size_t)blockDim.x + threadIdx.x, step = (size_t)gridDim.x * blockDim.x;
    if (i0 < (size_t)n_words) words[i0] = 0;
    if (i0 == 0) *dstats = 0;
    for (size_t i = i0; i < caps; i += step) L.pcap[i] = __uint_as_float(0x7f7f7f7fu);  // above any bound; pd too
    for (size_t i = i0; i < best; i += step) {
        L.pbest[i] = ~0ull;
        L.dir[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    for (size_t i = i0; i < flags; i += step) L.flag1[i] = -1;  // flag2 too
    for (size_t i = i0; i < zero; i += step) L.ctr[i] = 0;      // pown and pmiss too
}

// ---------------------------------------------------------------- items
// One thread per voxel pair.  A pair all of whose voxel pairs, once refined,
// are refined at every later LOD has one cap (its smallest upper bound can
// only fall); a voxel that is empty at a later LOD breaks that, and its pairs
// keep a cap per voxel pair (in vmx) instead.
__global__ void __launch_bounds__(256) k_lod_items(LodDev L, int k) {
    __shared__ unsigned cnt[8];
    __shared__ unsigned long long tps[8];
    __shared__ unsigned first;
    const JoinDev& d = L.d;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    unsigned* ctr = L.ctr + k * kLodCtrWords;
    // whole blocks step together: one slot claim and one sum per block
    for (int64_t v0 = blockIdx.x * (int64_t)blockDim.x; v0 < d.V; v0 += (int64_t)gridDim.x * blockDim.x) {
        const int64_t v = v0 + threadIdx.x;
        int p = 0, a = 0, b = 0;
        bool ok = false;
        if (v < d.V) {
            p = d.vpair[v];
            ok = d.valive[v] && d.pstat[p] == kUndecided;
        }
        uint32_t o1 = 0, n1 = 0, o2 = 0, n2 = 0;
        if (ok) {
            a = d.vpa[v];
            b = d.vpb[v];
            if (k == 0) {
                bool seen = false, bad = false;
                for (int m = 0; m < L.nl; ++m) {
                    const bool full = L.vt1[m][a + 1] > L.vt1[m][a] && L.vt2[m][b + 1] > L.vt2[m][b];
                    bad = bad || (seen && !full);
                    seen = seen || full;
                }
                if (bad) L.pown[p] = 1;
            }
            o1 = L.vt1[k][a]; n1 = L.vt1[k][a + 1] - o1;
            o2 = L.vt2[k][b]; n2 = L.vt2[k][b + 1] - o2;
            ok = n1 > 0 && n2 > 0;
        }
        const unsigned m = __ballot_sync(kFull, ok);
        unsigned long long tp = ok ? (unsigned long long)n1 * n2 : 0ull;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) tp += __shfl_xor_sync(kFull, tp, o);
        if (lane == 0) {
            cnt[wid] = __popc(m);
            tps[wid] = tp;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            unsigned c = 0;
            unsigned long long t = 0;
            for (int i = 0; i < 8; ++i) {
                const unsigned ci = cnt[i];
                cnt[i] = c;
                c += ci;
                t += tps[i];
            }
            if (c) {
                first = atomicAdd(L.n_items + k, c);
                atomicAdd(L.tri_pairs, t);
            }
        }
        __syncthreads();
        if (ok) {
            const unsigned w = first + cnt[wid] + __popc(m & ((1u << lane) - 1u));
            L.items[w] = RefineItem{o1, n1, o2, n2};
            L.ext[w] = make_int4((int)v, p, (int)cluster_base(o1, a), (int)cluster_base(o2, b));
            L.vox[w] = make_int2(a, b);
            // a voxel pair refined for the first time brings its core distance;
            // at the first LOD the pair's closest cores also name its seed
            const unsigned c = __float_as_uint(d.vmx[v]);
            if (k == 0) atomicMin(L.pbest + p, ((unsigned long long)c << 32) | w);
            else if (d.vupd[v] < 0) atomicMin((unsigned*)L.pcap + p, c);
        }
        if (m) {
            lod_claim(ok, a, k, L.flag1, L.list1, ctr + cList1, lane);
            if (L.self) lod_claim(ok, b, k, L.flag1, L.list1, ctr + cList1, lane);
            else lod_claim(ok, b, k, L.flag2, L.list2, ctr + cList2, lane);
        }
    }
}

// ---------------------------------------------------------------- clusters
__device__ __forceinline__ float grp8_sum(float v) {
#pragma unroll
    for (int o = 1; o < kCl; o <<= 1) v += __shfl_xor_sync(kFull, v, o);
    return v;
}

// One warp per voxel in use.
__global__ void __launch_bounds__(256) k_lod_clusters(LodDev L, int k) {
    const int lane = threadIdx.x & 31;
    const unsigned* ctr = L.ctr + k * kLodCtrWords;
    const unsigned n1 = ctr[cList1], n = n1 + (L.self ? 0u : ctr[cList2]);
    const unsigned nw = (gridDim.x * blockDim.x) >> 5;
    for (unsigned t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; t < n; t += nw) {
        const bool one = t < n1;
        const int vx = one ? L.list1[t] : L.list2[t - n1];
        const uint32_t* vt = one ? L.vt1[k] : L.vt2[k];
        const float4* tri = one ? L.tri1[k] : L.tri2[k];
        const uint32_t off = vt[vx], cnt = vt[vx + 1] - off;
        float4* cl = (one ? L.cl1 : L.cl2) + kClF4 * cluster_base(off, vx);
        float blx = FLT_MAX, bly = FLT_MAX, blz = FLT_MAX, bhx = -FLT_MAX, bhy = -FLT_MAX, bhz = -FLT_MAX;
        for (uint32_t base = 0; base < cnt; base += 32) {
            const bool ok = base + lane < cnt;
            // a missing triangle repeats the chunk's last one
            const float4* tp = tri + ((size_t)off + min(base + lane, cnt - 1)) * kTriF4;
            const float4 t0 = tp[0], t1 = tp[1], t2 = tp[2];
            const float lx = fminf(t0.x, fminf(t1.x, t2.x)), hx = fmaxf(t0.x, fmaxf(t1.x, t2.x));
            const float ly = fminf(t0.y, fminf(t1.y, t2.y)), hy = fmaxf(t0.y, fmaxf(t1.y, t2.y));
            const float lz = fminf(t0.z, fminf(t1.z, t2.z)), hz = fmaxf(t0.z, fmaxf(t1.z, t2.z));
            blx = fminf(blx, lx); bly = fminf(bly, ly); blz = fminf(blz, lz);
            bhx = fmaxf(bhx, hx); bhy = fmaxf(bhy, hy); bhz = fmaxf(bhz, hz);
            const float cx = 0.5f * (grp8_min(lx) + grp8_max(hx)), cy = 0.5f * (grp8_min(ly) + grp8_max(hy)),
                        cz = 0.5f * (grp8_min(lz) + grp8_max(hz));
            const float ex = t1.x - t0.x, ey = t1.y - t0.y, ez = t1.z - t0.z;
            const float fx = t2.x - t0.x, fy = t2.y - t0.y, fz = t2.z - t0.z;
            float nx = grp8_sum(ey * fz - ez * fy), ny = grp8_sum(ez * fx - ex * fz), nz = grp8_sum(ex * fy - ey * fx);
            const float nn = nx * nx + ny * ny + nz * nz;
            const float inv = nn > 1e-30f && nn < 1e30f ? rsqrtf(nn) : 0.f;  // no direction: a plain sphere
            nx *= inv; ny *= inv; nz *= inv;
            float w2 = 0.f, r2 = 0.f, th = 0.f;
            const float4 vv[3] = {t0, t1, t2};
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                const float x = vv[q].x - cx, y = vv[q].y - cy, z = vv[q].z - cz;
                const float s = x * nx + y * ny + z * nz, l2 = x * x + y * y + z * z;
                w2 = fmaxf(w2, l2);
                r2 = fmaxf(r2, l2 - s * s);
                th = fmaxf(th, fabsf(s));
            }
            w2 = grp8_max(w2);
            r2 = grp8_max(r2);
            th = grp8_max(th);
            const float ph = grp8_max(t0.w), h = grp8_min(t1.w);
            // inflated so that FP32 rounding keeps every vertex inside
            const float wl = sqrt_up(w2);
            if ((lane & (kCl - 1)) == 0 && ok) {
                float4* c = cl + (size_t)kClF4 * ((base + lane) / kCl);
                c[0] = make_float4(cx, cy, cz, sqrt_up(r2 + 1e-6f * w2) * 1.0001f + 1e-6f);
                c[1] = make_float4(nx, ny, nz, th * 1.0001f + 1e-5f * wl + 1e-6f);
                c[2] = make_float4(ph, h, 0.f, 0.f);
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            blx = fminf(blx, __shfl_xor_sync(kFull, blx, o));
            bly = fminf(bly, __shfl_xor_sync(kFull, bly, o));
            blz = fminf(blz, __shfl_xor_sync(kFull, blz, o));
            bhx = fmaxf(bhx, __shfl_xor_sync(kFull, bhx, o));
            bhy = fmaxf(bhy, __shfl_xor_sync(kFull, bhy, o));
            bhz = fmaxf(bhz, __shfl_xor_sync(kFull, bhz, o));
        }
        if (lane == 0) {
            float4* vb = (one ? L.vb1 : L.vb2) + 2 * (size_t)vx;
            vb[0] = make_float4(blx, bly, blz, 0.f);
            vb[1] = make_float4(bhx, bhy, bhz, 0.f);
        }
    }
}

// A lower bound of the distance of two clusters: the gap, along the line of
// their centres, between their extents (a disc of radius r and half thickness
// t with normal n reaches r sin + t cos from its centre).
struct Cluster {
    float4 s, n;
    float ph, h;
};
__device__ __forceinline__ Cluster load_cluster(const float4* __restrict__ c) {
    const float4 x = c[2];
    return Cluster{c[0], c[1], x.x, x.y};
}
__device__ __forceinline__ float cluster_gap(const Cluster& a, const Cluster& b) {
    const float x = b.s.x - a.s.x, y = b.s.y - a.s.y, z = b.s.z - a.s.z;
    const float d2 = x * x + y * y + z * z;
    const float inv = rsqrtf(fmaxf(d2, 1e-30f));
    const float ca = (a.n.x * x + a.n.y * y + a.n.z * z) * inv, cb = (b.n.x * x + b.n.y * y + b.n.z * z) * inv;
    // 2e-6: the rounding of the cosines, so that sin is never taken too small
    const float ra = a.s.w * sqrt_up(1.000002f - ca * ca) + a.n.w * fabsf(ca);
    const float rb = b.s.w * sqrt_up(1.000002f - cb * cb) + b.n.w * fabsf(cb);
    return d2 * inv - ra - rb;
}

// a gap widened by triangles' own Hausdorff values: (upper bound's, lower bound's)
template <int MODE>
__device__ __forceinline__ float2 widen(float gap, const Cluster& a, const Cluster& b) {
    return MODE == kTriH ? make_float2(gap + a.h + b.h, gap - a.ph - b.ph) : make_float2(gap, gap);
}

// kObjH: what is added for the upper bound (x, y, one after the other) and
// taken off for the lower one (z, in all).  Level 0 has no lower bound.
__device__ __forceinline__ float3 object_h(const LodDev& L, int p, int k) {
    if (L.level == 0) return make_float3(0.f, 0.f, -INFINITY);
    const int q = L.d.pq[p], t = L.d.pt[p], li = L.li[k];
    return make_float3(L.d.ophd1[q * 5 + li], L.d.ophd2[t * 5 + li], L.d.ohd1[q * 5 + li] + L.d.ohd2[t * 5 + li]);
}

// the running thresholds of an item: (cap, lower bound)
template <int MODE>
__device__ __forceinline__ float2 thresholds(const LodDev& L, int v, int p, float slack, float preset) {
    if (MODE == kLast) {
        // the pair's cap stands in until a distance below it is found
        float d = __ldcg(L.pd + p);
        if (!(L.pown[p] || L.pmiss[p])) d = fminf(d, L.pcap[p]);
        return make_float2(fminf(d + slack, preset), -INFINITY);
    }
    const float* cap = L.pown[p] ? L.d.vmx + v : L.pcap + p;
    return make_float2(__ldcg(cap), MODE == kObjH && L.level == 0 ? -INFINITY : __ldcg(L.d.vmn + v));
}
// the same, with the item's margin, on the scale of a widened gap; a bound that
// is not at or above its limit (NaN too) matters
template <int MODE>
__device__ __forceinline__ float2 gap_limits(const LodDev& L, int k, int p, float2 th, float mg) {
    float zt = th.x + mg, yt = th.y + mg;
    if (MODE == kObjH) {
        const float3 oh = object_h(L, p, k);
        zt -= oh.x + oh.y;
        yt += oh.z;
    }
    return make_float2(zt, yt);
}
__device__ __forceinline__ bool lower_to(float* at, float x) {
    if (!(x < __ldcg(at))) return false;
    return atomicMin((unsigned*)at, __float_as_uint(x)) > __float_as_uint(x);
}

// from the middle of triangle A to the middle of triangle B
__device__ __forceinline__ float4 tri_to_tri(const PreTri<float>& A, const PreTri<float>& B) {
    return make_float4(B.v[0].x + B.v[1].x + B.v[2].x - A.v[0].x - A.v[1].x - A.v[2].x,
                       B.v[0].y + B.v[1].y + B.v[2].y - A.v[0].y - A.v[1].y - A.v[2].y,
                       B.v[0].z + B.v[1].z + B.v[2].z - A.v[0].z - A.v[1].z - A.v[2].z, 0.f);
}

// largest |coordinate| of both voxels relative to o: rounding x - o is
// monotone in x, so the voxels' exact boxes give exactly the refine's value
__device__ __forceinline__ float item_rmax(const float4 alo, const float4 ahi, const float4 blo, const float4 bhi,
                                           const float4 o) {
    float r = fmaxf(fabsf(alo.x - o.x), fabsf(ahi.x - o.x));
    r = fmaxf(r, fmaxf(fabsf(alo.y - o.y), fabsf(ahi.y - o.y)));
    r = fmaxf(r, fmaxf(fabsf(alo.z - o.z), fabsf(ahi.z - o.z)));
    r = fmaxf(r, fmaxf(fabsf(blo.x - o.x), fabsf(bhi.x - o.x)));
    r = fmaxf(r, fmaxf(fabsf(blo.y - o.y), fabsf(bhi.y - o.y)));
    return fmaxf(r, fmaxf(fabsf(blo.z - o.z), fabsf(bhi.z - o.z)));
}

__device__ __forceinline__ void pre_rel(const float4* __restrict__ t, float4 o, PreTri<float>& P, float& ph, float& h) {
    const float4 t0 = t[0], t1 = t[1], t2 = t[2];
    pretri(P, v3(t0.x - o.x, t0.y - o.y, t0.z - o.z), v3(t1.x - o.x, t1.y - o.y, t1.z - o.z),
           v3(t2.x - o.x, t2.y - o.y, t2.z - o.z));
    ph = t0.w;
    h = t1.w;
}

__device__ __forceinline__ void pre_rel64(const float4* __restrict__ t, float4 o, PreTri<double>& P) {
    const float4 a = t[0], b = t[1], c = t[2];
    const double ox = o.x, oy = o.y, oz = o.z;
    pretri(P, v3<double>(a.x - ox, a.y - oy, a.z - oz), v3<double>(b.x - ox, b.y - oy, b.z - oz),
           v3<double>(c.x - ox, c.y - oy, c.z - oz));
}

// Margin, slack and preset of an item (uniform over a warp).  The margin
// covers the FP32 error of a bound and of the distance it bounds.  At the
// last LOD a voxel pair whose minimum is within twice the pair's error of the
// smallest must keep its exact minimum (it may be rechecked in FP64); the
// objects' boxes bound the coordinates of all of them.
template <int MODE>
__device__ __forceinline__ void item_margins(const LodDev& L, const RefineItem& it, const int4& x, const int2& vx,
                                             int k, float& rmax, float& mg, float& slack, float& preset) {
    const float4 o4 = L.tri1[k][(size_t)it.a_off * kTriF4];
    const float4* va = L.vb1 + 2 * (size_t)vx.x;
    const float4* vb = (L.self ? L.vb1 : L.vb2) + 2 * (size_t)vx.y;
    rmax = item_rmax(va[0], va[1], vb[0], vb[1], o4);
    mg = err_bound(rmax) + 1e-6f;
    slack = 0.f;
    preset = FLT_MAX;
    if (MODE == kLast) {
        const float* qb = L.box1 + 6 * (size_t)L.d.pq[x.y];
        const float* tb = L.box2 + 6 * (size_t)L.d.pt[x.y];
        float R = rmax;
#pragma unroll
        for (int c = 0; c < 3; ++c)
            R = fmaxf(R, fmaxf(fmaxf(fabsf(tb[3 + c] - qb[c]), fabsf(tb[c] - qb[3 + c])), qb[3 + c] - qb[c]));
        slack = 2.f * err_bound(1.3f * R) + 2e-6f;
        if (L.use_preset) preset = within_preset(L.d, x.y, vx.x, vx.y, L.tau);
    }
}

// ---------------------------------------------------------------- seeds
constexpr int kEvalBlock = 128;

// One warp per undecided pair: the voxel pair with the closest cores is taken
// for the one that holds the closest points, and the nearest 32 triangle
// pairs of its nearest cluster pair are evaluated.
template <int MODE>
__global__ void __launch_bounds__(kEvalBlock, 4) k_lod_seed(LodDev L, int k) {
    const int lane = threadIdx.x & 31;
    const unsigned nw = (gridDim.x * blockDim.x) >> 5;
    const float4* cl2 = L.self ? L.cl1 : L.cl2;
    for (unsigned p = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; p < (unsigned)L.d.P; p += nw) {
        const unsigned long long pb = L.pbest[p];
        if (pb == ~0ull) continue;  // nothing to refine
        const unsigned w = (unsigned)pb;
        const RefineItem it = L.items[w];
        const int4 x = L.ext[w];
        const int2 vx = L.vox[w];
        const float core = __uint_as_float((unsigned)(pb >> 32));
        float rmax, mg, slack, preset;
        item_margins<MODE>(L, it, x, vx, k, rmax, mg, slack, preset);
        const float3 oh = MODE == kObjH ? object_h(L, x.y, k) : make_float3(0.f, 0.f, 0.f);
        const unsigned nA = (it.a_cnt + kCl - 1) / kCl, nB = (it.b_cnt + kCl - 1) / kCl;
        const unsigned long long tot = (unsigned long long)nA * nB;
        float best = INFINITY;
        unsigned bi = 0, bj = 0;
        unsigned i = 0, j = lane;  // t = i * nB + j
        i = j / nB;
        j -= i * nB;
        for (unsigned long long t = lane; t < tot; t += 32) {
            const Cluster a = load_cluster(L.cl1 + kClF4 * ((size_t)x.z + i)),
                          b = load_cluster(cl2 + kClF4 * ((size_t)x.w + j));
            const float z = widen<MODE>(cluster_gap(a, b), a, b).x;
            if (z < best) {
                best = z;
                bi = i;
                bj = j;
            }
            j += 32;
            while (j >= nB) {
                j -= nB;
                ++i;
            }
        }
        float m = best;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) m = fminf(m, __shfl_xor_sync(kFull, m, o));
        // every voxel pair's core distance is one of its upper bounds
        if (lane == 0 && !L.pown[p]) L.pcap[p] = core;
        if (!(m < core + mg + slack)) continue;
        const int src = __ffs(__ballot_sync(kFull, best == m)) - 1;
        bi = __shfl_sync(kFull, bi, src);
        bj = __shfl_sync(kFull, bj, src);
        // each lane takes the nearer of its two triangle pairs by their centres
        float4 along = make_float4(0.f, 0.f, 0.f, 0.f);
        const unsigned ia = bi * kCl + (lane & 7);
        const unsigned b0 = bj * kCl + (lane >> 3), b1 = b0 + 4;
        if (ia < it.a_cnt && b0 < it.b_cnt) {
            const float4* ta = L.tri1[k] + ((size_t)it.a_off + ia) * kTriF4;
            const float4* tb0 = L.tri2[k] + ((size_t)it.b_off + b0) * kTriF4;
            const float4* tb1 = b1 < it.b_cnt ? L.tri2[k] + ((size_t)it.b_off + b1) * kTriF4 : tb0;
            const float ax = ta[0].x + ta[1].x + ta[2].x, ay = ta[0].y + ta[1].y + ta[2].y, az = ta[0].z + ta[1].z + ta[2].z;
            const float ux = tb0[0].x + tb0[1].x + tb0[2].x - ax, uy = tb0[0].y + tb0[1].y + tb0[2].y - ay,
                        uz = tb0[0].z + tb0[1].z + tb0[2].z - az;
            const float vx2 = tb1[0].x + tb1[1].x + tb1[2].x - ax, vy = tb1[0].y + tb1[1].y + tb1[2].y - ay,
                        vz = tb1[0].z + tb1[1].z + tb1[2].z - az;
            const bool second = vx2 * vx2 + vy * vy + vz * vz < ux * ux + uy * uy + uz * uz;
            const float4* tb = second ? tb1 : tb0;
            along = second ? make_float4(vx2, vy, vz, 0.f) : make_float4(ux, uy, uz, 0.f);
            const float4 o4 = L.tri1[k][(size_t)it.a_off * kTriF4];
            PreTri<float> A, B;
            float pa, ha, pb, hb;
            pre_rel(ta, o4, A, pa, ha);
            pre_rel(tb, o4, B, pb, hb);
            const float dd = sqrtf(tri_dist2(A, B));
            best = MODE == kTriH ? dd + ha + hb : MODE == kObjH ? dd + oh.x + oh.y : dd;
        } else {
            best = FLT_MAX;
        }
        const float up = __uint_as_float(__reduce_min_sync(kFull, __float_as_uint(best >= 0.f ? best : FLT_MAX)));
        if (up < FLT_MAX && lane == __ffs(__ballot_sync(kFull, best == up)) - 1) L.dir[p] = along;
        if (lane == 0) {
            if (MODE == kLast) L.pd[p] = up;
            else if (!L.pown[p]) L.pcap[p] = fminf(core, up);
            else L.d.vmx[x.x] = fminf(L.d.vmx[x.x], up);
        }
    }
}

// One side's share of a pair's two bounds (the pair's are the sums of two).
struct TriSide {
    float z, y;
};

// ---------------------------------------------------------------- cull
constexpr int kCullWarps = 8;
constexpr int kCullBuf = 96;  // tasks a warp collects before it claims queue slots (>= 63 + 32)
constexpr int kSide = 16;     // clusters of one side that are looked at together

// Item w is evaluated whole.  (Looked at first: an item can have thousands of
// entries that do not fit.)
__device__ __forceinline__ void go_whole(const LodDev& L, unsigned* ctr, unsigned w) {
    int* in_over = (int*)&L.mg[w].w;
    if (__ldcg(in_over) == 0 && atomicExch(in_over, 1) == 0) L.over[atomicAdd(ctr + cOver, 1u)] = w;
}

// Queue `cnt` of the warp's collected tasks.  Items whose tasks find the
// queue full go to the list of items that are evaluated whole, once each.
__device__ __forceinline__ void flush_tasks(const LodDev& L, unsigned* ctr, const LodTask* buf, int cnt, int lane,
                                            QueueClaims& queue) {
    __syncwarp();
    const unsigned base = queue.claim((unsigned)cnt, L.task_cap, [&](unsigned n) {
        unsigned at = 0;
        if (lane == 0) at = atomicAdd(ctr + cTasks, n);
        return __shfl_sync(kFull, at, 0);
    });
    for (int i = lane; i < cnt; i += 32) {
        const LodTask t = buf[i];
        if (base + i < L.task_cap) L.tasks[base + i] = t;
        else go_whole(L, ctr, t.w);
    }
    __syncwarp();
}

// An item as the cull reads it: the pair's direction, where projections on it
// start (the item's origin), the thresholds on the scale of a widened gap.
struct alignas(16) CullItem {
    float ux, uy, uz, ox;
    float oy, oz, zt, yt;
    uint32_t ca, cb, n, w;  // first clusters, cluster counts (A | B << 16), item
};

// What a cluster adds to a pair's two bounds along direction u: A clusters
// reach up to their largest projection, B clusters down to their smallest.
template <int MODE>
__device__ __forceinline__ TriSide cluster_side(const Cluster& c, const CullItem& T, bool isA) {
    const float x = c.s.x - T.ox, y = c.s.y - T.oy, z = c.s.z - T.oz;
    const float pr = x * T.ux + y * T.uy + z * T.uz;
    const float cu = c.n.x * T.ux + c.n.y * T.uy + c.n.z * T.uz;
    const float reach = c.s.w * sqrt_up(1.000002f - cu * cu) + c.n.w * fabsf(cu);
    const float g = (isA ? -pr : pr) - reach;
    return MODE == kTriH ? TriSide{g + c.h, g - c.ph} : TriSide{g, g};
}

// the smaller of two shares; NaN wins, so that what cannot be bounded goes on
__device__ __forceinline__ float least_of(float a, float b) { return b < a || b != b ? b : a; }

// Batches of up to 32 items per warp, in three steps:
// 1. one item a lane: margins, thresholds, what the update reads of the item;
// 2. side by side (4, 8 or 16 lanes a side, so 4, 2 or 1 items at a time) every
//    cluster's share of the bounds along the pair's direction: an item ends
//    here when the least shares of both sides together do not matter, and of
//    the others only the clusters that do with the other side's least go on
//    (voxels of more than 16 clusters skip this);
// 3. those in pairs, one a lane, along the line of their own centres.
// One item a warp and every cluster pair of it took twice as long (10-NN
// self-join of 3,000 nuclei, five LODs: 1.95 -> 1.11 ms): each item waited for
// its own chain of loads.  Going on to the triangles in this kernel (each
// loaded once per item) was faster by a fifth where items keep 15 cluster
// pairs and slower everywhere else, most where a LOD has few items.
template <int MODE>
__global__ void __launch_bounds__(kCullWarps * 32) k_lod_cull(LodDev L, int k, int pass, const unsigned* n_items,
                                                                int stamp) {
    __shared__ LodTask bufs[kCullWarps][kCullBuf];
    __shared__ CullItem recs[kCullWarps][32];
    __shared__ uint8_t lists[kCullWarps][4][2][kSide];  // clusters that go on, per item of a step and side
    const JoinDev& d = L.d;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const unsigned lt = (1u << lane) - 1u;
    LodTask* buf = bufs[wid];
    CullItem* rec = recs[wid];
    int bn = 0;
    QueueClaims queue;
    unsigned* ctr = L.ctr + pass * kLodCtrWords;
    const unsigned n = *n_items;
    const unsigned nw = gridDim.x * kCullWarps, gw = blockIdx.x * kCullWarps + wid;
    const unsigned batch = max(1u, min(32u, (n + nw - 1) / nw));
    const float4* cl2 = L.self ? L.cl1 : L.cl2;
    for (unsigned w0 = gw * batch; w0 < n; w0 += nw * batch) {
        const unsigned cnt = min(batch, n - w0);
        unsigned most = 0;
        if (lane < cnt) {
            const unsigned w = w0 + lane;
            const RefineItem it = L.items[w];
            const int4 x = L.ext[w];
            const int2 vx = L.vox[w];
            float rmax, mg, slack, preset;
            item_margins<MODE>(L, it, x, vx, k, rmax, mg, slack, preset);
            const float2 th = thresholds<MODE>(L, x.x, x.y, slack, preset);
            const float4 o4 = L.tri1[k][(size_t)it.a_off * kTriF4];
            const float4 u = __ldcg(L.dir + x.y);
            const float u2 = u.x * u.x + u.y * u.y + u.z * u.z;
            const float inv = u2 > 1e-30f && u2 < 1e30f ? rsqrtf(u2) : 0.f;
            const unsigned nA = (it.a_cnt + kCl - 1) / kCl, nB = (it.b_cnt + kCl - 1) / kCl;
            const float2 lim = gap_limits<MODE>(L, k, x.y, th, mg);
            const bool big = nA > 0xffffu || nB > 0xffffu;  // indices do not fit a task
            rec[lane] = CullItem{u.x * inv, u.y * inv, u.z * inv, o4.x, o4.y, o4.z, lim.x, lim.y,
                                 (unsigned)x.z, (unsigned)x.w, big ? 0u : nA | (nB << 16), w};
            most = big ? 0u : max(nA, nB);
            L.mg[w] = make_float4(mg, slack, preset, __int_as_float(big ? 1 : 0));
            if (big) L.over[atomicAdd(ctr + cOver, 1u)] = w;
            const int v = x.x;
            const float e = err_bound(rmax);
            d.vupd[v] = stamp;
            if (MODE == kLast) {
                L.vres[v] = FLT_MAX;
                d.vmx[v] = e;  // read by the update, which then sets both bounds
            } else {
                if (MODE == kObjH) L.vres[v] = FLT_MAX;
                // The voxel pair's own upper bound enters only its error term
                // (4 u of it); where it is not kept, the middle between the
                // least it can be and its core distance stands in.  That is
                // sound: the term has to cover the bounds that a decision
                // takes from this voxel pair.  Its lower bound only falls from
                // mn; its upper bound is the pair's only where it is the least
                // of all, so at most th.x and at most every core distance, and
                // the middle is not below that.  (Not the bits of the one-warp
                // form's term, which its own minimum enters.)
                const float mn = d.vmn[v], core = __ldcg(d.vmx + v);
                const float mx = L.pown[x.y] ? core : 0.5f * (core + fminf(core, fmaxf(mn, th.x)));
                d.verr[v] = fmaxf(d.verr[v], e + 4.f * kUnitRoundoff * fmaxf(fabsf(mn), fabsf(mx)));
            }
        }
        most = __reduce_max_sync(kFull, most);
        const int lg = most <= 4 ? 2 : most <= 8 ? 3 : 4;  // lanes a side
        const int g = 1 << lg, per = kSide >> lg;          // items a step
        __syncwarp();
        for (unsigned s0 = 0; s0 < cnt; s0 += per) {
            const int slot = lane >> (lg + 1);
            const bool isA = !((lane >> lg) & 1);
            const int idx = lane & (g - 1);
            const bool live = s0 + slot < cnt;
            const CullItem& T = rec[live ? s0 + slot : s0];
            const unsigned nA = T.n & 0xffffu, nB = T.n >> 16;
            const unsigned cn = live ? (isA ? nA : nB) : 0u;
            const bool wide = live && max(nA, nB) > (unsigned)kSide;
            TriSide s{INFINITY, INFINITY};
            if ((unsigned)idx < cn)
                s = cluster_side<MODE>(load_cluster((isA ? L.cl1 + kClF4 * (size_t)T.ca : cl2 + kClF4 * (size_t)T.cb) +
                                                    kClF4 * (size_t)idx), T, isA);
            TriSide least = s;
#pragma unroll
            for (int o = 1; o < kSide; o <<= 1) {
                if (o < g) {
                    least.z = least_of(least.z, __shfl_xor_sync(kFull, least.z, o));
                    if (MODE != kLast) least.y = least_of(least.y, __shfl_xor_sync(kFull, least.y, o));
                }
            }
            const float oz = __shfl_xor_sync(kFull, least.z, g);
            const float oy = MODE == kLast ? 0.f : __shfl_xor_sync(kFull, least.y, g);
            const bool item_on = wide || (live && cn > 0 && (!(least.z + oz >= T.zt) || (MODE != kLast && !(least.y + oy >= T.yt))));
            const bool keep = item_on && (unsigned)idx < cn && (!(s.z + oz >= T.zt) || (MODE != kLast && !(s.y + oy >= T.yt)));
            const unsigned on = __ballot_sync(kFull, item_on);
            if (!on) continue;
            const unsigned km = __ballot_sync(kFull, keep);
            const unsigned sm = (km >> (lane & ~(g - 1))) & ((1u << g) - 1u);
            if (keep) lists[wid][slot][isA ? 0 : 1][__popc(sm & ((1u << idx) - 1u))] = (uint8_t)idx;
            __syncwarp();
            for (int sl = 0; sl < per; ++sl) {
                if (!((on >> (sl * 2 * g)) & 1u)) continue;
                const CullItem I = rec[s0 + sl];
                const unsigned iA = I.n & 0xffffu, iB = I.n >> 16;
                const bool all = max(iA, iB) > (unsigned)kSide;
                const unsigned rows = all ? iA : __popc((km >> (sl * 2 * g)) & ((1u << g) - 1u));
                const unsigned cols = all ? iB : __popc((km >> (sl * 2 * g + g)) & ((1u << g) - 1u));
                const unsigned total = rows * cols;
                unsigned r = lane / max(cols, 1u), c = lane - r * max(cols, 1u);
                for (unsigned t0 = 0; t0 < total; t0 += 32) {
                    bool go = t0 + lane < total;
                    LodTask t{I.w, 0, 0.f, 0.f};
                    if (go) {
                        const unsigned i = all ? r : lists[wid][sl][0][r], j = all ? c : lists[wid][sl][1][c];
                        const Cluster a = load_cluster(L.cl1 + kClF4 * ((size_t)I.ca + i)),
                                      b = load_cluster(cl2 + kClF4 * ((size_t)I.cb + j));
                        const float2 zy = widen<MODE>(cluster_gap(a, b), a, b);
                        t = LodTask{I.w, (i << 16) | j, zy.x, zy.y};
                        go = !(t.z >= I.zt) || (MODE != kLast && !(t.y >= I.yt));
                    }
                    const unsigned m = __ballot_sync(kFull, go);
                    if (go) buf[bn + __popc(m & lt)] = t;
                    bn += __popc(m);
                    if (bn >= 64) {
                        flush_tasks(L, ctr, buf, bn, lane, queue);
                        bn = 0;
                    }
                    c += 32;
                    while (c >= cols) {
                        c -= cols;
                        ++r;
                    }
                }
            }
            __syncwarp();
        }
        __syncwarp();
    }
    if (bn > 0) flush_tasks(L, ctr, buf, bn, lane, queue);
}

// ---------------------------------------------------------------- triangle tests
// A cluster pair on a half warp: lanes 0-7 hold the A triangles, lanes 8-15
// the B triangles, each its share of the two bounds of a triangle pair: A's
// largest and B's smallest projection on the line of the two centres (taken
// relative to the A cluster's centre), with the triangle's own Hausdorff
// values.  A pair's bound is the sum of its two sides.  Any direction gives a
// lower bound of the distance; along this one it is off only by the square of
// the angle to the closest points' direction.
struct alignas(16) TaskDir {
    float ux, uy, uz, ax;
    float ay, az, zt, yt;   // a pair matters when its z is below zt or its y below yt
    uint32_t a0, b0, n, w;  // first triangles, counts (A | B << 8), item
};

template <int MODE>
__device__ __forceinline__ TaskDir task_dir(const LodDev& L, const float4* cl2, unsigned w, unsigned ci, unsigned cj,
                                            float2 lim, const int4& x) {
    const RefineItem it = L.items[w];
    const float4 ca = L.cl1[kClF4 * ((size_t)x.z + ci)], cb = cl2[kClF4 * ((size_t)x.w + cj)];
    const float ux = cb.x - ca.x, uy = cb.y - ca.y, uz = cb.z - ca.z;
    const float u2 = ux * ux + uy * uy + uz * uz;
    const float inv = u2 > 0.f ? rsqrtf(u2) : 0.f;
    const unsigned na = min(8u, it.a_cnt - ci * kCl), nb = min(8u, it.b_cnt - cj * kCl);
    return TaskDir{ux * inv, uy * inv, uz * inv, ca.x, ca.y, ca.z, lim.x, lim.y,
                   it.a_off + ci * kCl, it.b_off + cj * kCl, na | (nb << 8), w};
}

template <int MODE>
__device__ __forceinline__ TriSide tri_side(const TaskDir& T, const float4* __restrict__ tri1,
                                            const float4* __restrict__ tri2, int hl) {
    const bool isA = hl < 8;
    const unsigned i = hl & 7;
    if (i >= (isA ? T.n & 0xffu : T.n >> 8)) return TriSide{INFINITY, INFINITY};
    const float4* t = (isA ? tri1 + (size_t)T.a0 * kTriF4 : tri2 + (size_t)T.b0 * kTriF4) + i * kTriF4;
    const float4 t0 = t[0], t1 = t[1], t2 = t[2];
    const float p0 = (t0.x - T.ax) * T.ux + (t0.y - T.ay) * T.uy + (t0.z - T.az) * T.uz;
    const float p1 = (t1.x - T.ax) * T.ux + (t1.y - T.ay) * T.uy + (t1.z - T.az) * T.uz;
    const float p2 = (t2.x - T.ax) * T.ux + (t2.y - T.ay) * T.uy + (t2.z - T.az) * T.uz;
    const float g = isA ? -fmaxf(p0, fmaxf(p1, p2)) : fminf(p0, fminf(p1, p2));
    return MODE == kTriH ? TriSide{g + t1.w, g - t0.w} : TriSide{g, g};
}

// the least sum over a half warp's (A, B) triangle pairs
__device__ __forceinline__ float least_sum(float v) {
#pragma unroll
    for (int o = 1; o < kCl; o <<= 1) v = least_of(v, __shfl_xor_sync(kFull, v, o));
    return v + __shfl_xor_sync(kFull, v, 8);
}

constexpr int kTestWarps = 8;
constexpr int kTestBuf = 96;  // triangle pairs a warp collects before it claims queue slots (>= 63 + 32)

template <int MODE>
__global__ void __launch_bounds__(kTestWarps * 32, 5) k_lod_test(LodDev L, int k, int pass) {
    __shared__ TaskDir dirs[kTestWarps][32];
    __shared__ LodEval bufs[kTestWarps][kTestBuf];
    const int lane = threadIdx.x & 31, half = lane >> 4, hl = lane & 15, wid = threadIdx.x >> 5;
    const unsigned lt = (1u << lane) - 1u;
    TaskDir* dir = dirs[wid];
    LodEval* buf = bufs[wid];
    int bn = 0;
    unsigned* ctr = L.ctr + pass * kLodCtrWords;
    const unsigned n = min(ctr[cTasks], L.task_cap);
    // batches small enough that every warp of the grid gets some
    const unsigned nw = gridDim.x * kTestWarps, gw = blockIdx.x * kTestWarps + wid;
    const unsigned batch = max(1u, min(32u, (n + nw - 1) / nw));
    const float4* tri1 = L.tri1[k];
    const float4* tri2 = L.tri2[k];
    const float4* cl2 = L.self ? L.cl1 : L.cl2;
    auto flush = [&] {  // (at most 64 for each of the tasks: the counter does not wrap)
        __syncwarp();
        unsigned base = 0;
        if (lane == 0) base = atomicAdd(ctr + cEvals, (unsigned)bn);
        base = __shfl_sync(kFull, base, 0);
        for (int i = lane; i < bn; i += 32) {
            const LodEval e = buf[i];
            if (base + i < L.eval_cap) L.evals[base + i] = e;
            else go_whole(L, ctr, e.w);
        }
        __syncwarp();
        bn = 0;
    };
    for (unsigned t0 = gw * batch; t0 < n; t0 += nw * batch) {
        // one task a lane: does it still matter, and along which line
        bool have = lane < batch && t0 + lane < n;
        LodTask t{0, 0, 0.f, 0.f};
        int4 x = make_int4(0, 0, 0, 0);
        float2 lim = make_float2(0.f, 0.f);
        if (have) {
            t = L.tasks[t0 + lane];
            x = L.ext[t.w];
            const float4 g = L.mg[t.w];
            lim = gap_limits<MODE>(L, k, x.y, thresholds<MODE>(L, x.x, x.y, g.y, g.z), g.x);
            have = !(t.z >= lim.x) || (MODE != kLast && !(t.y >= lim.y));
            have = have && __float_as_int(g.w) == 0;  // (else its item is evaluated whole)
        }
        const unsigned m = __ballot_sync(kFull, have);
        if (!m) continue;
        __syncwarp();
        if (have) dir[__popc(m & lt)] = task_dir<MODE>(L, cl2, t.w, t.ij >> 16, t.ij & 0xffffu, lim, x);
        __syncwarp();
        const int cnt = __popc(m);
        for (int c = 0; c < cnt; c += 2) {
            const bool live = c + half < cnt;
            const TaskDir T = dir[live ? c + half : c];
            TriSide s = tri_side<MODE>(T, tri1, tri2, hl);
            if (!live) s = TriSide{INFINITY, INFINITY};
            const float zl = least_sum(s.z), yl = MODE == kLast ? 0.f : least_sum(s.y);
            if (!__any_sync(kFull, live && (!(zl >= T.zt) || (MODE != kLast && !(yl >= T.yt))))) continue;
            const int la = half * 16 + (hl & 7);
            const float za = __shfl_sync(kFull, s.z, la), ya = MODE == kLast ? 0.f : __shfl_sync(kFull, s.y, la);
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const int bj = 2 * r + (hl >> 3), lb = half * 16 + 8 + bj;
                const float z = za + __shfl_sync(kFull, s.z, lb);
                const float y = MODE == kLast ? 0.f : ya + __shfl_sync(kFull, s.y, lb);
                const bool ky = MODE != kLast && !(y >= T.yt);
                // (a bound that is not a number passes: a missing triangle's too, beside one that has none)
                const bool there = (hl & 7) < (int)(T.n & 0xffu) && bj < (int)(T.n >> 8);
                const bool keep = live && there && (!(z >= T.zt) || ky);
                const unsigned km = __ballot_sync(kFull, keep);
                if (!km) continue;
                if (keep) buf[bn + __popc(km & lt)] = LodEval{T.w, T.a0 + (hl & 7), T.b0 + bj, ky ? -INFINITY : z};
                bn += __popc(km);
                if (bn >= 64) flush();
            }
        }
    }
    if (bn > 0) flush();
}

// ---------------------------------------------------------------- evaluation
constexpr int kEvalQueue = 96;  // triangle pairs a warp collects (>= 31 + 64)

// Persistent warps: the queued triangle pairs that still matter, 32 at a time
// and one a lane; then the items whose tasks or triangle pairs found a queue
// full, each as a whole by one warp.
template <int MODE>
__global__ void __launch_bounds__(kEvalBlock, 4) k_lod_eval(LodDev L, int k, int pass) {
    __shared__ uint4 queues[kEvalBlock / 32][kEvalQueue];
    const JoinDev& d = L.d;
    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    uint4* q = queues[threadIdx.x >> 5];
    unsigned* ctr = L.ctr + pass * kLodCtrWords;
    const unsigned n = min(ctr[cEvals], L.eval_cap), n_over = ctr[cOver];
    if (n_over && blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(L.n_over, n_over);
    const float4* tri1 = L.tri1[k];
    const float4* tri2 = L.tri2[k];
    const float4* cl2 = L.self ? L.cl1 : L.cl2;
    unsigned long long evals = 0;
    int qn = 0;
    bool evals_left = n > 0, over_left = n_over > 0;
    unsigned ow = 0, onB = 1, todo = 0;  // the item that is evaluated whole: its current 32 cluster pairs
    unsigned long long obase = 0, opos = 0, otot = 0;
    for (;;) {
        if (evals_left) {
            unsigned e0 = 0;
            if (lane == 0) e0 = atomicAdd(ctr + cWork, 32u);
            e0 = __shfl_sync(kFull, e0, 0);
            evals_left = e0 < n;
            bool have = evals_left && e0 + lane < n;
            LodEval e{0, 0, 0, 0.f};
            if (have) {
                e = L.evals[e0 + lane];
                if (e.z > -INFINITY) {  // the caps may have come down since its test
                    const int4 x = L.ext[e.w];
                    const float4 g = L.mg[e.w];
                    have = !(e.z >= gap_limits<MODE>(L, k, x.y, thresholds<MODE>(L, x.x, x.y, g.y, g.z), g.x).x);
                }
            }
            const unsigned km = __ballot_sync(kFull, have);
            if (have) q[qn + __popc(km & lt)] = make_uint4(e.w, e.a, e.b, 0u);
            qn += __popc(km);
        } else if (over_left) {
            if (!todo && opos >= otot) {
                unsigned o = 0;
                if (lane == 0) o = atomicAdd(ctr + cWorkOver, 1u);
                o = __shfl_sync(kFull, o, 0);
                over_left = o < n_over;
                if (over_left) {
                    ow = L.over[o];
                    onB = (L.items[ow].b_cnt + kCl - 1) / kCl;
                    opos = 0;
                    otot = (unsigned long long)((L.items[ow].a_cnt + kCl - 1) / kCl) * onB;
                }
            }
            if (over_left) {
                const int4 x = L.ext[ow];
                const float4 g = L.mg[ow];
                const float2 lim = gap_limits<MODE>(L, k, x.y, thresholds<MODE>(L, x.x, x.y, g.y, g.z), g.x);
                if (!todo) {
                    bool have = false;
                    if (opos + lane < otot) {
                        const unsigned ci = (unsigned)((opos + lane) / onB);
                        const unsigned cj = (unsigned)((opos + lane) - (unsigned long long)ci * onB);
                        const Cluster a = load_cluster(L.cl1 + kClF4 * ((size_t)x.z + ci)),
                                      b = load_cluster(cl2 + kClF4 * ((size_t)x.w + cj));
                        const float2 zy = widen<MODE>(cluster_gap(a, b), a, b);
                        have = !(zy.x >= lim.x) || (MODE != kLast && !(zy.y >= lim.y));
                    }
                    todo = __ballot_sync(kFull, have);
                    obase = opos;
                    opos += 32;
                }
                if (todo) {
                    const unsigned long long t = obase + (__ffs(todo) - 1);
                    todo &= todo - 1;
                    const unsigned ci = (unsigned)(t / onB), cj = (unsigned)(t - (unsigned long long)ci * onB);
                    const TaskDir T = task_dir<MODE>(L, cl2, ow, ci, cj, lim, x);
                    const TriSide s = tri_side<MODE>(T, tri1, tri2, lane & 15);
#pragma unroll
                    for (int r = 0; r < 2; ++r) {
                        const int la = lane & 7, bj = 4 * r + (lane >> 3);
                        const float z = __shfl_sync(kFull, s.z, la) + __shfl_sync(kFull, s.z, 8 + bj);
                        const float y = __shfl_sync(kFull, s.y, la) + __shfl_sync(kFull, s.y, 8 + bj);
                        const bool keep = la < (int)(T.n & 0xffu) && bj < (int)(T.n >> 8) &&
                                          (!(z >= T.zt) || (MODE != kLast && !(y >= T.yt)));
                        const unsigned km = __ballot_sync(kFull, keep);
                        if (keep) q[qn + __popc(km & lt)] = make_uint4(ow, T.a0 + la, T.b0 + bj, 0u);
                        qn += __popc(km);
                    }
                }
            }
        }
        const bool fin = !evals_left && !over_left;
        while (qn >= 32 || (fin && qn > 0)) {
            const int take = min(qn, 32);
            __syncwarp();
            if (lane < take) {
                const uint4 e = q[lane];
                const float4 o4 = tri1[(size_t)L.items[e.x].a_off * kTriF4];
                PreTri<float> A, B;
                float pa, ha, pb, hb;
                pre_rel(tri1 + (size_t)e.y * kTriF4, o4, A, pa, ha);
                pre_rel(tri2 + (size_t)e.z * kTriF4, o4, B, pb, hb);
                const float dd = sqrtf(tri_dist2(A, B));
                const int4 x = L.ext[e.x];
                // a pair's new best also gives it its direction (racing writers may
                // mix theirs: the reader normalises, and any direction is valid)
                bool best = false;
                if (MODE == kTriH) {
                    best = lower_to(L.pown[x.y] ? d.vmx + x.x : L.pcap + x.y, dd + ha + hb);
                    lower_to(d.vmn + x.x, fmaxf(dd - pa - pb, 0.f));
                } else if (MODE == kObjH) {
                    const float3 o = object_h(L, x.y, k);
                    best = lower_to(L.pown[x.y] ? d.vmx + x.x : L.pcap + x.y, dd + o.x + o.y);
                    lower_to(L.vres + x.x, dd);
                } else {
                    // what is not below the threshold does not count as found:
                    // not every triangle pair up to it was looked at
                    const float4 g = L.mg[e.x];
                    if (dd < thresholds<MODE>(L, x.x, x.y, g.y, g.z).x) {
                        lower_to(L.pd + x.y, dd);
                        lower_to(L.vres + x.x, dd);
                    }
                }
                if (best) L.dir[x.y] = tri_to_tri(A, B);
                ++evals;
            }
            // up to 95 pairs: two moves to the front
            const uint4 m0 = lane + take < qn ? q[lane + take] : make_uint4(0u, 0u, 0u, 0u);
            const uint4 m1 = lane + 32 + take < qn ? q[lane + 32 + take] : make_uint4(0u, 0u, 0u, 0u);
            __syncwarp();
            qn -= take;
            if (lane < qn) q[lane] = m0;
            if (lane + 32 < qn) q[lane + 32] = m1;
            __syncwarp();
        }
        if (fin) break;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) evals += __shfl_xor_sync(kFull, evals, o);
    if (lane == 0 && evals) atomicAdd(L.n_full, evals);
}

// ---------------------------------------------------------------- update
// One warp per object pair.  LAST: the voxel pairs' distances become their
// bounds (kFar where nothing was near enough to matter).  A pair none of whose
// voxel pairs came below the hint its last LOD started from (bounds in the
// tile that do not hold) is left as it was and its items go through the last
// LOD once more without a hint; again != 0 is that second time.
template <bool LAST>
__global__ void __launch_bounds__(256) k_lod_update(LodDev L, int k, int stamp, int decide, int again) {
    const JoinDev& d = L.d;
    const int lane = threadIdx.x & 31;
    const int nw = (gridDim.x * blockDim.x) >> 5;
    unsigned* redo_ctr = L.ctr + (k + 1) * kLodCtrWords;
    if (again && redo_ctr[cRedo] == 0) return;
    for (int p = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; p < d.P; p += nw) {
        if (d.pstat[p] != kUndecided) continue;
        if (LAST && again && !L.pmiss[p]) continue;
        const int64_t b = d.pvp[p], e = d.pvp[p + 1];
        const bool own = L.pown[p];
        float minmax = INFINITY, mindist = FLT_MAX, err = 0.f, least = FLT_MAX;
        bool any = false;
        if (LAST) {
            for (int64_t v = b + lane; v < e; v += 32)
                if (d.valive[v] && d.vupd[v] == stamp) {
                    any = true;
                    least = fminf(least, L.vres[v]);
                }
            any = __any_sync(kFull, any);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) least = fminf(least, __shfl_xor_sync(kFull, least, o));
            if (!again && any && !(least < FLT_MAX)) {
                const float hint = own ? FLT_MAX : L.pcap[p];
                float most = -FLT_MAX;  // the largest preset: nothing below it needs no second look
                for (int64_t v = b + lane; v < e; v += 32)
                    if (d.valive[v] && d.vupd[v] == stamp)
                        most = fmaxf(most, L.use_preset ? within_preset(d, p, d.vpa[v], d.vpb[v], L.tau) : FLT_MAX);
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) most = fmaxf(most, __shfl_xor_sync(kFull, most, o));
                if (hint < most) {
                    for (int64_t v0 = b; v0 < e; v0 += 32) {
                        const int64_t v = v0 + lane;
                        const bool ok = v < e && d.valive[v] && d.vupd[v] == stamp;
                        const unsigned m = __ballot_sync(kFull, ok);
                        unsigned base = 0;
                        if (lane == 0 && m) base = atomicAdd(redo_ctr + cRedo, (unsigned)__popc(m));
                        base = __shfl_sync(kFull, base, 0);
                        if (ok) {
                            const unsigned w = base + __popc(m & ((1u << lane) - 1u));
                            const int va = d.vpa[v], vb = d.vpb[v];
                            const uint32_t o1 = L.vt1[k][va], o2 = L.vt2[k][vb];
                            L.items[w] = RefineItem{o1, L.vt1[k][va + 1] - o1, o2, L.vt2[k][vb + 1] - o2};
                            L.ext[w] = make_int4((int)v, p, (int)cluster_base(o1, va), (int)cluster_base(o2, vb));
                            L.vox[w] = make_int2(va, vb);
                        }
                    }
                    if (lane == 0) L.pmiss[p] = 1;
                    continue;
                }
            }
        }
        for (int64_t v = b + lane; v < e; v += 32) {
            if (!d.valive[v]) continue;
            const bool upd = d.vupd[v] == stamp;
            float mn = d.vmn[v], ve = d.verr[v];
            if (LAST && upd) {
                const float x = L.vres[v], ex = d.vmx[v];
                const bool near = x < FLT_MAX;
                mn = near ? x : kFar;
                ve = fmaxf(ve, near ? ex + 4.f * kUnitRoundoff * fabsf(x) : ex);
                d.vmn[v] = mn;
                d.vmx[v] = mn;
                d.verr[v] = ve;
                minmax = fminf(minmax, mn);
            }
            if (!LAST && upd) {
                if (L.level == 1) {
                    const float x = L.vres[v];
                    if (x < FLT_MAX) {
                        const int q = d.pq[p], t = d.pt[p], li = L.li[k];
                        mn = fminf(mn, x - d.ohd1[q * 5 + li] - d.ohd2[t * 5 + li]);
                        d.vmn[v] = mn;
                        ve = fmaxf(ve, 4.f * kUnitRoundoff * fabsf(mn));
                        d.verr[v] = ve;
                    }
                }
                any = true;
                if (own) minmax = fminf(minmax, d.vmx[v]);
            }
            mindist = fminf(mindist, mn);
            err = fmaxf(err, ve);
        }
        if (!LAST && __any_sync(kFull, any) && !own) minmax = L.pcap[p];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            minmax = fminf(minmax, __shfl_xor_sync(kFull, minmax, o));
            mindist = fminf(mindist, __shfl_xor_sync(kFull, mindist, o));
            err = fmaxf(err, __shfl_xor_sync(kFull, err, o));
        }
        // evict voxel pairs that cannot hold the minimum, except those whose
        // FP32 bounds overlap within the error band
        const float slack = 2.f * err;
        for (int64_t v = b + lane; v < e; v += 32)
            if (d.valive[v] && d.vmn[v] - slack > minmax) d.valive[v] = 0;
        if (lane == 0) {
            d.pmn[p] = mindist;
            d.pmx[p] = minmax;
            d.perr[p] = err;
            if (decide) {  // as k_within_decide
                float tau = L.tau;
                bool within = true;
                if (d.qk) {
                    const int q = d.pq[p];
                    within = d.qk[q] <= 0;
                    tau = d.qtau[q];
                }
                if (within) {
                    if (minmax + err <= tau) d.pstat[p] = kReported;
                    else if (mindist - err > tau) d.pstat[p] = kDropped;
                }
            }
        }
    }
}

// ---------------------------------------------------------------- exact
// The queued triangle pairs of a last-LOD pass over reported pairs, once all
// their FP32 distances are known: the one that holds a pair's minimum is in the
// queue (its gap is below every cap that ever stood) unless its item is in
// `over`.  A lane takes one: its gap against the pair's final cap, its FP32
// distance with its error against the same, and what is left in FP64.  A
// warp collects those, to run the FP64 distance with all its lanes.

__global__ void __launch_bounds__(kEvalBlock, 2) k_lod_f64(LodDev L, unsigned long long* __restrict__ exact,
                                                           unsigned* __restrict__ n_items) {
    __shared__ uint2 queues[kEvalBlock / 32][64];  // (entry, pair)
    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    uint2* q = queues[threadIdx.x >> 5];
    const unsigned n = min(L.ctr[cEvals], L.eval_cap);
    const unsigned nw = (gridDim.x * blockDim.x) >> 5, gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    int qn = 0;
    for (unsigned e0 = gw * 32; ; e0 += nw * 32) {
        const bool fin = e0 >= n;
        if (!fin) {
            bool have = e0 + lane < n;
            unsigned p = 0;
            if (have) {
                const LodEval e = L.evals[e0 + lane];
                const float4 g = L.mg[e.w];
                p = (unsigned)L.ext[e.w].y;
                if (!(__float_as_int(g.w) & kEvalFlag)) atomicOr((int*)&L.mg[e.w].w, kEvalFlag);
                const float lim = fminf(L.pd[p], L.pcap[p]) + g.y;
                have = !(e.z >= lim + g.x);
                if (have) {
                    const float4 o4 = L.tri1[0][(size_t)L.items[e.w].a_off * kTriF4];
                    PreTri<float> A, B;
                    float x0, x1, x2, x3;
                    pre_rel(L.tri1[0] + (size_t)e.a * kTriF4, o4, A, x0, x1);
                    pre_rel(L.tri2[0] + (size_t)e.b * kTriF4, o4, B, x2, x3);
                    have = !(sqrtf(tri_dist2(A, B)) - g.x > lim);
                    if (have && !(atomicOr((int*)&L.mg[e.w].w, kExactFlag) & kExactFlag)) atomicAdd(n_items, 1u);
                }
            }
            const unsigned m = __ballot_sync(kFull, have);
            if (have) q[qn + __popc(m & lt)] = make_uint2(e0 + lane, p);
            qn += __popc(m);
        }
        __syncwarp();
        while (qn >= 32 || (fin && qn > 0)) {
            const int take = min(qn, 32);
            if (lane < take) {
                const uint2 u = q[lane];
                const LodEval e = L.evals[u.x];
                const float4 o4 = L.tri1[0][(size_t)L.items[e.w].a_off * kTriF4];
                PreTri<double> A, B;
                pre_rel64(L.tri1[0] + (size_t)e.a * kTriF4, o4, A);
                pre_rel64(L.tri2[0] + (size_t)e.b * kTriF4, o4, B);
                // non-negative doubles order like their bit patterns
                atomicMin(exact + u.y, (unsigned long long)__double_as_longlong(sqrt(tri_dist2(A, B))));
            }
            const uint2 moved = lane + take < qn ? q[lane + take] : make_uint2(0, 0);
            __syncwarp();
            qn -= take;
            if (lane < qn) q[lane] = moved;
            __syncwarp();
        }
        if (fin) break;
    }
}

// counts[0]: items none of whose triangle pairs was queued; counts[1]: items
// with a triangle pair below the pair's cap
__global__ void k_lod_count(LodDev L, unsigned n, unsigned* __restrict__ counts) {
    unsigned none = 0, below = 0;
    for (unsigned w = blockIdx.x * blockDim.x + threadIdx.x; w < n; w += gridDim.x * blockDim.x) {
        none += !(__float_as_int(L.mg[w].w) & (kEvalFlag | 1));
        below += L.vres[w] < FLT_MAX;
    }
    none = __reduce_add_sync(kFull, none);
    below = __reduce_add_sync(kFull, below);
    if ((threadIdx.x & 31) == 0) {
        if (none) atomicAdd(counts, none);
        if (below) atomicAdd(counts + 1, below);
    }
}

int blocks_for(int64_t n, int per_block, int cap) {
    int64_t g = (n + per_block - 1) / per_block;
    if (g < 1) g = 1;
    return (int)(g > cap ? cap : g);
}

template <int MODE>
cudaError_t refine_pass(const LodDev& L, int k, int pass, const unsigned* n_items, int stamp, cudaStream_t s) {
    k_lod_cull<MODE><<<blocks_for(L.d.V, kCullWarps, L.num_sms * 4), kCullWarps * 32, 0, s>>>(L, k, pass, n_items,
                                                                                            stamp);
    k_lod_test<MODE><<<L.num_sms * 5, kTestWarps * 32, 0, s>>>(L, k, pass);
    k_lod_eval<MODE><<<L.num_sms * 4, kEvalBlock, 0, s>>>(L, k, pass);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_lod_init(const LodDev& L, unsigned* words, int n_words, unsigned long long* dstats, size_t caps_bytes,
                            size_t best_bytes, size_t flags_bytes, size_t zero_bytes, cudaStream_t s) {
    const size_t most = std::max({caps_bytes, 2 * best_bytes, flags_bytes, zero_bytes});
    k_lod_init<<<blocks_for((int64_t)(most / 4), 256, L.num_sms * 8), 256, 0, s>>>(L, words, n_words, dstats, caps_bytes / 4, best_bytes / 8,
                                                                           flags_bytes / 4, (zero_bytes + 3) / 4);
    return cudaGetLastError();
}

cudaError_t launch_lod_items(const LodDev& L, int k, cudaStream_t s) {
    k_lod_items<<<blocks_for(L.d.V, 256, L.num_sms * 32), 256, 0, s>>>(L, k);
    return cudaGetLastError();
}

cudaError_t launch_lod_refine(const LodDev& L, int k, int highest, cudaStream_t s) {
    const long nv = L.self ? L.nvox1 : L.nvox1 + L.nvox2;
    k_lod_clusters<<<blocks_for(nv < 2 * L.d.V ? nv : 2 * L.d.V, 8, L.num_sms * 8), 256, 0, s>>>(L, k);
    const int seed_blocks = blocks_for(L.d.P, kEvalBlock / 32, L.num_sms * 4);
    if (highest) {
        if (k == 0) k_lod_seed<kLast><<<seed_blocks, kEvalBlock, 0, s>>>(L, k);
        return refine_pass<kLast>(L, k, k, L.n_items + k, k, s);
    }
    if (L.level == 2) {
        if (k == 0) k_lod_seed<kTriH><<<seed_blocks, kEvalBlock, 0, s>>>(L, k);
        return refine_pass<kTriH>(L, k, k, L.n_items + k, k, s);
    }
    if (k == 0) k_lod_seed<kObjH><<<seed_blocks, kEvalBlock, 0, s>>>(L, k);
    return refine_pass<kObjH>(L, k, k, L.n_items + k, k, s);
}

cudaError_t launch_lod_update(const LodDev& L, int k, int highest, int decide, cudaStream_t s) {
    const int g = blocks_for(L.d.P, 8, L.num_sms * 32);
    if (highest) k_lod_update<true><<<g, 256, 0, s>>>(L, k, k, decide, 0);
    else k_lod_update<false><<<g, 256, 0, s>>>(L, k, k, decide, 0);
    return cudaGetLastError();
}

cudaError_t launch_lod_redo(const LodDev& L, int k, int decide, cudaStream_t s) {
    // the update counted the items at word cRedo of the pass after the last LOD's
    const cudaError_t e = refine_pass<kLast>(L, k, k + 1, L.ctr + (k + 1) * kLodCtrWords + cRedo, k, s);
    if (e != cudaSuccess) return e;
    k_lod_update<true><<<blocks_for(L.d.P, 8, L.num_sms * 32), 256, 0, s>>>(L, k, k, decide, 1);
    return cudaGetLastError();
}

__global__ void k_lod_chunks(unsigned* ctr, int64_t n, int64_t chunk, int n_chunks) {
    for (int c = threadIdx.x; c < n_chunks; c += blockDim.x)
        ctr[(size_t)c * kLodCtrWords + cRedo] = (unsigned)(n - c * chunk < chunk ? n - c * chunk : chunk);
}

cudaError_t launch_lod_exact_begin(const LodDev& L, int64_t chunk, int n_chunks, cudaStream_t s) {
    const long nv = L.self ? L.nvox1 : L.nvox1 + L.nvox2;
    k_lod_clusters<<<blocks_for(nv < 2 * L.d.V ? nv : 2 * L.d.V, 8, L.num_sms * 8), 256, 0, s>>>(L, 0);
    k_lod_chunks<<<1, 256, 0, s>>>(L.ctr, L.d.V, chunk, n_chunks);
    return cudaGetLastError();
}

cudaError_t launch_lod_exact(const LodDev& L, cudaStream_t s) {
    return refine_pass<kLast>(L, 0, 0, L.ctr + cRedo, 0, s);
}

cudaError_t launch_lod_f64(const LodDev& L, unsigned long long* exact, unsigned* n_f64, cudaStream_t s) {
    k_lod_f64<<<L.num_sms * 2, kEvalBlock, 0, s>>>(L, exact, n_f64);
    return cudaGetLastError();
}

cudaError_t launch_lod_exact_count(const LodDev& L, unsigned* counts, cudaStream_t s) {
    k_lod_count<<<blocks_for(L.d.V, 256, L.num_sms * 8), 256, 0, s>>>(L, (unsigned)L.d.V, counts);
    return cudaGetLastError();
}

}  // namespace tdp
