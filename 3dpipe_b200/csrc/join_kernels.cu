// join_kernels.cu -- the filter and LOD-loop kernels of the spatial join.
//
// Reference correspondence (paths inside lyuheng/3dpipe):
//   k_pair_bounds      voxel_pair_dist_kernel_for_all_aggregate_distance and the
//                      min reduction of the streaming kernels
//                      (src/geometry/computing_gpu.cu:1984-2043, :2155-2359),
//                      voxel bounds voxel_dist_core (:1606-1631)
//   k_within_decide    filter-time classification (src/join/WithinJoin.cpp:164-252)
//                      and the per-LOD within decision (WithinJoin.cpp:769-792)
//   k_knn_rank         evaluate_knn_kernel (computing_gpu.cu:105-151) + the confirm
//                      cap in candidate order (src/join/KNNJoin.cpp:133-202), a
//                      warp per query with the cap taken by ballot
//   k_count/write_vps  record_valid_voxel_pairs_streaming_{knn,within}
//                      (computing_gpu.cu:2604-2812): voxel pairs with
//                      min <= object min-max (and <= tau for within)
//   k_build_items      packing_data_stream's voxel-pair list (src/join/SpatialJoin.cpp:169-248),
//                      skipping voxels empty at this LOD (KNNJoin.cpp:1662)
//   k_apply_results    the per-voxel-pair bound update (KNNJoin.cpp:1668-1705)
//   k_pair_update      SpatialJoin::update_voxel_pair_list (SpatialJoin.cpp:48-69):
//                      object min over all voxel pairs, max over the updated ones,
//                      eviction of voxel pairs whose min exceeds that max
// The reference's block reductions in the filter assume a power-of-two block
// (computing_gpu.cu:2027-2033, blockDim = min(max_voxel_size, 1024)); the
// reductions here are exact for any voxel count.
#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>
#include <float.h>

#include "join_kernels.cuh"
#include "pair_rules.cuh"

namespace tdp {

namespace {

constexpr int kBlock = 256;

__device__ __forceinline__ float wmin(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fminf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// Squared box gap and squared core-core distance of two voxels (the terms of
// voxel_dist_core before its square roots).  Per axis the gap is
// max(0, alo - bhi, blo - ahi); for boxes with lo <= hi at most one of the two
// differences is positive, so this is the reference's branch
// (t2 < 0 ? t2^2 : t1 > 0 ? t1^2 : 0) with the same rounding.
__device__ __forceinline__ void vox_dist2(const float4 alo, const float4 ahi, const float4 ac, const float4 blo,
                                          const float4 bhi, const float4 bc, float& m, float& M) {
    const float gx = fmaxf(fmaxf(alo.x - bhi.x, blo.x - ahi.x), 0.f);
    const float gy = fmaxf(fmaxf(alo.y - bhi.y, blo.y - ahi.y), 0.f);
    const float gz = fmaxf(fmaxf(alo.z - bhi.z, blo.z - ahi.z), 0.f);
    const float dx = ac.x - bc.x, dy = ac.y - bc.y, dz = ac.z - bc.z;
    m = 0.f;
    M = 0.f;
    m += gx * gx;
    M += dx * dx;
    m += gy * gy;
    M += dy * dy;
    m += gz * gz;
    M += dz * dz;
}

// voxel_dist_core: box gap and core-core distance, a = tile-1 voxel, b = tile-2 voxel
__device__ __forceinline__ void vox_dist(const float4* __restrict__ va, const float4* __restrict__ vb, float& mn,
                                         float& mx) {
    float m, M;
    vox_dist2(va[0], va[1], va[2], vb[0], vb[1], vb[2], m, M);
    mn = sqrtf(m);
    mx = sqrtf(M);
}

// relative FP32 error of a box gap / core distance: a handful of roundings
constexpr float kVoxRel = 8.0f * kUnitRoundoff;

constexpr int kPBWarps = kBlock / 32;
constexpr int kPBCap = 64;    // tile-1 voxels staged per warp and pass
constexpr int kPBSmall = 24;  // below this many tile-2 voxels, lanes run over (a, b) pairs

// minimum / maximum over the warp (one instruction each on sm_100a)
__device__ __forceinline__ float rmin(float v) {
    float r;
    asm("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}
__device__ __forceinline__ float rmax(float v) {
    float r;
    asm("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}

// The box of some voxels' boxes and the box of their cores.
struct Extent {
    float3 lo, hi, clo, chi;
};
__device__ __forceinline__ Extent no_extent() {
    const float3 m = make_float3(FLT_MAX, FLT_MAX, FLT_MAX), n = make_float3(-FLT_MAX, -FLT_MAX, -FLT_MAX);
    return Extent{m, n, m, n};
}
__device__ __forceinline__ void extend(Extent& e, const float4 lo, const float4 hi, const float4 c) {
    e.lo = make_float3(fminf(e.lo.x, lo.x), fminf(e.lo.y, lo.y), fminf(e.lo.z, lo.z));
    e.hi = make_float3(fmaxf(e.hi.x, hi.x), fmaxf(e.hi.y, hi.y), fmaxf(e.hi.z, hi.z));
    e.clo = make_float3(fminf(e.clo.x, c.x), fminf(e.clo.y, c.y), fminf(e.clo.z, c.z));
    e.chi = make_float3(fmaxf(e.chi.x, c.x), fmaxf(e.chi.y, c.y), fmaxf(e.chi.z, c.z));
}
__device__ __forceinline__ void warp_extent(Extent& e) {
    e.lo = make_float3(rmin(e.lo.x), rmin(e.lo.y), rmin(e.lo.z));
    e.hi = make_float3(rmax(e.hi.x), rmax(e.hi.y), rmax(e.hi.z));
    e.clo = make_float3(rmin(e.clo.x), rmin(e.clo.y), rmin(e.clo.z));
    e.chi = make_float3(rmax(e.chi.x), rmax(e.chi.y), rmax(e.chi.z));
}
// Squared lower bounds of vox_dist2 over the voxels of e against voxel b.
// Rounded as vox_dist2 rounds: every step is monotone, so neither exceeds a
// value it bounds.
__device__ __forceinline__ void extent_dist2(const Extent& e, const float4 blo, const float4 bhi, const float4 bc,
                                             float& m, float& M) {
    const float gx = fmaxf(fmaxf(e.lo.x - bhi.x, blo.x - e.hi.x), 0.f);
    const float gy = fmaxf(fmaxf(e.lo.y - bhi.y, blo.y - e.hi.y), 0.f);
    const float gz = fmaxf(fmaxf(e.lo.z - bhi.z, blo.z - e.hi.z), 0.f);
    const float dx = fmaxf(fmaxf(e.clo.x - bc.x, bc.x - e.chi.x), 0.f);
    const float dy = fmaxf(fmaxf(e.clo.y - bc.y, bc.y - e.chi.y), 0.f);
    const float dz = fmaxf(fmaxf(e.clo.z - bc.z, bc.z - e.chi.z), 0.f);
    m = 0.f;
    M = 0.f;
    m += gx * gx;
    M += dx * dx;
    m += gy * gy;
    M += dy * dy;
    m += gz * gz;
    M += dz * dz;
}

// the within decision at the filter: its query's distance against the range
__device__ __forceinline__ uint8_t within_status(const JoinDev& d, int p, float mn, float mx, float err, float tau_all,
                                                 int tuned) {
    float tau = tau_all;
    if (d.qk) {
        const int q = d.pq[p];
        if (d.qk[q] > 0) return kUndecided;  // a kNN object of a mixed batch
        tau = d.qtau[q];
    }
    const float e = tuned ? err : 0.f;
    return mx + e <= tau ? kReported : mn - e > tau ? kDropped : kUndecided;
}

// Object-pair bounds: min over voxel pairs of the box gap and of the core
// distance.  The square root is correctly rounded and so monotone:
// min_i sqrt(x_i) == sqrt(min_i x_i) exactly, so the minima are taken over the
// squared values and each object pair takes two square roots.  The query
// object's voxels are staged in shared memory (one warp per object pair).
//
// Tile-2 voxels are taken 64 at a time.  Each is first bounded against the
// extent of all staged tile-1 voxels; then the one with the nearest possible
// core goes through them, a tile-1 voxel a lane, and again, until no bound is
// below a minimum.  A nucleus looks at 5 to 10 of a vessel's 200 voxels that
// way instead of all (291,000 pairs of 13 x 200 voxels: 0.82 -> 0.45 ms, which
// was issue-bound).  decide != 0 also takes the within decision.
__global__ void __launch_bounds__(kBlock) k_pair_bounds(JoinDev d, int decide, float tau_all, int tuned) {
    __shared__ float4 sa[kPBWarps][kPBCap * 3];
    __shared__ float4 sb[kPBWarps][kPBSmall * 3];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int nw = (gridDim.x * blockDim.x) >> 5;
    unsigned long long vp = 0;  // voxel pairs of this warp's object pairs (lane 0)
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < d.N1; q += gridDim.x * blockDim.x) d.qconf[q] = 0;
    for (int p = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; p < d.P; p += nw) {
        const int q = d.pq[p], t = d.pt[p];
        const uint32_t a0 = d.ovox1[q], a1 = d.ovox1[q + 1], b0 = d.ovox2[t], b1 = d.ovox2[t + 1];
        const int nb = (int)(b1 - b0);
        float m2 = FLT_MAX, M2 = FLT_MAX;
        bool early = false;  // reported before every voxel pair was seen
        const float etau = d.early_mixed ? (d.qk[q] == 0 ? d.qtau[q] : -1.f) : d.early_tau;
        if (nb < kPBSmall) {
            __syncwarp();
            for (int i = lane; i < nb * 3; i += 32) sb[w][i] = d.vox2[3 * (size_t)b0 + i];
        }
        for (uint32_t ac = a0; ac < a1 && !early; ac += kPBCap) {
            const int na = (int)min((uint32_t)kPBCap, a1 - ac);
            __syncwarp();
            for (int i = lane; i < na * 3; i += 32) sa[w][i] = d.vox1[3 * (size_t)ac + i];
            __syncwarp();
            if (nb >= kPBSmall) {
                Extent ext = no_extent();
                for (int i = lane; i < na; i += 32) extend(ext, sa[w][3 * i], sa[w][3 * i + 1], sa[w][3 * i + 2]);
                warp_extent(ext);
                for (int bb = 0; bb < nb && !early; bb += 64) {
                    // two tile-2 voxels a lane: their least possible values
                    float lm0 = 0.f, lM0 = 0.f, lm1 = 0.f, lM1 = 0.f;
                    bool u0 = bb + lane < nb, u1 = bb + 32 + lane < nb;  // not gone through yet
                    const float4* v0 = d.vox2 + 3 * ((size_t)b0 + bb + lane);
                    if (u0) extent_dist2(ext, __ldg(v0), __ldg(v0 + 1), __ldg(v0 + 2), lm0, lM0);
                    if (u1) extent_dist2(ext, __ldg(v0 + 96), __ldg(v0 + 97), __ldg(v0 + 98), lm1, lM1);
                    float bm = rmin(m2), bM = rmin(M2);
                    for (;;) {
                        // !(>=): a NaN bound is looked at
                        const bool n0 = u0 && (!(lm0 >= bm) || !(lM0 >= bM));
                        const bool n1 = u1 && (!(lm1 >= bm) || !(lM1 >= bM));
                        const float key = fminf(n0 ? lM0 : INFINITY, n1 ? lM1 : INFINITY);
                        const unsigned any = __ballot_sync(0xffffffffu, n0 || n1);
                        if (!any) break;
                        const float best = rmin(key);
                        const unsigned at = __ballot_sync(0xffffffffu, (n0 || n1) && !(key > best));
                        const int src = __ffs(at ? at : any) - 1;
                        const int hs = __shfl_sync(0xffffffffu, n0 && (!n1 || !(lM0 > lM1)) ? 0 : 1, src);
                        if (lane == src) (hs ? u1 : u0) = false;
                        const float4* v = d.vox2 + 3 * ((size_t)b0 + bb + 32 * hs + src);
                        const float4 lo = __ldg(v), hi = __ldg(v + 1), c = __ldg(v + 2);
                        for (int i = lane; i < na; i += 32) {
                            float m, M;
                            vox_dist2(sa[w][3 * i], sa[w][3 * i + 1], sa[w][3 * i + 2], lo, hi, c, m, M);
                            m2 = fminf(m2, m);
                            M2 = fminf(M2, M);
                        }
                        bm = rmin(m2);
                        bM = rmin(M2);
                    }
                    if (etau >= 0.f) {
                        // a core distance is a distance between two surface points,
                        // so it bounds the pair's distance from above: the tuned
                        // within decision (max + error band <= tau) is final
                        const float mx = sqrtf(M2);
                        early = __any_sync(0xffffffffu, mx + kVoxRel * mx <= etau);
                    }
                }
            } else if (nb > 0) {
                const int n = na * nb;
                int i = lane / nb, b = lane - i * nb;
                for (int k = lane; k < n; k += 32) {
                    float m, M;
                    vox_dist2(sa[w][3 * i], sa[w][3 * i + 1], sa[w][3 * i + 2], sb[w][3 * b], sb[w][3 * b + 1],
                              sb[w][3 * b + 2], m, M);
                    m2 = fminf(m2, m);
                    M2 = fminf(M2, M);
                    b += 32;
                    while (b >= nb) { b -= nb; ++i; }
                }
            }
        }
        m2 = rmin(m2);
        M2 = rmin(M2);
        if (lane != 0) continue;
        vp += (unsigned long long)(a1 - a0) * (b1 - b0);
        if (early) {
            const float mx = sqrtf(M2);
            d.pmn[p] = 0.f;  // not computed: the pair is decided
            d.pmx[p] = mx;
            d.perr[p] = kVoxRel * mx;
            d.pstat[p] = kReported;
            continue;
        }
        const float mn = m2 == FLT_MAX ? FLT_MAX : sqrtf(m2);
        const float mx = M2 == FLT_MAX ? FLT_MAX : sqrtf(M2);
        const float err = kVoxRel * fmaxf(mn, mx);
        d.pmn[p] = mn;
        d.pmx[p] = mx;
        d.perr[p] = err;
        d.pstat[p] = decide ? within_status(d, p, mn, mx, err, tau_all, tuned) : (uint8_t)kUndecided;
    }
    if (lane == 0 && vp && d.stat_vp) atomicAdd(d.stat_vp, vp);
}

__global__ void k_within_decide(JoinDev d, float tau_all, int tuned) {
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < d.P; p += gridDim.x * blockDim.x)
        if (d.pstat[p] == kUndecided) d.pstat[p] = within_status(d, p, d.pmn[p], d.pmx[p], d.perr[p], tau_all, tuned);
}

// One warp per query object.  Pass 1: each lane takes candidates lane,
// lane + 32, ... and applies the bulk rule against every other undecided
// candidate (CONFIRMED if fewer than K - confirmed candidates may be closer,
// REMOVED if at least that many are surely closer).  Pass 2: the cap in
// candidate order, 32 candidates at a time: a candidate is acted on while the
// confirmations before it (a ballot and a prefix count) leave an open slot,
// which is what the reference's sequential loop does (it stops at the first
// candidate that finds the K slots full).
__global__ void __launch_bounds__(kBlock) k_knn_rank(JoinDev d, int K_all, int tuned, int* __restrict__ st) {
    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    const int nw = (gridDim.x * blockDim.x) >> 5;
    for (int q = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; q < d.N1; q += nw) {
        const int K = d.qk ? d.qk[q] : K_all;
        if (K <= 0) continue;  // a within object of a mixed batch (warp-uniform)
        const int64_t b = d.qoff[q], e = d.qoff[q + 1];
        int conf = d.qconf[q];
        if (conf < K) {
            const int cand_left = K - conf;
            for (int64_t i = b + lane; i < e; i += 32) {
                if (d.pstat[i] != kUndecided) continue;
                const float ei = tuned ? d.perr[i] : 0.f;
                const float lo = d.pmn[i] - ei, hi = d.pmx[i] + ei;
                int sure = 0, maybe = 0;
                for (int64_t j = b; j < e; ++j) {
                    if (j == i || d.pstat[j] != kUndecided) continue;
                    const float ej = tuned ? d.perr[j] : 0.f;
                    if (lo >= d.pmx[j] + ej) ++sure;
                    if (!(hi <= d.pmn[j] - ej)) ++maybe;
                }
                st[i] = maybe < cand_left ? 1 : (sure >= cand_left ? 2 : 0);
            }
            __syncwarp();
            for (int64_t base = b; base < e && conf < K; base += 32) {
                const int64_t i = base + lane;
                const bool und = i < e && d.pstat[i] == kUndecided;
                const int s = und ? st[i] : 0;
                const unsigned cm = __ballot_sync(0xffffffffu, s == 1);
                if (und && conf + __popc(cm & lt) < K) {
                    if (s == 1) d.pstat[i] = kReported;
                    else if (s == 2) d.pstat[i] = kDropped;
                }
                conf = min(K, conf + __popc(cm));
            }
            if (lane == 0) d.qconf[q] = conf;
        }
        if (conf >= K)  // query complete: nothing left to refine for it
            for (int64_t i = b + lane; i < e; i += 32)
                if (d.pstat[i] == kUndecided) d.pstat[i] = kDropped;
        __syncwarp();
    }
}

// Voxel pairs of the undecided object pairs that can still matter.  A tile-2
// voxel goes through the tile-1 voxels only if it could pass against the
// extent of all of them; those that do are taken together, one voxel pair a
// lane.  Every voxel pair in turn, with a division each, took 417 us for both
// passes on 291,000 object pairs of 13 x 200 voxels (now 143), and 77 us where
// 1,800 such pairs leave few undecided, each in its own warp (now 29).
template <bool WRITE>
__global__ void __launch_bounds__(kBlock) k_vps(JoinDev d, int within_all, float tau_all, int tuned,
                                                 int64_t* __restrict__ cnt) {
    __shared__ uint32_t near[kBlock / 32][32];
    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    uint32_t* nr = near[threadIdx.x >> 5];
    const int nw = (gridDim.x * blockDim.x) >> 5;
    for (int p = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; p < d.P; p += nw) {
        if (d.pstat[p] != kUndecided) {
            if (!WRITE && lane == 0) cnt[p] = 0;
            continue;
        }
        const int q = d.pq[p], t = d.pt[p];
        const int within = d.qk ? d.qk[q] == 0 : within_all;
        const float tau = d.qk ? d.qtau[q] : tau_all;
        const uint32_t a0 = d.ovox1[q], b0 = d.ovox2[t];
        const uint32_t n1 = d.ovox1[q + 1] - a0, n2 = d.ovox2[t + 1] - b0;
        const float slack = tuned ? d.perr[p] : 0.f;
        const float lim = d.pmx[p] + slack;
        auto passes = [&](float m) { return (m - slack <= lim) && (!within || m - slack <= tau); };
        Extent ext = no_extent();
        for (uint32_t a = lane; a < n1; a += 32) {
            const float4* v = d.vox1 + 3 * (size_t)(a0 + a);
            extend(ext, v[0], v[1], v[2]);
        }
        warp_extent(ext);
        const float4 xlo = make_float4(ext.lo.x, ext.lo.y, ext.lo.z, 0.f), xhi = make_float4(ext.hi.x, ext.hi.y, ext.hi.z, 0.f);
        // aab::intersect: strict overlap on every axis
        auto overlap = [](const float4 alo, const float4 ahi, const float4 blo, const float4 bhi) {
            return !(blo.x >= ahi.x || bhi.x <= alo.x || blo.y >= ahi.y || bhi.y <= alo.y || blo.z >= ahi.z ||
                     bhi.z <= alo.z);
        };
        int64_t pos = WRITE ? d.pvp[p] : 0;
        int64_t count = 0;
        for (uint32_t bb = 0; bb < n2; bb += 32) {
            bool on = bb + lane < n2;
            if (on) {
                const float4* vb = d.vox2 + 3 * (size_t)(b0 + bb + lane);
                float m, M;
                extent_dist2(ext, vb[0], vb[1], vb[2], m, M);
                on = d.isect ? overlap(xlo, xhi, vb[0], vb[1]) : passes(sqrtf(m));
            }
            const unsigned bm = __ballot_sync(0xffffffffu, on);
            if (!bm) continue;
            __syncwarp();
            if (on) nr[__popc(bm & lt)] = b0 + bb + lane;
            __syncwarp();
            const uint64_t total = (uint64_t)__popc(bm) * n1;
            uint32_t s = lane / n1, a = lane - s * n1;
            for (uint64_t base = 0; base < total; base += 32) {
                bool keep = false;
                float m = 0.f, M = 0.f;
                uint32_t b = 0;
                if (base + lane < total) {
                    b = nr[s];
                    const float4* va = d.vox1 + 3 * (size_t)(a0 + a);
                    const float4* vb = d.vox2 + 3 * (size_t)b;
                    vox_dist(va, vb, m, M);
                    keep = d.isect ? overlap(va[0], va[1], vb[0], vb[1]) : passes(m);
                }
                const unsigned bal = __ballot_sync(0xffffffffu, keep);
                if (WRITE && keep) {
                    const int64_t w = pos + __popc(bal & lt);
                    d.vpa[w] = (int)(a0 + a);
                    d.vpb[w] = (int)b;
                    d.vpair[w] = p;
                    d.vmn[w] = m;
                    d.vmx[w] = M;
                    d.verr[w] = kVoxRel * fmaxf(m, M);
                    d.valive[w] = 1;
                    d.vupd[w] = -1;
                }
                pos += __popc(bal);
                count += __popc(bal);
                a += 32;
                while (a >= n1) {
                    a -= n1;
                    ++s;
                }
            }
        }
        if (!WRITE && lane == 0) cnt[p] = count;
    }
}

// One slot claim and one triangle-pair sum per warp: lane 0 adds the warp's
// item count and n1*n2 sum to the counters, the lanes write at the claimed
// base plus their rank among the warp's items.  (The items form a set: their
// order never changes a result.)
// preset != NULL (the tuned form's last LOD of a join with within queries):
// also write each item's preset (within_preset)
__global__ void k_build_items(JoinDev d, const uint32_t* __restrict__ vt1, const uint32_t* __restrict__ vt2,
                              RefineItem* __restrict__ items, int* __restrict__ item_vp, unsigned* __restrict__ counter,
                              float* __restrict__ preset, float tau_all) {
    // counter[0] = items, counter[2..3] = sum n1*n2 (u64)
    const int lane = threadIdx.x & 31;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    // every lane of a warp runs the same number of iterations (the bound is rounded up to whole warps)
    const int64_t vend = (d.V + 31) & ~(int64_t)31;
    for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < vend; v += stride) {
        bool ok = v < d.V && d.valive[v] && d.pstat[d.vpair[v]] == kUndecided;
        uint32_t o1 = 0, n1 = 0, o2 = 0, n2 = 0;
        int a = 0, b = 0;
        if (ok) {
            a = d.vpa[v];
            b = d.vpb[v];
            o1 = vt1[a]; n1 = vt1[a + 1] - o1;
            o2 = vt2[b]; n2 = vt2[b + 1] - o2;
            ok = n1 > 0 && n2 > 0;
        }
        const unsigned m = __ballot_sync(0xffffffffu, ok);
        if (!m) continue;
        unsigned long long tp = ok ? (unsigned long long)n1 * n2 : 0ull;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) tp += __shfl_xor_sync(0xffffffffu, tp, o);
        unsigned base = 0;
        if (lane == 0) {
            base = atomicAdd(counter, (unsigned)__popc(m));
            atomicAdd(reinterpret_cast<unsigned long long*>(counter + 2), tp);
        }
        base = __shfl_sync(0xffffffffu, base, 0);
        if (ok) {
            const unsigned w = base + __popc(m & ((1u << lane) - 1u));
            items[w] = RefineItem{o1, n1, o2, n2};
            item_vp[w] = (int)v;
            if (preset) preset[w] = within_preset(d, d.vpair[v], a, b, tau_all);
        }
    }
}

__global__ void k_apply_results(JoinDev d, const float4* __restrict__ res, const int* __restrict__ item_vp, int W_host,
                                const unsigned* W_dev, int highest, int level, int li, int stamp,
                                const float* __restrict__ preset) {
    const int W = W_dev ? (int)*W_dev : W_host;
    for (int w = blockIdx.x * blockDim.x + threadIdx.x; w < W; w += gridDim.x * blockDim.x) {
        const int v = item_vp[w];
        const float4 r = res[w];
        float mn = d.vmn[v], mx = d.vmx[v];
        const float e = err_bound(r.w);
        if (highest && preset) {
            const float pb = preset[w];
            if (pb < FLT_MAX && !(r.x < pb)) {
                d.vmn[v] = kFar;
                d.vmx[v] = kFar;
                d.verr[v] = fmaxf(d.verr[v], e);
                d.vupd[v] = stamp;
                continue;
            }
        }
        if (highest) {
            mn = r.x;
            mx = r.x;
        } else if (level == 2) {
            mn = fminf(mn, r.y);
            mx = fminf(mx, r.z);
        } else if (level == 1) {
            const int p = d.vpair[v];
            const int q = d.pq[p], t = d.pt[p];
            mn = fminf(mn, r.x - d.ohd1[q * 5 + li] - d.ohd2[t * 5 + li]);
            mx = fminf(mx, r.x + d.ophd1[q * 5 + li] + d.ophd2[t * 5 + li]);
        } else {
            mx = fminf(mx, r.x);
        }
        d.vmn[v] = mn;
        d.vmx[v] = mx;
        d.verr[v] = fmaxf(d.verr[v], e + 4.f * kUnitRoundoff * fmaxf(fabsf(mn), fabsf(mx)));
        d.vupd[v] = stamp;
    }
}

// undecided and reported pairs (whole warps)
__device__ __forceinline__ void count_status(const JoinDev& d, unsigned* __restrict__ c) {
    unsigned und = 0, rep = 0;
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < d.P; p += gridDim.x * blockDim.x) {
        und += d.pstat[p] == kUndecided;
        rep += d.pstat[p] == kReported;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        und += __shfl_xor_sync(0xffffffffu, und, o);
        rep += __shfl_xor_sync(0xffffffffu, rep, o);
    }
    if ((threadIdx.x & 31) == 0) {
        if (und) atomicAdd(c + 0, und);
        if (rep) atomicAdd(c + 1, rep);
    }
}

// ---- FP64 recheck (tuned form) of pairs still undecided after the last LOD ----
__global__ void k_recheck_items(JoinDev d, const uint32_t* __restrict__ vt1, const uint32_t* __restrict__ vt2,
                                RefineItem* __restrict__ items, int* __restrict__ item_vp, double* __restrict__ vexact,
                                unsigned* __restrict__ counter, unsigned* __restrict__ status) {
    count_status(d, status);
    for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < d.V; v += (int64_t)gridDim.x * blockDim.x) {
        if (!d.valive[v] || d.pstat[d.vpair[v]] != kUndecided) continue;
        vexact[v] = 1e300;
        const int a = d.vpa[v], b = d.vpb[v];
        const uint32_t o1 = vt1[a], n1 = vt1[a + 1] - o1, o2 = vt2[b], n2 = vt2[b + 1] - o2;
        if (!n1 || !n2) continue;
        const unsigned w = atomicAdd(counter, 1u);
        items[w] = RefineItem{o1, n1, o2, n2};
        item_vp[w] = (int)v;
    }
}

__global__ void __launch_bounds__(kBlock) k_recheck_pairs(JoinDev d, const double* __restrict__ vexact,
                                                          double* __restrict__ pexact, int within_all,
                                                          float tau_all) {
    const int lane = threadIdx.x & 31;
    const int nw = (gridDim.x * blockDim.x) >> 5;
    for (int p = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; p < d.P; p += nw) {
        if (d.pstat[p] != kUndecided) continue;
        double D = 1e300;
        for (int64_t v = d.pvp[p] + lane; v < d.pvp[p + 1]; v += 32)
            if (d.valive[v]) D = vexact[v] < D ? vexact[v] : D;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            double x = __shfl_xor_sync(0xffffffffu, D, o);
            D = x < D ? x : D;
        }
        if (lane == 0) {
            const int q = d.pq[p];
            const int within = d.qk ? d.qk[q] == 0 : within_all;
            const float tau = d.qk ? d.qtau[q] : tau_all;
            pexact[p] = D;
            d.pmn[p] = d.pmx[p] = (float)D;
            if (within) d.pstat[p] = D <= (double)tau ? kReported : kDropped;
        }
    }
}

// kNN: the still-undecided candidates of a query compete for its open slots by exact distance
__global__ void k_recheck_knn(JoinDev d, int K_all, const double* __restrict__ pexact) {
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < d.N1; q += gridDim.x * blockDim.x) {
        const int K = d.qk ? d.qk[q] : K_all;
        if (K <= 0) continue;
        const int64_t b = d.qoff[q], e = d.qoff[q + 1];
        int conf = d.qconf[q];
        while (conf < K) {
            int64_t best = -1;
            for (int64_t i = b; i < e; ++i)
                if (d.pstat[i] == kUndecided && (best < 0 || pexact[i] < pexact[best])) best = i;
            if (best < 0) break;
            d.pstat[best] = kReported;
            ++conf;
        }
        for (int64_t i = b; i < e; ++i)
            if (d.pstat[i] == kUndecided) d.pstat[i] = kDropped;
        d.qconf[q] = conf;
    }
}

// decide != 0: the within decision of k_within_decide is taken here too, for
// the within query objects, as soon as the pair's bounds are known (the tuned
// LOD loop; it saves a launch and a pass over the pairs per LOD)
__global__ void __launch_bounds__(kBlock) k_pair_update(JoinDev d, int stamp, int tuned, int decide, float tau_all) {
    const int lane = threadIdx.x & 31;
    const int nw = (gridDim.x * blockDim.x) >> 5;
    for (int p = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; p < d.P; p += nw) {
        if (d.pstat[p] != kUndecided) continue;
        const int64_t b = d.pvp[p], e = d.pvp[p + 1];
        float minmax = INFINITY, mindist = FLT_MAX, err = 0.f;
        for (int64_t v = b + lane; v < e; v += 32) {
            if (!d.valive[v]) continue;
            mindist = fminf(mindist, d.vmn[v]);
            err = fmaxf(err, d.verr[v]);
            if (d.vupd[v] == stamp) minmax = fminf(minmax, d.vmx[v]);
        }
        minmax = wmin(minmax);
        mindist = wmin(mindist);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) err = fmaxf(err, __shfl_xor_sync(0xffffffffu, err, o));
        // evict voxel pairs that cannot hold the minimum; the tuned form keeps any
        // whose FP32 bounds overlap within the error band
        const float slack = tuned ? 2.f * err : 0.f;
        for (int64_t v = b + lane; v < e; v += 32)
            if (d.valive[v] && d.vmn[v] - slack > minmax) d.valive[v] = 0;
        if (lane == 0) {
            d.pmn[p] = mindist;
            d.pmx[p] = minmax;
            d.perr[p] = err;
            if (decide) {  // as k_within_decide
                float tau = tau_all;
                bool within = true;
                if (d.qk) {
                    const int q = d.pq[p];
                    within = d.qk[q] <= 0;
                    tau = d.qtau[q];
                }
                if (within) {
                    const float e = tuned ? err : 0.f;
                    if (minmax + e <= tau) d.pstat[p] = kReported;
                    else if (mindist - e > tau) d.pstat[p] = kDropped;
                }
            }
        }
    }
}

__global__ void k_count_status(JoinDev d, unsigned* __restrict__ c) { count_status(d, c); }

// Result keys: query * n2 + result id for reported pairs, `none` (= n1 * n2)
// for the rest, so one radix sort over every pair puts the reported ones
// first, ordered by (query, result id); the payload is the pair index.
__global__ void k_collect_keys(JoinDev d, long long n2, unsigned long long none, unsigned long long* __restrict__ keys,
                               int* __restrict__ vals, unsigned* __restrict__ counter) {
    const int lane = threadIdx.x & 31;
    for (int64_t base = (int64_t)blockIdx.x * blockDim.x; base < d.P; base += (int64_t)gridDim.x * blockDim.x) {
        const int64_t p = base + threadIdx.x;
        const bool rep = p < d.P && d.pstat[p] == kReported;
        if (p < d.P) {
            keys[p] = rep ? (unsigned long long)d.pq[p] * (unsigned long long)n2 + (unsigned)d.pt[p] : none;
            vals[p] = (int)p;
        }
        const unsigned m = __ballot_sync(0xffffffffu, rep);
        if (lane == 0 && m) atomicAdd(counter, (unsigned)__popc(m));
    }
}

__device__ __forceinline__ void write_row(const JoinDev& d, const JoinRows& o, int64_t i, int q, int t, int64_t p,
                                          const double* __restrict__ pexact) {
    if (i >= o.cap) return;
    o.q[i] = q;
    o.t[i] = t;
    o.d[i] = d.pmx[p];
    if (o.d64) o.d64[i] = pexact ? pexact[p] : (double)d.pmx[p];
}
__device__ __forceinline__ void write_header(const JoinRows& o, unsigned rows) {  // one block
    if (threadIdx.x == 0) o.head->rows = rows;
    if (threadIdx.x < 32) o.head->counters[threadIdx.x] = o.counters[threadIdx.x];
    if (threadIdx.x < 2) o.head->stats[threadIdx.x] = o.stats[threadIdx.x];
    if (threadIdx.x == 2) o.head->stats[2] = *o.fetched;
}

__global__ void k_split(JoinDev d, const unsigned long long* __restrict__ keys, const int* __restrict__ vals,
                        long long n2, unsigned long long none, const double* __restrict__ pexact,
                        const unsigned* __restrict__ rows, JoinRows out) {
    if (blockIdx.x == 0) write_header(out, *rows);
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < d.P; i += (int64_t)gridDim.x * blockDim.x) {
        const unsigned long long k = keys[i];
        if (k == none) break;  // sorted: every later key is `none` too
        write_row(d, out, i, (int)(k / (unsigned long long)n2), (int)(k % (unsigned long long)n2), vals[i], pexact);
    }
}

// reported candidates of every query, one warp a query
__global__ void __launch_bounds__(kBlock) k_row_counts(JoinDev d, int64_t* __restrict__ cnt) {
    const int lane = threadIdx.x & 31;
    const int nw = (gridDim.x * blockDim.x) >> 5;
    for (int q = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; q < d.N1; q += nw) {
        int n = 0;
        for (int64_t p = d.qoff[q] + lane; p < d.qoff[q + 1]; p += 32) n += d.pstat[p] == kReported;
        n = __reduce_add_sync(0xffffffffu, n);
        if (lane == 0) cnt[q] = n;
    }
}

// The rows of every query, one warp a query: a pair's place is the number of
// reported candidates with a smaller result id (kNN lists are in order of
// distance; within lists are in order of id, and a place is a prefix count).
// off: the rows before each query; NULL: each block adds up the counts itself
// (a block's 4,096 counts are 16 loads a thread; the scan is two more launches).
__global__ void __launch_bounds__(kBlock) k_rows(JoinDev d, int knn_all, const int64_t* __restrict__ cnt,
                                                 const int64_t* __restrict__ off, const double* __restrict__ pexact,
                                                 JoinRows out) {
    __shared__ int64_t part[kBlock / 32], all;  // (all: apart from part, which other warps may still be adding up)
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const unsigned lt = (1u << lane) - 1u;
    for (int q0 = blockIdx.x * (kBlock / 32); q0 < d.N1; q0 += gridDim.x * (kBlock / 32)) {
        const int q = q0 + w;
        int64_t at = 0;
        if (off) {
            at = off[min(q, d.N1)];
        } else {
            int64_t n = 0;
            for (int k = threadIdx.x; k < q0; k += kBlock) n += cnt[k];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) n += __shfl_xor_sync(0xffffffffu, n, o);
            __syncthreads();
            if (lane == 0) part[w] = n;
            __syncthreads();
            for (int k = 0; k < kBlock / 32; ++k) at += part[k];
            for (int k = q0; k < min(q, d.N1); ++k) at += cnt[k];
        }
        if (q0 + kBlock / 32 >= d.N1) {  // the block of the last query
            if (q == d.N1 - 1 && lane == 0) all = at + cnt[q];
            __syncthreads();
            write_header(out, (unsigned)all);
        }
        if (q >= d.N1) continue;
        const int64_t b = d.qoff[q], e = d.qoff[q + 1];
        if (d.qk ? d.qk[q] > 0 : knn_all) {
            for (int64_t p = b + lane; p < e; p += 32) {
                if (d.pstat[p] != kReported) continue;
                const int t = d.pt[p];
                int before = 0;
#pragma unroll 4
                for (int64_t k = b; k < e; ++k) before += d.pstat[k] == kReported && d.pt[k] < t;
                write_row(d, out, at + before, q, t, p, pexact);
            }
        } else {
            for (int64_t p0 = b; p0 < e; p0 += 32) {
                const int64_t p = p0 + lane;
                const bool rep = p < e && d.pstat[p] == kReported;
                const unsigned m = __ballot_sync(0xffffffffu, rep);
                if (rep) write_row(d, out, at + __popc(m & lt), q, d.pt[p], p, pexact);
                at += __popc(m);
            }
        }
    }
}

int grid_for(int64_t n, int per_block, int cap = 148 * 32) {
    int64_t g = (n + per_block - 1) / per_block;
    if (g < 1) g = 1;
    if (g > cap) g = cap;
    return (int)g;
}

}  // namespace

cudaError_t launch_pair_bounds(const JoinDev& d, cudaStream_t s, int decide, float tau, int tuned) {
    if (d.P <= 0) return cudaSuccess;
    k_pair_bounds<<<grid_for(d.P, kBlock / 32), kBlock, 0, s>>>(d, decide, tau, tuned);
    return cudaGetLastError();
}
cudaError_t launch_within_decide(const JoinDev& d, float tau, int tuned, cudaStream_t s) {
    if (d.P <= 0) return cudaSuccess;
    k_within_decide<<<grid_for(d.P, 256), 256, 0, s>>>(d, tau, tuned);
    return cudaGetLastError();
}
cudaError_t launch_knn_rank(const JoinDev& d, int K, int tuned, int* st, cudaStream_t s) {
    if (d.N1 <= 0) return cudaSuccess;
    k_knn_rank<<<grid_for(d.N1, kBlock / 32, 148 * 32), kBlock, 0, s>>>(d, K, tuned, st);
    return cudaGetLastError();
}
cudaError_t launch_count_vps(const JoinDev& d, int within, float tau, int tuned, int64_t* cnt, cudaStream_t s) {
    if (d.P <= 0) return cudaSuccess;
    k_vps<false><<<grid_for(d.P, kBlock / 32), kBlock, 0, s>>>(d, within, tau, tuned, cnt);
    return cudaGetLastError();
}
cudaError_t launch_write_vps(const JoinDev& d, int within, float tau, int tuned, cudaStream_t s) {
    if (d.P <= 0) return cudaSuccess;
    k_vps<true><<<grid_for(d.P, kBlock / 32), kBlock, 0, s>>>(d, within, tau, tuned, nullptr);
    return cudaGetLastError();
}
cudaError_t launch_build_items(const JoinDev& d, const uint32_t* vt1, const uint32_t* vt2, RefineItem* items,
                               int* item_vp, unsigned* counter, cudaStream_t s, float* preset, float tau) {
    if (d.V <= 0) return cudaSuccess;
    k_build_items<<<grid_for(d.V, 256), 256, 0, s>>>(d, vt1, vt2, items, item_vp, counter, preset, tau);
    return cudaGetLastError();
}
cudaError_t launch_apply_results(const JoinDev& d, const float4* res, const int* item_vp, int W, int highest,
                                 int level, int li, int stamp, cudaStream_t s, const unsigned* W_dev,
                                 const float* preset) {
    if (W <= 0) return cudaSuccess;
    k_apply_results<<<grid_for(W, 256), 256, 0, s>>>(d, res, item_vp, W, W_dev, highest, level, li, stamp, preset);
    return cudaGetLastError();
}
cudaError_t launch_pair_update(const JoinDev& d, int stamp, int tuned, cudaStream_t s, int decide, float tau) {
    if (d.P <= 0) return cudaSuccess;
    k_pair_update<<<grid_for(d.P, kBlock / 32), kBlock, 0, s>>>(d, stamp, tuned, decide, tau);
    return cudaGetLastError();
}
cudaError_t launch_recheck_items(const JoinDev& d, const uint32_t* vt1, const uint32_t* vt2, RefineItem* items,
                                 int* item_vp, double* vexact, unsigned* counter, unsigned* status, cudaStream_t s) {
    if (d.V <= 0) return cudaSuccess;
    k_recheck_items<<<grid_for(d.V, 256), 256, 0, s>>>(d, vt1, vt2, items, item_vp, vexact, counter, status);
    return cudaGetLastError();
}
cudaError_t launch_recheck_finish(const JoinDev& d, double* vexact, double* pexact, int knn, int K, float tau,
                                  cudaStream_t s) {
    if (d.P > 0) k_recheck_pairs<<<grid_for(d.P, kBlock / 32), kBlock, 0, s>>>(d, vexact, pexact, !knn, tau);
    if ((knn || d.qk) && d.N1 > 0) k_recheck_knn<<<grid_for(d.N1, 128), 128, 0, s>>>(d, K, pexact);
    return cudaGetLastError();
}
cudaError_t launch_count_status(const JoinDev& d, unsigned* c, cudaStream_t s) {
    if (d.P <= 0) return cudaSuccess;
    k_count_status<<<grid_for(d.P, 256, 148 * 8), 256, 0, s>>>(d, c);
    return cudaGetLastError();
}
static int key_bits(unsigned long long none) {
    int b = 1;
    while (b < 64 && (none >> b)) ++b;
    return b;
}
cudaError_t collect_sort_bytes(int64_t P, long long n1, long long n2, size_t& bytes) {
    bytes = 0;
    if (P <= 0) return cudaSuccess;
    cub::DoubleBuffer<unsigned long long> k(nullptr, nullptr);
    cub::DoubleBuffer<int> v(nullptr, nullptr);
    return cub::DeviceRadixSort::SortPairs(nullptr, bytes, k, v, (int)P, 0,
                                           key_bits((unsigned long long)n1 * (unsigned long long)n2));
}
cudaError_t launch_collect(const JoinDev& d, long long n2, unsigned long long* keys[2], int* vals[2], void* temp,
                           size_t temp_bytes, unsigned* counter, const double* pexact, const JoinRows& out,
                           cudaStream_t s) {
    if (d.P <= 0) return cudaSuccess;
    const unsigned long long none = (unsigned long long)d.N1 * (unsigned long long)n2;
    k_collect_keys<<<grid_for(d.P, 256), 256, 0, s>>>(d, n2, none, keys[0], vals[0], counter);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    cub::DoubleBuffer<unsigned long long> k(keys[0], keys[1]);
    cub::DoubleBuffer<int> v(vals[0], vals[1]);
    e = cub::DeviceRadixSort::SortPairs(temp, temp_bytes, k, v, (int)d.P, 0, key_bits(none), s);
    if (e != cudaSuccess) return e;
    k_split<<<grid_for(d.P, 256), 256, 0, s>>>(d, k.Current(), v.Current(), n2, none, pexact, counter, out);
    return cudaGetLastError();
}
cudaError_t launch_collect_ranked(const JoinDev& d, int knn, int64_t* cnt, int64_t* off, void* temp, size_t temp_bytes,
                                  const double* pexact, const JoinRows& out, cudaStream_t s) {
    if (d.P <= 0) return cudaSuccess;
    k_row_counts<<<grid_for(d.N1, kBlock / 32), kBlock, 0, s>>>(d, cnt);
    cudaError_t e = cudaGetLastError();
    const bool own = d.N1 <= kOwnPrefix;
    if (e == cudaSuccess && !own) e = cudaMemsetAsync(cnt + d.N1, 0, 8, s);
    if (e == cudaSuccess && !own) e = scan_counts(cnt, off, d.N1, temp, temp_bytes, s);
    if (e != cudaSuccess) return e;
    k_rows<<<grid_for(d.N1, kBlock / 32), kBlock, 0, s>>>(d, knn, cnt, own ? nullptr : off, pexact, out);
    return cudaGetLastError();
}

namespace {
constexpr int kScanThreads = 1024, kScanSmall = 16 * kScanThreads;

// Exclusive scan of n counts by one block, each thread a run of them; the total
// goes to out[n] and, with *extra, to the host's page-locked words.
__global__ void __launch_bounds__(kScanThreads) k_scan_small(const int64_t* __restrict__ cnt, int64_t* __restrict__ out, int n,
                                                            const unsigned long long* __restrict__ extra,
                                                            unsigned long long* __restrict__ host) {
    __shared__ int64_t sums[kScanThreads / 32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int per = (n + kScanThreads - 1) / kScanThreads, b = min(n, (int)threadIdx.x * per), e = min(n, b + per);
    int64_t mine = 0;
    for (int i = b; i < e; ++i) mine += cnt[i];
    int64_t inc = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int64_t t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += t;
    }
    if (lane == 31) sums[w] = inc;
    __syncthreads();
    int64_t at = inc - mine;
    for (int k = 0; k < w; ++k) at += sums[k];
    for (int i = b; i < e; ++i) {
        const int64_t c = cnt[i];
        out[i] = at;
        at += c;
    }
    if (threadIdx.x == kScanThreads - 1) {
        out[n] = at;
        host[0] = (unsigned long long)at;
        if (extra) host[1] = *extra;
    }
}
}  // namespace

cudaError_t scan_to_host_bytes(int n, bool host_locked, size_t& bytes) {
    bytes = 0;
    return n <= kScanSmall && host_locked ? cudaSuccess : scan_counts(nullptr, nullptr, n, nullptr, bytes, nullptr);
}
cudaError_t scan_to_host(int64_t* cnt, int64_t* out, int n, void* temp, size_t temp_bytes, const unsigned long long* extra,
                         unsigned long long* host, bool host_locked, cudaStream_t s) {
    if (n <= kScanSmall && host_locked) {
        k_scan_small<<<1, kScanThreads, 0, s>>>(cnt, out, n, extra, host);
        return cudaGetLastError();
    }
    cudaError_t e = cudaMemsetAsync(cnt + n, 0, 8, s);
    if (e == cudaSuccess) e = scan_counts(cnt, out, n, temp, temp_bytes, s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(host, out + n, 8, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess && extra) e = cudaMemcpyAsync(host + 1, extra, 8, cudaMemcpyDeviceToHost, s);
    return e;
}

cudaError_t scan_counts(const int64_t* cnt, int64_t* out, int n, void* temp, size_t& temp_bytes, cudaStream_t s) {
    // exclusive scan of n+1 values (cnt[n] must be 0) so out[n] is the total
    return cub::DeviceScan::ExclusiveSum(temp, temp_bytes, cnt, out, n + 1, s);
}

}  // namespace tdp
