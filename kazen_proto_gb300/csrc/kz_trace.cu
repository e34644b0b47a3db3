// kz_trace.cu — sm_103a traversal kernels: batch intersection (closest,
// any, fetch counts) and the path tracer's closest-hit and shadow passes, as
// host-count kernels and as persistent kernels that refill idle lanes from a
// global cursor, for single renders and batched jobs.
#include "kz_stages.cuh"

// Resident 256-thread blocks per SM the persistent traversal kernels are
// compiled for (4: at most 64 registers a thread).
#ifndef KZ_TRACE_MINB
#define KZ_TRACE_MINB 4
#endif

namespace kz {
namespace {

// Blocks of a stage of at most `cap` rays: all that are resident, since few rays
// take a warp each; larger queues leave the rest idle (trace_blocks).
unsigned stage_grid(uint64_t cap, unsigned resident) {
    return (unsigned)std::min<uint64_t>(resident, (cap + 7) / 8);
}

// A node of the builder's layout (kz_bvh.h) to the traversal's (WideAxis,
// kz_traverse.cuh), in place; the same boxes, children and records.
__global__ void k_pack_nodes(uint4* nodes, uint32_t n) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    uint4* p = nodes + (size_t)i * 5;
    const uint4 h0 = p[0], h1 = p[1];
    uint32_t valid = 0;
#pragma unroll
    for (int s = 0; s < 8; ++s) {
        const uint32_t m = ((s < 4 ? h1.z : h1.w) >> (8 * (s & 3))) & 0xFFu;
        if (!((h0.w >> (24 + s)) & 1u)) valid |= (m >> 5) << (3 * s);
    }
    const auto scale = [&](int a) { return (((h0.w >> (8 * a)) & 0xFFu) + 15u) << 7; };
    p[0].w = scale(0) | scale(1) << 16;
    p[1].z = valid | (h0.w & 0xFF000000u);
    p[1].w = scale(2);
#pragma unroll
    for (int a = 2; a < 5; ++a) {
        const uint4 q = p[a];  // low planes of slots 0-3, 4-7, high planes of slots 0-3, 4-7
        p[a] = make_uint4(__byte_perm(q.x, q.z, 0x5140), __byte_perm(q.x, q.z, 0x7362),
                          __byte_perm(q.y, q.w, 0x5140), __byte_perm(q.y, q.w, 0x7362));
    }
}

// kz_intersect_any: rays (o, tmin, d, tmax) in, an occlusion byte out.
__global__ void __launch_bounds__(256, KZ_TRACE_MINB) k_intersect_any_persistent(DevScene s,
                                                                                 const kz_ray* __restrict__ rays,
                                                                                 unsigned long long n, uint8_t* occ,
                                                                                 unsigned long long* next,
                                                                                 uint32_t* status) {
    uint32_t dn = 0, dt = 0;
    persistent_any<false>(
        s, n, next,
        [&](unsigned long long k, TRay& r, float& tmax) {
            const float4* rp = reinterpret_cast<const float4*>(rays + k);
            const float4 a = __ldg(rp), b = __ldg(rp + 1);
            r = make_tray(mk(a.x, a.y, a.z), mk(b.x, b.y, b.z), a.w);
            tmax = b.w;
        },
        [&](unsigned long long k, int rc) {
            if (rc < 0) set_status(status, KZ_ERR_STACK);
            occ[k] = rc == 2 ? 1 : 0;
        },
        dn, dt);
}

__global__ void k_intersect_stats(DevScene s, const kz_ray* __restrict__ rays, uint64_t n,
                                  unsigned long long* counters, uint32_t* status) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t nn = 0, nt = 0;
    if (i < n) {
        const float4* rp = reinterpret_cast<const float4*>(rays + i);
        const float4 a = __ldg(rp), b = __ldg(rp + 1);
        TRay r = make_tray(mk(a.x, a.y, a.z), mk(b.x, b.y, b.z), a.w);
        HitRec h;
        if (!trace_closest<true>(s, r, b.w, h, nn, nt)) set_status(status, KZ_ERR_STACK);
    }
    // warp reduction, one atomic per warp
    unsigned long long a0 = nn, a1 = nt;
    for (int o = 16; o > 0; o >>= 1) {
        a0 += __shfl_down_sync(0xffffffffu, a0, o);
        a1 += __shfl_down_sync(0xffffffffu, a1, o);
    }
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(counters, a0);
        atomicAdd(counters + 1, a1);
    }
}

template <bool kCount>
__global__ void __launch_bounds__(256) k_trace_paths(DevScene s, PathSoA p, uint32_t n, DevCounters* ctr) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t dn = 0, dt = 0;
    if (i < n) {
        const float4 o = p.o4[i], d = p.d4[i];
        TRay r = make_tray(xyz(o), xyz(d), kRayEps);
        HitRec h;
        if (!trace_closest<kCount>(s, r, __int_as_float(0x7f800000), h, dn, dt)) {
            set_status(&ctr->status, KZ_ERR_STACK);
            h.rec = -1;
        }
        p.hit[i] = make_float4(h.t, h.u, h.v, __int_as_float(h.rec));
    }
    if (kCount) warp_count(dn, dt, &ctr->fetch[0]);
}

// Closest hits of the wavefront's paths. kFew: with the way of few rays beside
// the persistent loop; the kernel of wavefronts above the joint trace's size
// leaves it out, its registers cost the loop 2 % there.
template <bool kCount, bool kFew>
__device__ __forceinline__ void trace_paths(ClosestSmem& m, DevScene& s, PathSoA p, uint32_t n, DevCounters* ctr,
                                            uint32_t& dn, uint32_t& dt) {
    const auto load = [&](uint32_t k, TRay& r, float& tmax) {
        const float4 o = p.o4[k], d = p.d4[k];
        r = make_tray(xyz(o), xyz(d), kRayEps);
        tmax = __int_as_float(0x7f800000);
    };
    const auto store = [&](uint32_t k, const HitRec& h) {
        p.hit[k] = make_float4(h.t, h.u, h.v, __int_as_float(h.rec));
    };
    if (kFew && n <= kFewRays)
        few_closest(m, s, n, &ctr->trace_next, &ctr->status, load, store);
    else
        persistent_closest_in<kCount, false>(m, s, n, &ctr->trace_next, &ctr->status, load, store, dn, dt);
}

// The shadow rays queued in iteration `ctr`; an unoccluded one adds its
// contribution to the film (and to the guiding records).
template <bool kCount, bool kGuided, typename Smem>
__device__ __forceinline__ void trace_shadow(Smem& m, DevScene& s, ShadowSoA sq, DevCounters* ctr, float* film,
                                             double* film64, VRec* recs, NRec* nee, uint32_t max_depth, uint32_t& dn,
                                             uint32_t& dt) {
    const auto unoccluded = [&](uint32_t ray) {
        const float4 cc = sq.c4[ray];
        film_add(film, film64, __float_as_uint(sq.d4[ray].w), xyz(cc));
        if (kGuided && recs) {
            const uint32_t tag = __float_as_uint(cc.w);
            const uint64_t rb = (uint64_t)(tag >> 4) * max_depth;
            propagate(recs, rb, tag & 15u, xyz(cc));
            if (nee) nee[rb + (tag & 15u)].n.w = 1.f;
        }
    };
    const auto load = [&](uint32_t k, TRay& r, float& tmax) {
        const float4 o = sq.o4[k], d = sq.d4[k];
        r = make_tray(xyz(o), xyz(d), kRayEps);
        tmax = o.w;
    };
    const auto done = [&](uint32_t ray, int rc) {
        if (rc < 0) set_status(&ctr->status, KZ_ERR_STACK);
        if (rc == 1) unoccluded(ray);
    };
    const uint32_t n = ctr->queue.shadow;
    if (!kCount && n <= kFewRays)
        few_any(m, s, n, &ctr->shadow_next, load, done);
    else
        persistent_any_in<kCount, false>(m, s, n, &ctr->shadow_next, load, done, dn, dt);
}

template <bool kCount>
__global__ void __launch_bounds__(256, KZ_TRACE_MINB) k_trace_paths_persistent(DevScene s, PathSoA p,
                                                                               const uint32_t* n_active,
                                                                               DevCounters* ctr) {
    __shared__ ClosestSmem m;
    uint32_t dn = 0, dt = 0;
    trace_paths<kCount, false>(m, s, p, *n_active, ctr, dn, dt);
    if (kCount) warp_count(dn, dt, &ctr->fetch[0]);
}

// The new camera paths of an iteration: each warp takes 32 consecutive ones,
// generates them and traces them as a bundle; one that reaches over the end of
// an image row is traced as a bundle per row (as one it would be as wide as
// the image).
constexpr int kBundleWarps = 4;  // per block
__global__ void __launch_bounds__(32 * kBundleWarps, 8)
    k_camera_bundles(DevScene s, DevCamera cam, PathParams pp, PathSoA p, IterSlots it) {
    __shared__ uint2 stacks[kBundleWarps][kWarpStack];
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const NewPaths nw = new_paths(it, blockIdx.x * blockDim.x + threadIdx.x);
    const uint32_t skip = (uint32_t)nw.first & 31u;  // bundles start at multiples of 32 path ids
    for (;;) {
        uint32_t j = 0;
        if (lane == 0) j = atomicAdd(&it.cur->camera_next, 32u);
        j = __shfl_sync(0xFFFFFFFFu, j, 0);
        if (j >= nw.count + skip) break;
        const bool live = j + lane >= skip && j + lane < nw.count + skip;
        const uint32_t i = live ? j + lane - skip : 0u, k = nw.slot + i;
        const uint64_t pid = nw.first + i;
        const CameraPath c = camera_path(cam, pp, pid);
        if (live) store_camera_path(cam, p, k, pid, c);
        const uint32_t row = live ? (uint32_t)(pid / pp.spp / cam.W) : 0xFFFFFFFFu;
        HitRec h{__int_as_float(0x7f800000), 0.f, 0.f, KZ_INVALID_ID, -1};
        for (uint32_t todo = __ballot_sync(0xFFFFFFFFu, live); todo;) {
            const uint32_t lead = __ffs(todo) - 1;
            const bool mine = row == __shfl_sync(0xFFFFFFFFu, row, lead);
            todo &= ~__ballot_sync(0xFFFFFFFFu, mine);
            const f3 d = mk(__shfl_sync(0xFFFFFFFFu, c.d.x, lead), __shfl_sync(0xFFFFFFFFu, c.d.y, lead),
                            __shfl_sync(0xFFFFFFFFu, c.d.z, lead));
            const TRay r = make_tray(ld3(cam.eye), mine ? c.d : d, kRayEps);
            WarpRay w;
            bool aborted;
            if (warp_bundle(s, r, mine, stacks[warp], w, aborted)) {
                if (mine && !aborted && w.rec >= 0) h = HitRec{w.t, w.V / w.det, w.W / w.det, w.prim, w.rec};
            } else if (mine) {
                uint32_t dn = 0, dt = 0;
                aborted = !trace_closest<false>(s, r, __int_as_float(0x7f800000), h, dn, dt);
            }
            if (mine && aborted) set_status(&it.cur->status, KZ_ERR_STACK);
            __syncwarp();
        }
        if (live) p.hit[k] = make_float4(h.t, h.u, h.v, __int_as_float(h.rec));
    }
}

// An iteration's closest hits and the shadow rays of the iteration before,
// which depend on nothing of this one, in one launch: a warp that finds no
// path left goes on to the shadow rays, so that one tail of long rays is
// waited for instead of two, and the launch is one instead of two.
template <bool kGuided>
__global__ void __launch_bounds__(256, KZ_TRACE_MINB) k_trace_both(DevScene s, PathSoA p, const uint32_t* n_active,
                                                                   DevCounters* ctr, ShadowSoA sq, DevCounters* prev,
                                                                   float* film, double* film64, VRec* recs, NRec* nee,
                                                                   uint32_t max_depth) {
    __shared__ ClosestSmem m;
    uint32_t dn = 0, dt = 0;
    trace_paths<false, true>(m, s, p, *n_active, ctr, dn, dt);
    trace_shadow<false, kGuided>(m, s, sq, prev, film, film64, recs, nee, max_depth, dn, dt);
}

// kz_intersect_closest: rays (o, tmin, d, tmax) in, hit fields out.
__global__ void __launch_bounds__(256, KZ_TRACE_MINB) k_intersect_closest_persistent(DevScene s, const kz_ray* __restrict__ rays,
                                                                      unsigned long long n, kz_hits hits,
                                                                      unsigned long long* next, uint32_t* status) {
    uint32_t dn = 0, dt = 0;
    persistent_closest<false>(
        s, n, next, status,
        [&](unsigned long long k, TRay& r, float& tmax) {
            const float4* rp = reinterpret_cast<const float4*>(rays + k);
            const float4 a = __ldg(rp), b = __ldg(rp + 1);
            r = make_tray(mk(a.x, a.y, a.z), mk(b.x, b.y, b.z), a.w);
            tmax = b.w;
        },
        [&](unsigned long long k, const HitRec& h) { store_hit(s, hits, k, h); }, dn, dt);
}

// One ray per warp, for calls of few rays (kz_intersect_closest / _any).
constexpr int kFewWarps = 4;  // per block
template <bool kAny>
__global__ void __launch_bounds__(32 * kFewWarps) k_intersect_few(DevScene s, const kz_ray* __restrict__ rays,
                                                                  uint32_t n, kz_hits hits, uint8_t* occ,
                                                                  uint32_t* status) {
    __shared__ uint2 stacks[kFewWarps][kWarpStack];
    const uint32_t warp = threadIdx.x >> 5, k = blockIdx.x * kFewWarps + warp;
    if (k >= n) return;
    const float4* rp = reinterpret_cast<const float4*>(rays + k);
    const float4 a = __ldg(rp), b = __ldg(rp + 1);
    const TRay r = make_tray(mk(a.x, a.y, a.z), mk(b.x, b.y, b.z), a.w);
    uint2* stack = stacks[warp];
    if (kAny) {
        const int rc = warp_any(s, r, b.w, stack);
        if (rc < 0) set_status(status, KZ_ERR_STACK);
        if ((threadIdx.x & 31u) == 0) occ[k] = rc == 2 ? 1 : 0;
    } else if (!warp_closest(s, r, b.w, stack, [&](const HitRec& h) { store_hit(s, hits, k, h); })) {
        set_status(status, KZ_ERR_STACK);
    }
}

template <bool kCount>
__global__ void __launch_bounds__(256) k_trace_shadow(DevScene s, ShadowSoA sq, DevCounters* ctr, float* film,
                                                      double* film64) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t dn = 0, dt = 0;
    if (i < ctr->queue.shadow) {
        const float4 o = sq.o4[i], d = sq.d4[i];
        TRay r = make_tray(xyz(o), xyz(d), kRayEps);
        bool overflow;
        const bool occluded = trace_any<kCount>(s, r, o.w, overflow, dn, dt);
        if (overflow) set_status(&ctr->status, KZ_ERR_STACK);
        if (!occluded && !overflow) film_add(film, film64, __float_as_uint(d.w), xyz(sq.c4[i]));
    }
    if (kCount) warp_count(dn, dt, &ctr->fetch[2]);
}

// Persistent form of k_trace_shadow for the device-driven loop.
template <bool kCount, bool kGuided>
__global__ void __launch_bounds__(256, KZ_TRACE_MINB) k_trace_shadow_persistent(DevScene s, ShadowSoA sq, DevCounters* ctr,
                                                                 float* film, double* film64, VRec* recs, NRec* nee,
                                                                 uint32_t max_depth) {
    __shared__ AnySmem m;
    uint32_t dn = 0, dt = 0;
    trace_shadow<kCount, kGuided>(m, s, sq, ctr, film, film64, recs, nee, max_depth, dn, dt);
    if (kCount) warp_count(dn, dt, &ctr->fetch[2]);
}

// Batched jobs: as k_trace_both (prev == nullptr: closest hits only).
__global__ void __launch_bounds__(256, KZ_TRACE_MINB) k_trace_both_batch(const DevJob* __restrict__ jobs, PathSoA p,
                                                                         const uint32_t* n_active, DevCounters* ctr,
                                                                         ShadowSoA sq, DevCounters* prev) {
    __shared__ ClosestSmem m;
    batch_trace_paths(m, jobs, p, *n_active, ctr);
    if (prev) batch_trace_shadow(m, jobs, sq, prev);
}

__global__ void __launch_bounds__(256, KZ_TRACE_MINB) k_trace_shadow_batch(const DevJob* __restrict__ jobs,
                                                                           ShadowSoA sq, DevCounters* ctr) {
    __shared__ AnySmem m;
    batch_trace_shadow(m, jobs, sq, ctr);
}

}  // namespace

void launch_pack_nodes(uint4* nodes, uint32_t n, cudaStream_t st) {
    if (n) k_pack_nodes<<<grid_for(n, 256), 256, 0, st>>>(nodes, n);
}

void launch_intersect_closest(const DevScene& s, const kz_ray* rays, uint64_t n, kz_hits hits,
                              unsigned long long* next, uint32_t* status, cudaStream_t st) {
    if (!n) return;
    if (n <= few_rays(s)) {
        k_intersect_few<false><<<grid_for(n, kFewWarps), 32 * kFewWarps, 0, st>>>(s, rays, (uint32_t)n, hits, nullptr,
                                                                                 status);
        return;
    }
    static const unsigned g = resident_grid(k_intersect_closest_persistent, 256);
    k_intersect_closest_persistent<<<trace_blocks(n, g), 256, 0, st>>>(s, rays, n, hits,
                                                                                                     next, status);
}

void launch_intersect_any(const DevScene& s, const kz_ray* rays, uint64_t n, uint8_t* occ,
                          unsigned long long* next, uint32_t* status, cudaStream_t st) {
    if (!n) return;
    if (n <= few_rays(s)) {
        k_intersect_few<true><<<grid_for(n, kFewWarps), 32 * kFewWarps, 0, st>>>(s, rays, (uint32_t)n, kz_hits{}, occ,
                                                                                status);
        return;
    }
    static const unsigned g = resident_grid(k_intersect_any_persistent, 256);
    k_intersect_any_persistent<<<trace_blocks(n, g), 256, 0, st>>>(s, rays, n, occ,
                                                                                                 next, status);
}

void launch_intersect_stats(const DevScene& s, const kz_ray* rays, uint64_t n, unsigned long long* counters,
                            uint32_t* status, cudaStream_t st) {
    if (!n) return;
    k_intersect_stats<<<grid_for(n, 128), 128, 0, st>>>(s, rays, n, counters, status);
}

void launch_trace_paths(const DevScene& s, PathSoA p, uint32_t n, DevCounters* ctr, bool count, uint32_t block,
                        cudaStream_t st) {
    if (!n) return;
    if (count) k_trace_paths<true><<<grid_for(n, block), block, 0, st>>>(s, p, n, ctr);
    else k_trace_paths<false><<<grid_for(n, block), block, 0, st>>>(s, p, n, ctr);
}

void launch_camera_bundles(const DevScene& s, const DevCamera& cam, const PathParams& pp, PathSoA p,
                           const IterSlots& it, cudaStream_t st) {
    if (!it.cap) return;
    static const unsigned g = resident_grid(k_camera_bundles, 32 * kBundleWarps);
    k_camera_bundles<<<std::min(g, grid_for(it.cap, 32 * kBundleWarps)), 32 * kBundleWarps, 0, st>>>(s, cam, pp, p, it);
}

void launch_trace_paths_dev(const DevScene& s, PathSoA p, uint32_t cap, const uint32_t* n_active, DevCounters* ctr,
                            bool count, cudaStream_t st) {
    if (!cap) return;
    if (count) {
        static const unsigned g = resident_grid(k_trace_paths_persistent<true>, 256);
        k_trace_paths_persistent<true><<<stage_grid(cap, g), 256, 0, st>>>(s, p, n_active, ctr);
    } else {
        static const unsigned g = resident_grid(k_trace_paths_persistent<false>, 256);
        k_trace_paths_persistent<false><<<stage_grid(cap, g), 256, 0, st>>>(s, p, n_active, ctr);
    }
}

void launch_trace_both(const DevScene& s, PathSoA p, uint32_t cap, const uint32_t* n_active, DevCounters* ctr,
                       ShadowSoA sq, DevCounters* prev, float* film, double* film64, const GuideShade* gs,
                       uint32_t max_depth, cudaStream_t st) {
    if (!cap) return;
    if (gs) {
        static const unsigned g = resident_grid(k_trace_both<true>, 256);
        k_trace_both<true><<<stage_grid(cap, g), 256, 0, st>>>(
            s, p, n_active, ctr, sq, prev, film, film64, gs->recs, gs->nee, max_depth);
    } else {
        static const unsigned g = resident_grid(k_trace_both<false>, 256);
        k_trace_both<false><<<stage_grid(cap, g), 256, 0, st>>>(s, p, n_active, ctr, sq, prev,
                                                                                    film, film64, nullptr, nullptr, 0);
    }
}

void launch_trace_shadow_dev(const DevScene& s, ShadowSoA sq, uint32_t n_max, DevCounters* ctr, bool count,
                             float* film, double* film64, const GuideShade* gs, uint32_t max_depth, cudaStream_t st) {
    if (!n_max) return;
    if (gs) {
        static const unsigned g = resident_grid(k_trace_shadow_persistent<false, true>, 256);
        k_trace_shadow_persistent<false, true><<<stage_grid(n_max, g), 256, 0, st>>>(
            s, sq, ctr, film, film64, gs->recs, gs->nee, max_depth);
    } else if (count) {
        static const unsigned g = resident_grid(k_trace_shadow_persistent<true, false>, 256);
        k_trace_shadow_persistent<true, false><<<stage_grid(n_max, g), 256, 0, st>>>(
            s, sq, ctr, film, film64, nullptr, nullptr, 0);
    } else {
        static const unsigned g = resident_grid(k_trace_shadow_persistent<false, false>, 256);
        k_trace_shadow_persistent<false, false><<<stage_grid(n_max, g), 256, 0, st>>>(
            s, sq, ctr, film, film64, nullptr, nullptr, 0);
    }
}

void launch_trace_shadow(const DevScene& s, ShadowSoA sq, uint32_t n_max, DevCounters* ctr, bool count, float* film,
                         double* film64, uint32_t block, cudaStream_t st) {
    if (!n_max) return;
    if (count) k_trace_shadow<true><<<grid_for(n_max, block), block, 0, st>>>(s, sq, ctr, film, film64);
    else k_trace_shadow<false><<<grid_for(n_max, block), block, 0, st>>>(s, sq, ctr, film, film64);
}

static unsigned grid_trace_batch() {
    static const unsigned g = resident_grid(k_trace_both_batch, 256);
    return g;
}

static unsigned grid_shadow_batch() {
    static const unsigned g = resident_grid(k_trace_shadow_batch, 256);
    return g;
}

void prepare_batch_wavefront() {
    (void)grid_trace_batch();
    (void)grid_shadow_batch();
}

void launch_trace_both_batch(const DevJob* jobs, PathSoA p, uint32_t cap, const uint32_t* n_active, DevCounters* ctr,
                             ShadowSoA sq, DevCounters* prev, cudaStream_t st) {
    if (!cap) return;
    k_trace_both_batch<<<stage_grid(cap, grid_trace_batch()), 256, 0, st>>>(jobs, p, n_active,
                                                                                               ctr, sq, prev);
}

void launch_trace_shadow_batch(const DevJob* jobs, ShadowSoA sq, uint32_t cap, DevCounters* ctr, cudaStream_t st) {
    if (!cap) return;
    k_trace_shadow_batch<<<stage_grid(cap, grid_shadow_batch()), 256, 0, st>>>(jobs, sq, ctr);
}

}  // namespace kz
