// kz_stages.cuh — device helpers shared by the wavefront stage kernels
// (kz_trace.cu: traversal kernels; kz_kernels.cu: generation, shading and the
// loop kernels): path-state flags, warp-aggregated counters and appends, film
// accumulation, camera path generation, the shaded vertex (shade_vertex), job
// lookup for batched renders, the persistent closest-hit driver and grid
// sizing. Each translation unit gets its own copy (internal linkage).
//
// The wavefront stages restate PathIntegrator::Li
// (src/core/integrator.cpp:362-561 in kazen_proto) with the estimator
// corrections listed at the top of k_shade. Random numbers: PCG32 stream
// (seed, path id); a camera path first draws the pixel jitter (2 floats,
// Renderer::render, src/core/renderer.cpp:57), then 9 floats per shaded
// vertex in a fixed order whatever branches run:
//   [0] light pick  [1] light triangle  [2,3] point on triangle  [4] roulette
//   [5] lobe pick   [6,7,8] lobe sample
#pragma once

#include <algorithm>

#include "kz_guide.cuh"
#include "kz_internal.h"
#include "kz_traverse.cuh"

namespace kz {
namespace {

constexpr uint32_t kSpecularFlag = 1u << 8;
// Batched wavefront: bits 12-31 of a path's d4.w hold its job index (0 for a
// single render); continuations keep them, shadow rays carry the job in c4.w.
constexpr uint32_t kJobShift = 12;
constexpr uint32_t kJobMask = 0xFFFFF000u;

__device__ __forceinline__ void set_status(uint32_t* status, uint32_t code) {
    if (status) atomicCAS(status, 0u, code);
}

__device__ __forceinline__ f3 ld3(const float* p) { return mk(p[0], p[1], p[2]); }
__device__ __forceinline__ f3 xyz(float4 v) { return mk(v.x, v.y, v.z); }

// Warp-aggregated append: one atomic per warp, lanes get consecutive slots.
__device__ __forceinline__ uint32_t warp_append(bool pred, uint32_t* counter) {
    const unsigned mask = __activemask();
    const unsigned ballot = __ballot_sync(mask, pred);
    if (!pred) return 0xFFFFFFFFu;
    const int lane = threadIdx.x & 31;
    const int leader = __ffs(ballot) - 1;
    uint32_t base = 0;
    if (lane == leader) base = atomicAdd(counter, (uint32_t)__popc(ballot));
    base = __shfl_sync(ballot, base, leader);
    return base + (uint32_t)__popc(ballot & ((1u << lane) - 1u));
}

__device__ __forceinline__ void store_hit(const DevScene& s, kz_hits hits, uint64_t i, const HitRec& h) {
    hits.t[i] = h.t;
    uint32_t geom = KZ_INVALID_ID, local = KZ_INVALID_ID;
    if (h.rec >= 0) {
        geom = __float_as_uint(__ldg(s.tris + (size_t)h.rec * 3 + 1).w);
        local = h.prim - __ldg(s.geom_offset + geom);
    }
    hits.prim_id[i] = local;
    if (hits.geom_id) hits.geom_id[i] = geom;
    if (hits.u) hits.u[i] = h.u;
    if (hits.v) hits.v[i] = h.v;
}

// ------------------------------------------------------------------ wavefront stages
struct CameraPath {
    f3 d;
    unsigned long long rng;
};
__device__ __forceinline__ CameraPath camera_path(const DevCamera& cam, const PathParams& pp, uint64_t pid) {
    const uint64_t pix = pid / pp.spp;
    const uint32_t px = (uint32_t)(pix % cam.W), py = (uint32_t)(pix / cam.W);
    Pcg rng;
    rng.seed(pp.seed, pid);
    const float jx = rng.nextf(), jy = rng.nextf();
    // Camera::generate_ray (src/core/camera.cpp:5-37): horizontal fov,
    // row 0 at the top unless flipped.
    const float sx = ((float)px + jx) / (float)cam.W;
    const float sy = ((float)py + jy) / (float)cam.H;
    const float nx = 2.0f * sx - 1.0f;
    const float ny = cam.flip * ((1.0f - 2.0f * sy) / cam.aspect);
    const float cx = nx * cam.tan_half;
    const float cy = ny * cam.tan_half;
    return CameraPath{normalize(ld3(cam.x) * cx + ld3(cam.y) * cy + ld3(cam.z) * (-1.0f)), rng.state};
}
__device__ __forceinline__ void store_camera_path(const DevCamera& cam, PathSoA dst, uint32_t k, uint64_t pid,
                                                  const CameraPath& c) {
    dst.o4[k] = make_float4(cam.eye[0], cam.eye[1], cam.eye[2], 0.f);
    dst.d4[k] = make_float4(c.d.x, c.d.y, c.d.z, __uint_as_float(kSpecularFlag));
    dst.b4[k] = make_float4(1.f, 1.f, 1.f, __uint_as_float((uint32_t)pid));
    dst.rng[k] = c.rng;
}
__device__ __forceinline__ void generate_camera_path(const DevCamera& cam, const PathParams& pp, PathSoA dst,
                                                     uint32_t k, uint64_t pid) {
    store_camera_path(cam, dst, k, pid, camera_path(cam, pp, pid));
}

__device__ __forceinline__ void generate_ray_path(const kz_ray* __restrict__ rays, const PathParams& pp, PathSoA dst,
                                                  uint32_t k, uint64_t pid) {
    Pcg rng;
    rng.seed(pp.seed, pid);
    const kz_ray r = rays[pid];
    dst.o4[k] = make_float4(r.ox, r.oy, r.oz, 0.f);
    dst.d4[k] = make_float4(r.dx, r.dy, r.dz, __uint_as_float(kSpecularFlag));
    dst.b4[k] = make_float4(1.f, 1.f, 1.f, __uint_as_float((uint32_t)pid));
    dst.rng[k] = rng.state;
}

// Sums two per-thread counters over the warp; one 64-bit atomic each.
__device__ __forceinline__ void warp_count(uint32_t a, uint32_t b, unsigned long long* dst) {
    unsigned long long x = a, y = b;
    for (int o = 16; o > 0; o >>= 1) {
        x += __shfl_down_sync(0xffffffffu, x, o);
        y += __shfl_down_sync(0xffffffffu, y, o);
    }
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(dst, x);
        atomicAdd(dst + 1, y);
    }
}

// Shared memory of the persistent traversal loops: the closest-hit loop's
// first stack entries and warp-shared leaf arrays, and the any-hit loop's
// leaf arrays (blocks of 256 threads). A kernel that runs both loops one
// after the other (the single-launch batch kernel) overlays them.
struct ClosestSmem {
    uint2 stack[(KZ_SMEM_STACK > 0 ? KZ_SMEM_STACK : 1) * 256];
    float4 ray[2 * 256];
    unsigned long long key[256];
    uint32_t rec[256];
    float4 vwdt[256];
    uint4 ent[kClosestSteps * 256];
};
struct AnySmem {
    float4 ray[2 * 256];
    unsigned long long key[256];
    uint32_t rec[256];
    uint4 ent[kAnySteps * 256];
};
// The any-hit loop's arrays; a kernel that runs both loops, its warps in
// either at the same time, takes them from the closest-hit loop's (each warp
// keeps its own part of every array).
__device__ __forceinline__ LeafShare any_share(AnySmem& m) {
    return LeafShare{m.ray, m.key, m.rec, nullptr, m.ent + (threadIdx.x & ~31u) * kAnySteps};
}
__device__ __forceinline__ LeafShare any_share(ClosestSmem& m) {
    return LeafShare{m.ray, m.key, m.rec, nullptr, m.ent + (threadIdx.x & ~31u) * kClosestSteps};
}
static_assert(kAnySteps <= kClosestSteps, "the any-hit loop's lists must fit the closest-hit loop's");

// Closest hit of ray k through persistent_rays_shared: load(k, r, tmax) sets
// the ray up, store(k, hit) writes the result; m is the block's shared memory.
// `s` is the lane's scene; load may repoint it per ray (batched jobs:
// kOwnScene). The fetch-counting variant keeps one node per step, so that its
// counts are those of a sequential traversal.
template <bool kCount, bool kOwnScene, typename Ctr, typename Load, typename Store>
__device__ __forceinline__ void persistent_closest_in(ClosestSmem& m, DevScene& s, Ctr n, Ctr* next,
                                                      uint32_t* status, Load load, Store store, uint32_t& dn,
                                                      uint32_t& dt) {
#if KZ_SMEM_STACK > 0 && KZ_SMEM_STACK < KZ_WIDE_STACK
    uint2 stack_lm[kWideStack - KZ_SMEM_STACK];
    const SplitStack<KZ_SMEM_STACK> stack{m.stack, stack_lm};
#else
    uint2 stack_lm[kWideStack];
    const LocalStack stack{stack_lm};
#endif
    constexpr int K = kCount ? 1 : kClosestSteps;
    const LeafShare sh{m.ray, m.key, m.rec, m.vwdt, m.ent + (threadIdx.x & ~31u) * kClosestSteps};
    AnyState c;
    TRay r;
    WideDir dir;
    float tmax = 0.f, tcur = 0.f;
    Ctr ray = 0;
    persistent_rays_shared<K>(
        n, next, kTraceRefill,
        [&](Ctr k) {
            ray = k;
            load(k, r, tmax);
            dir = wide_dir(r);
            any_begin(c);
            tcur = tmax;
            publish_ray(sh, r);
            best_begin(sh, tmax);
        },
        [&](LeafGroup& lg) {
            if (visit_node<kCount>(s, r, dir, tcur, c, stack, lg, dn) < 0) return -1;
            if (kCount) dt += __popc(lg.bits);
            return group_pop(c, stack);
        },
        [&](const LeafGroup(&g)[K]) { closest_leaves<kOwnScene>(sh, s.tris, g, tcur); },
        [&](int rc) {
            if (rc == 0) return false;
            HitRec h;
            best_finish(sh, rc > 0, tmax, h);
            if (rc < 0) set_status(status, KZ_ERR_STACK);
            store(ray, h);
            return true;
        });
}

// A warp's stack where its pending groups lie otherwise (other warps of the
// block may be in the persistent loops).
template <typename Smem>
__device__ __forceinline__ uint2* warp_stack(Smem& m) {
    static_assert(kAnySteps * 32 * sizeof(uint4) >= kWarpStack * sizeof(uint2), "a warp's lists hold its stack");
    return reinterpret_cast<uint2*>(any_share(m).ent);
}

// The same with the block's own static shared memory.
template <bool kCount, bool kOwnScene = false, typename Ctr, typename Load, typename Store>
__device__ __forceinline__ void persistent_closest(DevScene& s, Ctr n, Ctr* next, uint32_t* status, Load load,
                                                   Store store, uint32_t& dn, uint32_t& dt) {
    __shared__ ClosestSmem m;
    persistent_closest_in<kCount, kOwnScene>(m, s, n, next, status, load, store, dn, dt);
}

// Any hit of ray k through persistent_rays_shared: load(k, r, tmax) sets the
// ray up, done(k, rc) gets 1 (no hit), 2 (hit) or -1 (aborted: miss).
template <bool kCount, bool kOwnScene, typename Smem, typename Ctr, typename Load, typename Done>
__device__ __forceinline__ void persistent_any_in(Smem& m, DevScene& s, Ctr n, Ctr* next, Load load, Done done,
                                                  uint32_t& dn, uint32_t& dt) {
    uint2 stack_lm[kWideStack];  // all local: with 4 or 8 entries in shared memory the shadow stage gained nothing
    const LocalStack stack{stack_lm};
    constexpr int K = kCount ? 1 : kAnySteps;
    const LeafShare sh = any_share(m);
    AnyState c;
    TRay r;
    WideDir dir;
    float tmax = 0.f;
    Ctr ray = 0;
    bool hit = false;
    persistent_rays_shared<K>(
        n, next, kAnyRefill,
        [&](Ctr k) {
            ray = k;
            load(k, r, tmax);
            dir = wide_dir(r);
            any_begin(c);
            publish_ray(sh, r);
            publish_tmax(sh, tmax);
        },
        [&](LeafGroup& lg) {
            if (visit_node<kCount>(s, r, dir, tmax, c, stack, lg, dn) < 0) return -1;
            return group_pop(c, stack);
        },
        [&](const LeafGroup(&g)[K]) {
            const uint32_t hits = any_leaves<kOwnScene>(sh, s.tris, g);
            hit = hits != 0u;
            if (kCount) dt += any_tested(g[0].bits, hits);
        },
        [&](int rc) {
            if (hit && rc >= 0) rc = 2;
            if (rc == 0) return false;
            done(ray, rc);
            return true;
        });
}

template <bool kCount, bool kOwnScene = false, typename Ctr, typename Load, typename Done>
__device__ __forceinline__ void persistent_any(DevScene& s, Ctr n, Ctr* next, Load load, Done done, uint32_t& dn,
                                               uint32_t& dt) {
    __shared__ AnySmem m;
    persistent_any_in<kCount, kOwnScene>(m, s, n, next, load, done, dn, dt);
}

// At most kFewRays rays, a warp per ray: load, store and done as in the
// persistent loops (load on every lane, store and done on one).
template <typename Load, typename Store>
__device__ __forceinline__ void few_closest(ClosestSmem& m, DevScene& s, uint32_t n, uint32_t* next, uint32_t* status,
                                            Load load, Store store) {
    warp_rays(n, next, [&](uint32_t k) {
        TRay r;
        float tmax;
        load(k, r, tmax);
        if (!warp_closest(s, r, tmax, warp_stack(m), [&](const HitRec& h) { store(k, h); }))
            set_status(status, KZ_ERR_STACK);
    });
}
template <typename Smem, typename Load, typename Done>
__device__ __forceinline__ void few_any(Smem& m, DevScene& s, uint32_t n, uint32_t* next, Load load, Done done) {
    warp_rays(n, next, [&](uint32_t k) {
        TRay r;
        float tmax;
        load(k, r, tmax);
        const int rc = warp_any(s, r, tmax, warp_stack(m));
        if ((threadIdx.x & 31u) == 0) done(k, rc);
    });
}

__device__ __forceinline__ void film_add(float* film, double* film64, uint32_t idx, f3 c) {
    atomicAdd(film + 3 * (size_t)idx, c.x);
    atomicAdd(film + 3 * (size_t)idx + 1, c.y);
    atomicAdd(film + 3 * (size_t)idx + 2, c.z);
    if (film64) {
        atomicAdd(film64 + 3 * (size_t)idx, (double)c.x);
        atomicAdd(film64 + 3 * (size_t)idx + 1, (double)c.y);
        atomicAdd(film64 + 3 * (size_t)idx + 2, (double)c.z);
    }
}

// DiscrectPDF::sample (src/base/dpdf.h:31-36): lower_bound over cdf[0..n].
__device__ __forceinline__ uint32_t cdf_sample(const float* cdf, uint32_t n, float u) {
    uint32_t lo = 0, cnt = n + 1;
    while (cnt > 0) {
        uint32_t step = cnt / 2, it = lo + step;
        if (__ldg(cdf + it) < u) {
            lo = it + 1;
            cnt -= step + 1;
        } else {
            cnt = step;
        }
    }
    int idx = (int)lo - 1;
    if (idx < 0) idx = 0;
    return min((uint32_t)idx, n - 1);
}

// One shaded vertex per thread. Estimator corrections relative to the
// reference loop (each one keeps the estimator unbiased):
//  * NEE uses f*|cos| once (the reference multiplies Diffuse's f*cos by cos
//    again, integrator.cpp:475-480) and divides by the light pick pdf inside
//    the MIS weight as well as outside;
//  * BSDF sampling divides by the direction pdf (integrator.cpp:503-505
//    multiplies by f only) and picks the lobe by its selection probability;
//  * emission hits weigh against the light pdf of the sampled direction
//    (integrator.cpp:452-462 reuses the previous light sample's pdf);
//  * max_depth counts shaded vertices (the reference steps depth twice per
//    loop, integrator.cpp:420,555).
// Guided mode (learned path guiding, not in the reference) additionally:
//  * on materials without delta lobes, samples the direction from the
//    network's vMF mixture with probability alpha and from the BSDF mixture
//    otherwise, with the one-sample MIS pdf alpha*q + (1-alpha)*p_bsdf in the
//    path weight, the NEE MIS weight and the next emission hit's MIS weight;
//  * records every such vertex (position, normal, direction, pdf,
//    throughput after it) and adds each later contribution, divided by that
//    throughput, to the vertex's incident-radiance estimate: the training
//    data of the network.
__device__ __forceinline__ void propagate(VRec* recs, uint64_t rbase, uint32_t depth, f3 c) {
    for (uint32_t k = 0; k < depth; ++k) {
        VRec& r = recs[rbase + k];
        if (r.n.w == 0.f) continue;
        const float4 b = r.beta;
        r.L.x += b.x > 0.f ? c.x / b.x : 0.f;
        r.L.y += b.y > 0.f ? c.y / b.y : 0.f;
        r.L.z += b.z > 0.f ? c.z / b.z : 0.f;
    }
}

// ------------------------------------------------------------------ textures
// OSL checkerboard (int() truncates, as the shader's int(fmod(..)) does) or
// a bilinear lookup with periodic wrap, texel centres at (i + 0.5) / w.
__device__ __noinline__ f3 tex_eval(const DevScene& s, int32_t k, float u, float v) {
    const DevTexture& tx = s.textures[k];
    if (!isfinite(u)) u = 0.f;
    if (!isfinite(v)) v = 0.f;
    if (tx.kind == KZ_TEX_CHECKER) {
        const float cs = fmodf(u * tx.scale_s, 2.f), ct = fmodf(v * tx.scale_t, 2.f);
        const int a = isfinite(cs) ? (int)cs : 0, b = isfinite(ct) ? (int)ct : 0;
        return (a ^ b) == 0 ? mk(tx.Ca[0], tx.Ca[1], tx.Ca[2]) : mk(tx.Cb[0], tx.Cb[1], tx.Cb[2]);
    }
    u -= floorf(u);
    v -= floorf(v);
    const float x = u * (float)tx.w - 0.5f, y = v * (float)tx.h - 0.5f;
    const float fx = floorf(x), fy = floorf(y);
    const float ax = x - fx, ay = y - fy;
    const uint32_t x0 = fx < 0.f ? tx.w - 1 : min((uint32_t)fx, tx.w - 1), x1 = x0 + 1 == tx.w ? 0 : x0 + 1;
    const uint32_t y0 = fy < 0.f ? tx.h - 1 : min((uint32_t)fy, tx.h - 1), y1 = y0 + 1 == tx.h ? 0 : y0 + 1;
    const float* d = s.tex_data + tx.offset;
    const f3 c00 = ld3(d + ((size_t)y0 * tx.w + x0) * 3), c10 = ld3(d + ((size_t)y0 * tx.w + x1) * 3);
    const f3 c01 = ld3(d + ((size_t)y1 * tx.w + x0) * 3), c11 = ld3(d + ((size_t)y1 * tx.w + x1) * 3);
    return (c00 * (1.f - ax) + c10 * ax) * (1.f - ay) + (c01 * (1.f - ax) + c11 * ax) * ay;
}

// Radiance of a ray leaving the scene: the environment in latitude-longitude form.
__device__ __noinline__ f3 env_radiance(const DevScene& s, f3 d) {
    f3 e = mk(s.env.x, s.env.y, s.env.z);
    if (s.env_tex >= 0) {
        const float u = 0.5f + atan2f(d.x, -d.z) * (0.5f * kInvPi);
        const float v = acosf(fminf(fmaxf(d.y, -1.f), 1.f)) * kInvPi;
        e = hmul(e, tex_eval(s, s.env_tex, u, v));
    }
    return e;
}

// Weight of lobe k at this vertex: the texture tint applies to the lobes
// that reference the material's texture.
__device__ __forceinline__ f3 lobe_weight(const kz_lobe& lb, bool textured, f3 tint) {
    const f3 w = ld3(lb.weight);
    return textured && lb.params[KZ_LOBE_TEXTURE_PARAM] != 0.f ? hmul(w, tint) : w;
}

struct ShadeOut {
    bool cont = false, shadow = false;
    float4 o_next, d_next, b_next, s_o, s_d, s_c;
    unsigned long long rng_next = 0;
    f3 Lsum = {0.f, 0.f, 0.f};  // contribution to the film pixel film_idx
    uint32_t film_idx = 0;
};

// Next-event estimation's light sample seen from P: the light picked by u0, its
// triangle by u1, the point on it by u2 and u3.
struct LightSample {
    f3 dir, Le;
    float dist, dist2, pdf;  // pdf in solid angle, with the pick probability
    bool point, lit;         // lit: P lies on the emitting side
};
__device__ __forceinline__ LightSample sample_light(const DevScene& s, f3 P, float u0, float u1, float u2, float u3) {
    const uint32_t nl = s.n_lights;
    const uint32_t li = min((uint32_t)(u0 * (float)nl), nl - 1);
    const DevLight lt = s.lights[li];
    LightSample r;
    // a point light (PointLight, light.cpp:18-31) has no triangles: its
    // position is the one light_tris record it names
    r.point = lt.tri_count == 0;
    f3 p, nlgt = mk(0.f, 0.f, 0.f);
    if (r.point) {
        p = xyz(__ldg(s.light_tris + (size_t)lt.tri_begin * 3));
    } else {
        const uint32_t kk = cdf_sample(s.light_cdf + lt.cdf_begin, lt.tri_count, u1);
        const float4* lq = s.light_tris + (size_t)(lt.tri_begin + kk) * 3;
        const f3 a0 = xyz(__ldg(lq)), a1 = xyz(__ldg(lq + 1)), a2 = xyz(__ldg(lq + 2));
        const float su0 = sqrtf(u2);
        const float bu0 = 1.f - su0;
        const float bv0 = u3 * su0;
        p = a0 * bu0 + a1 * bv0 + a2 * (1.f - bu0 - bv0);
        nlgt = normalize(cross(a1 - a0, a2 - a0));
    }
    const f3 lv = p - P;
    r.dist2 = dot(lv, lv);
    r.dist = sqrtf(r.dist2);
    r.dir = mk(lv.x / r.dist, lv.y / r.dist, lv.z / r.dist);
    const float cos_l = r.point ? 1.f : -dot(r.dir, nlgt);
    r.lit = cos_l > 0.f && r.dist2 > 0.f;
    // a delta light is picked with probability 1/nl and weighs no MIS
    r.pdf = r.point ? 1.0f / (float)nl : r.dist2 / (cos_l * lt.area) * (1.0f / (float)nl);
    r.Le = ld3(lt.Le);
    return r;
}

// Shading normal and point of a hit: the interpolated vertex normal, with the
// point moved off the flat triangle by the shadow-terminator offset (Hanika
// 2021), as TriangleMesh::post_hit does (shape.cpp:628-656); Ng and P as they
// are for a mesh without normals.
__device__ __forceinline__ void smooth_hit(const DevScene& s, int rec, const float4 hit, f3 v0, f3 v1, f3 v2, f3& Ns,
                                           f3& P) {
    const float4 m0 = __ldg(s.tri_nrm + (size_t)rec * 3);
    if (m0.w == 0.f) return;
    const f3 n0 = xyz(m0), n1 = xyz(__ldg(s.tri_nrm + (size_t)rec * 3 + 1)),
             n2 = xyz(__ldg(s.tri_nrm + (size_t)rec * 3 + 2));
    const float b0 = 1.f - hit.y - hit.z;
    Ns = normalize(n0 * b0 + n1 * hit.y + n2 * hit.z);
    const f3 Pb = v0 * b0 + v1 * hit.y + v2 * hit.z;
    const float e0 = fminf(0.f, dot(Pb - v0, n0)), e1 = fminf(0.f, dot(Pb - v1, n1)),
                e2 = fminf(0.f, dot(Pb - v2, n2));
    P = Pb - (n0 * (b0 * e0) + n1 * (hit.y * e1) + n2 * (hit.z * e2));
}

// Texture tint of a hit at its uv (interpolated vertex uvs; the barycentrics
// of vertices 1, 2 when the mesh has none).
__device__ __forceinline__ f3 hit_tint(const DevScene& s, int rec, const float4 hit, int32_t tex) {
    const float2 q0 = s.tri_uv[(size_t)rec * 3], q1 = s.tri_uv[(size_t)rec * 3 + 1], q2 = s.tri_uv[(size_t)rec * 3 + 2];
    const float b0 = 1.f - hit.y - hit.z;
    return tex_eval(s, tex, b0 * q0.x + hit.y * q1.x + hit.z * q2.x, b0 * q0.y + hit.y * q1.y + hit.z * q2.y);
}

// Weight of an emission hit against the light sample it competes with (MIS),
// or against nothing: after a specular bounce, and when only one of the two
// estimators runs.
__device__ __forceinline__ float emission_weight(const DevScene& s, const PathParams& pp, uint32_t geom, bool prev_spec,
                                                 float prev_pdf, float t, f3 d, f3 Ng) {
    if (prev_spec || pp.estimator == 2u) return 1.f;
    const int li = __ldg(s.geom_light + geom);
    if (li < 0) return 1.f;
    if (pp.estimator == 1u) return 0.f;  // this light was sampled directly
    const float cos_l = -dot(d, Ng);
    const float lpdf = (t * t) / (cos_l * s.lights[li].area) * (1.0f / (float)s.n_lights);
    return power_heuristic(prev_pdf, lpdf);
}

// A path that leaves the scene: throughput times the environment, without MIS
// (the environment is not sampled as a light), integrator.cpp:545-552.
__device__ __forceinline__ void shade_miss(const DevScene& s, const PathParams& pp, const float4 d4, const float4 b4,
                                           ShadeOut& out) {
    out.Lsum = hmul(xyz(b4), env_radiance(s, xyz(d4)));
    out.film_idx = __float_as_uint(b4.w) / pp.spp;
}

// One vertex of a plain material (kPlainClass: at most one lobe, diffuse about
// the shading normal), as shade_vertex shades it, bit for bit: with one lobe
// its selection probability is wsum / wsum, the lobe's value and pdf are both
// max(cos, 0) / pi, and neither the incident direction nor the frame is needed
// for the light sample. Most vertices of most scenes are of
// this kind, and the general function holds arrays over eight lobes and calls
// the 21-way lobe switch twice.
template <bool kAttr>
__device__ __forceinline__ void shade_plain(const DevScene& s, const PathParams& pp, const float4 hit, const float4 o4,
                                            const float4 d4, const float4 b4, unsigned long long rng_state,
                                            ShadeOut& out) {
    const int rec = __float_as_int(hit.w);
    const uint32_t pid = __float_as_uint(b4.w);
    const uint32_t flags = __float_as_uint(d4.w);
    const uint32_t depth = flags & 0xffu;
    Pcg rng;
    rng.state = rng_state;
    rng.inc = ((uint64_t)pid << 1u) | 1u;
    float u[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) u[k] = rng.nextf();

    const float4* tp = s.tris + (size_t)rec * 3;
    const float4 ta = __ldg(tp), tb = __ldg(tp + 1), tc = __ldg(tp + 2);
    const uint32_t m = __float_as_uint(tc.w);
    const f3 v0 = xyz(ta), v1 = xyz(tb), v2 = xyz(tc);
    const f3 Ng = normalize(cross(v1 - v0, v2 - v0)), d = xyz(d4);
    f3 N = Ng, P = xyz(o4) + d * hit.x;
    if (kAttr && s.tri_nrm) smooth_hit(s, rec, hit, v0, v1, v2, N, P);
    const float4 plain = __ldg(s.mat_plain + m);
    f3 lw = xyz(plain);
    if (kAttr && s.mat_tex) {
        const int32_t mtex = __ldg(s.mat_tex + m);
        if (mtex >= 0) lw = hmul(lw, hit_tint(s, rec, hit, mtex));
    }
    f3 beta = xyz(b4);
    out.film_idx = pid / pp.spp;
    if (plain.w != 0.f && dot(d, N) < 0.f)  // the material emits
        out.Lsum = hmul(beta, ld3(s.materials[m].Le)) *
                   emission_weight(s, pp, __float_as_uint(tb.w), (flags & kSpecularFlag) != 0, o4.w, hit.x, d, Ng);
    const float wsum = (lw.x * beta.x + lw.y * beta.y + lw.z * beta.z) * (1.f / (beta.x + beta.y + beta.z));
    if (!(wsum > 0.f)) return;
    const float lp = wsum <= 3.402823466e38f ? 1.f : __int_as_float(0x7fffffff);  // inf / inf

    if (pp.estimator != 2u && s.n_lights > 0) {
        const LightSample ls = sample_light(s, P, u[0], u[1], u[2], u[3]);
        if (ls.lit) {
            const float e = fmaxf(dot(ls.dir, N), 0.f) * kInvPi;
            const f3 f = lw * e;
            if (!is_zero(f)) {
                const float w = ls.point || pp.estimator == 1u ? 1.f : power_heuristic(ls.pdf, lp * e);
                const f3 Le_l = ls.point ? ls.Le * (1.f / (ls.dist2 * 0.1f)) : ls.Le;
                const f3 c = hmul(hmul(beta, f), Le_l) * (w / ls.pdf);
                out.shadow = true;
                out.s_o = make_float4(P.x, P.y, P.z, ls.dist - kRayEps);
                out.s_d = make_float4(ls.dir.x, ls.dir.y, ls.dir.z, __uint_as_float(out.film_idx));
                out.s_c = make_float4(c.x, c.y, c.z, __uint_as_float(flags >> kJobShift));
            }
        }
    }
    if (depth + 1 >= pp.max_depth) return;
    if (depth >= pp.rr_min) {
        const float prob = fminf(max_comp(beta) * 0.9025f, 0.99f);
        if (prob < u[4]) return;
        beta = beta * (1.f / prob);
    }
    const f3 wo = cosine_hemisphere(u[6], u[7]);
    const float e = fmaxf(wo.y, 0.f) * kInvPi;
    const float pdf = lp * e;
    if (!(pdf > 0.f)) return;
    beta = hmul(beta, (lw * e) * (1.f / pdf));
    if (is_zero(beta)) return;
    const f3 dn = normalize(Frame(N).to_world(wo));
    out.cont = true;
    out.o_next = make_float4(P.x, P.y, P.z, pdf);
    out.d_next = make_float4(dn.x, dn.y, dn.z, __uint_as_float((depth + 1) | (flags & kJobMask)));
    out.b_next = make_float4(beta.x, beta.y, beta.z, b4.w);
    out.rng_next = rng.state;
}

// One shaded path vertex: emission, next-event estimation (the shadow ray is
// returned, not traced), roulette and direction sampling. `raw` holds the
// guiding network's outputs for this path (guided mode only). kAttr = false
// compiles the vertex attributes out (texture tint, shading normals) for
// scenes that have neither.
template <bool kGuided, bool kAttr = true>
__device__ __forceinline__ void shade_vertex(const DevScene& s, const PathParams& pp, const float4 hit,
                                             const float4 o4, const float4 d4, const float4 b4,
                                             unsigned long long rng_state, const GuideShade& gs, const float* raw,
                                             ShadeOut& out) {
    const int rec = __float_as_int(hit.w);
    if (rec >= 0) {
        const uint32_t pid = __float_as_uint(b4.w);
        const uint32_t film_idx = pid / pp.spp;
        const uint32_t flags = __float_as_uint(d4.w);
        const uint32_t depth = flags & 0xffu;
        const bool prev_spec = (flags & kSpecularFlag) != 0;
        const float prev_pdf = o4.w;
        Pcg rng;
        rng.state = rng_state;
        rng.inc = ((uint64_t)pid << 1u) | 1u;
        float u[9];
#pragma unroll
        for (int k = 0; k < 9; ++k) u[k] = rng.nextf();

        const float4* tp = s.tris + (size_t)rec * 3;
        const float4 ta = __ldg(tp), tb = __ldg(tp + 1), tc = __ldg(tp + 2);
        const uint32_t geom = __float_as_uint(tb.w);
        const kz_material& mat = s.materials[__float_as_uint(tc.w)];
        const f3 v0 = xyz(ta), v1 = xyz(tb), v2 = xyz(tc);
        const f3 Ng = normalize(cross(v1 - v0, v2 - v0));
        const f3 d = xyz(d4);
        f3 P = xyz(o4) + d * hit.x;
        f3 Ns = Ng;
        if (kAttr && s.tri_nrm) smooth_hit(s, rec, hit, v0, v1, v2, Ns, P);
        const int32_t mtex = kAttr && s.mat_tex ? __ldg(s.mat_tex + __float_as_uint(tc.w)) : -1;
        const bool textured = mtex >= 0;
        const f3 tint = textured ? hit_tint(s, rec, hit, mtex) : mk(1.f, 1.f, 1.f);
        const Frame fr(Ns);
        const f3 wi = -fr.to_local(d);
        f3 beta = xyz(b4);
        f3 Lsum = mk(0.f, 0.f, 0.f);
        const uint32_t nl = s.n_lights;
        const uint64_t rbase = kGuided ? ((uint64_t)pid - gs.pass_first) * pp.max_depth : 0;

        // 1. emission (front face only, against the shading normal:
        // single_emissive_surface, integrator.cpp:454)
        const f3 Le = ld3(mat.Le);
        if (!is_zero(Le) && dot(d, Ns) < 0.f) {
            Lsum = Lsum + hmul(beta, Le) * emission_weight(s, pp, geom, prev_spec, prev_pdf, hit.x, d, Ng);
            // MIS-weighted, like the next-event samples it pairs with
            if (kGuided && gs.recs) propagate(gs.recs, rbase, depth, Lsum);
        }

        // lobe selection probabilities (CompositeClosure::compute_pdfs)
        const uint32_t nlobes = min(mat.n_lobes, (uint32_t)KZ_MAX_LOBES);
        float lp[KZ_MAX_LOBES];
        const float winv = 1.f / (beta.x + beta.y + beta.z);
        float wsum = 0.f;
        bool any_smooth = false, any_delta = false;
        for (uint32_t k = 0; k < nlobes; ++k) {
            const kz_lobe& lb = mat.lobes[k];
            const f3 lw = lobe_weight(lb, textured, tint);
            lp[k] = (lw.x * beta.x + lw.y * beta.y + lw.z * beta.z) * winv;
            wsum += lp[k];
            const bool dl = lobe_is_delta(lb.closure_id);
            any_smooth |= !dl;
            any_delta |= dl;
        }
        if (wsum > 0.f)
            for (uint32_t k = 0; k < nlobes; ++k) lp[k] /= wsum;
        const bool guided = kGuided && any_smooth && !any_delta && wsum > 0.f;
        VmfMixture mix;
        if (kGuided && guided)
            mixture_for_shading(raw, hmul(P - mk(s.box_lo.x, s.box_lo.y, s.box_lo.z), mk(s.box_inv.x, s.box_inv.y, s.box_inv.z)),
                                mk(1.f / s.box_inv.x, 1.f / s.box_inv.y, 1.f / s.box_inv.z), mix);
        const float alpha = gs.alpha;

        // 2. next-event estimation (none when sampling the BSDF only)
        if (pp.estimator != 2u && nl > 0 && any_smooth && wsum > 0.f) {
            const LightSample ls = sample_light(s, P, u[0], u[1], u[2], u[3]);
            const f3 ldir = ls.dir;
            const float dist = ls.dist, dist2 = ls.dist2, lpdf = ls.pdf;
            const bool point = ls.point;
            if (ls.lit) {
                const f3 wo = fr.to_local(ldir);
                f3 f = mk(0.f, 0.f, 0.f);
                float bpdf = 0.f;
                for (uint32_t k = 0; k < nlobes; ++k) {
                    const kz_lobe& lb = mat.lobes[k];
                    if (lobe_is_delta(lb.closure_id)) continue;
                    const LobeEval e = lobe_eval(lb, wi, wo);
                    f = f + hmul(lobe_weight(lb, textured, tint), e.f);
                    bpdf += lp[k] * e.pdf;
                }
                // the MIS partner of this light sample is the next direction,
                // sampled from the guide mixture; at the last vertex no
                // direction follows, so the weight is the plain one and the
                // guided image converges to the plain image at every depth
                if (kGuided && guided && depth + 1 < pp.max_depth)
                    bpdf = alpha * mixture_pdf_shading(mix, ldir) + (1.f - alpha) * bpdf;
                if (!is_zero(f)) {
                    const float w = point || pp.estimator == 1u ? 1.f : power_heuristic(lpdf, bpdf);
                    // PointLight::sample's falloff: radiance / (0.1 |d|^2)
                    const f3 Le_l = point ? ls.Le * (1.f / (dist2 * 0.1f)) : ls.Le;
                    const f3 c = hmul(hmul(beta, f), Le_l) * (w / lpdf);
                    out.shadow = true;
                    out.s_o = make_float4(P.x, P.y, P.z, dist - kRayEps);
                    out.s_d = make_float4(ldir.x, ldir.y, ldir.z, __uint_as_float(film_idx));
                    const uint32_t tag = kGuided ? (uint32_t)(((uint64_t)pid - gs.pass_first) << 4 | (depth & 15u))
                                                 : flags >> kJobShift;
                    out.s_c = make_float4(c.x, c.y, c.z, __uint_as_float(tag));
                    if (kGuided && gs.nee && guided) {
                        // training sample: the light direction with its
                        // MIS-weighted share of L*f*cos over the light pdf
                        const f3 fl = hmul(f, Le_l);
                        const float wt = (0.2126f * fl.x + 0.7152f * fl.y + 0.0722f * fl.z) * (w / lpdf);
                        const f3 p01 = hmul(P - mk(s.box_lo.x, s.box_lo.y, s.box_lo.z),
                                            mk(s.box_inv.x, s.box_inv.y, s.box_inv.z));
                        NRec& nr = gs.nee[rbase + depth];
                        nr.p = make_float4(p01.x, p01.y, p01.z, wt);
                        nr.n = make_float4(Ng.x, Ng.y, Ng.z, 0.f);
                        nr.d = make_float4(ldir.x, ldir.y, ldir.z, 0.f);
                    }
                }
            }
        }

        bool alive = depth + 1 < pp.max_depth;
        // 3. Russian roulette (integrator.cpp:491-498)
        if (alive && depth >= pp.rr_min) {
            const float prob = fminf(max_comp(beta) * 0.9025f, 0.99f);
            if (prob < u[4]) alive = false;
            else beta = beta * (1.f / prob);
        }
        // 4. direction sampling
        if (kGuided && guided && alive) {
            // one-sample MIS of the learned vMF mixture and the BSDF mixture
            f3 wo, wdir;
            bool ok = true;
            if (u[5] < alpha) {
                wdir = mixture_sample(mix, u[5] / alpha, u[6], u[7]);
                wo = fr.to_local(wdir);
            } else {
                const float us = (u[5] - alpha) / (1.f - alpha);
                uint32_t sel = nlobes - 1;
                float acc = 0.f;
                for (uint32_t k = 0; k < nlobes; ++k) {
                    acc += lp[k];
                    if (us < acc) {
                        sel = k;
                        break;
                    }
                }
                while (sel > 0 && lp[sel] == 0.f) --sel;
                const LobeSample smp = lobe_sample(mat.lobes[sel], wi, u[6], u[7], u[8]);
                ok = smp.valid;
                wo = smp.wo;
                wdir = normalize(fr.to_world(wo));
            }
            f3 f = mk(0.f, 0.f, 0.f);
            float pdf = 0.f;
            if (ok) {
                for (uint32_t k = 0; k < nlobes; ++k) {
                    const kz_lobe& lb = mat.lobes[k];
                    const LobeEval e = lobe_eval(lb, wi, wo);
                    f = f + hmul(lobe_weight(lb, textured, tint), e.f);
                    pdf += lp[k] * e.pdf;
                }
                pdf = alpha * mixture_pdf_shading(mix, wdir) + (1.f - alpha) * pdf;
            }
            alive = ok && pdf > 0.f && !is_zero(f);
            if (alive) {
                beta = hmul(beta, f * (1.f / pdf));
                alive = !is_zero(beta);
            }
            if (alive) {
                out.cont = true;
                out.o_next = make_float4(P.x, P.y, P.z, pdf);
                out.d_next = make_float4(wdir.x, wdir.y, wdir.z, __uint_as_float((depth + 1) | (flags & kJobMask)));
                out.b_next = make_float4(beta.x, beta.y, beta.z, b4.w);
                out.rng_next = rng.state;
            }
            if (alive && gs.recs) {
                VRec& r = gs.recs[rbase + depth];
                const f3 p01 = hmul(P - mk(s.box_lo.x, s.box_lo.y, s.box_lo.z),
                                    mk(s.box_inv.x, s.box_inv.y, s.box_inv.z));
                r.p = make_float4(p01.x, p01.y, p01.z, pdf);
                r.n = make_float4(Ng.x, Ng.y, Ng.z, 1.f);
                // d.w: luminance of f*|cos| along the sampled direction,
                // so the network learns the whole integrand L*f*cos
                r.d = make_float4(wdir.x, wdir.y, wdir.z, 0.2126f * f.x + 0.7152f * f.y + 0.0722f * f.z);
                r.beta = make_float4(beta.x, beta.y, beta.z, 0.f);
                r.L = make_float4(0.f, 0.f, 0.f, 0.f);
            }
        } else if (alive && wsum > 0.f) {
            // BSDF sample (one-sample mixture over the non-delta lobes)
            uint32_t sel = nlobes - 1;
            float acc = 0.f;
            for (uint32_t k = 0; k < nlobes; ++k) {
                acc += lp[k];
                if (u[5] < acc) {
                    sel = k;
                    break;
                }
            }
            while (sel > 0 && lp[sel] == 0.f) --sel;
            const kz_lobe& ls = mat.lobes[sel];
            const LobeSample smp = lobe_sample(ls, wi, u[6], u[7], u[8]);
            alive = smp.valid;
            f3 weight = mk(0.f, 0.f, 0.f);
            float pdf_dir = 0.f;
            if (alive) {
                if (smp.delta) {
                    weight = hmul(lobe_weight(ls, textured, tint), smp.weight) * (1.f / lp[sel]);
                } else {
                    f3 f = mk(0.f, 0.f, 0.f);
                    float pdf = 0.f;
                    for (uint32_t k = 0; k < nlobes; ++k) {
                        const kz_lobe& lb = mat.lobes[k];
                        if (lobe_is_delta(lb.closure_id)) continue;
                        // the sampled lobe's own value came with the sample
                        const LobeEval e = k == sel ? LobeEval{smp.f, smp.pdf} : lobe_eval(lb, wi, smp.wo);
                        f = f + hmul(lobe_weight(lb, textured, tint), e.f);
                        pdf += lp[k] * e.pdf;
                    }
                    alive = pdf > 0.f;
                    if (alive) weight = f * (1.f / pdf);
                    pdf_dir = pdf;
                }
            }
            if (alive) {
                beta = hmul(beta, weight);
                alive = !is_zero(beta);
            }
            if (alive) {
                const f3 dn = normalize(fr.to_world(smp.wo));
                out.cont = true;
                out.o_next = make_float4(P.x, P.y, P.z, pdf_dir);
                out.d_next = make_float4(
                    dn.x, dn.y, dn.z,
                    __uint_as_float((depth + 1) | (smp.delta ? kSpecularFlag : 0u) | (flags & kJobMask)));
                out.b_next = make_float4(beta.x, beta.y, beta.z, b4.w);
                out.rng_next = rng.state;
            }
        }
        out.Lsum = Lsum;
        out.film_idx = film_idx;
    } else if (s.has_env) {
        shade_miss(s, pp, d4, b4, out);
        if (kGuided && gs.recs) {
            const uint32_t depth = __float_as_uint(d4.w) & 0xffu;
            propagate(gs.recs, ((uint64_t)__float_as_uint(b4.w) - gs.pass_first) * pp.max_depth, depth, out.Lsum);
        }
    }
}

__device__ __forceinline__ uint32_t find_job(const DevJob* __restrict__ jobs, uint32_t n_jobs, unsigned long long g) {
    uint32_t lo = 0, hi = n_jobs;  // last job with path_begin <= g
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (jobs[mid].path_begin <= g) lo = mid;
        else hi = mid;
    }
    return lo;
}

// The traversal reads only these fields of a scene.
__device__ __forceinline__ void trace_fields(DevScene& dst, const DevScene& src) {
    dst.nodes = src.nodes;
    dst.tris = src.tris;
    dst.n_nodes = src.n_nodes;
    dst.n_tris = src.n_tris;
}

// ---- stages of the batched wavefront (jobs of several scenes in one
// wavefront), as device functions shared by the per-stage kernels and the
// single persistent kernel of KZ_BATCH_PERSISTENT.

// Closest hits of the wavefront's paths; each path's scene through its job.
__device__ __forceinline__ void batch_trace_paths(ClosestSmem& m, const DevJob* __restrict__ jobs, PathSoA p,
                                                  uint32_t n, DevCounters* ctr) {
    uint32_t dn = 0, dt = 0;
    DevScene ls;
    const auto load = [&](uint32_t k, TRay& r, float& tmax) {
        const float4 o = p.o4[k], d = p.d4[k];
        trace_fields(ls, jobs[__float_as_uint(d.w) >> kJobShift].scene);
        r = make_tray(xyz(o), xyz(d), kRayEps);
        tmax = __int_as_float(0x7f800000);
    };
    const auto store = [&](uint32_t k, const HitRec& h) {
        p.hit[k] = make_float4(h.t, h.u, h.v, __int_as_float(h.rec));
    };
    if (n <= kFewRays)
        few_closest(m, ls, n, &ctr->trace_next, &ctr->status, load, store);
    else
        persistent_closest_in<false, true>(m, ls, n, &ctr->trace_next, &ctr->status, load, store, dn, dt);
}

// Shadow rays of the wavefront; an unoccluded one adds its contribution to
// its job's film.
template <typename Smem>
__device__ __forceinline__ void batch_trace_shadow(Smem& m, const DevJob* __restrict__ jobs, ShadowSoA sq,
                                                   DevCounters* ctr) {
    uint32_t dn = 0, dt = 0;
    DevScene ls;
    const auto load = [&](uint32_t k, TRay& r, float& tmax) {
        const float4 o = sq.o4[k], d = sq.d4[k];
        trace_fields(ls, jobs[__float_as_uint(sq.c4[k].w)].scene);
        r = make_tray(xyz(o), xyz(d), kRayEps);
        tmax = o.w;
    };
    const auto done = [&](uint32_t ray, int rc) {
        if (rc < 0) set_status(&ctr->status, KZ_ERR_STACK);
        if (rc == 1)
            film_add(jobs[__float_as_uint(sq.c4[ray].w)].film, nullptr, __float_as_uint(sq.d4[ray].w),
                     xyz(sq.c4[ray]));
    };
    if (ctr->queue.shadow <= kFewRays)
        few_any(m, ls, ctr->queue.shadow, &ctr->shadow_next, load, done);
    else
        persistent_any_in<false, true>(m, ls, ctr->queue.shadow, &ctr->shadow_next, load, done, dn, dt);
}

// Camera path g (over all jobs) into slot k.
__device__ __forceinline__ void batch_generate(const DevJob* __restrict__ jobs, uint32_t n_jobs, PathSoA dst,
                                               unsigned long long g, uint32_t k) {
    const uint32_t job = find_job(jobs, n_jobs, g);
    const DevJob& J = jobs[job];
    generate_camera_path(J.cam, J.pp, dst, k, g - J.path_begin);
    dst.d4[k].w = __uint_as_float(__float_as_uint(dst.d4[k].w) | (job << kJobShift));
}

// New paths of an iteration of the device-driven loop, as every thread of its
// generating kernel works it out from the iteration before and the last one
// that generated; one of them (j == 0) leaves it for the kernels that follow.
struct NewPaths {
    unsigned long long first;  // path id
    uint32_t count, slot;
};
__device__ __forceinline__ NewPaths new_paths(const IterSlots& it, uint32_t j) {
    const uint32_t alive = it.prev->queue.next, room = it.cap - alive;
    const unsigned long long first = it.last_gen->next_path, left = it.total - first;
    const NewPaths n{first, (uint32_t)(left < room ? left : room), alive};
    if (j == 0) {
        it.cur->next_path = first + n.count;
        it.cur->n_active = alive + n.count;
    }
    return n;
}

// Counters of one iteration of the single-launch batch kernel: how many new
// paths fill the free slots (when `generate`), and the cursors reset.
__device__ __forceinline__ void plan_iteration(DevCounters* c, uint32_t cap, bool generate) {
    const uint64_t remaining = c->total - c->next_path;
    const uint32_t room = cap - c->n_active;
    const uint32_t n_new = generate ? (uint32_t)(remaining < room ? remaining : room) : 0u;
    c->gen_first = c->next_path;
    c->gen_count = n_new;
    c->gen_slot = c->n_active;
    c->next_path += n_new;
    c->n_active += n_new;
    c->n_append = 0;
    c->trace_next = 0;
    c->shadow_next = 0;
    if (c->n_active) {
        c->iterations += 1;
        c->path_bounces += c->n_active;
    }
}

// End of an iteration: the continuing paths become the next wavefront.
__device__ __forceinline__ void finish_iteration(DevCounters* c) {
    c->shadow_rays += c->queue.shadow;
    c->n_active = c->queue.next;
}

inline unsigned grid_for(uint64_t n, unsigned block) { return (unsigned)((n + block - 1) / block); }

// Slots of a vertex's continuing path and shadow ray in the two queues, one
// 64-bit atomic per warp for both. Every lane of the warp calls it.
struct AppendSlots {
    uint32_t cont, shadow;
};
__device__ __forceinline__ AppendSlots warp_append_pair(bool cont, bool shadow, DevCounters* ctr) {
    const uint32_t lane = threadIdx.x & 31u, lt = (1u << lane) - 1u;
    const uint32_t bc = __ballot_sync(0xFFFFFFFFu, cont), bs = __ballot_sync(0xFFFFFFFFu, shadow);
    unsigned long long base = 0;
    if (lane == 0 && (bc | bs))
        base = atomicAdd(&ctr->n_append, ((unsigned long long)__popc(bs) << 32) | (unsigned)__popc(bc));
    base = __shfl_sync(0xFFFFFFFFu, base, 0);
    return AppendSlots{(uint32_t)base + __popc(bc & lt), (uint32_t)(base >> 32) + __popc(bs & lt)};
}

__device__ __forceinline__ void store_next(const PathSoA& out, const ShadowSoA& sq, const ShadeOut& so,
                                           const AppendSlots& at) {
    if (so.cont) {
        out.o4[at.cont] = so.o_next;
        out.d4[at.cont] = so.d_next;
        out.b4[at.cont] = so.b_next;
        out.rng[at.cont] = so.rng_next;
    }
    if (so.shadow) {
        sq.o4[at.shadow] = so.s_o;
        sq.d4[at.shadow] = so.s_d;
        sq.c4[at.shadow] = so.s_c;
    }
}

// Blocks of `block` threads resident on the whole device for kernel f.
template <typename F>
static unsigned resident_grid(F f, unsigned block) {
    int dev = 0, sms = 0, per_sm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, f, (int)block, 0);
    return (unsigned)(sms > 0 ? sms : 1) * (unsigned)(per_sm > 0 ? per_sm : 1);
}

// Shading kind of a traced path: 0 a miss, 1 + the material's shading class
// (kz_internal.h) for a hit, kNoPath for a thread without one.
constexpr uint32_t kNoPath = 1u + kNumClasses, kNumKinds = kNoPath + 1u;
__device__ __forceinline__ uint32_t shade_kind(const DevScene& s, const float4 hit) {
    const int rec = __float_as_int(hit.w);
    if (rec < 0) return 0u;
    const uint32_t m = __float_as_uint(__ldg(reinterpret_cast<const float*>(s.tris + (size_t)rec * 3 + 2) + 3));
    return 1u + __ldg(s.mat_class + m);
}

// Regroups a block's paths by kind before they are shaded, so each warp runs
// one branch of the shading: a counting sort in shared memory; returns the
// path index this thread shades and sets `kind` to its kind. The order within
// a kind is arbitrary; each path's result is not. blockDim.x <= 256.
__device__ __forceinline__ uint32_t block_group_by_kind(uint32_t i, uint32_t& kind) {
    __shared__ uint32_t s_cnt[kNumKinds];
    __shared__ uint32_t s_perm[256];
    if (threadIdx.x < kNumKinds) s_cnt[threadIdx.x] = 0u;
    __syncthreads();
    const uint32_t rank = atomicAdd(&s_cnt[kind], 1u);
    __syncthreads();
    uint32_t first = 0u;
    for (uint32_t k = 0; k < kind; ++k) first += s_cnt[k];
    s_perm[first + rank] = threadIdx.x | (kind << 16);
    __syncthreads();
    const uint32_t p = s_perm[threadIdx.x];
    kind = p >> 16;
    return i - threadIdx.x + (p & 0xFFFFu);
}

// The one-kernel shading runs 6 blocks per SM (40 registers, ~860 bytes of
// spills to L1): it waits on dependent loads, and more warps hide more of
// them. Terrain frame shade stage, when this kernel shaded all of it, at 4 / 5 /
// 6 / 7 / 8 blocks per SM: 32.5 / 31.6 / 31.1 / 31.9 / 31.9 ms.
#ifndef KZ_SHADE_MIN_BLOCKS
#define KZ_SHADE_MIN_BLOCKS 6
#endif
// The guided variant at 3 blocks per SM (80 registers, ~200 bytes of spills):
// slit room 1024^2, 64 spp, shade stage 88.2 ms at 1 or 2 blocks (126 / 114
// registers), 80.9 ms at 3, 84.0 ms at 4 (64 registers, 728 bytes of spills).
#ifndef KZ_SHADE_GUIDED_MIN_BLOCKS
#define KZ_SHADE_GUIDED_MIN_BLOCKS 3
#endif
// Each block's paths are grouped by kind (miss, material shading class) before
// they are shaded: without it a warp holds several kinds and runs them in turn
// (8.2 of 32 lanes active against 19.7). (Also writing the continuing paths
// grouped by the octant of their next direction, one atomic per block,
// measured trace -3.0 ms but shade +4.2 ms: not kept.)
template <bool kGuided, bool kAttr = true>
__global__ void __launch_bounds__(256, kGuided ? KZ_SHADE_GUIDED_MIN_BLOCKS : KZ_SHADE_MIN_BLOCKS)
    k_shade(DevScene s, PathParams pp, PathSoA in, uint32_t n_in, PathSoA out,
                                               ShadowSoA sq, DevCounters* ctr, float* film, double* film64,
                                               GuideShade gs, const uint32_t* n_dev) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (n_dev) n_in = *n_dev;
    if (blockIdx.x * blockDim.x >= n_in) return;  // the grid covers the wavefront's capacity
    uint32_t kind = i < n_in ? shade_kind(s, in.hit[i]) : kNoPath;
    i = block_group_by_kind(i, kind);
    ShadeOut so;
    if (!kGuided && kind == 1u + kPlainClass)
        shade_plain<kAttr>(s, pp, in.hit[i], in.o4[i], in.d4[i], in.b4[i], in.rng[i], so);
    else if (i < n_in)
        shade_vertex<kGuided, kAttr>(s, pp, in.hit[i], in.o4[i], in.d4[i], in.b4[i], in.rng[i], gs,
                                     kGuided ? gs.raw + (size_t)i * kGuideOut : nullptr, so);
    if (!is_zero(so.Lsum)) film_add(film, film64, so.film_idx, so.Lsum);
    const AppendSlots at = warp_append_pair(so.cont, so.shadow, ctr);
    store_next(out, sq, so, at);
}

// ------------------------------------------------------------------ split shading
// Large wavefronts are shaded by two kernels. k_shade_plain goes over all
// paths once: it finishes the misses and the plain vertices itself and sorts
// the others into a queue per material class. k_shade_heavy then takes the
// queues 32 paths of one class at a time, the longest class first. In one
// kernel the general vertex sets the registers (40 with 860 bytes of spills),
// and a block waits for its slowest warp, which a Beckmann sample's FP64 search
// makes ten times slower than the rest. Both wait on dependent loads; the
// plain pass moves about 230 bytes a path, the heavy one is left with the lobe
// switch and FP64. Shade stage, one kernel before / two: terrain 1080p 30.8 /
// 18.8 ms, slit room 12.1 / 6.2 ms, 641 x 359 frame of mixed materials 16.3 /
// 2.8 ms, box room 0.59 / 0.36 ms.
// Blocks per SM, terrain + materials shade: plain (256 threads) 4 / 5 / 6 / 8:
// 27.5 / 27.6 / 28.1 / 32.8 ms; heavy (128 threads) 4 / 6 / 8 / 12: 27.8 /
// 27.6 / 27.4 / 28.3 ms.
#ifndef KZ_PLAIN_MIN_BLOCKS
#define KZ_PLAIN_MIN_BLOCKS 4
#endif
#ifndef KZ_HEAVY_MIN_BLOCKS
#define KZ_HEAVY_MIN_BLOCKS 8
#endif
constexpr int kHeavyThreads = 128;
// Paths a thread classifies between two rounds of shading. The plain ones are
// listed per block and shaded 256 at a time: where most bounces leave the scene,
// ten of 32 lanes were active otherwise. Two independent hit -> triangle ->
// class chains a thread also hide half of their waits. Shade stage, a path per
// lane / 2 / 4 / 8 a thread with the list: terrain 22.7 / 18.8 / 18.9 / 19.4 ms,
// slit room 6.47 / 6.21 / 6.21 / 6.41, mixed materials 2.92 / 2.82 / 2.84 / 2.92.
#ifndef KZ_PLAIN_CHUNK
#define KZ_PLAIN_CHUNK 2
#endif
constexpr uint32_t kPlainChunk = KZ_PLAIN_CHUNK;
static_assert(kPlainChunk * 32u <= 256u, "ranks within a warp are kept in a byte");

// Queue place of the k-th path of a heavy class: two arrays of the wavefront's
// capacity, each filled from both ends (a path is in one class only).
__device__ __forceinline__ uint32_t* heavy_slot(const HeavyQueue& q, uint32_t cls, uint32_t k) {
    uint32_t* a = q.paths + (cls >= 2u ? q.cap : 0u);
    return (cls & 1u) ? a + (q.cap - 1u - k) : a + k;
}

template <bool kAttr>
__global__ void __launch_bounds__(256, KZ_PLAIN_MIN_BLOCKS)
    k_shade_plain(DevScene s, PathParams pp, PathSoA in, PathSoA out, ShadowSoA sq, HeavyQueue hq, DevCounters* ctr,
                  const uint32_t* n_active, float* film, double* film64) {
    __shared__ uint32_t s_list[256 * (kPlainChunk + 1)];  // plain paths found and not yet shaded
    __shared__ uint32_t s_heavy[kHeavyClasses][8], s_plain[9];
    __shared__ unsigned long long s_app[2][8];  // per warp: appended paths and shadow rays; double buffered
    const uint32_t n = *n_active, lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, lt = (1u << lane) - 1u;
    // every block has paths before one takes several per thread
    const uint32_t per = min((uint32_t)kPlainChunk, n / (gridDim.x * 256u) + 1u);
    uint32_t found = 0, buf = 0;  // the list's length, the same in every thread
    for (uint32_t base = blockIdx.x * 256u * per; base < n; base += gridDim.x * 256u * per) {
        // ---- classify: misses are finished, the others listed or queued
        uint32_t mark[kPlainChunk];  // class << 8 | rank among the warp's; class 0 plain, c + 1 heavy c
        uint32_t cnt[1 + kHeavyClasses] = {};
#pragma unroll
        for (uint32_t k = 0; k < kPlainChunk; ++k) {
            const uint32_t i = base + k * 256u + threadIdx.x;
            mark[k] = ~0u;
            if (k >= per) continue;  // uniform over the block
            uint32_t cls = ~0u;
            if (i < n) {
                const uint32_t kind = shade_kind(s, in.hit[i]);
                if (kind) {
                    cls = kind - 1u;  // kPlainClass is 0
                } else if (s.has_env) {
                    ShadeOut so;
                    shade_miss(s, pp, in.d4[i], in.b4[i], so);
                    if (!is_zero(so.Lsum)) film_add(film, film64, so.film_idx, so.Lsum);
                }
            }
            const uint32_t classes = __any_sync(0xFFFFFFFFu, cls != ~0u && cls) ? 1u + kHeavyClasses : 1u;
#pragma unroll
            for (uint32_t c = 0; c < 1u + kHeavyClasses; ++c) {
                if (c >= classes) break;
                const uint32_t m = __ballot_sync(0xFFFFFFFFu, cls == c);
                if (cls == c) mark[k] = c << 8 | (cnt[c] + __popc(m & lt));
                cnt[c] += __popc(m);
            }
        }
        if (lane == 0) {
            s_plain[warp] = cnt[0];
#pragma unroll
            for (uint32_t c = 0; c < kHeavyClasses; ++c) s_heavy[c][warp] = cnt[1 + c];
        }
        __syncthreads();
        if (warp == 0) {  // lanes 8 c + w: warp w of class c; one atomic per class and block
            const uint32_t c = lane >> 3, w = lane & 7u;
            const uint32_t v = s_heavy[c][w];
            uint32_t incl = v;
#pragma unroll
            for (uint32_t o = 1; o < 8; o <<= 1) {
                const uint32_t x = __shfl_up_sync(0xFFFFFFFFu, incl, o, 8);
                if (w >= o) incl += x;
            }
            uint32_t first = 0;
            if (w == 7 && incl) first = atomicAdd(&ctr->heavy[c], incl);
            s_heavy[c][w] = __shfl_sync(0xFFFFFFFFu, first, 7, 8) + incl - v;
        } else if (warp == 1 && lane < 8) {
            const uint32_t v = s_plain[lane];
            uint32_t incl = v;
#pragma unroll
            for (uint32_t o = 1; o < 8; o <<= 1) {
                const uint32_t x = __shfl_up_sync(0xFFu, incl, o);
                if (lane >= o) incl += x;
            }
            s_plain[lane] = found + incl - v;
            if (lane == 7) s_plain[8] = found + incl;
        }
        __syncthreads();
#pragma unroll
        for (uint32_t k = 0; k < kPlainChunk; ++k) {
            if (mark[k] == ~0u) continue;
            const uint32_t i = base + k * 256u + threadIdx.x, c = mark[k] >> 8, r = mark[k] & 0xFFu;
            if (c == 0) s_list[s_plain[warp] + r] = i;
            else *heavy_slot(hq, c - 1u, s_heavy[c - 1u][warp] + r) = i;
        }
        found = s_plain[8];
        __syncthreads();
        // ---- shade full blocks of plain paths; what is left once no path follows
        const bool last = n - base <= gridDim.x * 256u * per;
        for (; found >= 256u || (last && found); buf ^= 1u) {
            const uint32_t take = min(found, 256u);
            found -= take;
            ShadeOut so;
            if (threadIdx.x < take) {
                const uint32_t i = s_list[found + threadIdx.x];
                shade_plain<kAttr>(s, pp, in.hit[i], in.o4[i], in.d4[i], in.b4[i], in.rng[i], so);
                if (!is_zero(so.Lsum)) film_add(film, film64, so.film_idx, so.Lsum);
            }
            // one atomic per block, not per warp
            const uint32_t bc = __ballot_sync(0xFFFFFFFFu, so.cont), bs = __ballot_sync(0xFFFFFFFFu, so.shadow);
            if (lane == 0) s_app[buf][warp] = ((unsigned long long)__popc(bs) << 32) | (unsigned)__popc(bc);
            __syncthreads();
            if (warp == 0 && lane < 8) {
                const unsigned long long v = s_app[buf][lane];
                unsigned long long incl = v, first = 0;
#pragma unroll
                for (uint32_t o = 1; o < 8; o <<= 1) {
                    const unsigned long long x = __shfl_up_sync(0xFFu, incl, o);
                    if (lane >= o) incl += x;
                }
                if (lane == 7 && incl) first = atomicAdd(&ctr->n_append, incl);
                s_app[buf][lane] = __shfl_sync(0xFFu, first, 7) + incl - v;
            }
            __syncthreads();
            const unsigned long long at = s_app[buf][warp];
            store_next(out, sq, so, AppendSlots{(uint32_t)at + __popc(bc & lt), (uint32_t)(at >> 32) + __popc(bs & lt)});
        }
        if (last) break;
    }
}

// The plain pass over jobs of several scenes: a path per lane. Listed, a path
// would look its job and that job's scene up twice, one dependent load after
// another: 24 jobs 5.82 ms a path per lane, 5.85 listed; 256 uneven jobs 563 and
// 565 ms.
template <bool kAttr>
__global__ void __launch_bounds__(256, KZ_PLAIN_MIN_BLOCKS)
    k_shade_plain_jobs(const DevJob* __restrict__ jobs, PathSoA in, PathSoA out, ShadowSoA sq, HeavyQueue hq,
                       DevCounters* ctr, const uint32_t* n_active) {
    // per warp: appended paths and shadow rays, then the four heavy classes; double buffered over the rounds
    __shared__ unsigned long long s_app[2][8];
    __shared__ uint32_t s_heavy[2][kHeavyClasses][8];
    const uint32_t n = *n_active, lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, lt = (1u << lane) - 1u;
    uint32_t buf = 0;
    for (uint32_t base = blockIdx.x * 256u; base < n; base += gridDim.x * 256u, buf ^= 1u) {
        const uint32_t i = base + threadIdx.x;
        ShadeOut so;
        uint32_t heavy = kHeavyClasses;  // none
        if (i < n) {
            const float4 hit = in.hit[i], d4 = in.d4[i];
            const DevJob* J = jobs + (__float_as_uint(d4.w) >> kJobShift);
            const DevScene& s = J->scene;
            const PathParams& pp = J->pp;
            const uint32_t kind = shade_kind(s, hit);
            if (kind == 1u + kPlainClass) shade_plain<kAttr>(s, pp, hit, in.o4[i], d4, in.b4[i], in.rng[i], so);
            else if (kind) heavy = kind - 2u;
            else if (s.has_env) shade_miss(s, pp, d4, in.b4[i], so);
            if (!is_zero(so.Lsum)) film_add(J->film, nullptr, so.film_idx, so.Lsum);
        }
        // one atomic per queue and block, not per warp
        const uint32_t bc = __ballot_sync(0xFFFFFFFFu, so.cont), bs = __ballot_sync(0xFFFFFFFFu, so.shadow);
        uint32_t bh = 0;  // this lane's class among the warp's
#pragma unroll
        for (uint32_t c = 0; c < kHeavyClasses; ++c) {
            const uint32_t b = __ballot_sync(0xFFFFFFFFu, heavy == c);
            if (heavy == c) bh = b;
            if (lane == 0) s_heavy[buf][c][warp] = __popc(b);
        }
        if (lane == 0) s_app[buf][warp] = ((unsigned long long)__popc(bs) << 32) | (unsigned)__popc(bc);
        __syncthreads();
        if (warp == 0) {  // lanes 8 c + w: warp w of class c
            const uint32_t c = lane >> 3, w = lane & 7u;
            const uint32_t v = s_heavy[buf][c][w];
            uint32_t incl = v;
#pragma unroll
            for (uint32_t o = 1; o < 8; o <<= 1) {
                const uint32_t x = __shfl_up_sync(0xFFFFFFFFu, incl, o, 8);
                if (w >= o) incl += x;
            }
            uint32_t first = 0;
            if (w == 7 && incl) first = atomicAdd(&ctr->heavy[c], incl);
            s_heavy[buf][c][w] = __shfl_sync(0xFFFFFFFFu, first, 7, 8) + incl - v;
        } else if (warp == 1 && lane < 8) {
            const unsigned long long v = s_app[buf][lane];
            unsigned long long incl = v, first = 0;
#pragma unroll
            for (uint32_t o = 1; o < 8; o <<= 1) {
                const unsigned long long x = __shfl_up_sync(0xFFu, incl, o);
                if (lane >= o) incl += x;
            }
            if (lane == 7 && incl) first = atomicAdd(&ctr->n_append, incl);
            s_app[buf][lane] = __shfl_sync(0xFFu, first, 7) + incl - v;
        }
        __syncthreads();
        const unsigned long long at = s_app[buf][warp];
        store_next(out, sq, so, AppendSlots{(uint32_t)at + __popc(bc & lt), (uint32_t)(at >> 32) + __popc(bs & lt)});
        if (heavy < kHeavyClasses) *heavy_slot(hq, heavy, s_heavy[buf][heavy][warp] + __popc(bh & lt)) = i;
    }
}

template <bool kAttr, bool kJobs>
__global__ void __launch_bounds__(kHeavyThreads, KZ_HEAVY_MIN_BLOCKS)
    k_shade_heavy(DevScene scene, PathParams params, const DevJob* __restrict__ jobs, PathSoA in, PathSoA out,
                  ShadowSoA sq, HeavyQueue hq, DevCounters* ctr, float* film, double* film64) {
    const uint32_t lane = threadIdx.x & 31u;
    for (;;) {
        uint32_t p = 0;
        if (lane == 0) p = atomicAdd(&ctr->heavy_next, 32u);
        p = __shfl_sync(0xFFFFFFFFu, p, 0);
        uint32_t cls = 0, n = 0;
        for (; cls < kHeavyClasses; ++cls) {  // each class's range is rounded up to whole warps
            n = ctr->heavy[cls];
            const uint32_t r = (n + 31u) & ~31u;
            if (p < r) break;
            p -= r;
        }
        if (cls == kHeavyClasses) break;
        ShadeOut so;
        if (p + lane < n) {
            const uint32_t i = *heavy_slot(hq, cls, p + lane);
            const float4 d4 = in.d4[i];
            const DevJob* J = kJobs ? jobs + (__float_as_uint(d4.w) >> kJobShift) : nullptr;
            shade_vertex<false, kAttr>(kJobs ? J->scene : scene, kJobs ? J->pp : params, in.hit[i], in.o4[i], d4,
                                       in.b4[i], in.rng[i], GuideShade{}, nullptr, so);
            if (!is_zero(so.Lsum)) film_add(kJobs ? J->film : film, kJobs ? nullptr : film64, so.film_idx, so.Lsum);
        }
        store_next(out, sq, so, warp_append_pair(so.cont, so.shadow, ctr));
    }
}

// Wavefronts from this capacity on are shaded by the two kernels; smaller ones
// by the one: there the second launch and its dependent queue cost what the
// split saves (65,537 Li rays of depth 5: 0.94 ms with one kernel, 1.01 with
// two; a 25,220-path preview of mixed materials 1.16 and 1.11).
#ifndef KZ_SPLIT_SHADING
#define KZ_SPLIT_SHADING (1u << 18)
#endif
struct SplitGrids {
    unsigned plain, heavy;
};
template <bool kAttr, bool kJobs>
static SplitGrids split_grids() {
    static const SplitGrids g = [] {
        const unsigned heavy = resident_grid(k_shade_heavy<kAttr, kJobs>, kHeavyThreads);
        if constexpr (kJobs) return SplitGrids{resident_grid(k_shade_plain_jobs<kAttr>, 256), heavy};
        else return SplitGrids{resident_grid(k_shade_plain<kAttr>, 256), heavy};
    }();
    return g;
}
template <bool kAttr, bool kJobs>
static int launch_split_shading(const DevScene& s, const PathParams& pp, const DevJob* jobs, PathSoA in, uint32_t cap,
                                PathSoA out, ShadowSoA sq, HeavyQueue hq, DevCounters* ctr,
                                const uint32_t* n_active, float* film, double* film64, bool heavy, cudaStream_t st) {
    const SplitGrids g = split_grids<kAttr, kJobs>();
    const unsigned plain = std::min(g.plain, grid_for(cap, 256));
    if constexpr (kJobs)
        k_shade_plain_jobs<kAttr><<<plain, 256, 0, st>>>(jobs, in, out, sq, hq, ctr, n_active);
    else
        k_shade_plain<kAttr><<<plain, 256, 0, st>>>(s, pp, in, out, sq, hq, ctr, n_active, film, film64);
    if (!heavy) return 1;
    k_shade_heavy<kAttr, kJobs><<<std::min(g.heavy, grid_for(cap, kHeavyThreads)), kHeavyThreads, 0, st>>>(
        s, pp, jobs, in, out, sq, hq, ctr, film, film64);
    return 2;
}

}  // namespace
}  // namespace kz
