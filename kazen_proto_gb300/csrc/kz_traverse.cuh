// kz_traverse.cuh — BVH traversal and watertight ray/triangle test (device).
//
// Replaces EmbreeAccel::intersect / occluded (src/core/accel.cpp:348-432,
// src/core/hitable.h:25-33) and the Moller-Trumbore routine
// (src/core/shape.cpp:373-450) with:
//  * the watertight test of S. Woop, C. Benthin, I. Wald, "Watertight
//    Ray/Triangle Intersection", JCGT 2(1), 2013 — double-sided, double
//    precision fallback when an edge function is exactly zero;
//  * closest hit in (tmin, tmax], equal t resolved to the smaller global
//    triangle id, so the result is independent of traversal order and of the
//    BVH shape (bit-exact against any exact restatement);
//  * an 8-wide BVH with quantized child boxes (80-byte nodes, five 16-byte
//    non-coherent loads), in the manner of H. Ylitie, T. Karras, S. Laine,
//    "Efficient Incoherent Ray Traversal on GPUs Through Compressed Wide
//    BVHs", HPG 2017: one node test yields a 32-bit mask of inner children
//    (visited in an octant-derived near-first order) and leaf triangles; a
//    stack of (child base, mask) groups in local memory.
// Box distances are widened by a margin above their rounding error (see
// wide_axis), so no box holding a hit at t <= t_best is culled.
#pragma once

#include "kz_bvh.h"
#include "kz_device.cuh"

namespace kz {

static_assert(kWideWords == 20, "a wide node is five 16-byte vectors");

struct TRay {
    f3 o, inv;
    float tmin;
    int kx, ky, kz;
    float Sx, Sy, Sz;
};

__device__ __forceinline__ float safe_inv(float c) {
    if (fabsf(c) < 1e-30f) c = copysignf(1e-30f, c);
    return 1.0f / c;
}

__device__ __forceinline__ TRay make_tray(f3 o, f3 d, float tmin) {
    TRay r;
    r.o = o;
    r.tmin = tmin;
    r.inv = mk(safe_inv(d.x), safe_inv(d.y), safe_inv(d.z));
    float ax = fabsf(d.x), ay = fabsf(d.y), az = fabsf(d.z);
    int kz = 0;
    float m = ax;
    if (ay > m) { kz = 1; m = ay; }
    if (az > m) { kz = 2; }
    int kx = kz + 1 == 3 ? 0 : kz + 1;
    int ky = kx + 1 == 3 ? 0 : kx + 1;
    float dz = comp(d, kz);
    if (dz < 0.f) { int t = kx; kx = ky; ky = t; }
    r.kx = kx; r.ky = ky; r.kz = kz;
    r.Sx = comp(d, kx) / dz;
    r.Sy = comp(d, ky) / dz;
    r.Sz = 1.0f / dz;
    return r;
}

// The component whose bit is set in a pair of bits (0: x, 1: y; neither: z).
__device__ __forceinline__ float pick_bits(float4 v, uint32_t k) { return (k & 1u) ? v.x : ((k & 2u) ? v.y : v.z); }

// The per-ray terms of the watertight test: the origin in the permuted axes
// (kx, ky, kz), the shear and the ray's lower bound.
struct TriRay {
    float okx, oky, okz, tmin;
    float Sx, Sy, Sz;
    uint32_t axes;  // pick_bits pairs of kx (bits 0-1), ky (2-3), kz (4-5)
};

__device__ __forceinline__ TriRay tri_ray(const TRay& r) {
    TriRay q;
    q.okx = comp(r.o, r.kx);
    q.oky = comp(r.o, r.ky);
    q.okz = comp(r.o, r.kz);
    q.tmin = r.tmin;
    q.Sx = r.Sx;
    q.Sy = r.Sy;
    q.Sz = r.Sz;
    q.axes = (r.kx == 2 ? 0u : 1u << r.kx) | (r.ky == 2 ? 0u : 4u << r.ky) | (r.kz == 2 ? 0u : 16u << r.kz);
    return q;
}

// Watertight test against a triangle record; t is valid when it returns true.
// The barycentric divisions are left to the caller: u = V / det, v = W / det
// for the hit that is kept.
__device__ __forceinline__ bool tri_test_t(const TriRay& r, float4 a, float4 b, float4 c, float& t, float& V_,
                                           float& W_, float& det_) {
    const float okx = r.okx, oky = r.oky, okz = r.okz;
    const uint32_t kx = r.axes, ky = r.axes >> 2, kz = r.axes >> 4;
    const float Akx = pick_bits(a, kx) - okx, Aky = pick_bits(a, ky) - oky, Akz = pick_bits(a, kz) - okz;
    const float Bkx = pick_bits(b, kx) - okx, Bky = pick_bits(b, ky) - oky, Bkz = pick_bits(b, kz) - okz;
    const float Ckx = pick_bits(c, kx) - okx, Cky = pick_bits(c, ky) - oky, Ckz = pick_bits(c, kz) - okz;
    const float Ax = Akx - r.Sx * Akz, Ay = Aky - r.Sy * Akz;
    const float Bx = Bkx - r.Sx * Bkz, By = Bky - r.Sy * Bkz;
    const float Cx = Ckx - r.Sx * Ckz, Cy = Cky - r.Sy * Ckz;
    float U = Cx * By - Cy * Bx;
    float V = Ax * Cy - Ay * Cx;
    float W = Bx * Ay - By * Ax;
    if (U == 0.f || V == 0.f || W == 0.f) {
        U = (float)((double)Cx * (double)By - (double)Cy * (double)Bx);
        V = (float)((double)Ax * (double)Cy - (double)Ay * (double)Cx);
        W = (float)((double)Bx * (double)Ay - (double)By * (double)Ax);
    }
    if ((U < 0.f || V < 0.f || W < 0.f) && (U > 0.f || V > 0.f || W > 0.f)) return false;
    const float det = U + V + W;
    if (det == 0.f) return false;
    const float T = U * (r.Sz * Akz) + V * (r.Sz * Bkz) + W * (r.Sz * Ckz);
    t = T / det;
    V_ = V;
    W_ = W;
    det_ = det;
    return true;
}
__device__ __forceinline__ bool tri_test_t(const TRay& r, float4 a, float4 b, float4 c, float& t, float& V_, float& W_,
                                           float& det_) {
    return tri_test_t(tri_ray(r), a, b, c, t, V_, W_, det_);
}

struct HitRec {
    float t, u, v;
    uint32_t prim;  // global triangle id, KZ_INVALID_ID on a miss
    int32_t rec;    // triangle record, -1 on a miss
};

// ---- 8-wide quantized BVH (layout in kz_bvh.h) ------------------------------
//
// A child box plane at p + q * 2^E on one axis is reached at
//   t(q) = (p + q 2^E - o) / d = b + q 2^E inv,  b = (p - o) inv.
// The byte q becomes f = 1 + q 2^-15 with one byte permute (0x3F80_qq00 as
// float bits), so t(q) = fma(f, A, B) with A = 2^(E+15) inv (exact: a power
// of two times inv) and B = b - A. Each term carries rounding error below
// 2^-24 (6 |b| + 3 |A|); the per-node margin 2^-16 (|b| + |A| / 32) exceeds it,
// so the near plane is lowered and the far plane raised by more than any
// rounding and no box holding a hit at t <= t_best is culled. An overflowing
// A or b turns the axis' distances into NaN, which the min/max below ignore:
// such an axis culls nothing.
// The device's copy of a node (pack_nodes, kz_trace.cu) holds the same boxes
// with the fields arranged so that a slot costs no decoding:
//   w0..w2   p
//   w3       the x and y scales 2^(E+15) as the upper halves of their floats
//   w4, w5   first inner child, first triangle record
//   w6       bits 0-23: triangle k of leaf slot s at bit 3 s + k; bits 24-31
//            the inner-slot mask
//   w7       the z scale's upper half (bits 0-15)
//   w8..w19  per axis 4 words, word j: low and high plane bytes of slot 2 j,
//            then of slot 2 j + 1
// A slot that is hit sets its three triangle bits and its inner bit with one
// constant; an AND with w6 then keeps what the node holds. The near and far
// byte of a word are picked by the byte permute's own selector, which the
// ray's direction signs fix.
struct WideAxis {
    float A, Bn, Bf;
    uint4 q;
};

__device__ __forceinline__ WideAxis wide_axis(float p, float scale, float o, float inv, uint4 q) {
    WideAxis ax;
    ax.A = scale * inv;
    const float b = (p - o) * inv;
    const float B = b - ax.A;
    const float d = (fabsf(b) + fabsf(ax.A) * 0.03125f) * 1.52587890625e-05f;
    ax.Bn = B - d;
    ax.Bf = B + d;
    ax.q = q;
    return ax;
}

// Per-ray constants of the node test and of the visiting order.
struct WideDir {
    uint32_t sx, sy, sz;  // byte-permute selectors of the near plane of even slots
    uint32_t p2, p1, p0;  // inner bits (24-31) visited first at each level of the octant order
};

template <int kSlot>
__device__ __forceinline__ float wide_t(const WideAxis& ax, uint32_t sel, bool near_plane) {
    const uint32_t w = kSlot < 2 ? ax.q.x : kSlot < 4 ? ax.q.y : kSlot < 6 ? ax.q.z : ax.q.w;
    const uint32_t k = (sel ^ (near_plane ? 0u : 0x10u)) | ((kSlot & 1) ? 0x20u : 0u);
    return fmaf(__uint_as_float(__byte_perm(w, 0x3F800000u, k)), ax.A, near_plane ? ax.Bn : ax.Bf);
}

// Two-input minima and maxima on purpose: with the three-input forms, or the
// planes in packed FP32 pairs, the trace stage of the terrain frame took 86.7
// and 86.9 ms against 82.2 (fewer instructions, but more registers than the
// 64 that keep 32 warps on an SM).
template <int kSlot>
__device__ __forceinline__ void wide_slot(const WideAxis& X, const WideAxis& Y, const WideAxis& Z, const WideDir& dir,
                                          float tmin, float tcur, uint32_t& hits) {
    const float tn = fmaxf(fmaxf(fmaxf(wide_t<kSlot>(X, dir.sx, true), tmin), wide_t<kSlot>(Y, dir.sy, true)),
                           wide_t<kSlot>(Z, dir.sz, true));
    const float tf = fminf(fminf(fminf(wide_t<kSlot>(X, dir.sx, false), tcur), wide_t<kSlot>(Y, dir.sy, false)),
                           wide_t<kSlot>(Z, dir.sz, false));
    if (tn <= tf) hits |= (7u << (3 * kSlot)) | (1u << (24 + kSlot));
}

// Leaf triangles pending for a warp-wide test: bits of the node's triangle
// mask that are hit, the mask itself (a triangle's record is the base plus
// its rank in the mask) and the base.
struct LeafGroup {
    uint32_t bits, valid, base;
};

__device__ __forceinline__ uint32_t leaf_record(uint32_t base, uint32_t valid, uint32_t bit) {
    return base + __popc(valid & ((1u << bit) - 1u));
}

// Tests the 8 child boxes of a node: the inner children hit (bits 24-31, with
// the inner-slot mask in bits 0-7) and the triangles of the leaves hit.
__device__ __forceinline__ uint32_t wide_node(const uint4* __restrict__ np, const TRay& r, const WideDir& dir,
                                              float tcur, uint32_t& child_base, LeafGroup& lg) {
    const uint4 h0 = __ldg(np), h1 = __ldg(np + 1);
    const uint4 qx = __ldg(np + 2), qy = __ldg(np + 3), qz = __ldg(np + 4);
    const WideAxis X = wide_axis(__uint_as_float(h0.x), __uint_as_float(h0.w << 16), r.o.x, r.inv.x, qx);
    const WideAxis Y = wide_axis(__uint_as_float(h0.y), __uint_as_float(h0.w & 0xFFFF0000u), r.o.y, r.inv.y, qy);
    const WideAxis Z = wide_axis(__uint_as_float(h0.z), __uint_as_float(h1.w << 16), r.o.z, r.inv.z, qz);
    uint32_t hits = 0;
    wide_slot<0>(X, Y, Z, dir, r.tmin, tcur, hits);
    wide_slot<1>(X, Y, Z, dir, r.tmin, tcur, hits);
    wide_slot<2>(X, Y, Z, dir, r.tmin, tcur, hits);
    wide_slot<3>(X, Y, Z, dir, r.tmin, tcur, hits);
    wide_slot<4>(X, Y, Z, dir, r.tmin, tcur, hits);
    wide_slot<5>(X, Y, Z, dir, r.tmin, tcur, hits);
    wide_slot<6>(X, Y, Z, dir, r.tmin, tcur, hits);
    wide_slot<7>(X, Y, Z, dir, r.tmin, tcur, hits);
    hits &= h1.z;
    child_base = h1.x;
    lg.bits = hits & 0x00FFFFFFu;
    lg.valid = h1.z & 0x00FFFFFFu;
    lg.base = h1.y;
    return (hits & 0xFF000000u) | (h1.z >> 24);
}

// A ray visits its inner children in the order of slot ^ m, largest first,
// with m = 7 for the octant it enters first (slot bits set on the axes whose
// direction is negative): at each level the half its direction enters first.
__device__ __forceinline__ WideDir wide_dir(const TRay& r) {
    const bool nx = r.inv.x < 0.f, ny = r.inv.y < 0.f, nz = r.inv.z < 0.f;
    WideDir d;
    d.sx = nx ? 0x7614u : 0x7604u;
    d.sy = ny ? 0x7614u : 0x7604u;
    d.sz = nz ? 0x7614u : 0x7604u;
    d.p2 = nz ? 0xF0000000u : 0x0F000000u;
    d.p1 = ny ? 0xCC000000u : 0x33000000u;
    d.p0 = nx ? 0xAA000000u : 0x55000000u;
    return d;
}

// Next inner child of a node group (base, bits): bits 24-31 the remaining
// hits by slot, bits 0-7 the node's inner-slot mask.
__device__ __forceinline__ uint32_t wide_pop_child(uint32_t base, uint32_t& bits, const WideDir& dir) {
    uint32_t m = bits & 0xFF000000u;
    if (m & dir.p2) m &= dir.p2;
    if (m & dir.p1) m &= dir.p1;
    if (m & dir.p0) m &= dir.p0;  // one bit is left
    bits ^= m;
    return base + __popc(bits & ((m >> 24) - 1u));
}

// Traversal stack of node groups: a per-thread local array (LocalStack), or
// its first kSmem entries in shared memory, entry i of thread t at
// i * blockDim.x + t, and the rest local (SplitStack).
struct LocalStack {
    uint2* p;
    __device__ __forceinline__ uint2 get(int i) const { return p[i]; }
    __device__ __forceinline__ void put(int i, uint2 e) const { p[i] = e; }
};
template <int kSmem>
struct SplitStack {
    uint2* sm;
    uint2* lm;
    __device__ __forceinline__ uint2 get(int i) const {
        return i < kSmem ? sm[i * blockDim.x + threadIdx.x] : lm[i - kSmem];
    }
    __device__ __forceinline__ void put(int i, uint2 e) const {
        if (i < kSmem) sm[i * blockDim.x + threadIdx.x] = e;
        else lm[i - kSmem] = e;
    }
};

// Closest-hit traversal state, advanced one node at a time (closest_step) so
// that persistent kernels can interleave rays; trace_closest runs it to the
// end. The barycentric divisions are deferred to closest_finish (for the kept
// hit only).
struct ClosestState {
    float t, V, W, det;
    uint32_t prim;
    int32_t rec;
    uint32_t gbase, gbits;  // current node group
    uint32_t visits;
    int sp;
};

__device__ __forceinline__ void closest_begin(ClosestState& c, float tmax) {
    c.t = tmax;
    c.V = c.W = 0.f;
    c.det = 1.f;
    c.prim = KZ_INVALID_ID;
    c.rec = -1;
    c.gbase = 0;
    c.gbits = 0x80000000u;  // the root as the only child of a virtual node
    c.visits = 0;
    c.sp = 0;
}

// Visits one node and tests its leaf triangles. Returns 0 while nodes remain,
// 1 when the traversal is complete, -1 if it must abort: the stack would
// overflow (the builder bounds the depth by the stack size), more nodes are
// visited than the tree holds, or a record index is out of range (a corrupt
// node array).
template <bool kCount, typename Stack>
__device__ __forceinline__ int closest_step(const DevScene& s, const TRay& r, const WideDir& dir, ClosestState& c,
                                            const Stack& stack, uint32_t& nnode, uint32_t& ntri) {
    const uint32_t node = wide_pop_child(c.gbase, c.gbits, dir);
    if (c.gbits > 0x00FFFFFFu) {
        if (c.sp >= kWideStack) return -1;
        stack.put(c.sp++, make_uint2(c.gbase, c.gbits));
    }
    if (++c.visits > s.n_nodes || node >= s.n_nodes) return -1;
    LeafGroup lg;
    c.gbits = wide_node(s.nodes + (size_t)node * 5, r, dir, c.t, c.gbase, lg);
    if (kCount) ++nnode;
    uint32_t tbits = lg.bits;
    while (tbits) {
        const uint32_t rec = leaf_record(lg.base, lg.valid, __ffs(tbits) - 1);
        tbits &= tbits - 1u;
        if (rec >= s.n_tris) return -1;
        const float4* tp = s.tris + (size_t)rec * 3;
        const float4 a = __ldg(tp), b = __ldg(tp + 1), cc = __ldg(tp + 2);
        if (kCount) ++ntri;
        float t, V, W, det;
        if (!tri_test_t(r, a, b, cc, t, V, W, det)) continue;
        const uint32_t prim = __float_as_uint(a.w);
        if (t > r.tmin && (t < c.t || (t == c.t && prim < c.prim))) {
            c.t = t;
            c.V = V;
            c.W = W;
            c.det = det;
            c.prim = prim;
            c.rec = (int32_t)rec;
        }
    }
    while (c.gbits <= 0x00FFFFFFu && c.sp > 0) {
        const uint2 e = stack.get(--c.sp);
        c.gbase = e.x;
        c.gbits = e.y;
    }
    return c.gbits <= 0x00FFFFFFu ? 1 : 0;
}

// Hit record of a finished traversal; an aborted one (ok == false) misses.
__device__ __forceinline__ void closest_finish(const ClosestState& c, bool ok, float tmax, HitRec& h) {
    if (!ok || c.rec < 0) {
        h.t = ok ? c.t : tmax;
        h.u = h.v = 0.f;
        h.prim = KZ_INVALID_ID;
        h.rec = -1;
        return;
    }
    h.t = c.t;
    h.u = c.V / c.det;
    h.v = c.W / c.det;
    h.prim = c.prim;
    h.rec = c.rec;
}

// Closest hit in (tmin, tmax]. Returns false if the traversal aborted
// (closest_step == -1); the caller reports KZ_ERR_STACK and the ray misses.
template <bool kCount>
__device__ bool trace_closest(const DevScene& s, const TRay& r, float tmax, HitRec& h, uint32_t& nnode,
                              uint32_t& ntri) {
    const WideDir dir = wide_dir(r);
    uint2 stack[kWideStack];
    ClosestState c;
    closest_begin(c, tmax);
    int rc;
    do {
        rc = closest_step<kCount>(s, r, dir, c, LocalStack{stack}, nnode, ntri);
    } while (rc == 0);
    closest_finish(c, rc > 0, tmax, h);
    return rc > 0;
}

// Any-hit traversal state, advanced one node at a time like ClosestState.
struct AnyState {
    uint32_t gbase, gbits;
    uint32_t visits;
    int sp;
};

__device__ __forceinline__ void any_begin(AnyState& c) {
    c.gbase = 0;
    c.gbits = 0x80000000u;
    c.visits = 0;
    c.sp = 0;
}

// One node of an any-hit query in (tmin, tmax]: 0 while nodes remain, 1 no
// hit (complete), 2 hit, -1 abort (as closest_step).
template <bool kCount, typename Stack>
__device__ __forceinline__ int any_step(const DevScene& s, const TRay& r, const WideDir& dir, float tmax, AnyState& c,
                                        const Stack& stack, uint32_t& nnode, uint32_t& ntri) {
    const uint32_t node = wide_pop_child(c.gbase, c.gbits, dir);
    if (c.gbits > 0x00FFFFFFu) {
        if (c.sp >= kWideStack) return -1;
        stack.put(c.sp++, make_uint2(c.gbase, c.gbits));
    }
    if (++c.visits > s.n_nodes || node >= s.n_nodes) return -1;
    LeafGroup lg;
    c.gbits = wide_node(s.nodes + (size_t)node * 5, r, dir, tmax, c.gbase, lg);
    if (kCount) ++nnode;
    uint32_t tbits = lg.bits;
    while (tbits) {
        const uint32_t rec = leaf_record(lg.base, lg.valid, __ffs(tbits) - 1);
        tbits &= tbits - 1u;
        if (rec >= s.n_tris) return -1;
        const float4* tp = s.tris + (size_t)rec * 3;
        if (kCount) ++ntri;
        float t, V, W, det;
        if (tri_test_t(r, __ldg(tp), __ldg(tp + 1), __ldg(tp + 2), t, V, W, det) && t > r.tmin && t <= tmax)
            return 2;
    }
    while (c.gbits <= 0x00FFFFFFu && c.sp > 0) {
        const uint2 e = stack.get(--c.sp);
        c.gbase = e.x;
        c.gbits = e.y;
    }
    return c.gbits <= 0x00FFFFFFu ? 1 : 0;
}

// Any hit in (tmin, tmax]; `overflow` is set when the traversal aborted
// (any_step == -1; the caller reports KZ_ERR_STACK).
template <bool kCount>
__device__ bool trace_any(const DevScene& s, const TRay& r, float tmax, bool& overflow, uint32_t& nnode,
                          uint32_t& ntri) {
    const WideDir dir = wide_dir(r);
    uint2 stack[kWideStack];
    AnyState c;
    any_begin(c);
    int rc;
    do {
        rc = any_step<kCount>(s, r, dir, tmax, c, LocalStack{stack}, nnode, ntri);
    } while (rc == 0);
    overflow = rc < 0;
    return rc == 2;
}

// ---- warp-shared leaf tests ---------------------------------------------------
//
// In the persistent kernels a traversal step is split into a node part
// (a few node tests per lane; the leaf triangles they hit are left
// pending) and a warp-wide part in which all 32 lanes, busy or idle, test the
// pending (ray, triangle) pairs of the whole warp, 32 at a time. A per-lane
// triangle loop would run for the warp's largest leaf count with a few lanes
// active; sharing the pairs spreads them over the warp.
//
// What bounds these loops is the issue rate (ncu, terrain frame: 79 % of the
// issue slots, ALU pipe 69 %), so the split follows the instructions: one node
// test a step leaves some 12 pairs for 32 lanes, two or three fill them. The
// nodes of a step cull against the bound of the step before, which costs a
// few visits more than it saves only from four on. Trace + shadow stages of
// the terrain frame at 1 / 2 / 3 / 4 nodes a step: 132.6 / 105.0 / 102.2 /
// 104.5 ms (135.7 before, with decoded slots and a searched pair list); any hit
// on 2^24 incoherent rays at 2 / 3 now: 5.44 / 5.34 ms, the terrain frame's
// shadow launches 22.75 / 22.09 ms; closest hit at 2 / 3 / 4: 8.55 / 8.39 /
// 8.94 ms.
//
// Each lane publishes its ray (TriRay) in shared memory when it starts one.
// The closest hit is exact and independent of which lane tested what:
// candidates are combined by a 64-bit atomicMin of (t in a total order, global
// triangle id) on the owner's slot, the lexicographic minimum that the
// sequential loop keeps (smaller t, then smaller id), then the lane whose
// candidate won writes its record, its unrounded t and the barycentric terms.
#ifndef KZ_CLOSEST_STEPS
#define KZ_CLOSEST_STEPS 3
#endif
#ifndef KZ_ANY_STEPS
#define KZ_ANY_STEPS 3
#endif
constexpr int kClosestSteps = KZ_CLOSEST_STEPS, kAnySteps = KZ_ANY_STEPS;

struct LeafShare {
    float4* ray;              // [2 * 256]: (okx, oky, okz, tmin), (Sx, Sy, Sz, axes)
    unsigned long long* key;  // [256] closest: best (t, id); any hit: tmax bits
    uint32_t* rec;            // [256] closest: record of the best; any hit: mask of the triangles hit
    float4* vwdt;             // [256] closest: V, W, det, t of the best
    uint4* ent;               // [steps * 32] this warp's pending groups: bits, valid, base, start | lane << 16
};

__device__ __forceinline__ void publish_ray(const LeafShare& sh, const TRay& r) {
    const TriRay q = tri_ray(r);
    sh.ray[2 * threadIdx.x] = make_float4(q.okx, q.oky, q.okz, q.tmin);
    sh.ray[2 * threadIdx.x + 1] =
        make_float4(q.Sx, q.Sy, q.Sz, __uint_as_float(q.axes));
}

__device__ __forceinline__ TriRay shared_ray(const LeafShare& sh, uint32_t slot) {
    const float4 a = sh.ray[2 * slot], b = sh.ray[2 * slot + 1];
    TriRay q;
    q.okx = a.x;
    q.oky = a.y;
    q.okz = a.z;
    q.tmin = a.w;
    q.Sx = b.x;
    q.Sy = b.y;
    q.Sz = b.z;
    q.axes = __float_as_uint(b.w);
    return q;
}

// (t, id) as one 64-bit key whose unsigned order is float order of t (-0 as
// +0), then id.
__device__ __forceinline__ unsigned long long hit_key(float t, uint32_t prim) {
    const uint32_t u = __float_as_uint(t == 0.f ? 0.f : t);
    const uint32_t o = (u & 0x80000000u) ? ~u : (u | 0x80000000u);
    return ((unsigned long long)o << 32) | prim;
}

// Position of the (k+1)-th set bit of m (k < popc(m), m below bit 31).
__device__ __forceinline__ uint32_t nth_set_bit(uint32_t m, uint32_t k) {
    uint32_t pos = 0;
#pragma unroll
    for (uint32_t s = 16; s; s >>= 1)
        if ((uint32_t)__popc(m & ((1u << (pos + s)) - 1u)) <= k) pos += s;
    return pos;
}

// The pending pairs of a warp as one list: lane by lane, group by group, bit
// by bit. publish_groups writes each non-empty group with the position of its
// first pair; pair p then belongs to the group with the largest start <= p,
// found as the rank of p in a bit mask of the starts (one warp-wide OR and one
// population count, instead of a search).
template <int K>
__device__ __forceinline__ uint32_t publish_groups(const LeafShare& sh, const LeafGroup (&g)[K], uint32_t (&start)[K]) {
    const uint32_t lane = threadIdx.x & 31u, lt = (1u << lane) - 1u;
    uint32_t cnt = 0;
#pragma unroll
    for (int k = 0; k < K; ++k) cnt += __popc(g[k].bits);
    uint32_t incl = cnt;
#pragma unroll
    for (uint32_t o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, incl, o);
        if (lane >= o) incl += v;
    }
    uint32_t rank = 0, at = incl - cnt;
#pragma unroll
    for (int k = 0; k < K; ++k) rank += __popc(__ballot_sync(0xFFFFFFFFu, g[k].bits != 0) & lt);
#pragma unroll
    for (int k = 0; k < K; ++k) {
        start[k] = at;
        if (g[k].bits) {
            sh.ent[rank++] = make_uint4(g[k].bits, g[k].valid, g[k].base, at | (lane << 16));
            at += __popc(g[k].bits);
        }
    }
    return __shfl_sync(0xFFFFFFFFu, incl, 31);
}

// Pair base + lane of the list (base a multiple of 32, the rounds in order;
// `seen` counts the groups that started in earlier rounds): its owner lane and
// record, and its bit in the owner's mask. Every lane must call it.
struct LeafPair {
    uint32_t owner, bit, rec;
    bool live;
};
template <int K>
__device__ __forceinline__ LeafPair leaf_pair(const LeafShare& sh, const LeafGroup (&g)[K], const uint32_t (&start)[K],
                                              uint32_t base, uint32_t total, uint32_t& seen) {
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t m = 0;
#pragma unroll
    for (int k = 0; k < K; ++k)
        if (g[k].bits && start[k] - base < 32u) m |= 1u << (start[k] - base);
    m = __reduce_or_sync(0xFFFFFFFFu, m);
    const uint32_t idx = seen + __popc(m & (0xFFFFFFFFu >> (31u - lane))) - 1u;
    seen += __popc(m);
    LeafPair lp;
    lp.owner = 0;
    lp.bit = 0;
    lp.rec = 0;
    lp.live = base + lane < total;
    if (lp.live) {
        const uint4 e = sh.ent[idx];
        lp.bit = nth_set_bit(e.x, base + lane - (e.w & 0xFFFFu));
        lp.owner = e.w >> 16;
        lp.rec = leaf_record(e.z, e.y, lp.bit);
    }
    return lp;
}

// Node part of a step: visits one node, culling boxes beyond tcur; its leaf
// triangles are left in lg for the warp-wide test. Returns -1 on an abort (as
// closest_step), else 0.
template <bool kCount, typename Stack>
__device__ __forceinline__ int visit_node(const DevScene& s, const TRay& r, const WideDir& dir, float tcur, AnyState& c,
                                          const Stack& stack, LeafGroup& lg, uint32_t& nnode) {
    const uint32_t node = wide_pop_child(c.gbase, c.gbits, dir);
    if (c.gbits > 0x00FFFFFFu) {
        if (c.sp >= kWideStack) return -1;
        stack.put(c.sp++, make_uint2(c.gbase, c.gbits));
    }
    if (++c.visits > s.n_nodes || node >= s.n_nodes) return -1;
    c.gbits = wide_node(s.nodes + (size_t)node * 5, r, dir, tcur, c.gbase, lg);
    if (kCount) ++nnode;
    if (lg.bits && (uint64_t)lg.base + __popc(lg.valid) > s.n_tris) {
        lg.bits = 0;
        return -1;
    }
    return 0;
}

// Next node group from the stack: 1 when the traversal is complete, else 0.
template <typename State, typename Stack>
__device__ __forceinline__ int group_pop(State& c, const Stack& stack) {
    while (c.gbits <= 0x00FFFFFFu && c.sp > 0) {
        const uint2 e = stack.get(--c.sp);
        c.gbase = e.x;
        c.gbits = e.y;
    }
    return c.gbits <= 0x00FFFFFFu ? 1 : 0;
}

// The triangle array of the pair's owner: with kOwnScene each owner's array
// is fetched from its lane (batched jobs trace different scenes in one warp).
template <bool kOwnScene>
__device__ __forceinline__ const float4* owner_tris(const float4* tris, uint32_t owner) {
    if (!kOwnScene) return tris;
    const uint64_t tv = reinterpret_cast<uint64_t>(tris);
    const uint32_t lo = __shfl_sync(0xFFFFFFFFu, (uint32_t)tv, owner);
    const uint32_t hi = __shfl_sync(0xFFFFFFFFu, (uint32_t)(tv >> 32), owner);
    return reinterpret_cast<const float4*>(((uint64_t)hi << 32) | lo);
}

template <int K>
__device__ __forceinline__ bool any_bits(const LeafGroup (&g)[K]) {
    uint32_t b = 0;
#pragma unroll
    for (int k = 0; k < K; ++k) b |= g[k].bits;
    return b != 0;
}

// The best hit of a lane's ray is kept in shared memory: its key, and, once
// there is one, its record and barycentric terms. A NaN bound accepts nothing.
__device__ __forceinline__ void best_begin(const LeafShare& sh, float tmax) {
    sh.key[threadIdx.x] = tmax == tmax ? hit_key(tmax, KZ_INVALID_ID) : 0ull;
    sh.rec[threadIdx.x] = 0xFFFFFFFFu;
}

// t of a key (a -0 comes back as +0)
__device__ __forceinline__ float key_t(unsigned long long key) {
    const uint32_t o = (uint32_t)(key >> 32);
    return __uint_as_float((o & 0x80000000u) ? o & 0x7FFFFFFFu : ~o);
}

// Hit record of the lane's finished traversal; an aborted one (ok == false)
// misses. The barycentric divisions are made for the kept hit only.
__device__ __forceinline__ void best_finish(const LeafShare& sh, bool ok, float tmax, HitRec& h) {
    const int32_t rec = (int32_t)sh.rec[threadIdx.x];
    h.t = tmax;
    h.u = h.v = 0.f;
    h.prim = KZ_INVALID_ID;
    h.rec = -1;
    if (!ok || rec < 0) return;
    const float4 w = sh.vwdt[threadIdx.x];
    h.t = w.w;
    h.u = w.x / w.z;
    h.v = w.y / w.z;
    h.prim = (uint32_t)sh.key[threadIdx.x];
    h.rec = rec;
}

// Warp-wide closest-hit leaf tests; every lane of the warp calls it, lanes
// without pending triangles with empty groups. `tris` is the calling lane's
// triangle array; tcur becomes the lane's best t.
template <bool kOwnScene, int K>
__device__ __forceinline__ void closest_leaves(const LeafShare& sh, const float4* tris, const LeafGroup (&g)[K],
                                               float& tcur) {
    const bool mine = any_bits(g);
    if (__ballot_sync(0xFFFFFFFFu, mine) == 0) return;
    const uint32_t lane = threadIdx.x & 31u, wbase = threadIdx.x - lane;
    uint32_t start[K], seen = 0;
    const uint32_t total = publish_groups(sh, g, start);
    __syncwarp();
    for (uint32_t base = 0; base < total; base += 32) {
        const LeafPair lp = leaf_pair(sh, g, start, base, total, seen);
        const float4* tp = owner_tris<kOwnScene>(tris, lp.owner);
        const uint32_t slot = wbase + lp.owner;
        bool cand = false;
        unsigned long long key = 0;
        float t = 0.f, V = 0.f, W = 0.f, det = 0.f;
        if (lp.live) {
            const TriRay q = shared_ray(sh, slot);
            const float4* tr = tp + (size_t)lp.rec * 3;
            const float4 a = __ldg(tr), b = __ldg(tr + 1), cc = __ldg(tr + 2);
            if (tri_test_t(q, a, b, cc, t, V, W, det) && t > q.tmin) {
                key = hit_key(t, __float_as_uint(a.w));
                cand = key < atomicMin(sh.key + slot, key);
            }
        }
        __syncwarp();
        if (cand && sh.key[slot] == key) {
            sh.rec[slot] = lp.rec;
            sh.vwdt[slot] = make_float4(V, W, det, t);
        }
        __syncwarp();
    }
    if (mine) tcur = fminf(tcur, key_t(sh.key[threadIdx.x]));
}

// Triangles a sequential any-hit loop over tbits (lowest bit first) tests
// before it stops at the first hit of `hits`.
__device__ __forceinline__ uint32_t any_tested(uint32_t tbits, uint32_t hits) {
    return hits ? __popc(tbits & (((hits & (0u - hits)) << 1) - 1u)) : __popc(tbits);
}

// Warp-wide any-hit leaf tests: the mask of the lane's pending triangles
// (bits of its groups) with a hit in (tmin, tmax]. The lane's tmax is in key[]
// as float bits (publish_tmax).
__device__ __forceinline__ void publish_tmax(const LeafShare& sh, float tmax) {
    sh.key[threadIdx.x] = __float_as_uint(tmax);
}
template <bool kOwnScene, int K>
__device__ __forceinline__ uint32_t any_leaves(const LeafShare& sh, const float4* tris, const LeafGroup (&g)[K]) {
    const bool mine = any_bits(g);
    if (__ballot_sync(0xFFFFFFFFu, mine) == 0) return 0u;
    const uint32_t lane = threadIdx.x & 31u, wbase = threadIdx.x - lane;
    uint32_t start[K], seen = 0;
    const uint32_t total = publish_groups(sh, g, start);
    if (mine) sh.rec[threadIdx.x] = 0u;
    __syncwarp();
    for (uint32_t base = 0; base < total; base += 32) {
        const LeafPair lp = leaf_pair(sh, g, start, base, total, seen);
        const float4* tp = owner_tris<kOwnScene>(tris, lp.owner);
        const uint32_t slot = wbase + lp.owner;
        if (lp.live) {
            const TriRay q = shared_ray(sh, slot);
            const float tmax = __uint_as_float((uint32_t)sh.key[slot]);
            const float4* tr = tp + (size_t)lp.rec * 3;
            float t, V, W, det;
            if (tri_test_t(q, __ldg(tr), __ldg(tr + 1), __ldg(tr + 2), t, V, W, det) && t > q.tmin && t <= tmax)
                atomicOr(sh.rec + slot, 1u << lp.bit);
        }
    }
    __syncwarp();
    const uint32_t hits = mine ? sh.rec[threadIdx.x] : 0u;
    __syncwarp();
    return hits;
}

// Persistent ray loop: each warp keeps its lanes busy by fetching new rays
// (one atomic per warp) whenever at least `refill` of its lanes are idle,
// instead of running until its slowest ray ends. Warp-synchronous: one ballot
// per step; start(k) sets up ray k on the calling lane, step() advances it by
// one node and returns true once the ray is finished and its result written.
// Every traversal is bounded, so a warp leaves once the queue [0, n) is
// drained. Refilling only in groups (8 lanes) keeps the set-up code from
// running for one or two lanes at a time.
// Stack entries of a persistent closest-hit thread kept in shared memory
// (16 KB per block of 256 threads at 8). Measured: the terrain frame's trace
// stage 130.6 -> 129.7 ms, the incoherent-ray microbenchmark 1.190 -> 1.242
// Grays/s; the any-hit kernels keep the local stack (their frame stage lost
// 1 % with it).
#ifndef KZ_SMEM_STACK
#define KZ_SMEM_STACK 8
#endif

#ifndef KZ_TRACE_REFILL
#define KZ_TRACE_REFILL 8
#endif
constexpr uint32_t kTraceRefill = KZ_TRACE_REFILL;
// Refill group of the any-hit (shadow ray) kernels.
#ifndef KZ_ANY_REFILL
#define KZ_ANY_REFILL KZ_TRACE_REFILL
#endif
constexpr uint32_t kAnyRefill = KZ_ANY_REFILL;

// node(lg) runs on the busy lanes and returns -1 on an abort, 0 while nodes
// remain and 1 when none do; leaves(groups) runs on all 32 lanes; finish(rc)
// on the busy lanes returns true once the ray is finished and its result
// written.
//
// A queue that does not fill the grid: blocks beyond its share leave at once
// (256 rays a block, but 8 a block, one a warp, while that leaves SMs without
// one), and of each warp only the first ceil(n / warps) lanes take rays; the
// others help with the leaf tests. Reached by calls of more rays than take a warp
// each, by stage timing and fetch counting, and by wavefronts above 2^23 paths.
// With / without the spread: 16,385 closest hits through 250,000 triangles 148 / 169
// us, 20,000 through a 525,000-triangle terrain 73 / 83, through 36 triangles 28 / 34
// (any hits, 12,288); 32 x 32 x 4 paths of depth 5 with stage timing 0.49 / 0.57 ms,
// counted 0.52 / 0.72. Rays over all resident blocks instead: 65,537 Li rays 600 us
// against 540 over 257 blocks, since the warps' steps, not the longest ray, are
// waited for there.
constexpr uint32_t kSpreadBlocks = 152;  // the SMs of a GB300: a rule of speed only
template <typename Ctr>
__host__ __device__ __forceinline__ uint32_t trace_blocks(Ctr n, uint32_t most) {
    const Ctr full = (n + 255) / 256, spread = n < 8 * kSpreadBlocks ? (n + 7) / 8 : kSpreadBlocks;
    const Ctr want = full > spread ? full : spread;
    return want < most ? (uint32_t)want : most;
}

template <int K, typename Ctr, typename Start, typename Node, typename Leaves, typename Finish>
__device__ __forceinline__ void persistent_rays_shared(Ctr n, Ctr* next, uint32_t refill, Start start, Node node,
                                                       Leaves leaves, Finish finish) {
    const uint32_t blocks = trace_blocks(n, gridDim.x);
    if (blockIdx.x >= blocks) return;
    const uint32_t lane = threadIdx.x & 31u, warps = blocks * (blockDim.x >> 5);
    const uint32_t take = n >= (Ctr)warps * 32u ? 32u : (uint32_t)((n + (warps - 1u)) / warps);
    const uint32_t takers = 0xFFFFFFFFu >> (32u - (take ? take : 1u));
    refill = min(refill, take);
    bool busy = false, more = true;
    for (;;) {
        const uint32_t idle = __ballot_sync(0xFFFFFFFFu, !busy) & takers;
        if (!more && idle == takers) break;
        const uint32_t n_idle = __popc(idle);
        if (more && n_idle >= refill) {
            Ctr base = 0;
            if (lane == 0) base = atomicAdd(next, (Ctr)n_idle);
            base = __shfl_sync(0xFFFFFFFFu, base, 0);
            if (base + n_idle >= n) more = false;
            if (!busy && ((takers >> lane) & 1u)) {
                const Ctr k = base + __popc(idle & ((1u << lane) - 1u));
                if (k < n) {
                    busy = true;
                    start(k);
                }
            }
        }
        LeafGroup g[K];
        int rc = busy ? 0 : 1;
#pragma unroll
        for (int k = 0; k < K; ++k) {
            g[k].bits = g[k].valid = g[k].base = 0;
            if (rc == 0) rc = node(g[k]);
        }
        leaves(g);
        if (busy && finish(rc)) busy = false;
    }
}

// ---- one ray per warp ------------------------------------------------------------
//
// A handful of rays cannot fill the device: the call takes as long as its
// longest ray, and a ray of the loops above waits some 80 instructions of one
// node's eight slots, one after the other, at every step. Here a warp takes
// one ray: four nodes of its stack at a time, a lane per slot, and every lane
// tests its own slot's triangles. The boxes, the triangle test and the order
// of hits are the same, so the results are the same bits. 64 picked rays from
// host memory through 20,000 triangles: 105 -> 39 us a call (with the copies gone,
// kz_api.cu), 65,537 Li rays of depth 5, whose later iterations have few: 536 ->
// 443 us.
// Entries of a warp's stack; a ray that needs more falls back on the sequential
// loop (a test build's small stack is small here too).
constexpr int kWarpStack = kWideStack < kWideDepthCap ? kWideStack : 128;

struct WarpRay {
    float t;  // the lane's best, with its terms
    float V, W, det;
    uint32_t prim;
    int32_t rec;
};

// Traverses one ray with the whole warp; `stack`: its kWarpStack entries of node
// and entry distance, in shared memory. Returns 1 when it is complete (closest:
// each lane holds the best of its own triangles; any hit: none found), 2 on a
// hit (any hit), 0 if the stack was too small, -1 on an abort (as closest_step).
template <bool kAny>
__device__ __forceinline__ int warp_traverse(const DevScene& s, const TRay& r, float tmax, uint2* stack, WarpRay& h) {
    const uint32_t lane = threadIdx.x & 31u, up = 3u - (lane >> 3), lt = (1u << lane) - 1u;
    const uint32_t flip = 7u ^ ((r.inv.x < 0.f ? 1u : 0u) | (r.inv.y < 0.f ? 2u : 0u) | (r.inv.z < 0.f ? 4u : 0u));
    const uint32_t slot = (lane & 7u) ^ flip;  // the nearest octant in the highest lane, pushed last
    const TriRay q = tri_ray(r);
    const WideDir dir = wide_dir(r);
    h.t = tmax;
    h.V = h.W = 0.f;
    h.det = 1.f;
    h.prim = KZ_INVALID_ID;
    h.rec = -1;
    float tcur = tmax;
    uint32_t sp = 1, visits = 0;
    if (lane == 0) stack[0] = make_uint2(0u, __float_as_uint(r.tmin));
    __syncwarp();
    while (sp) {
        // one node at a time when the stack might not hold four nodes' children
        const uint32_t n = (int)sp > kWarpStack - 32 && kWarpStack > 32 ? 1u : min(sp, 4u);
        visits += n;
        if (visits > s.n_nodes) return -1;
        const uint2 e = up < n ? stack[sp - 1u - up] : make_uint2(0u, 0u);
        bool alive = up < n && !(__uint_as_float(e.y) > tcur);
        if (__any_sync(0xFFFFFFFFu, alive && e.x >= s.n_nodes)) return -1;
        sp -= n;
        __syncwarp();
        uint32_t child = 0, tri = 0, leaf = 0;
        float tn = 0.f;
        bool inner = false;
        if (alive) {
            const uint4* np = s.nodes + (size_t)e.x * 5;
            const uint4 h0 = __ldg(np), h1 = __ldg(np + 1);
            const uint32_t* w = reinterpret_cast<const uint32_t*>(np + 2) + (slot >> 1);
            const uint32_t odd = (slot & 1u) << 5;
            const auto axis = [&](float p, float scale, float o, float inv, uint32_t word, uint32_t sel, float& lo,
                                  float& hi) {
                const WideAxis ax = wide_axis(p, scale, o, inv, make_uint4(0u, 0u, 0u, 0u));
                lo = fmaf(__uint_as_float(__byte_perm(word, 0x3F800000u, sel | odd)), ax.A, ax.Bn);
                hi = fmaf(__uint_as_float(__byte_perm(word, 0x3F800000u, (sel ^ 0x10u) | odd)), ax.A, ax.Bf);
            };
            float xn, xf, yn, yf, zn, zf;
            axis(__uint_as_float(h0.x), __uint_as_float(h0.w << 16), r.o.x, r.inv.x, __ldg(w), dir.sx, xn, xf);
            axis(__uint_as_float(h0.y), __uint_as_float(h0.w & 0xFFFF0000u), r.o.y, r.inv.y, __ldg(w + 4), dir.sy, yn,
                 yf);
            axis(__uint_as_float(h0.z), __uint_as_float(h1.w << 16), r.o.z, r.inv.z, __ldg(w + 8), dir.sz, zn, zf);
            tn = fmaxf(fmaxf(fmaxf(xn, r.tmin), yn), zn);
            const float tf = fminf(fminf(fminf(xf, tcur), yf), zf);
            if (tn <= tf) {
                inner = (h1.z >> (24 + slot)) & 1u;
                child = h1.x + __popc((h1.z >> 24) & ((1u << slot) - 1u));
                const uint32_t valid = h1.z & 0x00FFFFFFu;
                leaf = (valid >> (3u * slot)) & 7u;
                tri = leaf_record(h1.y, valid, 3u * slot);
            }
        }
        const uint32_t in = __ballot_sync(0xFFFFFFFFu, inner);
        if (sp + __popc(in) > (uint32_t)kWarpStack) return 0;
        if (inner) stack[sp + __popc(in & lt)] = make_uint2(child, __float_as_uint(tn));
        sp += __popc(in);
        __syncwarp();
        if (!__any_sync(0xFFFFFFFFu, leaf != 0)) continue;
        bool hit = false, out = false;
        for (; leaf; leaf &= leaf - 1u, ++tri) {  // a leaf's triangles are consecutive
            if (tri >= s.n_tris) {
                out = true;
                break;
            }
            const float4* tp = s.tris + (size_t)tri * 3;
            const float4 a = __ldg(tp), b = __ldg(tp + 1), c = __ldg(tp + 2);
            float t, V, W, det;
            if (!tri_test_t(q, a, b, c, t, V, W, det) || !(t > r.tmin)) continue;
            if (kAny) {
                hit |= t <= tmax;
            } else {
                const uint32_t prim = __float_as_uint(a.w);
                if (t < h.t || (t == h.t && prim < h.prim)) {
                    h.t = t;
                    h.V = V;
                    h.W = W;
                    h.det = det;
                    h.prim = prim;
                    h.rec = (int32_t)tri;
                }
            }
        }
        if (__any_sync(0xFFFFFFFFu, out)) return -1;
        if (kAny) {
            if (__any_sync(0xFFFFFFFFu, hit)) return 2;
        } else {
            tcur = fminf(tcur, key_t((unsigned long long)__reduce_min_sync(
                                         0xFFFFFFFFu, (uint32_t)(hit_key(h.t, 0u) >> 32)) << 32));
        }
    }
    return 1;
}

// ---- a bundle of 32 rays per warp ---------------------------------------------------
//
// Rays of one origin and neighbouring directions (the samples of a camera's
// pixel) visit the same nodes. The warp tests a box once for all of them, with
// the interval of their inverse directions on each axis and the largest of
// their bounds, a lane per slot of four nodes; the triangles of a leaf are then tested by
// every lane against its own ray. A box is culled only if every ray's own test
// would cull it, and a ray's hits are compared as in the sequential loop, so
// the results are the same bits. Camera rays of the 1080p terrain frame, 64 spp:
// 15 nodes and 7 triangles a bundle in 6 steps, where each ray alone visits 11
// and tests 4; 22.5 -> 15.8 ms, of which some 3 write the paths' state.
//
// That holds while the rays of a bundle stay together. In an image whose pixels
// are coarse against the scene (a small image, or a scene seen from afar) a
// bundle's beam covers thousands of triangles, of which each ray meets a few; so
// a bundle gives up, and its rays are traced each on its own lane, once its steps
// and triangle tests and four times the entries on its stack exceed kBundleWork
// (a wide beam is told by its stack before it has spent the work). Frames of depth
// 5, ms, without a limit / work alone up to 64 / up to 192 / this / without bundles:
// 2.2 M triangle terrain 8 x 8, 8 spp 230 / 0.29 / 0.35 / 0.32 / 0.22, 64 x 64, 8 spp
// 13.6 / 0.40 / 0.46 / 0.43 / 0.35, 512 x 512, 8 spp 2.65 / 1.93 / 2.03 / 2.00 / 1.79,
// 960 x 540, 8 spp from 20 times as far 18.0 / 0.67 / 0.73 / 0.66 / 0.59, 1080p, 8 spp
// 13.44 / 13.63 / 13.49 / 13.49 / 14.64, 64 spp of depth 8 98.2 / 98.8 / 98.5 / 98.5 /
// 109.5; slit room 64 x 64, 8 spp 0.463 / - / 0.473 / 0.465 / 0.400; mixed materials
// 641 x 359, 16 spp 7.46 / 7.50 / 7.46 / 7.46 / 7.74.
#ifndef KZ_BUNDLE_WORK
#define KZ_BUNDLE_WORK 192
#endif
constexpr uint32_t kBundleWork = KZ_BUNDLE_WORK;

// Smallest and largest of a float over the warp (no NaN).
__device__ __forceinline__ float warp_min(float v) {
    const uint32_t o = (uint32_t)(hit_key(v, 0u) >> 32);
    return key_t((unsigned long long)__reduce_min_sync(0xFFFFFFFFu, o) << 32);
}
__device__ __forceinline__ float warp_max(float v) {
    const uint32_t o = (uint32_t)(hit_key(v, 0u) >> 32);
    return key_t((unsigned long long)__reduce_max_sync(0xFFFFFFFFu, o) << 32);
}

// Closest hits of the warp's rays, all from r.o with r.tmin, unbounded. Lanes
// without a ray pass live = false and a copy of another lane's ray. False if
// the bundle gave up or the stack was too small (nothing is set then); on an
// abort (as closest_step) the rays miss and *aborted is set.
__device__ __forceinline__ bool warp_bundle(const DevScene& s, const TRay& r, bool live, uint2* stack, WarpRay& h,
                                            bool& aborted) {
    const uint32_t lane = threadIdx.x & 31u, up = 3u - (lane >> 3), lt = (1u << lane) - 1u;
    const float inf = __int_as_float(0x7f800000);
    f3 lo = mk(warp_min(r.inv.x), warp_min(r.inv.y), warp_min(r.inv.z));
    f3 hi = mk(warp_max(r.inv.x), warp_max(r.inv.y), warp_max(r.inv.z));
    // an axis whose directions change sign: the steepest of each side instead
    const auto sides = [&](float inv, float& l, float& h) {
        if (!(l < 0.f && h > 0.f)) return false;
        l = warp_max(inv < 0.f ? inv : -inf);
        h = warp_min(inv > 0.f ? inv : inf);
        return true;
    };
    const bool mx = sides(r.inv.x, lo.x, hi.x), my = sides(r.inv.y, lo.y, hi.y), mz = sides(r.inv.z, lo.z, hi.z);
    const uint32_t flip = 7u ^ ((lo.x < 0.f ? 1u : 0u) | (lo.y < 0.f ? 2u : 0u) | (lo.z < 0.f ? 4u : 0u));
    const uint32_t slot = (lane & 7u) ^ flip;
    const TriRay q = tri_ray(r);
    h.t = live ? inf : -inf;
    h.V = h.W = 0.f;
    h.det = 1.f;
    h.prim = KZ_INVALID_ID;
    h.rec = -1;
    aborted = false;
    float tcur = inf;
    uint32_t sp = 1, visits = 0, work = 0;
    if (lane == 0) stack[0] = make_uint2(0u, __float_as_uint(r.tmin));
    __syncwarp();
    while (sp) {
        if (++work + 4u * sp > kBundleWork) return false;
        const uint32_t n = (int)sp > kWarpStack - 32 && kWarpStack > 32 ? 1u : min(sp, 4u);
        visits += n;
        const uint2 e = up < n ? stack[sp - 1u - up] : make_uint2(0u, 0u);
        const bool alive = up < n && !(__uint_as_float(e.y) > tcur);
        if (visits > s.n_nodes || __any_sync(0xFFFFFFFFu, alive && e.x >= s.n_nodes)) {
            aborted = true;
            break;
        }
        sp -= n;
        __syncwarp();
        uint32_t child = 0, tri = 0, leaf = 0;
        float tn = 0.f;
        bool inner = false;
        if (alive) {
            const uint4* np = s.nodes + (size_t)e.x * 5;
            const uint4 h0 = __ldg(np), h1 = __ldg(np + 1);
            const uint32_t* w = reinterpret_cast<const uint32_t*>(np + 2) + (slot >> 1);
            const uint32_t odd = (slot & 1u) << 4;
            tn = r.tmin;
            float tf = tcur;
            const auto axis = [&](float p, float scale, float o, float i0, float i1, bool mixed, uint32_t word) {
                scale *= 3.0517578125e-05f;  // the node keeps 2^15 times its quantum
                const float b = p - o;
                const float a0 = b + (float)((word >> odd) & 0xFFu) * scale;
                const float a1 = b + (float)((word >> (odd + 8u)) & 0xFFu) * scale;
                const float d = (fabsf(b) + scale * 1024.f) * fmaxf(fabsf(i0), fabsf(i1)) * 1.52587890625e-05f;
                if (mixed) {  // reached once the steepest direction towards the box gets there, never left
                    const float near = a0 > 0.f ? a0 * i1 : a1 < 0.f ? a1 * i0 : -inf;
                    tn = fmaxf(tn, near - d);
                    return;
                }
                const float near = i0 < 0.f ? a1 : a0, far = i0 < 0.f ? a0 : a1;
                tn = fmaxf(tn, fminf(near * i0, near * i1) - d);
                tf = fminf(tf, fmaxf(far * i0, far * i1) + d);
            };
            axis(__uint_as_float(h0.x), __uint_as_float(h0.w << 16), r.o.x, lo.x, hi.x, mx, __ldg(w));
            axis(__uint_as_float(h0.y), __uint_as_float(h0.w & 0xFFFF0000u), r.o.y, lo.y, hi.y, my, __ldg(w + 4));
            axis(__uint_as_float(h0.z), __uint_as_float(h1.w << 16), r.o.z, lo.z, hi.z, mz, __ldg(w + 8));
            if (!(tn > tf)) {
                inner = (h1.z >> (24 + slot)) & 1u;
                child = h1.x + __popc((h1.z >> 24) & ((1u << slot) - 1u));
                const uint32_t valid = h1.z & 0x00FFFFFFu;
                leaf = (valid >> (3u * slot)) & 7u;
                tri = leaf_record(h1.y, valid, 3u * slot);
            }
        }
        const uint32_t in = __ballot_sync(0xFFFFFFFFu, inner);
        if (sp + __popc(in) > (uint32_t)kWarpStack) return false;
        if (inner) stack[sp + __popc(in & lt)] = make_uint2(child, __float_as_uint(tn));
        sp += __popc(in);
        __syncwarp();
        uint32_t leaves = __ballot_sync(0xFFFFFFFFu, leaf != 0);
        if (!leaves) continue;
        while (leaves) {
            const uint32_t l = 31u - __clz(leaves);  // the nearest first
            leaves ^= 1u << l;
            const uint32_t first = __shfl_sync(0xFFFFFFFFu, tri, l), count = __popc(__shfl_sync(0xFFFFFFFFu, leaf, l));
            if ((uint64_t)first + count > s.n_tris) {
                aborted = true;
                break;
            }
            work += count;
            for (uint32_t k = first; k < first + count; ++k) {
                const float4* tp = s.tris + (size_t)k * 3;
                const float4 a = __ldg(tp), b = __ldg(tp + 1), c = __ldg(tp + 2);
                float t, V, W, det;
                if (!tri_test_t(q, a, b, c, t, V, W, det) || !(t > r.tmin)) continue;
                const uint32_t prim = __float_as_uint(a.w);
                if (t < h.t || (t == h.t && prim < h.prim)) {
                    h.t = t;
                    h.V = V;
                    h.W = W;
                    h.det = det;
                    h.prim = prim;
                    h.rec = (int32_t)k;
                }
            }
        }
        if (aborted) break;
        __syncwarp();
        tcur = warp_max(h.t);
    }
    return true;
}

// The best of the lanes' hits, in the lane that holds it; true there. (Both
// reductions are taken by every lane, whether it holds a hit or not.)
__device__ __forceinline__ bool warp_best(const WarpRay& h) {
    const uint32_t o = h.rec >= 0 ? (uint32_t)(hit_key(h.t, 0u) >> 32) : 0xFFFFFFFFu;
    const uint32_t o_min = __reduce_min_sync(0xFFFFFFFFu, o);
    const bool first = h.rec >= 0 && o == o_min;
    const uint32_t prim_min = __reduce_min_sync(0xFFFFFFFFu, first ? h.prim : KZ_INVALID_ID);
    return first && h.prim == prim_min;
}

// Closest hit of one ray with the whole warp: calls store(hit) on one lane;
// false on an abort (the hit is a miss then).
template <typename Store>
__device__ __forceinline__ bool warp_closest(const DevScene& s, const TRay& r, float tmax, uint2* stack,
                                             Store store) {
    WarpRay w;
    const int rc = warp_traverse<false>(s, r, tmax, stack, w);
    HitRec h{tmax, 0.f, 0.f, KZ_INVALID_ID, -1};
    bool mine = (threadIdx.x & 31u) == 0, ok = rc >= 0;
    if (rc == 1) {
        const bool best = warp_best(w);
        if (__any_sync(0xFFFFFFFFu, best)) mine = best;
        if (best) h = HitRec{w.t, w.V / w.det, w.W / w.det, w.prim, w.rec};
    } else if (rc == 0 && mine) {
        uint32_t dn = 0, dt = 0;
        ok = trace_closest<false>(s, r, tmax, h, dn, dt);
    }
    if (mine) store(h);
    return __all_sync(0xFFFFFFFFu, ok);
}

// Any hit of one ray with the whole warp: 1 none, 2 a hit, -1 aborted.
__device__ __forceinline__ int warp_any(const DevScene& s, const TRay& r, float tmax, uint2* stack) {
    WarpRay w;
    int rc = warp_traverse<true>(s, r, tmax, stack, w);
    if (rc == 0) {
        if ((threadIdx.x & 31u) == 0) {
            uint32_t dn = 0, dt = 0;
            bool overflow;
            rc = trace_any<false>(s, r, tmax, overflow, dn, dt) ? 2 : overflow ? -1 : 1;
        }
        rc = __shfl_sync(0xFFFFFFFFu, rc, 0);
    }
    return rc;
}

// The warps of a persistent kernel take the rays [0, n) one at a time:
// ray(k) runs on the whole warp.
template <typename Ctr, typename Ray>
__device__ __forceinline__ void warp_rays(Ctr n, Ctr* next, Ray ray) {
    for (;;) {
        Ctr k = 0;
        if ((threadIdx.x & 31u) == 0) k = atomicAdd(next, (Ctr)1);
        k = __shfl_sync(0xFFFFFFFFu, k, 0);
        if (k >= n) break;
        ray(k);
    }
}

}  // namespace kz
