// kz_closures.cu — batch closure kernels (kz_closure_eval_batch /
// kz_closure_sample_batch): one lobe, incident and outgoing direction per
// query, in the reference or the integrator convention (kz_device.cuh).
//
// Queries come in any order of closure kinds, and the kinds are branches of
// one switch: a warp of 32 arbitrary queries runs most of the 21 branches with
// one or two lanes each, the FP64 Beckmann sampler among them. So a block
// stages a tile of queries in shared memory (coalesced), groups them by kind
// with a counting sort, and each thread then works on queries of the sorted
// order; results replace their query's own inputs in the tile and leave
// coalesced. Values are those of the ungrouped kernel, bit for bit.
//
// 1,000,003 queries over 21 kinds (221 bytes each over both calls, 33 us at
// the measured copy rate): evaluation 567 -> 140 us, sampling 4,856 -> 700 us.
// The sampling that is left is bound by FP64: the Beckmann slope search of
// one query in ten, on an FP64 rate of two lanes a clock and SM.
#include "kz_stages.cuh"

namespace kz {
namespace {

constexpr int kClosureThreads = 256;
constexpr int kLobeWords = sizeof(kz_lobe) / 4;
constexpr int kLobeStride = kLobeWords + 1;  // words; odd, so that a word of 32 records lies in 32 banks
constexpr int kKinds = 32;

// Bin of a lobe in the grouping: its closure id (all below 27 but the
// conductor's), the Beckmann form of the two microfacet kinds apart.
__device__ __forceinline__ uint32_t closure_kind(uint32_t id, float dist) {
    if (id == KZ_CLOSURE_KP_GLOSS || id == KZ_CLOSURE_KP_GLASS)
        return dist == (float)KZ_DIST_BECKMANN ? id + 10u : id;
    return id < 27u ? id : id == KZ_CLOSURE_CONDUCTOR_GGX ? 27u : 31u;
}

// A tile of kItems * 256 queries: lobes, two directions each (for sampling
// the second holds the uniforms), and the sorted order.
template <int kItems>
struct ClosureTile {
    static constexpr int kN = kItems * kClosureThreads;
    uint32_t lobe[kN * kLobeStride];
    float a[kN * 3], b[kN * 3];
    uint16_t order[kN];
    uint32_t count[kKinds];
};

// Loads the tile's m queries and groups them by kind.
template <int kItems>
__device__ __forceinline__ void load_tile(ClosureTile<kItems>& t, const kz_lobe* lobes, const float* a, const float* b,
                                          uint64_t first, uint32_t m) {
    const uint32_t tid = threadIdx.x;
    const uint32_t* lw = reinterpret_cast<const uint32_t*>(lobes + first);
    for (uint32_t k = tid; k < m * kLobeWords; k += kClosureThreads)
        t.lobe[(k / kLobeWords) * kLobeStride + k % kLobeWords] = __ldg(lw + k);
    for (uint32_t k = tid; k < 3 * m; k += kClosureThreads) {
        t.a[k] = __ldg(a + 3 * first + k);
        t.b[k] = __ldg(b + 3 * first + k);
    }
    if (tid < kKinds) t.count[tid] = 0u;
    __syncthreads();
    uint32_t kind[kItems], rank[kItems];
#pragma unroll
    for (int j = 0; j < kItems; ++j) {
        const uint32_t q = tid + j * kClosureThreads;
        if (q < m) {
            const kz_lobe& l = *reinterpret_cast<const kz_lobe*>(t.lobe + q * kLobeStride);
            kind[j] = closure_kind(l.closure_id, l.params[0]);
            rank[j] = atomicAdd(&t.count[kind[j]], 1u);
        }
    }
    __syncthreads();
    if (tid < kKinds) {  // exclusive prefix over the kinds (the first warp)
        const uint32_t c = t.count[tid];
        uint32_t incl = c;
#pragma unroll
        for (uint32_t o = 1; o < kKinds; o <<= 1) {
            const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, incl, o);
            if (tid >= o) incl += v;
        }
        t.count[tid] = incl - c;
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kItems; ++j) {
        const uint32_t q = tid + j * kClosureThreads;
        if (q < m) t.order[t.count[kind[j]] + rank[j]] = (uint16_t)q;
    }
    __syncthreads();
}

__device__ __forceinline__ void put3(float* p, f3 v) {
    p[0] = v.x;
    p[1] = v.y;
    p[2] = v.z;
}

template <int kItems>
__global__ void __launch_bounds__(kClosureThreads) k_closure_eval(const kz_lobe* __restrict__ lobes,
                                                                  const float* __restrict__ wi,
                                                                  const float* __restrict__ wo, uint64_t n, int conv,
                                                                  float* f, float* pdf) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    ClosureTile<kItems>& t = *reinterpret_cast<ClosureTile<kItems>*>(smem_raw);
    const uint64_t first = (uint64_t)blockIdx.x * t.kN;
    const uint32_t m = (uint32_t)min((uint64_t)t.kN, n - first);
    load_tile(t, lobes, wi, wo, first, m);
#pragma unroll 1
    for (uint32_t k = threadIdx.x; k < m; k += kClosureThreads) {
        const uint32_t q = t.order[k];
        const kz_lobe& l = *reinterpret_cast<const kz_lobe*>(t.lobe + q * kLobeStride);
        const f3 a = ld3(t.a + 3 * q), b = ld3(t.b + 3 * q);
        const LobeEval e = conv == KZ_CONVENTION_REFERENCE ? lobe_eval_reference<true>(l, a, b) : lobe_eval(l, a, b);
        put3(t.a + 3 * q, e.f);
        t.b[q * 3] = e.pdf;
    }
    __syncthreads();
    for (uint32_t k = threadIdx.x; k < 3 * m; k += kClosureThreads) f[3 * first + k] = t.a[k];
    for (uint32_t k = threadIdx.x; k < m; k += kClosureThreads) pdf[first + k] = t.b[3 * k];
}

template <int kItems>
__global__ void __launch_bounds__(kClosureThreads) k_closure_sample(const kz_lobe* __restrict__ lobes,
                                                                    const float* __restrict__ wi,
                                                                    const float* __restrict__ u, uint64_t n, float* wo,
                                                                    float* weight, float* pdf, uint8_t* flags) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    ClosureTile<kItems>& t = *reinterpret_cast<ClosureTile<kItems>*>(smem_raw);
    const uint64_t first = (uint64_t)blockIdx.x * t.kN;
    const uint32_t m = (uint32_t)min((uint64_t)t.kN, n - first);
    load_tile(t, lobes, wi, u, first, m);
#pragma unroll 1
    for (uint32_t k = threadIdx.x; k < m; k += kClosureThreads) {
        const uint32_t q = t.order[k];
        uint32_t* rec = t.lobe + q * kLobeStride;
        const LobeSample s = lobe_sample(*reinterpret_cast<const kz_lobe*>(rec), ld3(t.a + 3 * q), t.b[3 * q],
                                         t.b[3 * q + 1], t.b[3 * q + 2]);
        put3(t.a + 3 * q, s.wo);
        put3(t.b + 3 * q, s.weight);
        rec[0] = __float_as_uint(s.pdf);
        rec[1] = (s.valid ? 1u : 0u) | (s.delta ? 2u : 0u);
    }
    __syncthreads();
    for (uint32_t k = threadIdx.x; k < 3 * m; k += kClosureThreads) {
        wo[3 * first + k] = t.a[k];
        weight[3 * first + k] = t.b[k];
    }
    for (uint32_t k = threadIdx.x; k < m; k += kClosureThreads) {
        pdf[first + k] = __uint_as_float(t.lobe[k * kLobeStride]);
        flags[first + k] = (uint8_t)t.lobe[k * kLobeStride + 1];
    }
}

// Queries per thread: four (a tile of 1,024 holds about 45 of each of 23
// kinds, more than a warp) once that still gives every SM two tiles, else
// one, so that small batches spread over more SMs.
#ifndef KZ_CLOSURE_ITEMS
#define KZ_CLOSURE_ITEMS 4
#endif
bool wide_tiles(uint64_t n) { return n >= (uint64_t)2 * 152 * KZ_CLOSURE_ITEMS * kClosureThreads; }

// Tiles above 48 KB need the limit raised (on the current device and context,
// so with each launch).
template <typename F>
void allow_smem(F f, size_t bytes) {
    cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

}  // namespace

void launch_closure_eval(const kz_lobe* lobes, const float* wi, const float* wo, uint64_t n, int convention,
                         float* f, float* pdf, cudaStream_t st) {
    if (!n) return;
    if (wide_tiles(n)) {
        using T = ClosureTile<KZ_CLOSURE_ITEMS>;
        allow_smem(k_closure_eval<KZ_CLOSURE_ITEMS>, sizeof(T));
        k_closure_eval<KZ_CLOSURE_ITEMS><<<grid_for(n, T::kN), kClosureThreads, sizeof(T), st>>>(lobes, wi, wo, n,
                                                                                              convention, f, pdf);
    } else {
        using T = ClosureTile<1>;
        k_closure_eval<1><<<grid_for(n, T::kN), kClosureThreads, sizeof(T), st>>>(lobes, wi, wo, n, convention, f,
                                                                                 pdf);
    }
}
void launch_closure_sample(const kz_lobe* lobes, const float* wi, const float* u, uint64_t n, float* wo,
                           float* weight, float* pdf, uint8_t* flags, cudaStream_t st) {
    if (!n) return;
    if (wide_tiles(n)) {
        using T = ClosureTile<KZ_CLOSURE_ITEMS>;
        allow_smem(k_closure_sample<KZ_CLOSURE_ITEMS>, sizeof(T));
        k_closure_sample<KZ_CLOSURE_ITEMS><<<grid_for(n, T::kN), kClosureThreads, sizeof(T), st>>>(
            lobes, wi, u, n, wo, weight, pdf, flags);
    } else {
        using T = ClosureTile<1>;
        k_closure_sample<1><<<grid_for(n, T::kN), kClosureThreads, sizeof(T), st>>>(lobes, wi, u, n, wo, weight, pdf,
                                                                                   flags);
    }
}

}  // namespace kz
