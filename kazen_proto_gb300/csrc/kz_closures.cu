// kz_closures.cu — batch closure kernels (kz_closure_eval_batch /
// kz_closure_sample_batch): one lobe, incident and outgoing direction per
// query, in the reference or the integrator convention (kz_device.cuh).
//
// Queries come in any order of closure kinds, and the kinds are branches of
// one switch: a warp of 32 arbitrary queries runs most of the 21 branches with
// one or two lanes each, the FP64 Beckmann sampler among them. So a block
// groups a tile of queries by kind with a counting sort in shared memory, and
// its warps work through the sorted order, the FP64 searches first. Directions
// and results move coalesced through the tile, results in place of their
// query's own inputs. Values are those of the ungrouped kernel, bit for bit.
//
// 1,000,003 queries over 21 kinds (221 bytes each over both calls, 33 us at
// the measured copy rate), evaluation and sampling: 5,450 -> 490 us, 87 of it
// evaluation. Bound by instruction fetch (21 branches, a few warps in each at a
// time: 13 % of the issue slots busy in sampling) and by the wait of every tile
// for its Beckmann slope searches, one query in ten; not by FP64 throughput, nor
// by memory: Beckmann queries alone (1.8 us a thousand) and the others alone
// (0.07) add up to some 235 us. The lobes themselves stay out of the tile: with
// them in it two blocks fit an SM instead of four, and fewer searches were in
// flight (717 us; 860 with the searches last).
//
// A tile of one kind, or of few queries, is not sorted, and its results go
// straight to memory. A batch of one kind then takes as long as in an ungrouped
// kernel up to 311,296 queries, and 1.1 to 1.25 times as long above a million
// (diffuse ones 0.85 to 0.95 times): the tile's barriers and staging, and four
// queries a thread. GGX glass, 262,144 queries, both calls: 105 -> 82 us (80
// ungrouped); principled specular, 4,000,000: 484 -> 463 (395).
#include "kz_stages.cuh"

namespace kz {
namespace {

constexpr int kClosureThreads = 256;
constexpr int kClosureBlocks = 4;  // per SM: 64 registers a thread
constexpr int kKinds = 32;

// Bin of a lobe in the grouping: by closure id, largest first (all are below 27
// but the conductor's), the Beckmann form of the two microfacet kinds in bins
// of its own before them: a tile starts with the FP64 searches, which take as
// long as the rest of it, and its other warps work through the rest meanwhile.
__device__ __forceinline__ uint32_t closure_kind(uint32_t id, float dist) {
    if (id == KZ_CLOSURE_KP_GLOSS || id == KZ_CLOSURE_KP_GLASS)
        return dist == (float)KZ_DIST_BECKMANN ? 21u - id : 31u - id;
    return id < 27u ? 31u - id : id == KZ_CLOSURE_CONDUCTOR_GGX ? 4u : 0u;
}

// A tile of kItems * 256 queries: two directions each (for sampling the second
// holds the uniforms), the sorted order, and what a result does not fit into
// its inputs. Lobes stay in global memory: a thread reads its query's whole
// record, two sectors, and the kinds read before have brought one of them near.
template <int kItems>
struct ClosureTile {
    static constexpr int kN = kItems * kClosureThreads;
    float a[kN * 3], b[kN * 3], pdf[kN];
    uint16_t order[kN];
    uint8_t flags[kN];
    uint32_t count[kKinds], start[kKinds], kind0, next;
};

// The warps of a block take the sorted queries 32 at a time; returns the
// lane's place in the order (m or more: none), done once the warp's first is.
template <typename Tile>
__device__ __forceinline__ bool next_queries(Tile& t, uint32_t m, uint32_t& k) {
    uint32_t first = 0;
    if ((threadIdx.x & 31u) == 0) first = atomicAdd(&t.next, 32u);
    first = __shfl_sync(0xFFFFFFFFu, first, 0);
    k = first + (threadIdx.x & 31u);
    return first < m;
}

// Loads the tile's m queries and groups them by kind. False, with no order
// written, if they are all of one kind or at most kUnsorted: three warps are too
// few to hold a kind each, and a short call is as long as its barriers. Evaluation
// and sampling of 21 kinds sorted / unsorted (and in an ungrouped kernel): 48
// queries 137 / 114 us (115), 65 129 / 116 (118), 96 131 / 121 (124), but six
// microfacet kinds and diffuse 112 112 / 127 (129), 128 108 / 131 (133).
constexpr uint32_t kUnsorted = 96;
template <int kItems>
__device__ __forceinline__ bool load_tile(ClosureTile<kItems>& t, const kz_lobe* lobes, const float* a, const float* b,
                                          uint64_t first, uint32_t m) {
    const uint32_t tid = threadIdx.x;
    uint32_t kind[kItems], rank[kItems];
    for (uint32_t k = tid; k < 3 * m; k += kClosureThreads) {
        t.a[k] = __ldg(a + 3 * first + k);
        t.b[k] = __ldg(b + 3 * first + k);
    }
    if (tid < kKinds) t.count[tid] = 0u;
    if (tid == 0) t.next = 0u;
    __syncthreads();
    if (m <= kUnsorted) return false;
#pragma unroll
    for (int j = 0; j < kItems; ++j) {
        const uint32_t q = tid + j * kClosureThreads;
        if (q < m) {
            kind[j] = closure_kind(lobes[first + q].closure_id, lobes[first + q].params[0]);
            rank[j] = atomicAdd(&t.count[kind[j]], 1u);
        }
    }
    if (tid == 0) t.kind0 = kind[0];
    __syncthreads();
    if (t.count[t.kind0] == m) return false;
    if (tid < kKinds) {  // exclusive prefix over the kinds (the first warp)
        const uint32_t c = t.count[tid];
        uint32_t incl = c;
#pragma unroll
        for (uint32_t o = 1; o < kKinds; o <<= 1) {
            const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, incl, o);
            if (tid >= o) incl += v;
        }
        t.start[tid] = incl - c;
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kItems; ++j) {
        const uint32_t q = tid + j * kClosureThreads;
        if (q < m) t.order[t.start[kind[j]] + rank[j]] = (uint16_t)q;
    }
    __syncthreads();
    return true;
}

__device__ __forceinline__ void put3(float* p, f3 v) {
    p[0] = v.x;
    p[1] = v.y;
    p[2] = v.z;
}

template <int kItems>
__global__ void __launch_bounds__(kClosureThreads, kClosureBlocks) k_closure_eval(const kz_lobe* __restrict__ lobes,
                                                                  const float* __restrict__ wi,
                                                                  const float* __restrict__ wo, uint64_t n, int conv,
                                                                  float* f, float* pdf) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    ClosureTile<kItems>& t = *reinterpret_cast<ClosureTile<kItems>*>(smem_raw);
    const uint64_t first = (uint64_t)blockIdx.x * t.kN;
    const uint32_t m = (uint32_t)min((uint64_t)t.kN, n - first);
    if (!load_tile(t, lobes, wi, wo, first, m)) {
#pragma unroll 1
        for (uint32_t q = threadIdx.x; q < m; q += kClosureThreads) {
            const uint64_t i = first + q;
            const kz_lobe& l = lobes[i];
            const f3 a = ld3(t.a + 3 * q), b = ld3(t.b + 3 * q);
            const LobeEval e = conv == KZ_CONVENTION_REFERENCE ? lobe_eval_reference<true>(l, a, b) : lobe_eval(l, a, b);
            put3(f + 3 * i, e.f);
            pdf[i] = e.pdf;
        }
        return;
    }
    for (uint32_t k; next_queries(t, m, k);) {
        if (k >= m) continue;
        const uint32_t q = t.order[k];
        const kz_lobe& l = lobes[first + q];
        const f3 a = ld3(t.a + 3 * q), b = ld3(t.b + 3 * q);
        const LobeEval e = conv == KZ_CONVENTION_REFERENCE ? lobe_eval_reference<true>(l, a, b) : lobe_eval(l, a, b);
        put3(t.a + 3 * q, e.f);
        t.pdf[q] = e.pdf;
    }
    __syncthreads();
    for (uint32_t k = threadIdx.x; k < 3 * m; k += kClosureThreads) f[3 * first + k] = t.a[k];
    for (uint32_t k = threadIdx.x; k < m; k += kClosureThreads) pdf[first + k] = t.pdf[k];
}

template <int kItems>
__global__ void __launch_bounds__(kClosureThreads, kClosureBlocks) k_closure_sample(const kz_lobe* __restrict__ lobes,
                                                                    const float* __restrict__ wi,
                                                                    const float* __restrict__ u, uint64_t n, float* wo,
                                                                    float* weight, float* pdf, uint8_t* flags) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    ClosureTile<kItems>& t = *reinterpret_cast<ClosureTile<kItems>*>(smem_raw);
    const uint64_t first = (uint64_t)blockIdx.x * t.kN;
    const uint32_t m = (uint32_t)min((uint64_t)t.kN, n - first);
    if (!load_tile(t, lobes, wi, u, first, m)) {
#pragma unroll 1
        for (uint32_t q = threadIdx.x; q < m; q += kClosureThreads) {
            const uint64_t i = first + q;
            const kz_lobe& l = lobes[i];
            const LobeSample s = lobe_sample(l, ld3(t.a + 3 * q), t.b[3 * q], t.b[3 * q + 1], t.b[3 * q + 2]);
            put3(wo + 3 * i, s.wo);
            put3(weight + 3 * i, s.weight);
            pdf[i] = s.pdf;
            flags[i] = (uint8_t)((s.valid ? 1 : 0) | (s.delta ? 2 : 0));
        }
        return;
    }
    for (uint32_t k; next_queries(t, m, k);) {
        if (k >= m) continue;
        const uint32_t q = t.order[k];
        const kz_lobe& l = lobes[first + q];
        const LobeSample s = lobe_sample(l, ld3(t.a + 3 * q), t.b[3 * q], t.b[3 * q + 1], t.b[3 * q + 2]);
        put3(t.a + 3 * q, s.wo);
        put3(t.b + 3 * q, s.weight);
        t.pdf[q] = s.pdf;
        t.flags[q] = (uint8_t)((s.valid ? 1 : 0) | (s.delta ? 2 : 0));
    }
    __syncthreads();
    for (uint32_t k = threadIdx.x; k < 3 * m; k += kClosureThreads) {
        wo[3 * first + k] = t.a[k];
        weight[3 * first + k] = t.b[k];
    }
    for (uint32_t k = threadIdx.x; k < m; k += kClosureThreads) {
        pdf[first + k] = t.pdf[k];
        flags[first + k] = t.flags[k];
    }
}

// Queries per thread, 1, 2 or 4: as few as keep all tiles of a batch resident at
// once (kClosureBlocks an SM), four above that. A larger tile holds more of each
// kind, but leaves fewer warps to wait for their lobes, which is all that a batch
// of one kind does. Evaluation and sampling at 1 / 2 / 4 (and ungrouped), us a pair
// of calls: 21 kinds, 65,536 queries 169 / 150 / 139 (408), 100,000 170 / 170 / 156
// (541), 200,000 287 / 195 / 191 (1,027), 262,144 342 / 212 / 200 (1,265), 600,000
// 858 / 514 / 272 (3,161); one kind (GGX glass) 100,000 55 / 68 / 94 (59), 262,144
// 77 / 83 / 102 (80), 600,000 120 / 125 / 127 (121); five principled kinds 100,000
// 51 / 53 / 56 (62), 600,000 100 / 80 / 73 (131). (Lines at 2^16 and 2^18 queries
// made batches of one kind up to 1.3 times as slow as ungrouped.)
int items_per_thread(uint64_t n) {
    static const uint64_t wave = [] {
        int dev = 0, sms = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        return (uint64_t)(sms > 0 ? sms : 1) * kClosureBlocks * kClosureThreads;
    }();
    return n <= wave ? 1 : n <= 2 * wave ? 2 : 4;
}

template <int kItems>
void run_eval(const kz_lobe* lobes, const float* wi, const float* wo, uint64_t n, int conv, float* f, float* pdf,
              cudaStream_t st) {
    using T = ClosureTile<kItems>;
    k_closure_eval<kItems><<<grid_for(n, T::kN), kClosureThreads, sizeof(T), st>>>(lobes, wi, wo, n, conv, f, pdf);
}
template <int kItems>
void run_sample(const kz_lobe* lobes, const float* wi, const float* u, uint64_t n, float* wo, float* weight,
                float* pdf, uint8_t* flags, cudaStream_t st) {
    using T = ClosureTile<kItems>;
    k_closure_sample<kItems><<<grid_for(n, T::kN), kClosureThreads, sizeof(T), st>>>(lobes, wi, u, n, wo, weight, pdf,
                                                                                   flags);
}
static_assert(sizeof(ClosureTile<4>) <= 48 * 1024, "a tile fits the default shared memory limit");

}  // namespace

void launch_closure_eval(const kz_lobe* lobes, const float* wi, const float* wo, uint64_t n, int convention,
                         float* f, float* pdf, cudaStream_t st) {
    if (!n) return;
    const int k = items_per_thread(n);
    (k == 1 ? run_eval<1> : k == 2 ? run_eval<2> : run_eval<4>)(lobes, wi, wo, n, convention, f, pdf, st);
}
void launch_closure_sample(const kz_lobe* lobes, const float* wi, const float* u, uint64_t n, float* wo,
                           float* weight, float* pdf, uint8_t* flags, cudaStream_t st) {
    if (!n) return;
    const int k = items_per_thread(n);
    (k == 1 ? run_sample<1> : k == 2 ? run_sample<2> : run_sample<4>)(lobes, wi, u, n, wo, weight, pdf, flags, st);
}

}  // namespace kz
