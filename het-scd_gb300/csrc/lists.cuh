// Id lists by class: the ids 0..n-1 that belong to each of K classes, ascending,
// all K lists one after the other in one array.
//
// The engine sorts rows, improves vertices and counts triangles by length class,
// so every graph needs about thirty such lists. Built one class at a time (a scan
// of the class's flags over all ids, then a scatter) they were most of a small
// run's launches, buffers and host reads (a scan, a scatter, a copied count and
// two buffers for each). Here one pass counts all classes of a tile of ids by
// ballots, one scan over the (class, tile) counts places them, and one pass
// writes them: three launches for all the lists of a call, one for up to
// LISTS_ONE ids, and one host read of the K+1 bounds.
#pragma once

#include "primitives.cuh"

namespace scd {

constexpr int LISTS_WARPS = 8, LISTS_STEPS = 8;
constexpr uint32_t LISTS_TILE = LISTS_WARPS * 32 * LISTS_STEPS;
constexpr int LISTS_ONE_WARPS = 32, LISTS_ONE_STEPS = 16;
constexpr uint32_t LISTS_ONE = LISTS_ONE_WARPS * 32 * LISTS_ONE_STEPS;

// The class masks of a warp's steps x 32 (steps <= STEPS) consecutive ids from `first` on (bit
// k: the id is in class k), and in lane k < K the number of the warp's ids in class k.
template <int K, int STEPS, typename F>
__device__ __forceinline__ uint32_t warp_masks(F f, uint32_t n, uint32_t first, uint32_t steps, uint32_t (&m)[STEPS]) {
    static_assert(K <= 32, "a lane per class");
    const uint32_t lane = threadIdx.x & 31;
    uint32_t cnt = 0;
#pragma unroll
    for (int i = 0; i < STEPS; i++) {
        const uint32_t id = first + i * 32 + lane;
        m[i] = (uint32_t)i < steps && id < n ? f[id] : 0u;
    }
#pragma unroll
    for (int i = 0; i < STEPS; i++) {
        if ((uint32_t)i >= steps) break;
#pragma unroll
        for (int k = 0; k < K; k++) {
            const uint32_t c = __popc(__ballot_sync(FULL, (m[i] >> k) & 1u));
            if (lane == (uint32_t)k) cnt += c;
        }
    }
    return cnt;
}

// writes the warp's ids; lane k holds the list position of the warp's first id of class k
template <int K, int STEPS>
__device__ __forceinline__ void warp_scatter(uint32_t first, uint32_t steps, const uint32_t (&m)[STEPS], uint32_t pos,
                                             uint32_t *lists) {
    const uint32_t lane = threadIdx.x & 31;
    const unsigned lt = lanemask_lt();
#pragma unroll
    for (int i = 0; i < STEPS; i++) {
        if ((uint32_t)i >= steps) break;
#pragma unroll
        for (int k = 0; k < K; k++) {
            const unsigned b = __ballot_sync(FULL, (m[i] >> k) & 1u);
            const uint32_t p = __shfl_sync(FULL, pos, k);
            if ((m[i] >> k) & 1u) lists[p + __popc(b & lt)] = first + i * 32 + lane;
            if (lane == (uint32_t)k) pos += __popc(b);
        }
    }
}

template <int K, typename F>
__global__ void __launch_bounds__(LISTS_WARPS * 32)
k_lists_count(F f, uint32_t n, uint32_t tiles, uint32_t *hist) {
    __shared__ uint32_t sm[LISTS_WARPS][K];
    const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    uint32_t m[LISTS_STEPS];
    const uint32_t cnt = warp_masks<K>(f, n, blockIdx.x * LISTS_TILE + w * 32 * LISTS_STEPS, LISTS_STEPS, m);
    if (lane < K) sm[w][lane] = cnt;
    __syncthreads();
    if (threadIdx.x < K) {
        uint32_t t = 0;
        for (int j = 0; j < LISTS_WARPS; j++) t += sm[j][threadIdx.x];
        hist[(size_t)threadIdx.x * tiles + blockIdx.x] = t;
    }
}

template <int K, typename F>
__global__ void __launch_bounds__(LISTS_WARPS * 32)
k_lists_scatter(F f, uint32_t n, uint32_t tiles, const uint32_t *__restrict__ at, uint32_t *lists, uint32_t *bounds) {
    __shared__ uint32_t sm[LISTS_WARPS][K];
    const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint32_t first = blockIdx.x * LISTS_TILE + w * 32 * LISTS_STEPS;
    uint32_t m[LISTS_STEPS];
    const uint32_t cnt = warp_masks<K>(f, n, first, LISTS_STEPS, m);
    if (lane < K) sm[w][lane] = cnt;
    __syncthreads();
    if (threadIdx.x < K) {
        uint32_t run = at[(size_t)threadIdx.x * tiles + blockIdx.x];
        for (int j = 0; j < LISTS_WARPS; j++) {
            const uint32_t t = sm[j][threadIdx.x];
            sm[j][threadIdx.x] = run;
            run += t;
        }
    }
    if (blockIdx.x == 0 && threadIdx.x <= K) bounds[threadIdx.x] = at[(size_t)threadIdx.x * tiles];
    __syncthreads();
    warp_scatter<K>(first, LISTS_STEPS, m, lane < K ? sm[w][lane] : 0u, lists);
}

// up to LISTS_ONE ids: counts and lists in one CTA
template <int K, typename F>
__global__ void __launch_bounds__(LISTS_ONE_WARPS * 32)
k_lists_one(F f, uint32_t n, uint32_t *lists, uint32_t *bounds) {
    __shared__ uint32_t sm[LISTS_ONE_WARPS][K], base[K + 1];
    const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint32_t steps = (n + LISTS_ONE_WARPS * 32 - 1) / (LISTS_ONE_WARPS * 32), first = w * 32 * steps;
    uint32_t m[LISTS_ONE_STEPS];
    const uint32_t cnt = warp_masks<K>(f, n, first, steps, m);
    if (lane < K) sm[w][lane] = cnt;
    __syncthreads();
    if (threadIdx.x < K) {
        uint32_t run = 0;
        for (int j = 0; j < LISTS_ONE_WARPS; j++) {
            const uint32_t t = sm[j][threadIdx.x];
            sm[j][threadIdx.x] = run;
            run += t;
        }
        base[threadIdx.x] = run;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t run = 0;
        for (int k = 0; k <= K; k++) {
            const uint32_t t = k < K ? base[k] : 0u;
            base[k] = run;
            bounds[k] = run;
            run += t;
        }
    }
    __syncthreads();
    warp_scatter<K>(first, steps, m, lane < K ? sm[w][lane] + base[lane] : 0u, lists);
}

// The K lists into `lists` (room for every membership), list k at
// [bounds[k], bounds[k+1]) (bounds: K+1 device words).  f[id] is the id's class mask.
template <int K, typename F>
void build_lists(F f, uint32_t n, uint32_t *lists, uint32_t *bounds, cudaStream_t s) {
    if (n <= LISTS_ONE) {
        k_lists_one<K, F><<<1, LISTS_ONE_WARPS * 32, 0, s>>>(f, n, lists, bounds);
        CK_LAUNCH("k_lists_one");
        return;
    }
    const uint32_t tiles = (n + LISTS_TILE - 1) / LISTS_TILE;
    DevBuf<uint32_t> hist((size_t)K * tiles + 1, s);
    k_lists_count<K, F><<<tiles, LISTS_WARPS * 32, 0, s>>>(f, n, tiles, hist.get());
    CK_LAUNCH("k_lists_count");
    scan_exclusive<uint32_t>((const uint32_t *)hist.get(), hist.get(), (size_t)K * tiles, s);
    k_lists_scatter<K, F><<<tiles, LISTS_WARPS * 32, 0, s>>>(f, n, tiles, hist.get(), lists, bounds);
    CK_LAUNCH("k_lists_scatter");
}

}  // namespace scd
