// Device-wide building blocks written for this engine (no CUB/moderngpu):
// exclusive scan, stable LSD radix sort of 32/64-bit keys with optional
// 32-bit payloads, max-reduce, and stream-ordered temporary buffers.
//
// These replace the moderngpu primitives the reference GPU path calls
// (Scan, SegSortKeysFromIndices, ReduceByKey, Reduce; src/cuda.cu:205-345).
#pragma once

#include <mutex>
#include <utility>

#include "common.cuh"

namespace scd {

// ---------------------------------------------------------------------------
// stream-ordered temporary device buffers

// Blocks of up to 1 MB that a context keeps between its temporaries instead of returning each to
// the device's pool: a cudaMallocAsync and its free are 1.8 us of host time, and a call on a
// small graph, bound by the host, makes about ninety of them. Sizes are powers of two; at most
// 64 blocks of a size and 32 MB together are kept, the rest and (at the context's end) all of
// them go back. A block is only handed out again for work on the stream it was used on, later in
// that stream, as cudaFreeAsync and cudaMallocAsync on one stream would. The calls of a resident
// set do not use it (their temporaries come from the pool). Locked: a block may go back from
// another thread than the one that takes the next.
class BlockCache {
public:
    static constexpr int LOW = 9, HIGH = 20, SIZES = HIGH - LOW + 1, SLOTS = 64;
    static constexpr size_t KEEP = 32u << 20;
    cudaStream_t stream = nullptr;   // of the context

    static int size_of(size_t bytes) {   // SIZES: too large to keep
        int k = 0;
        while (k < SIZES && bytes > ((size_t)1 << (LOW + k))) k++;
        return k;
    }
    void *get(int k) {
        {
            std::lock_guard<std::mutex> hold(lock_);
            if (n_[k]) {
                kept_ -= (size_t)1 << (LOW + k);
                return block_[k][--n_[k]];
            }
        }
        void *p = nullptr;
        CK(cudaMallocAsync(&p, (size_t)1 << (LOW + k), stream));
        return p;
    }
    void put(void *p, int k) {
        {
            std::lock_guard<std::mutex> hold(lock_);
            if (n_[k] < SLOTS && kept_ + ((size_t)1 << (LOW + k)) <= KEEP) {
                kept_ += (size_t)1 << (LOW + k);
                block_[k][n_[k]++] = p;
                return;
            }
        }
        cudaFreeAsync(p, stream);
    }
    void give_back() {
        std::lock_guard<std::mutex> hold(lock_);
        for (int k = 0; k < SIZES; k++)
            while (n_[k]) cudaFreeAsync(block_[k][--n_[k]], stream);
        kept_ = 0;
    }
    // the cache of the context whose call this thread is in
    static BlockCache *&current() {
        static thread_local BlockCache *c = nullptr;
        return c;
    }

private:
    std::mutex lock_;
    void *block_[SIZES][SLOTS];
    int n_[SIZES] = {};
    size_t kept_ = 0;
};

template <typename T>
struct DevBuf {
    T *p = nullptr;
    size_t n = 0;
    cudaStream_t s = nullptr;
    BlockCache *cache = nullptr;   // the block came from it (size class k), else from the device's pool
    int k = 0;
    DevBuf() = default;
    DevBuf(size_t count, cudaStream_t stream) { alloc(count, stream); }
    void alloc(size_t count, cudaStream_t stream) {
        release();
        s = stream;
        n = count;
        if (!count) return;
        BlockCache *c = BlockCache::current();
        k = BlockCache::size_of(count * sizeof(T));
        if (c && c->stream == stream && k < BlockCache::SIZES) {
            p = (T *)c->get(k);
            cache = c;
        } else {
            CK(cudaMallocAsync((void **)&p, count * sizeof(T), stream));
        }
    }
    void release() {
        if (p && cache) cache->put(p, k);
        else if (p) cudaFreeAsync(p, s);
        p = nullptr;
        cache = nullptr;
        n = 0;
    }
    ~DevBuf() { release(); }
    DevBuf(const DevBuf &) = delete;
    DevBuf &operator=(const DevBuf &) = delete;
    DevBuf(DevBuf &&o) noexcept { *this = std::move(o); }
    DevBuf &operator=(DevBuf &&o) noexcept {
        release();
        p = o.p; n = o.n; s = o.s; cache = o.cache; k = o.k;
        o.p = nullptr; o.cache = nullptr; o.n = 0;
        return *this;
    }
    T *get() const { return p; }
};

// ---------------------------------------------------------------------------
// exclusive scan: out[0..n] with out[n] = total (n+1 outputs)
//
// Most scans here are short (a run makes about a hundred, most of them over the
// vertices or a list of them), so what bounds one is its launches, not its
// bytes: up to SCAN_ONE outputs a single CTA does it in one launch; above, two
// launches (every CTA's sum, then every CTA adds up the sums before its own and
// scans its range), which also reads the input twice instead of writing the
// output twice.

constexpr int SCAN_THREADS = 256;
constexpr int SCAN_ITEMS = 8;
constexpr int SCAN_TILE = SCAN_THREADS * SCAN_ITEMS;
constexpr int SCAN_ONE_THREADS = 1024;
constexpr int SCAN_ONE_ITEMS = 16;
constexpr size_t SCAN_ONE = (size_t)SCAN_ONE_THREADS * SCAN_ONE_ITEMS;
constexpr size_t SCAN_MAX_CTAS = 152 * 8;   // each reads the sums of the ones before it

template <int THREADS, typename T>
__device__ __forceinline__ T block_exclusive_scan(T v, T *total, T *smem_warp /*[THREADS / 32 + 1]*/) {
    constexpr int WARPS = THREADS / 32;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    T inc = warp_inclusive_scan(v);
    if (lane == 31) smem_warp[warp] = inc;
    __syncthreads();
    if (warp == 0) {
        T w = lane < WARPS ? smem_warp[lane] : T(0);
        T wi = warp_inclusive_scan(w);
        if (lane < WARPS) smem_warp[lane] = wi - w;
        if (lane == WARPS - 1) smem_warp[WARPS] = wi;
    }
    __syncthreads();
    T res = smem_warp[warp] + inc - v;
    *total = smem_warp[WARPS];
    __syncthreads();
    return res;
}

// out[base .. base + THREADS * ITEMS) of the exclusive scan that starts at `run`; returns the tile's total
template <int THREADS, int ITEMS, typename T, typename In>
__device__ __forceinline__ T scan_tile(In in, size_t n, size_t base, T run, T *out, T *sw) {
    const size_t first = base + (size_t)threadIdx.x * ITEMS;
    T v[ITEMS];
    T sum = 0;
#pragma unroll
    for (int i = 0; i < ITEMS; i++) {
        v[i] = first + i < n ? T(in[first + i]) : T(0);
        sum += v[i];
    }
    T total;
    run += block_exclusive_scan<THREADS>(sum, &total, sw);
#pragma unroll
    for (int i = 0; i < ITEMS; i++) {
        if (first + i <= n) out[first + i] = run;
        run += v[i];
    }
    return total;
}

template <typename T, typename In>
__global__ void __launch_bounds__(SCAN_THREADS) k_scan_tile(In in, size_t n, T *out) {
    __shared__ T sw[SCAN_THREADS / 32 + 1];
    scan_tile<SCAN_THREADS, SCAN_ITEMS>(in, n, 0, T(0), out, sw);
}

template <typename T, typename In>
__global__ void __launch_bounds__(SCAN_ONE_THREADS) k_scan_one(In in, size_t n, T *out) {
    __shared__ T sw[SCAN_ONE_THREADS / 32 + 1];
    scan_tile<SCAN_ONE_THREADS, SCAN_ONE_ITEMS>(in, n, 0, T(0), out, sw);
}

// sums[b] = sum of CTA b's range of per_cta tiles
template <typename T, typename In>
__global__ void __launch_bounds__(SCAN_THREADS) k_scan_sums(In in, size_t n, uint32_t per_cta, T *sums) {
    __shared__ T sw[SCAN_THREADS / 32];
    const size_t lo = (size_t)blockIdx.x * per_cta * SCAN_TILE;
    const size_t hi = min(n, lo + (size_t)per_cta * SCAN_TILE);
    T sum = 0;
#pragma unroll 4
    for (size_t i = lo + threadIdx.x; i < hi; i += SCAN_THREADS) sum += T(in[i]);
    sum = warp_sum(sum);
    if ((threadIdx.x & 31) == 0) sw[threadIdx.x >> 5] = sum;
    __syncthreads();
    if (threadIdx.x == 0) {
        T t = 0;
        for (int w = 0; w < SCAN_THREADS / 32; w++) t += sw[w];
        sums[blockIdx.x] = t;
    }
}

template <typename T, typename In>
__global__ void __launch_bounds__(SCAN_THREADS) k_scan_out(In in, size_t n, uint32_t per_cta, const T *sums, T *out) {
    __shared__ T sw[SCAN_THREADS / 32 + 1];
    T before = 0, run;
    for (uint32_t b = threadIdx.x; b < blockIdx.x; b += SCAN_THREADS) before += sums[b];
    block_exclusive_scan<SCAN_THREADS>(before, &run, sw);   // run: the sums of all CTAs before this one
    for (uint32_t k = 0; k < per_cta; k++) {
        const size_t base = ((size_t)blockIdx.x * per_cta + k) * SCAN_TILE;
        if (base > n) break;
        run += scan_tile<SCAN_THREADS, SCAN_ITEMS>(in, n, base, run, out, sw);
    }
}

// in may be a pointer or any functor-like indexable; out must hold n+1 entries
// (out == in is allowed: every CTA reads its range before it writes it).
template <typename T, typename In>
void scan_exclusive(In in, T *out, size_t n, cudaStream_t s) {
    if (n + 1 <= (size_t)SCAN_TILE) {
        k_scan_tile<T, In><<<1, SCAN_THREADS, 0, s>>>(in, n, out);
        CK_LAUNCH("k_scan_tile");
        return;
    }
    if (n + 1 <= SCAN_ONE) {
        k_scan_one<T, In><<<1, SCAN_ONE_THREADS, 0, s>>>(in, n, out);
        CK_LAUNCH("k_scan_one");
        return;
    }
    const size_t tiles = (n + 1 + SCAN_TILE - 1) / SCAN_TILE;
    const uint32_t per_cta = (uint32_t)((tiles + SCAN_MAX_CTAS - 1) / SCAN_MAX_CTAS);
    const unsigned ctas = (unsigned)((tiles + per_cta - 1) / per_cta);
    DevBuf<T> sums(ctas, s);
    k_scan_sums<T, In><<<ctas, SCAN_THREADS, 0, s>>>(in, n, per_cta, sums.get());
    CK_LAUNCH("k_scan_sums");
    k_scan_out<T, In><<<ctas, SCAN_THREADS, 0, s>>>(in, n, per_cta, sums.get(), out);
    CK_LAUNCH("k_scan_out");
}

// ---------------------------------------------------------------------------
// reductions

template <typename T>
__global__ void k_reduce_max(const T *in, size_t n, T *out) {
    T m = 0;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        m = in[i] > m ? in[i] : m;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        T u = __shfl_xor_sync(FULL, m, o);
        m = u > m ? u : m;
    }
    if ((threadIdx.x & 31) == 0) atomicMax(out, m);
}

// ---------------------------------------------------------------------------
// stable LSD radix sort, 8-bit digits.
//
// A tile is RS_WARPS*32*RS_ITEMS keys; warp w of a tile owns the contiguous
// run [w*32*RS_ITEMS, (w+1)*32*RS_ITEMS) and walks it 32 keys at a time, so
// (step, lane) order equals input order and __match_any_sync ranking keeps the
// sort stable.
//
// What bounds a sort is its launches for all but the largest graphs, so there are
// three forms by size:
//   one tile         one CTA makes every pass in shared memory, one launch;
//   <= RS_FUSED      one launch a pass: every CTA adds up the digit counts of the
//     tiles          tiles before its own (at most RS_FUSED reads a thread), and
//                    counts the next pass's digits by output tile as it writes;
//   more             per pass the tiles' digit counts, a scan of them, and the
//                    move: the counts before a tile are too many to add up again
//                    in every CTA.

constexpr int RS_WARPS = 8;
constexpr int RS_THREADS = RS_WARPS * 32;
constexpr int RS_ITEMS = 8;
constexpr int RS_TILE = RS_THREADS * RS_ITEMS;
constexpr size_t RS_FUSED = 128;   // tiles
static_assert(RS_THREADS == 256, "one thread per digit");

// Digit counts of the tile at blockIdx.x: to hist[digit * tiles + tile] (for the scan)
// or, tile_major, to hist[tile * 256 + digit].
template <typename K>
__global__ void __launch_bounds__(RS_THREADS) k_rs_upsweep(const K *keys, size_t n, int shift,
                                                           unsigned mask, uint32_t *hist,
                                                           size_t tiles, bool tile_major) {
    __shared__ uint32_t cnt[RS_WARPS][256];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int i = threadIdx.x; i < RS_WARPS * 256; i += RS_THREADS) (&cnt[0][0])[i] = 0;
    __syncthreads();
    const size_t base = (size_t)blockIdx.x * RS_TILE + (size_t)warp * 32 * RS_ITEMS;
#pragma unroll 4
    for (int k = 0; k < RS_ITEMS; k++) {
        size_t idx = base + (size_t)k * 32 + lane;
        bool valid = idx < n;
        unsigned d = valid ? (unsigned)(keys[idx] >> shift) & mask : 0u;
        if (valid) atomicAdd(&cnt[warp][d], 1u);
    }
    __syncthreads();
    const int d = threadIdx.x;
    uint32_t s = 0;
#pragma unroll
    for (int w = 0; w < RS_WARPS; w++) s += cnt[w][d];
    hist[tile_major ? (size_t)blockIdx.x * 256 + d : (size_t)d * tiles + blockIdx.x] = s;
}

// The lanes that hold the same digit (below mask + 1, a power of two) as this one, among the
// lanes of `valid`: a vote per bit. (__match_any_sync goes once round per distinct value, and
// the digits of a warp's 32 keys are nearly all distinct.)
__device__ __forceinline__ unsigned same_digit(unsigned d, unsigned mask, unsigned valid) {
    unsigned peers = valid;
#pragma unroll
    for (int b = 0; b < 8; b++) {
        if (!((mask >> b) & 1u)) break;
        const unsigned vote = __ballot_sync(FULL, (d >> b) & 1u);
        peers &= (d >> b) & 1u ? vote : ~vote;
    }
    return peers;
}

// Stable rank of every key of a tile within its digit and warp (rank[k]); cnt[w][d] becomes
// the digit's keys in the warps before w, returns the tile's keys of digit threadIdx.x.
// `count` keys of the tile are valid.  Starts and ends with a barrier's worth of order.
// A warp's keys are `items` (<= RS_ITEMS) rounds of 32 consecutive ones from warp * 32 * items on.
template <int WARPS, typename K>
__device__ __forceinline__ uint32_t rs_rank(const K (&key)[RS_ITEMS], uint32_t count, uint32_t items, int shift,
                                            unsigned mask, uint32_t (&cnt)[WARPS][256], uint32_t (&rank)[RS_ITEMS]) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned lt = lanemask_lt();
    for (int i = threadIdx.x; i < WARPS * 256; i += WARPS * 32) (&cnt[0][0])[i] = 0;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < RS_ITEMS; k++) {
        if ((uint32_t)k >= items) break;
        const bool valid = (uint32_t)(warp * 32 * items + k * 32 + lane) < count;
        const unsigned d = valid ? (unsigned)(key[k] >> shift) & mask : 0u;
        const unsigned peers = same_digit(d, mask, __ballot_sync(FULL, valid));   // (of an invalid lane: unused)
        const int leader = (__ffs(peers) - 1) & 31;
        uint32_t before = 0;
        if (valid && lane == leader) {
            before = cnt[warp][d];
            cnt[warp][d] = before + __popc(peers);
        }
        before = __shfl_sync(FULL, before, leader);
        rank[k] = before + __popc(peers & lt);
        __syncwarp();
    }
    __syncthreads();
    uint32_t total = 0;
    if (WARPS == 8 || threadIdx.x < 256) {
#pragma unroll
        for (int w = 0; w < WARPS; w++) {
            const uint32_t c = cnt[w][threadIdx.x];
            cnt[w][threadIdx.x] = total;
            total += c;
        }
    }
    return total;
}

// exclusive sum over the first 256 threads (sw: RS_WARPS words; v is 0 in any others)
__device__ __forceinline__ uint32_t rs_scan256(uint32_t v, uint32_t *sw) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t inc = warp_inclusive_scan(v);
    if (lane == 31 && warp < RS_WARPS) sw[warp] = inc;
    __syncthreads();
    uint32_t off = 0;
    for (int w = 0; w < RS_WARPS && w < warp; w++) off += sw[w];
    __syncthreads();
    return off + inc - v;
}

// Ranks every key of the tile stably by digit, reorders the tile in shared
// memory, then writes it out in tile order so that keys of one digit leave as
// one contiguous run (coalesced) at the digit's global offset.
// FUSED: `hist` holds the tile-major digit counts of this pass (the offsets are
// summed up here) and next_hist, if not null, receives those of the next pass;
// else `hist` holds the scanned digit-major offsets.
template <typename K, bool HAS_VALS, bool FUSED>
__global__ void __launch_bounds__(RS_THREADS, 4) k_rs_downsweep(const K *keys_in, const uint32_t *vals_in,
                                                                K *keys_out, uint32_t *vals_out,
                                                                size_t n, int shift, unsigned mask,
                                                                const uint32_t *hist, size_t tiles,
                                                                uint32_t *next_hist, int next_shift,
                                                                unsigned next_mask) {
    __shared__ uint32_t cnt[RS_WARPS][256];
    __shared__ uint32_t tile_start[256];   // first tile position of each digit
    __shared__ uint32_t glob[256];         // global position of that first key
    __shared__ uint32_t sw[RS_WARPS];
    __shared__ K skeys[RS_TILE];
    __shared__ uint32_t svals[HAS_VALS ? RS_TILE : 1];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const size_t tile_base = (size_t)blockIdx.x * RS_TILE;
    const uint32_t count = (uint32_t)min((size_t)RS_TILE, n - tile_base);
    const uint32_t first = warp * 32 * RS_ITEMS + lane;
    K key[RS_ITEMS];
    uint32_t val[RS_ITEMS], rank[RS_ITEMS];
#pragma unroll
    for (int k = 0; k < RS_ITEMS; k++) {
        const bool valid = first + k * 32 < count;
        key[k] = valid ? keys_in[tile_base + first + k * 32] : K(0);
        if (HAS_VALS) val[k] = valid ? vals_in[tile_base + first + k * 32] : 0u;
    }
    if constexpr (FUSED) {
        uint32_t before = 0, all = 0;
#pragma unroll 8
        for (uint32_t t = 0; t < (uint32_t)tiles; t++) {
            const uint32_t h = hist[t * 256 + threadIdx.x];
            if (t < blockIdx.x) before += h;
            all += h;
        }
        glob[threadIdx.x] = rs_scan256(all, sw) + before;
    } else {
        glob[threadIdx.x] = hist[(size_t)threadIdx.x * tiles + blockIdx.x];
    }
    const uint32_t total = rs_rank<RS_WARPS>(key, count, RS_ITEMS, shift, mask, cnt, rank);
    tile_start[threadIdx.x] = rs_scan256(total, sw);
    __syncthreads();
#pragma unroll
    for (int k = 0; k < RS_ITEMS; k++) {
        if (first + k * 32 < count) {
            const unsigned d = (unsigned)(key[k] >> shift) & mask;
            const uint32_t p = tile_start[d] + cnt[warp][d] + rank[k];
            skeys[p] = key[k];
            if (HAS_VALS) svals[p] = val[k];
        }
    }
    __syncthreads();
    for (uint32_t i0 = warp * 32; i0 < count; i0 += RS_THREADS) {
        const uint32_t i = i0 + lane;
        const bool valid = i < count;
        const K kk = valid ? skeys[i] : K(0);
        uint32_t dst = 0;
        if (valid) {
            const unsigned d = (unsigned)(kk >> shift) & mask;
            dst = glob[d] + (i - tile_start[d]);
            keys_out[dst] = kk;
            if (HAS_VALS) vals_out[dst] = svals[i];
        }
        if (FUSED && next_hist) {   // equal keys leave together: one atomic per counter and warp
            const uint32_t at = valid ? (dst / RS_TILE) * 256 + ((unsigned)(kk >> next_shift) & next_mask) : INVALID;
            const unsigned peers = __match_any_sync(FULL, at);
            if (valid && lane == __ffs(peers) - 1) atomicAdd(next_hist + at, (uint32_t)__popc(peers));
        }
    }
}

// up to one tile: every pass in one CTA
template <typename K, bool HAS_VALS>
__global__ void __launch_bounds__(RS_THREADS) k_rs_one(K *keys, uint32_t *vals, uint32_t n, int begin_bit, int end_bit) {
    __shared__ uint32_t cnt[RS_WARPS][256];
    __shared__ uint32_t tile_start[256], sw[RS_WARPS];
    __shared__ K skeys[RS_TILE];
    __shared__ uint32_t svals[HAS_VALS ? RS_TILE : 1];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t first = warp * 32 * RS_ITEMS + lane;
    K key[RS_ITEMS];
    uint32_t val[RS_ITEMS], rank[RS_ITEMS];
#pragma unroll
    for (int k = 0; k < RS_ITEMS; k++) {
        const bool valid = first + k * 32 < n;
        key[k] = valid ? keys[first + k * 32] : K(0);
        val[k] = HAS_VALS && valid ? vals[first + k * 32] : 0u;
    }
    for (int b = begin_bit; b < end_bit; b += 8) {
        const unsigned mask = (1u << (end_bit - b < 8 ? end_bit - b : 8)) - 1u;
        const uint32_t total = rs_rank<RS_WARPS>(key, n, RS_ITEMS, b, mask, cnt, rank);
        tile_start[threadIdx.x] = rs_scan256(total, sw);
        __syncthreads();
#pragma unroll
        for (int k = 0; k < RS_ITEMS; k++)
            if (first + k * 32 < n) {
                const unsigned d = (unsigned)(key[k] >> b) & mask;
                const uint32_t p = tile_start[d] + cnt[warp][d] + rank[k];
                skeys[p] = key[k];
                if (HAS_VALS) svals[p] = val[k];
            }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < RS_ITEMS; k++)
            if (first + k * 32 < n) {
                key[k] = skeys[first + k * 32];
                if (HAS_VALS) val[k] = svals[first + k * 32];
            }
        __syncthreads();
    }
#pragma unroll
    for (int k = 0; k < RS_ITEMS; k++)
        if (first + k * 32 < n) {
            keys[first + k * 32] = key[k];
            if (HAS_VALS) vals[first + k * 32] = val[k];
        }
}

template <typename K, bool HAS_VALS>
void radix_sort_impl(K *keys, uint32_t *vals, size_t n, int begin_bit, int end_bit, cudaStream_t s) {
    if (n <= (size_t)RS_TILE) {
        k_rs_one<K, HAS_VALS><<<1, RS_THREADS, 0, s>>>(keys, vals, (uint32_t)n, begin_bit, end_bit);
        CK_LAUNCH("k_rs_one");
        return;
    }
    const size_t tiles = (n + RS_TILE - 1) / RS_TILE;
    const int passes = (end_bit - begin_bit + 7) / 8;
    const bool fused = tiles <= RS_FUSED;
    DevBuf<K> kt(n, s);
    DevBuf<uint32_t> vt(HAS_VALS ? n : 0, s);
    DevBuf<uint32_t> hist(fused ? 256 * tiles * passes : 256 * tiles + 1, s);
    K *kin = keys, *kout = kt.get();
    uint32_t *vin = vals, *vout = vt.get(), *h = hist.get();
    if (fused && passes > 1) CK(cudaMemsetAsync(h + 256 * tiles, 0, 4 * 256 * tiles * (passes - 1), s));
    for (int p = 0; p < passes; p++) {
        const int b = begin_bit + 8 * p, nb = b + 8;
        const auto mask_at = [&](int bit) { return (1u << (end_bit - bit < 8 ? end_bit - bit : 8)) - 1u; };
        if (!fused || p == 0) {
            k_rs_upsweep<K><<<(unsigned)tiles, RS_THREADS, 0, s>>>(kin, n, b, mask_at(b), h, tiles, fused);
            CK_LAUNCH("k_rs_upsweep");
        }
        if (fused) {
            const bool more = p + 1 < passes;
            k_rs_downsweep<K, HAS_VALS, true><<<(unsigned)tiles, RS_THREADS, 0, s>>>(
                kin, vin, kout, vout, n, b, mask_at(b), h, tiles, more ? h + 256 * tiles : nullptr, more ? nb : 0,
                more ? mask_at(nb) : 0u);
            h += 256 * tiles;
        } else {
            scan_exclusive<uint32_t, const uint32_t *>(h, h, 256 * tiles, s);
            k_rs_downsweep<K, HAS_VALS, false><<<(unsigned)tiles, RS_THREADS, 0, s>>>(kin, vin, kout, vout, n, b,
                                                                                     mask_at(b), h, tiles, nullptr, 0, 0u);
        }
        CK_LAUNCH("k_rs_downsweep");
        K *tk = kin; kin = kout; kout = tk;
        uint32_t *tv = vin; vin = vout; vout = tv;
    }
    if (passes & 1) {
        CK(cudaMemcpyAsync(keys, kin, n * sizeof(K), cudaMemcpyDeviceToDevice, s));
        if (HAS_VALS) CK(cudaMemcpyAsync(vals, vin, n * sizeof(uint32_t), cudaMemcpyDeviceToDevice, s));
    }
}

// Sorts keys[0..n) (and vals, if non-null) by bits [begin_bit, end_bit).
// n must be < 2^32.  Uses one temporary copy of the arrays.
template <typename K>
void radix_sort(K *keys, uint32_t *vals, size_t n, int begin_bit, int end_bit, cudaStream_t s) {
    if (n < 2 || end_bit <= begin_bit) return;
    if (n >= (size_t(1) << 32)) throw Error(SCD_ERR_LIMIT, "radix_sort: more than 2^32 keys");
    if (vals) radix_sort_impl<K, true>(keys, vals, n, begin_bit, end_bit, s);
    else radix_sort_impl<K, false>(keys, nullptr, n, begin_bit, end_bit, s);
}

}  // namespace scd
