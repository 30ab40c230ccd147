// Row-wise CSR construction for the preprocessing (src/convert.cpp:252-268 and
// 417-455: sort, de-duplicate, write both directions with sorted rows).
//
// Instead of one global sort of 64-bit (row, value) keys, whose every radix
// pass moves every entry, the entries are placed by a counting sort on the row
// (row lengths, offsets, one scatter) and then every row is sorted on its own:
//   rows of length <= 512     a warp, bitonic network in registers and
//                             shuffles (1, 2, 4, 8 or 16 values per lane);
//   513 .. 4096               a CTA, radix sort in shared memory (as many
//                             8-bit passes as the row numbers have bytes);
//   longer rows               a CTA sets a bit per value in a shared bitmap of
//                             the row numbers and reads it back in order.
// With de-duplication a repeated value of a row becomes INVALID (anywhere in the
// row) and the number of distinct values of the row is written out; the callers
// skip the holes.
#include "engine.cuh"
#include "lists.cuh"

namespace scd {

namespace {

constexpr unsigned TPB = 256;
constexpr uint32_t WARP_ROW = 32, MID_ROW = 512, HALF_ROW = 2048, BIG_ROW = 4096;

// sorts G values, one a lane of a group, ascending
template <int G>
__device__ __forceinline__ uint32_t bitonic(uint32_t v, int gl) {
#pragma unroll
    for (int k = 2; k <= G; k <<= 1) {
#pragma unroll
        for (int j = k >> 1; j > 0; j >>= 1) {
            const uint32_t o = __shfl_xor_sync(FULL, v, j);
            const bool asc = (gl & k) == 0, low = (gl & j) == 0;
            v = (low == asc) ? min(v, o) : max(v, o);
        }
    }
    return v;
}

struct RowShared {
    uint32_t beg[TPB / 32][32], meta[TPB / 32][32];   // first entry; length << 5 | lane of the row
};

// rows [first, last) of the warp's table, G lanes a row
template <int G>
__device__ __forceinline__ void sort_group(const RowShared &sh, uint32_t first, uint32_t last, uint32_t r0, uint32_t *vals,
                                           bool dedup, uint32_t *udeg) {
    constexpr uint32_t PER_WARP = 32 / G;
    const int lane = threadIdx.x & 31, gl = lane % G, w = threadIdx.x >> 5;
    const auto entry = [&](uint32_t i0, uint32_t &beg, uint32_t &meta) {
        const uint32_t i = i0 + lane / G;
        beg = i < last ? sh.beg[w][i] : 0u;
        meta = i < last ? sh.meta[w][i] : 0u;
        return (uint32_t)gl < meta >> 5 ? vals[beg + gl] : INVALID;
    };
    uint32_t beg, meta, v = entry(first, beg, meta);
    for (uint32_t i0 = first; i0 < last; i0 += PER_WARP) {
        uint32_t nbeg, nmeta;
        const uint32_t next = entry(i0 + PER_WARP, nbeg, nmeta);   // (of other rows)
        v = bitonic<G>(v, gl);
        const uint32_t prev = __shfl_up_sync(FULL, v, 1, G);
        const bool in = (uint32_t)gl < meta >> 5, keep = in && (!dedup || gl == 0 || v != prev);
        if (in) vals[beg + gl] = keep ? v : INVALID;
        const unsigned kb = __ballot_sync(FULL, keep) >> (lane - gl) & (G == 32 ? FULL : (1u << (G & 31)) - 1u);
        if (udeg && gl == 0 && meta) udeg[r0 + (meta & 31)] = __popc(kb);
        v = next;
        beg = nbeg;
        meta = nmeta;
    }
}

// Every row of length <= 32: a warp takes `rows` consecutive ones, reads their bounds in one
// coalesced step and sorts those of more than 16 entries one at a time, of 9..16 two and of
// up to 8 four at a time, the next ones' entries on their way meanwhile. (Bound by the
// exchange stages: 15 for 32 values whatever the row's length, 10 for 16, 6 for 8. One row
// a warp: Chung-Lu 4M, both sorts, 870 us, 96 planted graphs 850 us; so 357 and 554 us.)
__global__ void __launch_bounds__(TPB)
k_sort_rows_warp(const uint32_t *__restrict__ off, uint32_t nrows, uint32_t rows, uint32_t *vals, bool dedup,
                 uint32_t *udeg) {
    __shared__ RowShared sh;
    const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5, warps = (gridDim.x * blockDim.x) >> 5;
    const unsigned lt = lanemask_lt();
    const uint32_t units = nrows / rows + (nrows % rows != 0);
    for (uint32_t unit = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; unit < units; unit += warps) {
        const uint32_t r0 = unit * rows, r = r0 + lane;
        uint32_t beg = 0, len = 0;
        if (lane < min(rows, nrows - r0)) {
            beg = off[r];
            len = off[r + 1] - beg;
            if (len == 0 && udeg) udeg[r] = 0;
            if (len > WARP_ROW) len = 0;
        }
        const unsigned m32 = __ballot_sync(FULL, len > 16), m16 = __ballot_sync(FULL, len > 8) & ~m32,
                       m8 = __ballot_sync(FULL, len > 0) & ~(m32 | m16);
        const uint32_t n32 = __popc(m32), n16 = n32 + __popc(m16), n8 = n16 + __popc(m8);
        if (len) {
            const uint32_t at = len > 16 ? __popc(m32 & lt) : len > 8 ? n32 + __popc(m16 & lt) : n16 + __popc(m8 & lt);
            sh.beg[w][at] = beg;
            sh.meta[w][at] = len << 5 | lane;
        }
        __syncwarp();
        if (n32) sort_group<32>(sh, 0, n32, r0, vals, dedup, udeg);
        if (n16 > n32) sort_group<16>(sh, n32, n16, r0, vals, dedup, udeg);
        if (n8 > n16) sort_group<8>(sh, n16, n8, r0, vals, dedup, udeg);
        __syncwarp();
    }
}

// rows of one list with 32 < len <= 32 * E: one warp per row, E values per lane
// (value index = lane * E + i), bitonic network in registers
template <int E>
__global__ void __launch_bounds__(TPB)
k_sort_rows_warp_e(const uint32_t *__restrict__ list, uint32_t count, const uint32_t *__restrict__ off, uint32_t *vals,
                   bool dedup, uint32_t *udeg) {
    const int lane = threadIdx.x & 31;
    const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < count; w += warps) {
        const uint32_t r = list[w], beg = off[r], len = off[r + 1] - beg;
        uint32_t v[E];
#pragma unroll
        for (int i = 0; i < E; i++) {
            const uint32_t idx = lane * E + i;
            v[i] = idx < len ? vals[beg + idx] : INVALID;
        }
#pragma unroll
        for (int k = 2; k <= 32 * E; k <<= 1) {
#pragma unroll
            for (int j = k >> 1; j > 0; j >>= 1) {
                if (j >= E) {   // partner in lane ^ (j / E)
#pragma unroll
                    for (int i = 0; i < E; i++) {
                        const int idx = lane * E + i;
                        const uint32_t o = __shfl_xor_sync(FULL, v[i], j / E);
                        const bool asc = (idx & k) == 0, low = (idx & j) == 0;
                        v[i] = (low == asc) ? min(v[i], o) : max(v[i], o);
                    }
                } else {        // partner in this lane: i ^ j
#pragma unroll
                    for (int i = 0; i < E; i++) {
                        const int q = i ^ j;
                        if (q > i) {
                            const bool asc = ((lane * E + i) & k) == 0;
                            const uint32_t x = v[i], y = v[q];
                            if ((x > y) == asc) {
                                v[i] = y;
                                v[q] = x;
                            }
                        }
                    }
                }
            }
        }
        const uint32_t last_prev = __shfl_up_sync(FULL, v[E - 1], 1);
        uint32_t kept = 0;
#pragma unroll
        for (int i = 0; i < E; i++) {
            const uint32_t idx = lane * E + i;
            const uint32_t prev = i ? v[i - 1] : last_prev;
            const bool keep = idx < len && (!dedup || idx == 0 || v[i] != prev);
            if (idx < len) vals[beg + idx] = keep ? v[i] : INVALID;
            kept += keep;
        }
        kept = warp_sum(kept);
        if (udeg && lane == 0) udeg[r] = kept;
    }
}

// rows of one list with len <= 256 * W: one CTA of W warps per row, LSD radix sort of the row
// numbers (`bits` of them) in shared memory. (A bitonic network over 4096 values is 78
// exchange stages, three radix passes are a third of its instructions; the counters of a
// pass are W x 256 whatever the row's length, hence the two sizes. R-MAT scale 22, both
// sorts, rows of 513 to 4096: 2.5 ms by the network, 2.2 with one size of 16 warps and ranks
// by __match_any_sync, 1.66 ms so; 1.54 ms with four times the resident CTAs, handed out as
// rows end.)
template <int W>
__global__ void __launch_bounds__(W * 32, 64 / W)
k_sort_rows_radix(const uint32_t *__restrict__ list, uint32_t count, const uint32_t *__restrict__ off, int bits,
                  uint32_t *vals, bool dedup, uint32_t *udeg) {
    __shared__ uint32_t cnt[W][256];
    __shared__ uint32_t start[256], sw[RS_WARPS], sh[W * 32 * RS_ITEMS], kept_at[W];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int width = (bits + (bits + 7) / 8 - 1) / ((bits + 7) / 8);   // even digits
    for (uint32_t i = blockIdx.x; i < count; i += gridDim.x) {
        const uint32_t r = list[i], beg = off[r], len = off[r + 1] - beg;
        const uint32_t items = (len + (W * 32) - 1) / (W * 32), first = warp * 32 * items + lane;
        uint32_t key[RS_ITEMS], rank[RS_ITEMS];
#pragma unroll
        for (int k = 0; k < RS_ITEMS; k++)
            key[k] = (uint32_t)k < items && first + k * 32 < len ? vals[beg + first + k * 32] : 0u;
        for (int b = 0; b < bits; b += width) {
            const unsigned mask = (1u << min(width, bits - b)) - 1u;
            const uint32_t total = rs_rank<W>(key, len, items, b, mask, cnt, rank);
            const uint32_t at = rs_scan256(total, sw);
            if (threadIdx.x < 256) start[threadIdx.x] = at;
            __syncthreads();
#pragma unroll
            for (int k = 0; k < RS_ITEMS; k++)
                if ((uint32_t)k < items && first + k * 32 < len) {
                    const unsigned d = (key[k] >> b) & mask;
                    sh[start[d] + cnt[warp][d] + rank[k]] = key[k];
                }
            __syncthreads();
            if (b + width < bits) {
#pragma unroll
                for (int k = 0; k < RS_ITEMS; k++)
                    if ((uint32_t)k < items && first + k * 32 < len) key[k] = sh[first + k * 32];
                __syncthreads();
            }
        }
        uint32_t kept = 0;
        for (uint32_t t = threadIdx.x; t < len; t += W * 32) {
            const uint32_t v = sh[t];
            const bool keep = !dedup || t == 0 || v != sh[t - 1];
            vals[beg + t] = keep ? v : INVALID;
            kept += keep;
        }
        kept = warp_sum(kept);
        if (lane == 0) kept_at[warp] = kept;
        __syncthreads();
        if (threadIdx.x == 0 && udeg) {
            uint32_t t = 0;
            for (int w = 0; w < W; w++) t += kept_at[w];
            udeg[r] = t;
        }
        __syncthreads();
    }
}

// Rows of one list with len > 4096, all of distinct values or to be de-duplicated: one CTA per
// row. A row's values, row numbers below nrows, set bits in a shared bitmap; the warps count
// and then list its blocks of 32 words in turn, a word a lane (in turn, because the ids of
// the densest part of a skewed graph are close together). The distinct values come first in
// the row, INVALID after them. Bound by shared memory: a row costs len bit sets and twice
// nrows/32 word reads, whatever its order; the network and radix passes it replaces cost
// log^2 or five rounds of len (R-MAT scale 22, both sorts, rows above 4096: 3.3 -> 0.93 ms).
// Row numbers beyond the bitmap are taken in ranges, each of which reads the row again
// from its copy in `src` (src_off: the rows' places in it; nullptr: one range, from vals).
constexpr int BITMAP_THREADS = 1024;
constexpr uint32_t BITMAP_WORDS = 54 * 1024;   // 216 KB (at most two blocks of 32 a thread)
constexpr uint32_t BITMAP_RANGES = 16;         // beyond: radix sort (every range walks the bitmap once more)
static_assert(BITMAP_WORDS / 32 <= 2 * BITMAP_THREADS, "a scan of two counts a thread");
constexpr size_t bitmap_bytes(uint64_t words) { return (words + words / 32) * 4; }

__global__ void __launch_bounds__(BITMAP_THREADS)
k_sort_rows_bitmap(const uint32_t *__restrict__ list, uint32_t count, const uint32_t *__restrict__ off, uint32_t nrows,
                   uint32_t words, const uint32_t *__restrict__ src, const uint32_t *__restrict__ src_off,
                   uint32_t *vals, uint32_t *udeg) {
    extern __shared__ uint32_t bits[];   // words (a multiple of 32), then a count per block of 32 words
    __shared__ uint32_t sw[BITMAP_THREADS / 32 + 1];
    uint32_t *blk = bits + words;
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, blocks = words / 32;
    for (uint32_t w = threadIdx.x; w < words; w += BITMAP_THREADS) bits[w] = 0;
    __syncthreads();
    for (uint32_t i = blockIdx.x; i < count; i += gridDim.x) {
        const uint32_t r = list[i], beg = off[r], len = off[r + 1] - beg;
        const uint32_t *row = src ? src + src_off[i] : vals + beg;
        uint32_t done = 0;
        for (uint64_t lo = 0; lo < nrows; lo += (uint64_t)words * 32) {
#pragma unroll 4
            for (uint32_t t = threadIdx.x; t < len; t += BITMAP_THREADS) {
                const uint32_t v = row[t] - (uint32_t)lo;   // (below the range: wraps to above it)
                if (v >> 5 < words) atomicOr(bits + (v >> 5), 1u << (v & 31));
            }
            __syncthreads();
#pragma unroll 4
            for (uint32_t b = warp; b < blocks; b += BITMAP_THREADS / 32) {
                const uint32_t c = __reduce_add_sync(FULL, (uint32_t)__popc(bits[b * 32 + lane]));
                if (lane == 0) blk[b] = c;
            }
            __syncthreads();
            const uint32_t b0 = 2 * threadIdx.x, c0 = b0 < blocks ? blk[b0] : 0u, c1 = b0 + 1 < blocks ? blk[b0 + 1] : 0u;
            uint32_t total;
            const uint32_t at0 = block_exclusive_scan<BITMAP_THREADS>(c0 + c1, &total, sw);
            if (b0 < blocks) blk[b0] = at0;
            if (b0 + 1 < blocks) blk[b0 + 1] = at0 + c0;
            __syncthreads();
            for (uint32_t b = warp; b < blocks; b += BITMAP_THREADS / 32) {
                uint32_t w = bits[b * 32 + lane];
                if (!__any_sync(FULL, w != 0)) continue;
                const uint32_t c = __popc(w);
                uint32_t at = beg + done + blk[b] + warp_inclusive_scan(c) - c;
                if (w) bits[b * 32 + lane] = 0;
                for (; w; w &= w - 1) vals[at++] = (uint32_t)lo + (b * 32 + lane) * 32 + __ffs(w) - 1;
            }
            done += total;
            __syncthreads();
        }
        for (uint32_t t = done + threadIdx.x; t < len; t += BITMAP_THREADS) vals[beg + t] = INVALID;
        if (threadIdx.x == 0 && udeg) udeg[r] = done;
    }
}

// the listed rows one after the other (koff: their places), in pieces of 4096 entries
__global__ void k_copy_rows(const uint32_t *__restrict__ list, uint32_t count, const uint32_t *__restrict__ off,
                            const uint32_t *__restrict__ koff, uint32_t total, const uint32_t *__restrict__ vals,
                            uint32_t *out) {
    constexpr uint32_t PIECE = 4096;
    for (uint64_t p0 = (uint64_t)blockIdx.x * PIECE; p0 < total; p0 += (uint64_t)gridDim.x * PIECE) {
        const uint32_t p1 = (uint32_t)min((uint64_t)total, p0 + PIECE);
        uint32_t lo = 0, hi = count;   // last row that starts at or before p0
        while (hi - lo > 1) {
            const uint32_t mid = (lo + hi) >> 1;
            if (koff[mid] <= p0) lo = mid;
            else hi = mid;
        }
        for (uint32_t i = lo; i < count && koff[i] < p1; i++) {
            const uint32_t beg = off[list[i]], k0 = koff[i], a = max((uint32_t)p0, k0), e = min(p1, koff[i + 1]);
            for (uint32_t p = a + threadIdx.x; p < e; p += blockDim.x) out[p] = vals[beg + (p - k0)];
        }
    }
}

// the length classes of the longer rows: (32, 64], (64, 128], (128, 256], (256, 512],
// (512, 2048], (2048, 4096] and above; shorter rows are in no class
constexpr int ROW_CLASSES = 7;
struct RowClassOf {
    const uint32_t *off;
    __device__ uint32_t operator[](size_t r) const {
        const uint32_t len = off[r + 1] - off[r];
        if (len <= WARP_ROW) return 0u;
        return 1u << ((len > 64) + (len > 128) + (len > 256) + (len > MID_ROW) + (len > HALF_ROW) +
                     (len > BIG_ROW));
    }
};

struct RowLenOf {
    const uint32_t *list, *off;
    __device__ uint32_t operator[](size_t i) const { return off[list[i] + 1] - off[list[i]]; }
};

// long rows of a graph of very many rows: key = (rank of the row in the list) << vbits | value
// (values are row numbers, < 2^vbits)
template <typename K>
__global__ void k_big_keys(const uint32_t *__restrict__ list, uint32_t count, const uint32_t *__restrict__ off,
                           const uint32_t *__restrict__ koff, const uint32_t *__restrict__ vals, int vbits, K *keys) {
    for (uint32_t i = blockIdx.x; i < count; i += gridDim.x) {
        const uint32_t r = list[i], beg = off[r], len = off[r + 1] - beg, k0 = koff[i];
        for (uint32_t t = threadIdx.x; t < len; t += blockDim.x) keys[k0 + t] = ((K)i << vbits) | vals[beg + t];
    }
}

template <typename K>
__global__ void k_big_back(const K *__restrict__ keys, int vbits, uint32_t total, const uint32_t *__restrict__ list,
                           const uint32_t *__restrict__ off, const uint32_t *__restrict__ koff, uint32_t *vals,
                           bool dedup, uint32_t *udeg) {
    for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < total; p += gridDim.x * blockDim.x) {
        const K key = keys[p];
        const uint32_t i = (uint32_t)(key >> vbits), v = (uint32_t)(key & (((K)1 << vbits) - 1));
        const uint32_t t = p - koff[i], r = list[i];
        const bool keep = !dedup || t == 0 || keys[p - 1] != key;
        vals[off[r] + t] = keep ? v : INVALID;
        if (udeg) {
            const unsigned peers = __match_any_sync(__activemask(), i);
            const unsigned kb = __ballot_sync(__activemask(), keep) & peers;
            if ((threadIdx.x & 31) == (unsigned)(__ffs(peers) - 1) && kb) atomicAdd(udeg + r, (uint32_t)__popc(kb));
        }
    }
}

__global__ void k_zero_rows(const uint32_t *__restrict__ list, uint32_t count, uint32_t *udeg) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x) udeg[list[i]] = 0;
}

template <typename K>
void sort_big_rows(const uint32_t *list, uint32_t count, const uint32_t *off, const uint32_t *koff, uint32_t total,
                   int vbits, int bits, uint32_t *vals, bool dedup, uint32_t *udeg, cudaStream_t s) {
    DevBuf<K> keys(total, s);
    k_big_keys<K><<<grid_for(count, 1, 152 * 8), TPB, 0, s>>>(list, count, off, koff, vals, vbits, keys.get());
    CK_LAUNCH("k_big_keys");
    radix_sort<K>(keys.get(), nullptr, total, 0, bits, s);
    if (udeg) {
        k_zero_rows<<<grid_for(count, TPB), TPB, 0, s>>>(list, count, udeg);
        CK_LAUNCH("k_zero_rows");
    }
    k_big_back<K><<<grid_for(total, TPB), TPB, 0, s>>>(keys.get(), vbits, total, list, off, koff, vals, dedup, udeg);
    CK_LAUNCH("k_big_back");
}

void prepare_sort_kernels() {
    static thread_local int done_device = -1;
    int dev = 0;
    CK(cudaGetDevice(&dev));
    if (done_device == dev) return;
    CK(cudaFuncSetAttribute((const void *)k_sort_rows_bitmap, cudaFuncAttributeMaxDynamicSharedMemorySize,
                            (int)bitmap_bytes(BITMAP_WORDS)));
    done_device = dev;
}

}  // namespace

void sort_rows(Ctx &c, const uint32_t *off, uint32_t nrows, uint32_t *vals, bool dedup, uint32_t *udeg,
               cudaStream_t s) {
    if (nrows == 0) return;
    uint32_t rows = 1;   // a warp's, as many as leave every SM 64 warps
    while (rows < 32 && (uint64_t)rows * 2 * NUM_SMS_HINT * 64 <= nrows) rows <<= 1;
    k_sort_rows_warp<<<grid_for(((uint64_t)nrows + rows - 1) / rows * 32, TPB), TPB, 0, s>>>(off, nrows, rows, vals, dedup,
                                                                                        udeg);
    CK_LAUNCH("k_sort_rows_warp");
    c.launches++;
    // the longer rows, listed by length class (one host read for all the counts)
    prepare_sort_kernels();
    DevBuf<uint32_t> lists(nrows, s), bounds(ROW_CLASSES + 1, s);
    build_lists<ROW_CLASSES>(RowClassOf{off}, nrows, lists.get(), bounds.get(), s);
    c.launches++;
    uint32_t *hb = c.host_u32 + HOST_PLAN;
    CK(cudaMemcpyAsync(hb, bounds.get(), 4 * (ROW_CLASSES + 1), cudaMemcpyDeviceToHost, s));
    CK(cudaStreamSynchronize(s));
    uint32_t cnt[ROW_CLASSES];
    const uint32_t *list[ROW_CLASSES];
    for (int k = 0; k < ROW_CLASSES; k++) {
        cnt[k] = hb[k + 1] - hb[k];
        list[k] = lists.get() + hb[k];
    }
    if (cnt[0]) {
        k_sort_rows_warp_e<2><<<grid_for((uint64_t)cnt[0] * 32, TPB), TPB, 0, s>>>(list[0], cnt[0], off, vals,
                                                                                dedup, udeg);
        CK_LAUNCH("k_sort_rows_warp64");
        c.launches++;
    }
    if (cnt[1]) {
        k_sort_rows_warp_e<4><<<grid_for((uint64_t)cnt[1] * 32, TPB), TPB, 0, s>>>(list[1], cnt[1], off, vals,
                                                                                dedup, udeg);
        CK_LAUNCH("k_sort_rows_warp128");
        c.launches++;
    }
    if (cnt[2]) {
        k_sort_rows_warp_e<8><<<grid_for((uint64_t)cnt[2] * 32, TPB), TPB, 0, s>>>(list[2], cnt[2], off, vals,
                                                                                dedup, udeg);
        CK_LAUNCH("k_sort_rows_warp256");
        c.launches++;
    }
    if (cnt[3]) {
        k_sort_rows_warp_e<16><<<grid_for((uint64_t)cnt[3] * 32, TPB), TPB, 0, s>>>(list[3], cnt[3], off, vals,
                                                                                 dedup, udeg);
        CK_LAUNCH("k_sort_rows_warp512");
        c.launches++;
    }
    const int vbits = ceil_log2(nrows < 2 ? 2 : nrows);   // values are row numbers
    if (cnt[4]) {
        k_sort_rows_radix<8><<<grid_for(cnt[4], 1, 152 * 32), 256, 0, s>>>(list[4], cnt[4], off, vbits, vals, dedup, udeg);
        CK_LAUNCH("k_sort_rows_radix2048");
        c.launches++;
    }
    if (cnt[5]) {
        k_sort_rows_radix<16><<<grid_for(cnt[5], 1, 152 * 16), 512, 0, s>>>(list[5], cnt[5], off, vbits, vals, dedup, udeg);
        CK_LAUNCH("k_sort_rows_radix4096");
        c.launches++;
    }
    if (!cnt[6]) return;
    const uint64_t words = ((uint64_t)nrows + 1023) / 1024 * 32, ranges = (words + BITMAP_WORDS - 1) / BITMAP_WORDS;
    if (ranges == 1) {
        int per_sm = 0;
        CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, (const void *)k_sort_rows_bitmap, BITMAP_THREADS,
                                                         bitmap_bytes(words)));
        k_sort_rows_bitmap<<<grid_for(cnt[6], 1, 152 * (per_sm > 0 ? per_sm : 1)), BITMAP_THREADS, bitmap_bytes(words), s>>>(
            list[6], cnt[6], off, nrows, (uint32_t)words, nullptr, nullptr, vals, udeg);
        CK_LAUNCH("k_sort_rows_bitmap");
        c.launches++;
        return;
    }
    DevBuf<uint32_t> koff((size_t)cnt[6] + 1, s);
    scan_exclusive<uint32_t>(RowLenOf{list[6], off}, koff.get(), cnt[6], s);
    uint32_t *htotal = c.host_u32 + HOST_PLAN;
    CK(cudaMemcpyAsync(htotal, koff.get() + cnt[6], 4, cudaMemcpyDeviceToHost, s));
    CK(cudaStreamSynchronize(s));
    const uint32_t total = *htotal;
    if (ranges <= BITMAP_RANGES) {
        const uint32_t per_range = (uint32_t)((words / 32 + ranges - 1) / ranges * 32);   // even ranges
        DevBuf<uint32_t> copy(total, s);
        k_copy_rows<<<grid_for(total, 4096, 152 * 8), TPB, 0, s>>>(list[6], cnt[6], off, koff.get(), total, vals,
                                                                copy.get());
        CK_LAUNCH("k_copy_rows");
        k_sort_rows_bitmap<<<grid_for(cnt[6], 1, 152), BITMAP_THREADS, bitmap_bytes(per_range), s>>>(
            list[6], cnt[6], off, nrows, per_range, copy.get(), koff.get(), vals, udeg);
        CK_LAUNCH("k_sort_rows_bitmap");
        c.launches += 2;
        return;
    }
    // the keys are as wide as the row ranks and the values need: in 32 bits a pass moves half the bytes
    const int bits = vbits + ceil_log2(cnt[6] < 2 ? 2 : cnt[6]);
    if (bits <= 32) sort_big_rows<uint32_t>(list[6], cnt[6], off, koff.get(), total, vbits, bits, vals, dedup, udeg, s);
    else sort_big_rows<uint64_t>(list[6], cnt[6], off, koff.get(), total, vbits, bits, vals, dedup, udeg, s);
    c.launches += 3;
}

}  // namespace scd
