// Triangle counting around the dense core of a skewed graph, by row bitmaps.
//
// The vertices of degree > T (the core D) are closed under the degree
// orientation: every out-list of a member lies in D. With D small, its adjacency
// is a square bit matrix, one row of |D| bits per member, and two kinds of
// triangle need no walk:
//   * all three vertices in D (the lowest-ordered one is): the triangles of D on an
//     edge a - b are the population count of row a AND row b;
//   * the lowest-ordered vertex a outside, the other two in D: with the members among
//     a's out-neighbours as a bit row, the triangles on a - b are the population
//     count of that row AND row b.
// Those counts are every output there is to produce: an edge lies on a triangle iff
// its count is positive, a vertex's triangles are the sum of its edges' counts (halved
// where both of the triangle's edges at the vertex are counted). No triangle is looked
// at one by one, no position is looked up and nothing is added per hit, which is what
// the walks of triangles.cu spend their instructions on; they keep the edges a -> b
// with b outside D, and those of short out-lists. (What the second kind does not give is
// the flag of the edge between the two members; nearly all of those lie on a triangle
// inside D, and the few that do not are kept as open bits that the second kind looks
// at too.)
//
// Cost and choice of T: an edge costs |D|/32 word operations however many neighbours
// its ends have, a walk costs the shorter out-list. k_dense_pick weighs the two over
// every T (see there).
//
// Kernels: a row in registers (4Q words a lane), the other rows stream from L2 as
// 16-byte loads of 512 bytes a warp, two edges in flight; three words go through a
// carry-save adder before they are counted (population counts issue at a quarter of
// the rate of logic operations). Inside D a CTA per row and a warp per edge; outside a
// warp per vertex, its row built in shared memory.
//
// Measured on R-MAT scale 22 (54 M final edges), the whole preprocessing count: 24.4 ms
// by walks alone; 13.3 ms with a core of 12,131 members (inside it 0.54 ms, around it
// 2.3 ms, the walks that stay 9.9 ms). A core of 32,651 counted inside only: 18.5 ms; the
// rows then no longer stay in L2 (3.8 against 5.3 T word operations/s). Chung-Lu 4M:
// 13.4 -> 6.3 ms, R-MAT scale 19: 2.03 -> 1.33 ms.
#include <algorithm>

#include "engine.cuh"
#include "lists.cuh"

namespace scd {

namespace {

constexpr uint32_t DENSE_BINS = 8192;    // degrees from here on share the last bin
constexpr uint32_t DENSE_LOW = 64;       // no core below this degree
constexpr uint32_t DENSE_MAX = 32768;    // members: rows of 4 KB, a matrix of 128 MB
constexpr uint32_t DENSE_STEP = 4096;    // a row is padded to this many bits: 32 lanes x 16 bytes
constexpr uint64_t DENSE_SAMPLE = 1u << 20;   // edges looked at to weigh the cores, about

constexpr uint32_t DENSE_SAMPLE_DEG = 4096;    // longest row a warp looks at

// Per degree d (the last bin: and above): the vertices, their out-edges and the squares of their
// out-degrees; and, from a sample of the vertices of out-degree > lo and degree <=
// DENSE_SAMPLE_DEG, of their edges a -> b with walk length w = min(d+(a), d+(b)):
struct DegreeBins {
    uint32_t *count;
    uint64_t *edges;
    uint64_t *squares;
    long long *walk;       // + w at deg(a), - w at deg(b): its sum below d is that of the edges with deg(a) < d <= deg(b)
    long long *crossing;   // the same for the number of edges
    static constexpr size_t WORDS = 5 * (size_t)DENSE_BINS;   // 64-bit words for all of them
    __host__ __device__ explicit DegreeBins(uint64_t *p)
        : count((uint32_t *)p), edges(p + DENSE_BINS), squares(p + 2 * DENSE_BINS),
          walk((long long *)p + 3 * DENSE_BINS), crossing((long long *)p + 4 * DENSE_BINS) {}
};

__device__ __forceinline__ uint32_t degree_bin(uint32_t d) { return min(d, DENSE_BINS - 1); }
__device__ __forceinline__ void add64(long long *p, long long v) { atomicAdd((unsigned long long *)p, (unsigned long long)v); }

__global__ void k_degree_bins(const uint32_t *__restrict__ olen, const uint32_t *__restrict__ deg, uint32_t n,
                              DegreeBins h) {
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
        const uint32_t d = deg[v];
        if (d <= DENSE_LOW) continue;
        atomicAdd(h.count + degree_bin(d), 1u);
        const unsigned long long l = olen[v];
        atomicAdd((unsigned long long *)h.edges + degree_bin(d), l);
        atomicAdd((unsigned long long *)h.squares + degree_bin(d), l * l);
    }
}

// one warp per row of the symmetric rows off/vals (INVALID holes) whose vertex is in the
// sample.  u -> v iff (deg v, v) > (deg u, u).
__global__ void __launch_bounds__(256)
k_edge_bins(const uint32_t *__restrict__ off, const uint32_t *__restrict__ vals, const uint32_t *__restrict__ olen,
            const uint32_t *__restrict__ deg, uint32_t n, uint32_t every, uint32_t lo, DegreeBins h) {
    const uint32_t lane = threadIdx.x & 31, warps = (gridDim.x * blockDim.x) >> 5;
    for (uint64_t s = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; s * every < n; s += warps) {
        const uint32_t u = (uint32_t)(s * every), la = olen[u];
        const uint32_t du = deg[u];
        if (la <= lo || du > DENSE_SAMPLE_DEG) continue;
        const uint32_t beg = off[u], end = off[u + 1];
        unsigned long long sum = 0, edges = 0;
        for (uint32_t i0 = beg; i0 < end; i0 += 32) {
            const uint32_t i = i0 + lane, v = i < end ? vals[i] : INVALID;
            const uint32_t dv = v != INVALID ? deg[v] : 0u;
            const bool out = dv > du || (dv == du && v != INVALID && v > u);
            const uint32_t w = out ? min(la, olen[v]) : 0u;
            sum += w;
            edges += out;
            // deg(b)'s bin: one addition per bin and warp
            const uint32_t bin = out ? degree_bin(dv) : INVALID;
            const unsigned peers = __match_any_sync(FULL, bin);
            const uint32_t ws = __reduce_add_sync(peers, w);
            if (out && lane == __ffs(peers) - 1) {
                add64(h.walk + bin, -(long long)ws);
                add64(h.crossing + bin, -(long long)__popc(peers));
            }
        }
        sum = warp_sum(sum);
        edges = warp_sum(edges);
        if (lane == 0) {
            add64(h.walk + degree_bin(du), (long long)sum);
            add64(h.crossing + degree_bin(du), (long long)edges);
        }
    }
}

// the padded row length of a core of k members, in bits
__host__ __device__ inline uint32_t dense_bits(uint32_t k) { return (k + DENSE_STEP - 1) / DENSE_STEP * DENSE_STEP; }

// pick[0] = members, pick[1] = T (degree > T) of the core that saves the most time, or
// 0 members.  The walks inside it are taken as two thirds of the squares of the
// out-degrees (0.60 to 0.76 of them on R-MAT and Chung-Lu cores), those from outside
// into it come from the sample.  In picoseconds on this device: ITEM per walked item
// saved; per word
// operation WORD, or WORD_FAR when the matrix is beyond about half of L2; FILL per matrix
// byte (two matrices cleared, one filled); FIXED for the launches.
__global__ void __launch_bounds__(1024) k_dense_pick(DegreeBins h, float every, uint32_t *pick) {
    constexpr float ITEM = 2.0f, WORD = 0.2f, WORD_FAR = 0.27f, FILL = 0.6f, FIXED = 60e6f;
    constexpr int PER = DENSE_BINS / 1024;
    __shared__ uint64_t sw[33];
    __shared__ unsigned long long best;
    uint64_t c[PER], e[PER], in[PER], wk[PER], cr[PER], sc = 0, se = 0, si = 0, sk = 0, sr = 0, tot;
    const uint32_t top = DENSE_BINS - 1 - threadIdx.x * PER;   // thread 0 holds the highest degrees
#pragma unroll
    for (int i = 0; i < PER; i++) {
        c[i] = h.count[top - i];
        e[i] = h.edges[top - i];
        in[i] = h.squares[top - i];
        wk[i] = (uint64_t)h.walk[top - i];
        cr[i] = (uint64_t)h.crossing[top - i];
        sc += c[i];
        se += e[i];
        si += in[i];
        sk += wk[i];
        sr += cr[i];
    }
    if (threadIdx.x == 0) best = 0;
    sc = block_exclusive_scan<1024>(sc, &tot, sw);
    se = block_exclusive_scan<1024>(se, &tot, sw);
    si = block_exclusive_scan<1024>(si, &tot, sw);
    sk = block_exclusive_scan<1024>(sk, &tot, sw);   // all bins add up to 0: the sum below d is minus that from d on
    sr = block_exclusive_scan<1024>(sr, &tot, sw);
    unsigned long long mine = 0;   // (gain in ns << 13) | degree of the lowest bin of the core
#pragma unroll
    for (int i = 0; i < PER; i++) {
        sc += c[i];
        se += e[i];
        si += in[i];
        sk += wk[i];
        sr += cr[i];
        const uint32_t d = top - i;
        if (!c[i] || sc > DENSE_MAX || d <= DENSE_LOW) continue;
        const float kp = (float)dense_bits((uint32_t)sc);
        const float items = 0.67f * (float)si - (float)(long long)sk * every;
        const float words = ((float)se - (float)(long long)sr * every) * (kp / 32.f);
        const float gain = ITEM * items - (kp <= 20480.f ? WORD : WORD_FAR) * words - FILL * (kp / 8.f) * kp - FIXED;
        if (gain > 0.f) {
            const unsigned long long key = ((unsigned long long)(gain * 1e-3f) << 13) | d;
            mine = key > mine ? key : mine;
        }
    }
    if (mine) atomicMax(&best, mine);
    __syncthreads();
    const unsigned long long b = best;
    if (b == 0) {
        if (threadIdx.x == 0) pick[0] = pick[1] = 0;
        return;
    }
    // the members: everything from that bin up (the thread that holds it knows)
    const uint32_t d = (uint32_t)(b & (DENSE_BINS - 1));
    if (d <= top && d + PER > top) {
        uint64_t k = sc;   // includes all of this thread's bins: take the lower ones off
#pragma unroll
        for (int i = 0; i < PER; i++)
            if (top - i < d) k -= c[i];
        pick[0] = (uint32_t)k;
        pick[1] = d - 1;
    }
}

struct InDense {
    const uint32_t *deg;
    uint32_t bound;
    __device__ uint32_t operator[](size_t v) const { return deg[v] > bound; }
};

// num[v] of the members (INVALID for the others); walk[v] = out-degree, 0 for members
__global__ void k_dense_num(const uint32_t *__restrict__ verts, uint32_t k, uint32_t *num, uint32_t *walk) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < k; i += gridDim.x * blockDim.x) {
        num[verts[i]] = i;
        walk[verts[i]] = 0;
    }
}

// both directions of every edge of the core into the matrix; one warp per member
__global__ void __launch_bounds__(256)
k_dense_fill(Oriented o, const uint32_t *__restrict__ verts, uint32_t k, const uint32_t *__restrict__ num,
             uint32_t words, uint32_t *bits) {
    const uint32_t lane = threadIdx.x & 31, warps = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < k; r += warps) {
        const uint32_t a = verts[r], beg = o.beg[a], len = o.len[a];
        for (uint32_t i = lane; i < len; i += 32) {
            const uint32_t c = num[o.adj[beg + i]];
            atomicOr(bits + (size_t)r * words + (c >> 5), 1u << (c & 31));
            atomicOr(bits + (size_t)c * words + (r >> 5), 1u << (r & 31));
        }
    }
}

// carry-save adder: x + y + z = s + 2c per bit
__device__ __forceinline__ void csa(uint32_t x, uint32_t y, uint32_t z, uint32_t &s, uint32_t &c) {
    s = x ^ y ^ z;
    c = (x & y) | (x & z) | (y & z);
}

// population count of a AND b over Q 16-byte words
template <int Q>
__device__ __forceinline__ uint32_t and_count(const uint4 (&a)[Q], const uint4 (&b)[Q]) {
    uint32_t w[4 * Q];
#pragma unroll
    for (int i = 0; i < Q; i++) {
        w[4 * i] = a[i].x & b[i].x;
        w[4 * i + 1] = a[i].y & b[i].y;
        w[4 * i + 2] = a[i].z & b[i].z;
        w[4 * i + 3] = a[i].w & b[i].w;
    }
    uint32_t ones = 0, twos = 0;
    int i = 0;
#pragma unroll
    for (; i + 3 <= 4 * Q; i += 3) {
        uint32_t s, c;
        csa(w[i], w[i + 1], w[i + 2], s, c);
        ones += __popc(s);
        twos += __popc(c);
    }
#pragma unroll
    for (; i < 4 * Q; i++) ones += __popc(w[i]);
    return ones + 2 * twos;
}

constexpr int DENSE_WARPS = 8;

// The counts of row ra with the rows of the lanes in `who` (lane j of it: member c of that
// lane), two rows in flight; each of those lanes gets its own count.
template <int Q>
__device__ __forceinline__ uint32_t row_counts(const uint4 (&ra)[Q], const uint4 *__restrict__ bits, uint32_t c,
                                               unsigned who) {
    const uint32_t lane = threadIdx.x & 31;
    uint32_t t = 0;
    while (who) {   // (an odd last row is paired with itself)
        const int j0 = __ffs(who) - 1;
        who &= who - 1;
        const int j1 = who ? __ffs(who) - 1 : j0;
        who &= who - 1;
        const uint4 *p0 = bits + (size_t)__shfl_sync(FULL, c, j0) * (32 * Q) + lane;
        const uint4 *p1 = bits + (size_t)__shfl_sync(FULL, c, j1) * (32 * Q) + lane;
        uint4 b0[Q], b1[Q];
#pragma unroll
        for (int q = 0; q < Q; q++) b0[q] = __ldg(p0 + q * 32);
#pragma unroll
        for (int q = 0; q < Q; q++) b1[q] = __ldg(p1 + q * 32);
        // both counts are at most 32768, so their sums over the warp fit 16 bits each
        const uint32_t both = __reduce_add_sync(FULL, and_count<Q>(ra, b0) | (and_count<Q>(ra, b1) << 16));
        if (lane == (uint32_t)j1) t = both >> 16;
        if (lane == (uint32_t)j0) t = both & 0xffffu;
    }
    return t;
}

// sums[r] += counts of r's edges; flag of every edge with a positive count.  Every edge is
// counted at its out-slot.  Q: 16-byte words of a row per lane.
template <int Q>
__global__ void __launch_bounds__(DENSE_WARPS * 32)
k_tc_dense(Oriented o, const uint32_t *__restrict__ verts, uint32_t k, const uint32_t *__restrict__ num,
           const uint4 *__restrict__ bits, uint32_t *sums, uint8_t *flag, uint32_t *next_row) {
    __shared__ uint32_t s_row;
    const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    while (true) {
        if (threadIdx.x == 0) s_row = atomicAdd(next_row, 1u);
        __syncthreads();
        const uint32_t r = s_row;
        __syncthreads();
        if (r >= k) break;
        const uint32_t a = verts[r], beg = o.beg[a], len = o.len[a];
        if (w >= len) continue;   // (the barriers are all at the loop's head)
        uint4 ra[Q];
#pragma unroll
        for (int q = 0; q < Q; q++) ra[q] = bits[(size_t)r * (32 * Q) + q * 32 + lane];
        const uint32_t mine = (len - w + DENSE_WARPS - 1) / DENSE_WARPS;   // edges w, w + 8, ...
        uint32_t total = 0;
        for (uint32_t j0 = 0; j0 < mine; j0 += 32) {
            const uint32_t idx = (j0 + lane) * DENSE_WARPS + w;
            const bool in = j0 + lane < mine;
            const uint32_t c = in ? num[o.adj[beg + idx]] : 0u;
            const uint32_t t = row_counts<Q>(ra, bits, c, __ballot_sync(FULL, in));
            if (in && t) {
                flag[beg + idx] = 1;
                atomicAdd(sums + c, t);
                total += t;
            }
        }
        total = warp_sum(total);
        if (lane == 0 && total) atomicAdd(sums + r, total);
    }
}

// Edges of the core that lie on no triangle inside it: open bits in both rows, and the rows
// that have any.
__global__ void __launch_bounds__(256)
k_dense_open(Oriented o, const uint32_t *__restrict__ verts, uint32_t k, const uint32_t *__restrict__ num,
             uint32_t words, const uint8_t *__restrict__ flag, uint32_t *open, uint8_t *row_open) {
    const uint32_t lane = threadIdx.x & 31, warps = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < k; r += warps) {
        const uint32_t a = verts[r], beg = o.beg[a], len = o.len[a];
        for (uint32_t i = lane; i < len; i += 32) {
            if (flag[beg + i]) continue;
            const uint32_t c = num[o.adj[beg + i]];
            atomicOr(open + (size_t)r * words + (c >> 5), 1u << (c & 31));
            atomicOr(open + (size_t)c * words + (r >> 5), 1u << (r & 31));
            row_open[r] = row_open[c] = 1;
        }
    }
}

// flags the open edges whose bit has been cleared since
__global__ void __launch_bounds__(256)
k_dense_close(Oriented o, const uint32_t *__restrict__ verts, uint32_t k, const uint32_t *__restrict__ num,
              uint32_t words, const uint32_t *__restrict__ open, const uint8_t *__restrict__ row_open, uint8_t *flag) {
    const uint32_t lane = threadIdx.x & 31, warps = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < k; r += warps) {
        if (!row_open[r]) continue;
        const uint32_t a = verts[r], beg = o.beg[a], len = o.len[a];
        for (uint32_t i = lane; i < len; i += 32) {
            if (flag[beg + i]) continue;
            const uint32_t c = num[o.adj[beg + i]];
            if (!((open[(size_t)r * words + (c >> 5)] >> (c & 31)) & 1u)) flag[beg + i] = 1;
        }
    }
}

// Triangles a, b, c with b and c in the core and a, a vertex of va or vb (out-lists of more
// than the walks' short ones), outside: one warp per a.  tcount and flags of a - b.
template <int Q>
__global__ void __launch_bounds__(DENSE_WARPS * 32)
k_tc_fringe(Oriented o, const uint32_t *__restrict__ va, uint32_t na, const uint32_t *__restrict__ vb, uint32_t nb,
            const uint32_t *__restrict__ num, const uint4 *__restrict__ bits, uint32_t *open,
            const uint8_t *__restrict__ row_open, uint32_t *tcount, uint8_t *flag, uint32_t *next) {
    __shared__ __align__(16) uint32_t rows[DENSE_WARPS][128 * Q];
    const uint32_t lane = threadIdx.x & 31;
    uint32_t *row = rows[threadIdx.x >> 5];
    uint4 *row4 = reinterpret_cast<uint4 *>(row);
    while (true) {
        uint32_t i = 0;
        if (lane == 0) i = atomicAdd(next, 1u);
        i = __shfl_sync(FULL, i, 0);
        if (i >= na + nb) break;
        const uint32_t a = i < na ? va[i] : vb[i - na], beg = o.beg[a], len = o.len[a];
        __syncwarp();
#pragma unroll
        for (int q = 0; q < Q; q++) row4[q * 32 + lane] = make_uint4(0, 0, 0, 0);
        __syncwarp();
        uint32_t members = 0;
        for (uint32_t j = lane; j < len; j += 32) {
            const uint32_t c = num[o.adj[beg + j]];
            if (c != INVALID) {
                atomicOr(row + (c >> 5), 1u << (c & 31));
                members++;
            }
        }
        __syncwarp();
        if (__reduce_add_sync(FULL, members) < 2) continue;
        uint4 ra[Q];
#pragma unroll
        for (int q = 0; q < Q; q++) ra[q] = row4[q * 32 + lane];
        uint32_t total = 0;
        for (uint32_t j0 = 0; j0 < len; j0 += 32) {
            const uint32_t j = j0 + lane;
            const uint32_t b = j < len ? o.adj[beg + j] : 0u;
            const uint32_t c = j < len ? num[b] : INVALID;
            const unsigned who = __ballot_sync(FULL, c != INVALID);
            const uint32_t t = row_counts<Q>(ra, bits, c, who);
            if (c != INVALID && t) {
                flag[beg + j] = 1;
                atomicAdd(tcount + o.at(b), t);
                total += t;
            }
            // open edges of b that end at another of a's members lie on a triangle with a
            unsigned look = __ballot_sync(FULL, c != INVALID && row_open[c]);
            for (; look; look &= look - 1) {
                uint32_t *ob = open + (size_t)__shfl_sync(FULL, c, __ffs(look) - 1) * (128 * Q);
                for (uint32_t x = lane; x < 128 * Q; x += 32) {
                    const uint32_t m = row[x];
                    if (m && (ob[x] & m)) atomicAnd(ob + x, ~m);
                }
            }
        }
        total = warp_sum(total);   // every triangle at a is counted at both of its edges there
        if (lane == 0 && total) atomicAdd(tcount + o.at(a), total / 2);
    }
}

// the triangles at a member: half the counts of its edges
__global__ void k_dense_counts(const uint32_t *__restrict__ verts, uint32_t k, const uint32_t *__restrict__ sums,
                               Spread at, uint32_t *tcount) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < k; i += gridDim.x * blockDim.x)
        if (sums[i]) atomicAdd(tcount + at(verts[i]), sums[i] / 2);
}

template <typename F>
unsigned dense_grid(F *kernel, uint64_t ctas) {
    int per_sm = 0;
    CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, (const void *)kernel, DENSE_WARPS * 32, 0));
    return (unsigned)std::min<uint64_t>(std::max<uint64_t>(ctas, 1), (uint64_t)NUM_SMS_HINT * std::max(per_sm, 1));
}

struct DenseBuffers {
    const uint32_t *bits;
    uint32_t *open, *sums;
    uint8_t *row_open;
};

template <int Q>
void launch_dense(const Oriented &o, const DenseCore &d, const TcPlan &plan, const DenseBuffers &m, uint32_t *tcount,
                  uint8_t *flag, uint32_t *ctr, cudaStream_t s) {
    const uint4 *bits = reinterpret_cast<const uint4 *>(m.bits);
    const unsigned grid = grid_for((uint64_t)d.n * 32, 256);
    k_tc_dense<Q><<<dense_grid(k_tc_dense<Q>, d.n), DENSE_WARPS * 32, 0, s>>>(o, d.verts.get(), d.n, d.num.get(), bits,
                                                                             m.sums, flag, ctr);
    CK_LAUNCH("k_tc_dense");
    const uint32_t na = plan.nfwd[2], nb = plan.nfwd[1];   // the longer out-lists first
    if (na + nb == 0) return;
    k_dense_open<<<grid, 256, 0, s>>>(o, d.verts.get(), d.n, d.num.get(), 128 * Q, flag, m.open, m.row_open);
    CK_LAUNCH("k_dense_open");
    k_tc_fringe<Q><<<dense_grid(k_tc_fringe<Q>, ((uint64_t)na + nb + DENSE_WARPS - 1) / DENSE_WARPS), DENSE_WARPS * 32, 0,
                     s>>>(o, plan.verts[2], na, plan.verts[1], nb, d.num.get(), bits, m.open, m.row_open, tcount, flag,
                          ctr + 1);
    CK_LAUNCH("k_tc_fringe");
    k_dense_close<<<grid, 256, 0, s>>>(o, d.verts.get(), d.n, d.num.get(), 128 * Q, m.open, m.row_open, flag);
    CK_LAUNCH("k_dense_close");
}

}  // namespace

void tc_dense_pick(Ctx &c, const uint32_t *off, const uint32_t *vals, uint64_t entries, const uint32_t *olen,
                   const uint32_t *deg, uint32_t n, uint32_t *pick, cudaStream_t s) {
    DevBuf<uint64_t> bins(DegreeBins::WORDS, s);
    CK(cudaMemsetAsync(bins.get(), 0, DegreeBins::WORDS * 8, s));
    const DegreeBins h(bins.get());
    k_degree_bins<<<grid_for(n, 256, 152 * 16), 256, 0, s>>>(olen, deg, n, h);
    CK_LAUNCH("k_degree_bins");
    const uint32_t every = (uint32_t)(1 + entries / 2 / DENSE_SAMPLE);
    k_edge_bins<<<grid_for((uint64_t)(n / every + 1) * 32, 256, 152 * 16), 256, 0, s>>>(off, vals, olen, deg, n, every,
                                                                                       tc_short_lists(c), h);
    CK_LAUNCH("k_edge_bins");
    k_dense_pick<<<1, 1024, 0, s>>>(h, (float)every, pick);
    CK_LAUNCH("k_dense_pick");
    c.launches += 3;
}

void tc_dense_setup(Ctx &c, const Oriented &o, const uint32_t *deg, uint32_t members, uint32_t bound, DenseCore &d,
                    cudaStream_t s) {
    d = DenseCore();
    if (!members) return;
    const size_t matrix = (size_t)members * (dense_bits(members) / 32);
    try {   // (up to 256 MB)
        d.bits.alloc(2 * matrix, s);
        d.sums.alloc(members, s);
        d.row_open.alloc(members, s);
    } catch (const Error &e) {
        if (e.status != SCD_ERR_OOM) throw;
        cudaGetLastError();
        d = DenseCore();
        return;
    }
    d.n = members;
    d.bound = bound;
    d.verts.alloc(members, s);
    d.num.alloc(o.n, s);
    d.walk.alloc(o.n, s);
    DevBuf<uint32_t> bounds(2, s);
    build_lists<1>(InDense{deg, bound}, o.n, d.verts.get(), bounds.get(), s);
    CK(cudaMemsetAsync(d.num.get(), 0xff, 4 * (size_t)o.n, s));
    CK(cudaMemcpyAsync(d.walk.get(), o.len, 4 * (size_t)o.n, cudaMemcpyDeviceToDevice, s));
    k_dense_num<<<grid_for(members, 256), 256, 0, s>>>(d.verts.get(), members, d.num.get(), d.walk.get());
    CK_LAUNCH("k_dense_num");
    c.launches += 2;
}

void tc_dense_count(Ctx &c, const Oriented &o, const TcPlan &plan, uint32_t *tcount, uint8_t *flag, uint32_t *ctr,
                    cudaStream_t s) {
    PhaseScope ph(c, "tc_dense");
    const DenseCore &d = plan.dense;
    const uint32_t words = dense_bits(d.n) / 32;
    const size_t matrix = (size_t)d.n * words;
    CK(cudaMemsetAsync(d.bits.get(), 0, 8 * matrix, s));
    CK(cudaMemsetAsync(d.sums.get(), 0, 4 * (size_t)d.n, s));
    CK(cudaMemsetAsync(d.row_open.get(), 0, d.n, s));
    k_dense_fill<<<grid_for((uint64_t)d.n * 32, 256), 256, 0, s>>>(o, d.verts.get(), d.n, d.num.get(), words, d.bits.get());
    CK_LAUNCH("k_dense_fill");
    const DenseBuffers m{d.bits.get(), d.bits.get() + matrix, d.sums.get(), d.row_open.get()};
    switch (words / 128) {
    case 1: launch_dense<1>(o, d, plan, m, tcount, flag, ctr, s); break;
    case 2: launch_dense<2>(o, d, plan, m, tcount, flag, ctr, s); break;
    case 3: launch_dense<3>(o, d, plan, m, tcount, flag, ctr, s); break;
    case 4: launch_dense<4>(o, d, plan, m, tcount, flag, ctr, s); break;
    case 5: launch_dense<5>(o, d, plan, m, tcount, flag, ctr, s); break;
    case 6: launch_dense<6>(o, d, plan, m, tcount, flag, ctr, s); break;
    case 7: launch_dense<7>(o, d, plan, m, tcount, flag, ctr, s); break;
    default: launch_dense<8>(o, d, plan, m, tcount, flag, ctr, s); break;
    }
    k_dense_counts<<<grid_for(d.n, 256), 256, 0, s>>>(d.verts.get(), d.n, d.sums.get(), o.at, tcount);
    CK_LAUNCH("k_dense_counts");
    c.launches += 6;
}

}  // namespace scd
