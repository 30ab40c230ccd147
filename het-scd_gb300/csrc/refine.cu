// Community statistics (collect_stats, src/scd.cpp:57-111), the WCC metric
// (compute_wcc, src/wcc.cpp:31-141) and the clustering coefficient p_ext
// (src/graph.cpp:57-68); the label improvement itself is in improve.cu.
//
// wcc: the internal out-lists (out-neighbours with the vertex's own label), the
// oriented triangle count on them (internal triangles per vertex and the flags
// of internal edges on one), per-vertex sums, per-vertex WCC terms and a
// fixed-order (deterministic) tree reduction.
#include "engine.cuh"
#include "rows.cuh"
#include "exact_div.cuh"
#include "gain.cuh"

namespace scd {

namespace {

constexpr unsigned TPB = 256;

// ---- collect_stats ---------------------------------------------------------

// A row segment for one warp: a whole short row or one piece of a long row.
struct RowSeg {
    uint32_t v, row0, beg, end;   // vertex, start of its row, [beg, end) of the segment in adj
    bool first, live;             // first segment of the row
};

__device__ __forceinline__ RowSeg chunk_seg(const RowWork &rw, uint32_t c, const uint32_t *indices) {
    uint32_t lo = 0, hi = rw.nlong;   // last row whose first chunk is <= c
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (rw.chunk_off[mid] <= c) lo = mid;
        else hi = mid;
    }
    const uint32_t k = c - rw.chunk_off[lo];
    RowSeg r;
    r.v = rw.llong[lo];
    const uint32_t b0 = indices[r.v], e0 = indices[r.v + 1];
    r.row0 = b0;
    r.beg = b0 + k * RowWork::CHUNK;
    r.end = min(e0, r.beg + RowWork::CHUNK);
    r.first = k == 0;
    r.live = true;
    return r;
}

// collect_stats for one row segment: sizes once per vertex, ext/int from the segment
template <int G>
__device__ __forceinline__ void stats_seg(RowSeg r, const uint32_t *adj, const uint32_t *labels, Stats st,
                                          LabelFilter skip) {
    const int gl = (threadIdx.x & 31) % G;
    const uint32_t l = r.live ? labels[r.v] : INVALID;
    const bool live = l != INVALID && !skip.frozen(r.v);
    uint32_t same = 0;
    if (live)
        for (uint32_t i = r.beg + gl; i < r.end; i += G) same += labels[adj[i]] == l;
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) same += __shfl_xor_sync(FULL, same, o);
    if (live && gl == 0) {
        const uint32_t len = r.end - r.beg;
        if (r.first) atomicAdd(st.sizes + l, 1);
        if (len - same) atomicAdd(st.ext + l, (int)(len - same));
        if (same) atomicAdd(st.intl + l, (int)same);
    }
}

// collect_stats (src/scd.cpp:57-111): rows of degree <= 256 as 32-row streams in id
// order, the rows longer than 256 as RowWork chunks after them
__global__ void __launch_bounds__(TPB)
k_stats(uint32_t n, RowWork rw, const uint32_t *__restrict__ indices, const uint32_t *__restrict__ adj,
        const uint32_t *__restrict__ labels, Stats st, LabelFilter skip) {
    const int lane = threadIdx.x & 31;
    const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
    const uint32_t groups = (n + 31) / 32, nchunks = rw.nchunks;
    for (uint32_t w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < groups + nchunks; w += warps) {
        if (w >= groups) {   // a piece of a long row
            stats_seg<32>(chunk_seg(rw, w - groups, indices), adj, labels, st, skip);
            continue;
        }
        const uint32_t r = w * 32 + lane;
        uint32_t b = 0, deg = 0, l = INVALID;
        if (r < n) {
            b = indices[r];
            deg = indices[r + 1] - b;
            l = labels[r];
            if (skip.frozen(r)) l = INVALID;
        }
        const bool mine = l != INVALID && deg <= RowWork::CHUNK;   // long rows: chunk units
        const RowStream rs(mine ? deg : 0u);
        uint32_t same = 0;
        for (uint32_t t0 = 0; t0 < rs.total; t0 += 32) {
            const uint32_t t = t0 + lane;
            const int j = rs.owner(t < rs.total ? t : rs.total - 1);
            const uint32_t pos = __shfl_sync(FULL, b, j) + (t - __shfl_sync(FULL, rs.pre, j));
            const uint32_t lj = __shfl_sync(FULL, l, j);
            const bool hit = t < rs.total && labels[adj[pos]] == lj;
            same += __popc(__ballot_sync(FULL, hit) & rs.my_lanes(t0));
        }
        if (mine) {
            atomicAdd(st.sizes + l, 1);
            if (deg - same) atomicAdd(st.ext + l, (int)(deg - same));
            if (same) atomicAdd(st.intl + l, (int)same);
        }
    }
}

// ---- WCC ---------------------------------------------------------------------

// int_tri_deg for one row segment: its out-slots (the first nlow entries of the row)
template <int G>
__device__ __forceinline__ void intdeg_seg(RowSeg r, const uint32_t *nlow, const uint32_t *adj, const uint8_t *flag,
                                           int32_t *itdeg, LabelFilter skip) {
    const int gl = (threadIdx.x & 31) % G;
    const bool live = r.live && !skip.frozen(r.v);
    uint32_t edges = 0;
    if (live) {
        const uint32_t stop = min(r.end, r.row0 + nlow[r.v]);
        for (uint32_t i = r.beg + gl; i < stop; i += G) {
            if (flag[i]) {
                atomicAdd(itdeg + adj[i], 1);
                edges++;
            }
        }
    }
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) edges += __shfl_xor_sync(FULL, edges, o);
    if (live && gl == 0 && edges) atomicAdd(itdeg + r.v, (int)edges);
}

// int_tri_deg (src/wcc.cpp:124-126): per vertex, the internal edges that lie on an
// internal triangle, counted from the out-slot flags of both endpoints; the out-slots
// of rows of degree <= 256 as streams of up to 32 rows in id order, longer rows as RowWork
// chunks. (A stream's steps are a chain of dependent loads: small graphs have fewer rows in
// one, so that every SM has its warps. 10,000 vertices, 32 rows 15 us, 4 rows 6 us.)
__global__ void __launch_bounds__(TPB)
k_internal_degrees(uint32_t n, uint32_t rows, RowWork rw, const uint32_t *__restrict__ indices, const uint32_t *__restrict__ nlow,
                   const uint32_t *__restrict__ adj, const uint8_t *__restrict__ flag, int32_t *itdeg,
                   LabelFilter skip) {
    const int lane = threadIdx.x & 31;
    const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
    const uint32_t groups = n / rows + (n % rows != 0), nchunks = rw.nchunks;
    for (uint32_t w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < groups + nchunks; w += warps) {
        if (w >= groups) {   // a piece of a long row
            intdeg_seg<32>(chunk_seg(rw, w - groups, indices), nlow, adj, flag, itdeg, skip);
            continue;
        }
        const uint32_t u = w * rows + lane;
        uint32_t b = 0, len = 0;
        if (lane < (int)rows && u < n && !skip.frozen(u)) {
            b = indices[u];
            if (indices[u + 1] - b <= RowWork::CHUNK) len = nlow[u];
        }
        const RowStream rs(len);
        uint32_t edges = 0;
        for (uint32_t t0 = 0; t0 < rs.total; t0 += 32) {
            const uint32_t t = t0 + lane;
            const int j = rs.owner(t < rs.total ? t : rs.total - 1);
            const uint32_t pos = __shfl_sync(FULL, b, j) + (t - __shfl_sync(FULL, rs.pre, j));
            const bool f = t < rs.total && flag[pos];
            if (f) atomicAdd(itdeg + adj[pos], 1);
            edges += __popc(__ballot_sync(FULL, f) & rs.my_lanes(t0));
        }
        if (edges) atomicAdd(itdeg + u, (int)edges);
    }
}

constexpr int WCC_ITEMS = 8;
constexpr int WCC_CHUNK = TPB * WCC_ITEMS;

// WCC_p of src/wcc.cpp:129-134
__device__ __forceinline__ double wcc_term(uint32_t p, const uint32_t *labels, const Stats &st,
                                           const int32_t *tri, const int32_t *tri_deg, const uint32_t *itcount,
                                           const int32_t *itdeg, double alpha) {
    const uint32_t l = labels[p];
    if (l == INVALID) return 0.0;
    const int size = st.sizes[l], td = tri_deg[p];
    if (size <= 2 || td == 0) return 0.0;
    const int it = (int)(2u * itcount[p]), itd = itdeg[p];   // int_tri = 2 x internal triangles
    const int nom = imul_wrap(it, td), t = tri[p], out = size - 1 - itd;
    // The FP64 pipe bound this kernel (conversions and a division of ten operations a vertex at
    // about two a clock and SM). With alpha 1, the default, the term is a quotient of integers:
    // it is made without that pipe where the FP64 product t * sum would be exact. Measured: 96
    // planted graphs, all steps, 1223 -> 440 us; Chung-Lu 4M 184 -> 55 us; 10,000 vertices
    // (five blocks) 19 -> 9 us.
    if (alpha == 1.0 && nom >= 0 && t > 0) {
        const long long sum = (long long)td + out;
        if (sum > 0) {
            const unsigned long long den = (unsigned long long)t * (unsigned long long)sum;   // < 2^63
            if (den < 1ull << 53) return nom ? exact_div((uint32_t)nom, den) : 0.0;
        }
    }
    const double den = dmul((double)t, dadd((double)td, dmul(alpha, (double)out)));
    return den != 0.0 ? ddiv((double)nom, den) : 0.0;
}

__device__ __forceinline__ double block_sum_fixed(double v, double *sh) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = dadd(v, __shfl_xor_sync(FULL, v, o));
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
    __syncthreads();
    double r = 0.0;
    if (threadIdx.x == 0)
        for (int w = 0; w < (int)(blockDim.x >> 5); w++) r = dadd(r, sh[w]);
    __syncthreads();
    return r;
}

// Graph-aligned blocks: block b sums WCC_CHUNK consecutive vertices of graph
// blk_gid[b], counted from that graph's first vertex, so every graph's sum has
// the same shape as when the graph is processed alone: eight consecutive terms by one
// thread, 32 threads by shuffles, eight warps in order. The terms themselves (a chain of
// FP64 operations that ends in a division) are made two by a thread, not eight: a small graph
// has few blocks, and the chains were its time (1000 vertices, one block: 15 -> 8 us).
constexpr int WCC_TERM_THREADS = 1024;

__global__ void __launch_bounds__(WCC_TERM_THREADS)
k_wcc_partial(const uint32_t *__restrict__ fin_off, const uint32_t *__restrict__ blk_off,
              const uint32_t *__restrict__ blk_gid, const uint32_t *__restrict__ labels, Stats st,
              const int32_t *__restrict__ tri, const int32_t *__restrict__ tri_deg,
              const uint32_t *__restrict__ itcount, const int32_t *__restrict__ itdeg, double alpha,
              double *partial, const uint8_t *__restrict__ active) {
    __shared__ double sh[TPB / 32];
    __shared__ double terms[WCC_CHUNK + WCC_CHUNK / WCC_ITEMS];   // a gap after every thread's eight: no bank conflicts
    const uint32_t g = blk_gid[blockIdx.x];
    if (active && !active[g]) return;   // a graph of the batch that stopped iterating
    const uint32_t end = fin_off[g + 1], base = fin_off[g] + (blockIdx.x - blk_off[g]) * WCC_CHUNK;
    for (uint32_t i = threadIdx.x; i < WCC_CHUNK; i += WCC_TERM_THREADS)
        terms[i + i / WCC_ITEMS] =
            base + i < end ? wcc_term(base + i, labels, st, tri, tri_deg, itcount, itdeg, alpha) : 0.0;
    __syncthreads();
    if (threadIdx.x >= TPB) return;
    double s = 0.0;
#pragma unroll
    for (int i = 0; i < WCC_ITEMS; i++) s = dadd(s, terms[threadIdx.x * (WCC_ITEMS + 1) + i]);   // (+ 0.0 past the end)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s = dadd(s, __shfl_xor_sync(FULL, s, o));
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = s;
    asm volatile("bar.sync 1, %0;" ::"n"(TPB) : "memory");   // the first TPB threads only
    if (threadIdx.x == 0) {
        double r = 0.0;
        for (int w = 0; w < TPB / 32; w++) r = dadd(r, sh[w]);
        partial[blockIdx.x] = r;
    }
}

// src/main.cpp:68-81 for a graph still iterating (thread 0 of its CTA of k_wcc_final: a launch
// of its own was 3 us of a small graph's step): count the iteration, remember whether it beat
// the best WCC, stop when it is below best*(1+threshold)
__device__ __forceinline__ void batch_step_of(uint32_t g, double w, const BatchStep &st) {
    st.improved[g] = 0;
    if (!st.active[g]) return;
    const double b = st.best[g];
    const int it = ++st.iters[g];
    if (st.trace && it <= st.max_trace) st.trace[(size_t)g * st.max_trace + it - 1] = w;
    if (w > b) st.improved[g] = 1;
    if (w < dmul(b, dadd(1.0, st.threshold))) {
        st.active[g] = 0;
    } else {
        st.best[g] = w;
        atomicAdd(st.n_active, 1u);
    }
}

// one block per graph: fixed-order sum of the graph's partials, divided by its n
__global__ void __launch_bounds__(TPB) k_wcc_final(const double *__restrict__ partial,
                                                   const uint32_t *__restrict__ blk_off,
                                                   const uint32_t *__restrict__ fin_off, double *out,
                                                   const uint8_t *active, BatchStep step) {
    __shared__ double sh[TPB / 32];
    const uint32_t g = blockIdx.x;
    if (active && !active[g]) {
        if (step.active && threadIdx.x == 0) step.improved[g] = 0;
        return;
    }
    const uint32_t p0 = blk_off[g], parts = blk_off[g + 1] - p0, n = fin_off[g + 1] - fin_off[g];
    double s = 0.0;
    for (uint32_t i = threadIdx.x; i < parts; i += TPB) s = dadd(s, partial[p0 + i]);
    double r = block_sum_fixed(s, sh);
    if (threadIdx.x) return;
    r = n > 0 ? ddiv(r, (double)n) : 0.0;
    out[g] = r;
    if (step.active) batch_step_of(g, r, step);
}

// ---- p_ext ---------------------------------------------------------------------

__global__ void k_pext_terms(uint32_t n, const uint32_t *__restrict__ indices, const int32_t *__restrict__ tri,
                             double *term) {
    for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x) {
        const uint32_t d = indices[p + 1] - indices[p];
        term[p] = d > 1 ? ddiv((double)tri[p], dmul((double)d, dsub((double)d, 1.0))) : 0.0;
    }
}

// The reference's single-thread order (src/graph.cpp:59-68 at one thread),
// s = ((t0 + t1) + t2) + ..., reproduced bit for bit without a 1.2M-long chain
// of dependent FP64 adds (67 cycles each on GB300).  All terms are >= 0 (zero
// for degree <= 1, which leaves s unchanged).  While s stays in one binade
// [2^e, 2^(e+1)) it is an integer S times u = 2^(e-52), and fl(s + t) is
// (S + round(t/u)) * u with round-to-nearest of the exact t/u — unless t/u has
// a fractional part of exactly 1/2 (then ties-to-even depends on S) or the sum
// leaves the binade.  So one CTA walks the terms in tiles of 8192: integer
// roundings + a block prefix sum give every in-binade partial sum exactly, and
// only the first tie or binade crossing in a tile is done with a real DADD,
// after which the tile restarts from the next term.
//
// Bound: one SM walks a graph's terms, so the rounding must not use the FP64
// pipe (2 operations a clock and SM: scale, floor and subtract of 8192 terms
// were 13 of the 25 us a tile took).  t/u is the term's 53-bit mantissa shifted
// right by the exponent distance: the quotient, the remainder and the tie are
// three 64-bit integer operations.  The first SEQ_HEAD terms, where s doubles
// every few terms and each doubling would restart a tile, are added one by one.
constexpr int SEQ_THREADS = 1024;
constexpr int SEQ_ITEMS = 8;
constexpr int SEQ_TILE = SEQ_THREADS * SEQ_ITEMS;
constexpr uint32_t SEQ_HEAD = 32;

// r = round-to-nearest of t / 2^(e-52) for 0 <= t < 2^(e+1); true: t needs a real
// addition instead (negative or not finite, not below 2^(e+1), or halfway between
// two multiples)
__device__ __forceinline__ bool seq_round(double t, int e, long long *r) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(t);
    *r = 0;
    if ((b << 1) == 0) return false;   // +0 or -0
    const int field = (int)(b >> 52) & 0x7ff;
    if (b >> 63 || field == 0x7ff) return true;
    const unsigned long long mant = (b & ((1ull << 52) - 1)) | (field ? 1ull << 52 : 0ull);
    const int sh = e + 1023 - (field ? field : 1);   // t = mant * 2^(e - 52 - sh)
    if (sh < 0) return true;
    if (sh > 53) return false;         // t is below half a unit
    const unsigned long long q = mant >> sh, twice = (mant - (q << sh)) << 1, unit = 1ull << sh;
    *r = (long long)(q + (twice > unit));
    return twice == unit;
}

__global__ void __launch_bounds__(SEQ_THREADS)
k_sequential_sum_exact(const double *__restrict__ terms, const uint32_t *__restrict__ seg_off, double *out) {
    // one block per segment (graph): sum of terms[seg_off[g] .. seg_off[g+1]) / length
    const double *term = terms + seg_off[blockIdx.x];
    const uint32_t n = seg_off[blockIdx.x + 1] - seg_off[blockIdx.x];
    const double divisor = (double)n;
    __shared__ long long warp_tot[SEQ_THREADS / 32];
    __shared__ double s_val;
    __shared__ uint32_t s_pos, s_event;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const long long TWO53 = 1ll << 53;
    __shared__ double head[SEQ_HEAD];
    const uint32_t nhead = min(n, SEQ_HEAD);
    if (threadIdx.x < nhead) head[threadIdx.x] = term[threadIdx.x];
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = 0.0;
        for (uint32_t p = 0; p < nhead; p++) s = dadd(s, head[p]);
        s_val = s;
        s_pos = nhead;
    }
    __syncthreads();
    while (true) {
        const uint32_t pos = s_pos;
        if (pos >= n) break;
        const double s = s_val;
        if (s == 0.0) {   // on to the first term that is not zero
            __syncthreads();   // s_val and s_pos are read
            if (threadIdx.x == 0) s_event = INVALID;
            __syncthreads();
            const uint32_t end = min(n, pos + (uint32_t)SEQ_TILE);
            uint32_t at = INVALID;
            for (uint32_t i = pos + threadIdx.x; i < end && at == INVALID; i += SEQ_THREADS)
                if (term[i] != 0.0) at = i;
            if (at != INVALID) atomicMin(&s_event, at);
            __syncthreads();
            if (threadIdx.x == 0) {
                s_pos = s_event == INVALID ? end : s_event + 1;
                if (s_event != INVALID) s_val = dadd(s, term[s_event]);
            }
            __syncthreads();
            continue;
        }
        if (!(s >= 1e-290) || s > 1e300) {
            // not a positive number well inside the normal range (e.g. after a negative term): one plain step
            __syncthreads();
            if (threadIdx.x == 0) {
                s_val = dadd(s, term[pos]);
                s_pos = pos + 1;
            }
            __syncthreads();
            continue;
        }
        const int e = (int)((__double_as_longlong(s) >> 52) & 0x7ff) - 1023;   // s in [2^e, 2^(e+1))
        const double u = __longlong_as_double((long long)(1023 - 52 + e) << 52);   // 2^(e-52)
        const long long S = (__double_as_longlong(s) & ((1ll << 52) - 1)) | (1ll << 52);   // s / u
        const uint32_t base = pos + threadIdx.x * SEQ_ITEMS;
        long long r[SEQ_ITEMS];
        bool ev[SEQ_ITEMS];
        long long local = 0;
#pragma unroll
        for (int i = 0; i < SEQ_ITEMS; i++) {
            r[i] = 0;
            ev[i] = false;
            if (base + i < n) ev[i] = seq_round(term[base + i], e, &r[i]);
            local += r[i];
        }
        // block exclusive scan of the per-thread totals
        long long inc = local;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            long long v = __shfl_up_sync(FULL, inc, o);
            if (lane >= o) inc += v;
        }
        if (lane == 31) warp_tot[warp] = inc;
        if (threadIdx.x == 0) s_event = INVALID;
        __syncthreads();
        if (warp == 0) {
            long long w = warp_tot[lane];
            long long wi = w;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                long long v = __shfl_up_sync(FULL, wi, o);
                if (lane >= o) wi += v;
            }
            warp_tot[lane] = wi - w;   // exclusive offset of each warp
        }
        __syncthreads();
        long long run = S + warp_tot[warp] + (inc - local);   // value before this thread's first item
        uint32_t first_event = INVALID;
        long long before_event = 0;
#pragma unroll
        for (int i = 0; i < SEQ_ITEMS; i++) {
            if (base + i < n && first_event == INVALID) {
                if (ev[i] || run + r[i] >= TWO53) {
                    first_event = base + i;
                    before_event = run;
                } else {
                    run += r[i];
                }
            }
        }
        if (first_event != INVALID) atomicMin(&s_event, first_event);
        __syncthreads();
        const uint32_t evi = s_event;
        if (evi == INVALID) {
            const uint32_t last = min(n, pos + (uint32_t)SEQ_TILE) - 1;
            if (last >= base && last < base + SEQ_ITEMS) {   // owner of the tile's last term
                s_val = dmul((double)run, u);
                s_pos = last + 1;
            }
        } else if (first_event == evi) {
            s_val = dadd(dmul((double)before_event, u), term[evi]);
            s_pos = evi + 1;
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) out[blockIdx.x] = ddiv(s_val, divisor);
}

__global__ void k_pext_tree(const uint32_t *__restrict__ fin_off, const uint32_t *__restrict__ blk_off,
                            const uint32_t *__restrict__ blk_gid, const double *__restrict__ term, double *partial) {
    __shared__ double sh[TPB / 32];
    const uint32_t g = blk_gid[blockIdx.x];
    const uint32_t end = fin_off[g + 1];
    const uint32_t base = fin_off[g] + (blockIdx.x - blk_off[g]) * WCC_CHUNK + threadIdx.x * WCC_ITEMS;
    double s = 0.0;
#pragma unroll
    for (int i = 0; i < WCC_ITEMS; i++)
        if (base + i < end) s = dadd(s, term[base + i]);
    double r = block_sum_fixed(s, sh);
    if (threadIdx.x == 0) partial[blockIdx.x] = r;
}

// ---- per-graph loop control ---------------------------------------------------

__global__ void k_copy_improved(uint32_t n, const uint32_t *__restrict__ gid, const uint8_t *__restrict__ improved,
                                const uint32_t *__restrict__ labels, uint32_t *best) {
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x)
        if (improved[gid ? gid[v] : 0]) best[v] = labels[v];
}

__global__ void k_batch_reset(uint32_t G, const uint32_t *__restrict__ fin_off, const double *__restrict__ wcc,
                              double *best, uint8_t *active, int32_t *iters) {
    for (uint32_t g = blockIdx.x * blockDim.x + threadIdx.x; g < G; g += gridDim.x * blockDim.x) {
        best[g] = wcc[g];
        active[g] = fin_off[g + 1] > fin_off[g];
        iters[g] = 0;
    }
}

}  // namespace

void copy_improved(Ctx &c) {
    if (!c.g.n) return;
    k_copy_improved<<<grid_for(c.g.n, TPB), TPB, 0, c.stream>>>(c.g.n, c.b.gid, c.b.improved, c.labels, c.best);
    CK_LAUNCH("k_copy_improved");
    c.launches++;
}

void batch_reset(Ctx &c) {
    Batch &b = c.b;
    k_batch_reset<<<grid_for(b.G, TPB), TPB, 0, c.stream>>>(b.G, b.fin_off, b.wcc, b.best_wcc, b.active, b.iters);
    CK_LAUNCH("k_batch_reset");
    c.launches++;
}

namespace {

// a vertex of label l and degree deg with c internal out-edges
__device__ __forceinline__ void add_stats(const Stats &st, uint32_t l, uint32_t deg, uint32_t c) {
    atomicAdd(st.sizes + l, 1);
    if (deg - 2 * c) atomicAdd(st.ext + l, (int)(deg - 2 * c));
    if (c) atomicAdd(st.intl + l, (int)(2 * c));
}

// One pass over the out-lists of a labelling, for the internal triangle count and for
// the community statistics.
//
// LISTS: the internal out-lists, i.e. the out-neighbours of v that carry v's (valid)
// label, in order, at v's CSR offset (length 0 for unlabelled vertices and those of
// converged graphs). The internal triangles of compute_wcc (src/wcc.cpp:84-127) are
// exactly the triangles of that subgraph, so the count walks internal lists only instead
// of filtering whole out-lists. The counters and flags the count starts from are cleared
// on the way.
// STATS: collect_stats (src/scd.cpp:57-111) of a symmetric graph without loops. An
// internal edge is an out-edge of one of its two ends and internal for both, so with c
// internal out-edges at v the row's share of the sums is +1 vertex, +2c internal and
// +deg - 2c external entries: half the neighbours are looked at, and in one iteration
// the same look gives the lists.
//
// Out-lists above the register groups' (the vertices of `longer`) have a warp each. Of the
// others a warp takes `rows` vertices: its lanes read their labels and bounds in one
// coalesced step; then a group of 8 lanes walks one out-list (most are short, and ids being
// degree ranks, the vertices of a warp have lists of similar length), the next four lists'
// neighbours on their way meanwhile. Bound by the latency of the dependent loads (label,
// bounds, neighbour, its label), which one vertex per group at a time paid in full.
// Measured (statistics + lists of a step): 96 planted graphs, 2.6 M vertices, 130 + 227 ->
// 195 us; Chung-Lu 500k, statistics alone 123 -> 30 us; R-MAT scale 20 89 + 40 -> 80 us.
template <bool LISTS, bool STATS>
__global__ void __launch_bounds__(TPB)
k_internal_lists(uint32_t n, uint32_t rows, WarpRows longer, uint32_t most_short,
                 const uint32_t *__restrict__ indices, const uint32_t *__restrict__ nlow, const uint32_t *__restrict__ adj, LabelFilter lf, uint32_t *ilen, uint32_t *iadj, uint8_t *flag,
                 uint32_t *itcount, int32_t *itdeg, Stats st, InternalWork work, uint32_t above) {
    const uint32_t lane = threadIdx.x & 31, gl = lane & 7, grp = lane >> 3;
    const uint32_t warps = (gridDim.x * blockDim.x) >> 5, units = n / rows + (n % rows != 0);
    const unsigned gmask = 0xffu << (grp * 8), lt = (1u << lane) - 1u;
    // entries of the work lists, a warp's 32 at a time (one atomic a vertex on one address would
    // be the kernel's time): lane i of the pending ones holds entry i
    uint32_t pend_v[InternalWork::K] = {}, pend_c[InternalWork::K] = {}, pend[InternalWork::K] = {};
    const auto flush = [&](int k) {
        uint32_t at = 0;
        if (lane == 0) at = atomicAdd(work.count + k, pend[k]);
        at = __shfl_sync(FULL, at, 0) + lane;
        if (lane < pend[k]) {
            work.verts[k][at] = pend_v[k];
            if (k >= 1) work.chunk[k][at] = pend_c[k];
        }
        pend[k] = 0;
    };
    for (uint32_t unit = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; unit < longer.total + units; unit += warps) {
        if (unit < longer.total) {
            const uint32_t v = longer[unit], l = lf.labels[v], beg = indices[v], len = nlow[v];
            const bool on = l != INVALID && !lf.frozen(v);
            uint32_t c = 0;
            if (on) {
                uint32_t w = lane < len ? adj[beg + lane] : INVALID;
                for (uint32_t i = lane; i - lane < len; i += 32) {
                    const uint32_t cw = w;
                    w = i + 32 < len ? adj[beg + i + 32] : INVALID;
                    const bool keep = cw != INVALID && lf.labels[cw] == l;
                    const unsigned kb = __ballot_sync(FULL, keep);
                    if (LISTS && keep) {
                        const uint32_t p = beg + c + __popc(kb & lt);
                        iadj[p] = cw;
                        flag[p] = 0;
                    }
                    c += __popc(kb);
                }
            }
            if (LISTS && lane == 0) ilen[v] = c;
            if (LISTS && c > above && len <= InternalWork::LONGEST) {
                const uint32_t chunks = c <= InternalWork::MID ? 1u : (c + InternalWork::CHUNK - 1) / InternalWork::CHUNK;
                for (uint32_t ch = 0; ch < chunks; ch++) {
#pragma unroll
                    for (int k = 0; k < InternalWork::K; k++) {
                        const uint32_t kk = (c > InternalWork::MID) + (c > InternalWork::CTA);
                        if (kk != (uint32_t)k) continue;
                        if (lane == pend[k]) {
                            pend_v[k] = v;
                            pend_c[k] = ch;
                        }
                        if (++pend[k] == 32) flush(k);
                    }
                }
            }
            if (STATS && on && lane == 0) add_stats(st, l, indices[v + 1] - beg, c);
            continue;
        }
        const uint32_t u = unit - longer.total, v = u * rows + lane, nrows = min(rows, n - u * rows);
        const bool in = lane < nrows;
        const uint32_t l = in ? lf.labels[v] : INVALID;
        bool on = l != INVALID && !lf.frozen(v);
        uint32_t beg = 0, len = in ? nlow[v] : 0u, deg = 0, cnt = 0;
        const bool shorter = len <= most_short;   // (the others have a warp)
        on = on && shorter;
        if (!on) len = 0;
        if (on) {
            beg = indices[v];
            if (STATS) deg = indices[v + 1] - beg;
        }
        uint32_t b = __shfl_sync(FULL, beg, grp), ln = __shfl_sync(FULL, len, grp);
        uint32_t w = gl < ln ? adj[b + gl] : INVALID;   // rows beyond nrows have length 0
        for (uint32_t s0 = 0; s0 < nrows; s0 += 4) {
            const uint32_t lr = __shfl_sync(FULL, l, s0 + grp), cb = b, cln = ln;
            uint32_t cw = w;
            if (s0 + 4 < nrows) {
                b = __shfl_sync(FULL, beg, s0 + 4 + grp);
                ln = __shfl_sync(FULL, len, s0 + 4 + grp);
                w = gl < ln ? adj[b + gl] : INVALID;
            }
            const uint32_t most = __reduce_max_sync(FULL, cln);
            uint32_t c = 0;
            for (uint32_t i = 0; i < most; i += 8) {
                const bool keep = cw != INVALID && lf.labels[cw] == lr;
                const unsigned kb = __ballot_sync(FULL, keep) & gmask;
                if (LISTS && keep) {
                    const uint32_t p = cb + c + __popc(kb & lt);
                    iadj[p] = cw;
                    flag[p] = 0;
                }
                c += __popc(kb);
                cw = i + 8 + gl < cln ? adj[cb + i + 8 + gl] : INVALID;
            }
            const uint32_t mine = __shfl_sync(FULL, c, ((lane - s0) & 3) * 8);
            if (lane >= s0 && lane < s0 + 4) cnt = mine;
        }
        if (LISTS && in) {
            if (shorter) ilen[v] = cnt;
            itcount[v] = 0;
            itdeg[v] = 0;
        }
        if (STATS && on) add_stats(st, l, deg, cnt);
    }
    if (LISTS) {
#pragma unroll
        for (int k = 0; k < InternalWork::K; k++)
            if (pend[k]) flush(k);
    }
}

// rows a warp takes: as many as leave every SM its 32 warps
uint32_t rows_a_warp(uint32_t n) {
    uint32_t rows = 4;
    while (rows < 32 && (uint64_t)rows * 2 * NUM_SMS_HINT * 32 <= n) rows <<= 1;
    return rows;
}

template <bool LISTS, bool STATS>
void launch_internal_lists(Ctx &c, LabelFilter lf, const Stats &st) {
    const Graph &g = c.g;
    const uint32_t rows = rows_a_warp(g.n);
    WarpRows longer{};
    for (int k = 0; k < WarpRows::K; k++)   // the longest first
        longer.set(k, c.wplan.verts[TcPlan::K - 1 - k], c.wplan.nverts[TcPlan::K - 1 - k]);
    static_assert(TcPlan::K == WarpRows::K, "the buckets above the register groups");
    k_internal_lists<LISTS, STATS><<<grid_for((((uint64_t)g.n + rows - 1) / rows + longer.total) * 32, TPB,
                                              NUM_SMS_HINT * 16), TPB, 0, c.stream>>>(
        g.n, rows, longer, c.wplan.small_max, g.indices, g.nlow, g.adj, lf, c.int_len, c.int_adj, c.slot_flag, c.itcount,
        c.itdeg, st, c.iwork, InternalWork::above(g.distinct));
    CK_LAUNCH("k_internal_lists");
}

// statistics from the out-lists alone: a symmetric graph (Graph::symmetric) whose longest
// out-list is no hub's whole row (a graph whose ids are not degree ranks may have such ones,
// and k_stats spreads them over warps)
bool stats_from_out_lists(const Ctx &c) { return c.g.symmetric && c.wplan.nverts[TcPlan::K - 1] == 0; }

}  // namespace

void collect_stats(Ctx &c, const uint32_t *labels, Stats &st, bool frozen_graphs) {
    const Graph &g = c.g;
    cudaStream_t s = c.stream;
    const size_t bytes = (size_t)(c.num_comms ? c.num_comms : 1) * 4;
    CK(cudaMemsetAsync(st.sizes, 0, bytes, s));
    CK(cudaMemsetAsync(st.ext, 0, bytes, s));
    CK(cudaMemsetAsync(st.intl, 0, bytes, s));
    if (g.n == 0) return;
    PhaseScope ph(c, "stats");
    const LabelFilter skip{nullptr, c.b.gid, frozen_graphs ? c.b.active : nullptr};
    if (stats_from_out_lists(c)) {
        launch_internal_lists<false, true>(c, LabelFilter{labels, skip.gid, skip.active}, st);
    } else {
        k_stats<<<grid_for(((uint64_t)(g.n + 31) / 32 + g.rows.nchunks) * 32, TPB), TPB, 0, s>>>(
            g.n, g.rows, g.indices, g.adj, labels, st, skip);
        CK_LAUNCH("k_stats");
    }
    c.launches++;
}

void launch_wcc(Ctx &c, const uint32_t *labels, const Stats &st, bool frozen_graphs, bool with_stats,
                const BatchStep &step) {
    const Graph &g = c.g;
    cudaStream_t s = c.stream;
    if (step.active) CK(cudaMemsetAsync(step.n_active, 0, 4, s));
    if (g.n == 0) {   // (no graph is active)
        CK(cudaMemsetAsync(c.b.wcc, 0, sizeof(double) * c.b.G, s));
        return;
    }
    PhaseScope ph(c, "wcc");
    const Batch &b = c.b;
    const uint8_t *active = frozen_graphs ? b.active : nullptr;
    const LabelFilter lf{labels, b.gid, active};
    CK(cudaMemsetAsync(c.work_counter, 0, 64, s));   // the lists' counts and the kernels' unit counters
    if (with_stats) launch_internal_lists<true, true>(c, lf, st);
    else launch_internal_lists<true, false>(c, lf, st);
    const Oriented o{g.indices, c.int_len, c.int_adj, g.n};
    count_internal_triangles(c, o, c.itcount, c.slot_flag);
    const uint32_t rows = rows_a_warp(g.n);
    k_internal_degrees<<<grid_for((((uint64_t)g.n + rows - 1) / rows + g.rows.nchunks) * 32, TPB), TPB, 0, s>>>(
        g.n, rows, g.rows, g.indices, c.int_len, c.int_adj, c.slot_flag, c.itdeg, lf);
    CK_LAUNCH("k_internal_degrees");
    c.launches++;
    if (b.blocks) {
        k_wcc_partial<<<b.blocks, WCC_TERM_THREADS, 0, s>>>(b.fin_off, b.blk_off, b.blk_gid, labels, st, g.tri, g.tri_deg,
                                               c.itcount, c.itdeg, c.alpha, c.wcc_part, active);
        CK_LAUNCH("k_wcc_partial");
    }
    k_wcc_final<<<b.G, TPB, 0, s>>>(c.wcc_part, b.blk_off, b.fin_off, b.wcc, active, step);
    CK_LAUNCH("k_wcc_final");
    c.launches += 3;
}

// statistics (st cleared by improve) and WCC of the labels of an iteration
void launch_stats_wcc(Ctx &c, const uint32_t *labels, Stats &st, bool frozen_graphs, const BatchStep &step) {
    const bool fused = stats_from_out_lists(c);
    if (!fused) collect_stats(c, labels, st, frozen_graphs);
    launch_wcc(c, labels, st, frozen_graphs, fused, step);
}

double read_wcc(Ctx &c) {
    CK(cudaMemcpyAsync(c.wcc_host, c.b.wcc, sizeof(double), cudaMemcpyDeviceToHost, c.stream));
    CK(cudaStreamSynchronize(c.stream));
    return *c.wcc_host;
}

double compute_wcc(Ctx &c, const uint32_t *labels, const Stats &st) {
    launch_wcc(c, labels, st);
    return read_wcc(c);
}

// FP32 enclosure of every p_ext (directed conversions), for the interval gains
__global__ void k_pe32(uint32_t G, const double *__restrict__ p_ext, float2 *pe32) {
    for (uint32_t g = blockIdx.x * blockDim.x + threadIdx.x; g < G; g += gridDim.x * blockDim.x)
        pe32[g] = make_float2(__double2float_rd(p_ext[g]), __double2float_ru(p_ext[g]));
}

// p_ext of every graph on the side stream: the index-ordered sum is one CTA per
// graph and runs alongside the initial partition and WCC on the main stream;
// join_p_ext (before the first improvement) and host_p_ext (host reads) wait for it.
void compute_p_ext(Ctx &c) {
    Graph &g = c.g;
    Batch &b = c.b;
    cudaStream_t s = c.side;
    if (!c.pext_ready) CK(cudaEventCreateWithFlags(&c.pext_ready, cudaEventDisableTiming));
    CK(cudaEventRecord(c.pext_ready, c.stream));   // the graph arrays are ready
    CK(cudaStreamWaitEvent(s, c.pext_ready, 0));
    DevBuf<double> term(g.n ? g.n : 1, s);
    if (g.n) {
        k_pext_terms<<<grid_for(g.n, TPB), TPB, 0, s>>>(g.n, g.indices, g.tri, term.get());
        CK_LAUNCH("k_pext_terms");
        c.launches++;
    }
    if ((c.flags & SCD_FLAG_PEXT_TREE) && g.n) {
        DevBuf<double> part(b.blocks ? b.blocks : 1, s);
        if (b.blocks) {
            k_pext_tree<<<b.blocks, TPB, 0, s>>>(b.fin_off, b.blk_off, b.blk_gid, term.get(), part.get());
            CK_LAUNCH("k_pext_tree");
        }
        k_wcc_final<<<b.G, TPB, 0, s>>>(part.get(), b.blk_off, b.fin_off, b.p_ext, nullptr, BatchStep{});
        CK_LAUNCH("k_wcc_final");
        c.launches += 2;
        // (an empty graph's p_ext is 0 here, NaN in the index-ordered mode like the reference's 0/0)
    } else {
        k_sequential_sum_exact<<<b.G, SEQ_THREADS, 0, s>>>(term.get(), b.fin_off, b.p_ext);
        CK_LAUNCH("k_sequential_sum_exact");
        c.launches++;
    }
    k_pe32<<<grid_for(b.G, TPB), TPB, 0, s>>>(b.G, b.p_ext, b.pe32);
    CK_LAUNCH("k_pe32");
    c.launches++;
    term.release();
    CK(cudaEventRecord(c.pext_ready, s));
    c.pext_join_pending = true;
    c.pext_host_valid = false;
}

void join_p_ext(Ctx &c) {
    if (!c.pext_join_pending) return;
    CK(cudaStreamWaitEvent(c.stream, c.pext_ready, 0));
    c.pext_join_pending = false;
}

void host_p_ext(Ctx &c) {
    if (c.pext_host_valid) return;
    Batch &b = c.b;
    b.h_p_ext.assign(b.G, 0.0);
    if (c.pext_ready) CK(cudaEventSynchronize(c.pext_ready));
    if (b.G && b.p_ext) CK(cudaMemcpy(b.h_p_ext.data(), b.p_ext, sizeof(double) * b.G, cudaMemcpyDeviceToHost));
    c.g.p_ext = b.G ? b.h_p_ext[0] : 0.0;
    c.pext_host_valid = true;
}

}  // namespace scd
