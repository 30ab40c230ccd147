// Initial partition on the device (create_initial_partition,
// src/scd.cpp:113-171).
//
// The reference sorts vertices by ((cc, deg), id) descending and walks them
// sequentially: a still-unlabelled vertex opens the next label and claims its
// unlabelled neighbours.  Exact parallel form used here: a vertex is a seed iff
// no neighbour earlier in the order is a seed (the lexicographically-first
// maximal independent set of that order); a seed's label is its rank among the
// seeds; a non-seed takes the label of its earliest seed neighbour (that seed
// reached it first).  The order comes from two stable LSD radix sorts:
// the degree (from descending ids) then the cc bits (positive doubles order like their bit patterns).
// The independent set is found in rounds: an undecided vertex becomes a
// non-seed as soon as an earlier neighbour is a seed, and a seed once every
// earlier neighbour is a decided non-seed.
#include <algorithm>

#include "engine.cuh"
#include "rows.cuh"

namespace scd {

namespace {

constexpr unsigned TPB = 256;
constexpr uint8_t UNDECIDED = 0, SEED = 1, NONSEED = 2;

// the vertices in descending id order with the keys maxd - degree: a stable sort of
// them gives (degree, id) descending
__global__ void k_order_keys(uint32_t n, const uint32_t *__restrict__ indices, uint32_t maxd, uint32_t *keys,
                             uint32_t *vals) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint32_t v = n - 1 - i;
        keys[i] = maxd - (indices[v + 1] - indices[v]);
        vals[i] = v;
    }
}

// cc = tri / (deg * (deg - 1.0)) (src/scd.cpp:129-131); key = ~bits so that
// ascending order is cc descending
__global__ void k_cc_keys(uint32_t n, const uint32_t *__restrict__ order, const uint32_t *__restrict__ indices,
                          const int32_t *__restrict__ tri, uint64_t *keys) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint32_t v = order[i];
        const uint32_t d = indices[v + 1] - indices[v];
        const double cc = __ddiv_rn((double)tri[v], __dmul_rn((double)d, __dsub_rn((double)d, 1.0)));
        keys[i] = ~(uint64_t)__double_as_longlong(cc);
    }
}

__global__ void k_graph_keys(uint32_t n, const uint32_t *__restrict__ order, const uint32_t *__restrict__ gid,
                             uint64_t *keys) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) keys[i] = gid[order[i]];
}

// label offset of every graph: the seed rank at the graph's first position
__global__ void k_comm_off(uint32_t G, const uint32_t *__restrict__ fin_off, const uint32_t *__restrict__ rank,
                           uint32_t *comm_off) {
    for (uint32_t g = blockIdx.x * blockDim.x + threadIdx.x; g <= G; g += gridDim.x * blockDim.x)
        comm_off[g] = rank[fin_off[g]];
}

__global__ void k_positions(uint32_t n, const uint32_t *__restrict__ order, uint32_t *pos) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) pos[order[i]] = i;
}

// vertices of degree > HUB_DEG are scanned by a whole CTA (k_mis_round_hub, k_claim_hub):
// a hub has thousands of earlier neighbours, one warp would walk them one load chain at a time
constexpr uint32_t HUB_DEG = 4096, HUB_TPB = 1024;

// The vertices of degree 33 .. HUB_DEG (four degree classes, the longest rows first) have a
// warp each; several of their rows in one warp, consecutive in id order, would be a long
// serial tail. Rows of up to 32 neighbours are taken `rows` at a time by a warp
// (k_mis_round, k_claim_labels): its lanes read the state, position and bounds of
// consecutive vertices in one coalesced step, and the next row's neighbours are fetched
// while a row is looked at, so a row costs two dependent gathers instead of five loads in a
// chain (these kernels are bound by that latency, not by their bytes: the first round of 96
// planted graphs, 2.6 M vertices, took 1.58 ms with a warp and the whole chain per row, 0.67
// ms so). Few rows for small graphs, so that every SM has warps.
inline uint32_t rows_per_warp(uint32_t n) {
    uint32_t r = 1;
    while (r < 32 && (uint64_t)r * 2 * NUM_SMS_HINT * 32 <= n) r <<= 1;
    return r;
}

// one row of a round for a warp, its first 32 neighbours in w: what becomes of the vertex
// at position pv (UNDECIDED: an earlier neighbour is still undecided)
__device__ __forceinline__ uint8_t mis_row(uint32_t w, uint32_t beg, uint32_t deg, uint32_t pv,
                                           const uint32_t *__restrict__ adj, const uint32_t *__restrict__ pos,
                                           const uint8_t *state) {
    const uint32_t lane = threadIdx.x & 31;
    bool open = false;
    for (uint32_t i0 = 0;;) {
        bool s = false, u = false;
        if (w != INVALID) {
            if (pos[w] < pv) {
                const uint8_t st = ((const volatile uint8_t *)state)[w];
                s = st == SEED;
                u = st == UNDECIDED;
            }
        }
        if (__any_sync(FULL, s)) return NONSEED;
        open = open || __any_sync(FULL, u);
        i0 += 32;
        if (i0 >= deg) return open ? UNDECIDED : SEED;
        w = i0 + lane < deg ? adj[beg + i0 + lane] : INVALID;
    }
}

// Units: the longer rows, then groups of `rows` consecutive vertices (their rows of up to 32).
__global__ void __launch_bounds__(TPB)
k_mis_round(uint32_t n, uint32_t rows, WarpRows wr, const uint32_t *__restrict__ indices,
            const uint32_t *__restrict__ adj, const uint32_t *__restrict__ pos, uint8_t *state, uint32_t *undecided) {
    const uint32_t lane = threadIdx.x & 31, warps = (gridDim.x * blockDim.x) >> 5;
    const uint32_t groups = n / rows + (n % rows != 0);
    uint32_t left = 0;   // rows of this warp still undecided
    for (uint32_t unit = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; unit < wr.total + groups; unit += warps) {
        if (unit < wr.total) {
            const uint32_t v = wr[unit];
            if (((volatile uint8_t *)state)[v] != UNDECIDED) continue;   // warp-uniform: only this warp writes it
            const uint32_t beg = indices[v], deg = indices[v + 1] - beg;
            const uint8_t to = mis_row(adj[beg + lane], beg, deg, pos[v], adj, pos, state);
            if (to == UNDECIDED) left++;
            else if (lane == 0) state[v] = to;
            continue;
        }
        const uint32_t first = (unit - wr.total) * rows, mine = first + lane;
        uint32_t my_beg = 0, my_deg = 0, my_pos = 0;
        bool look = lane < rows && mine < n && ((volatile uint8_t *)state)[mine] == UNDECIDED;
        if (look) {
            my_beg = indices[mine];
            my_deg = indices[mine + 1] - my_beg;
            my_pos = pos[mine];
            look = my_deg <= 32;
        }
        unsigned todo = __ballot_sync(FULL, look);
        uint32_t next_w = INVALID;   // this lane's neighbour in the next row
        if (todo) {
            const int j = __ffs(todo) - 1;
            const uint32_t b = __shfl_sync(FULL, my_beg, j), d = __shfl_sync(FULL, my_deg, j);
            if (lane < d) next_w = adj[b + lane];
        }
        while (todo) {
            const int j = __ffs(todo) - 1;
            todo &= todo - 1;
            const uint32_t beg = __shfl_sync(FULL, my_beg, j), deg = __shfl_sync(FULL, my_deg, j),
                           pv = __shfl_sync(FULL, my_pos, j);
            const uint32_t w = next_w;
            next_w = INVALID;
            if (todo) {
                const int k = __ffs(todo) - 1;
                const uint32_t b = __shfl_sync(FULL, my_beg, k), d = __shfl_sync(FULL, my_deg, k);
                if (lane < d) next_w = adj[b + lane];
            }
            const uint8_t to = mis_row(w, beg, deg, pv, adj, pos, state);
            if (to == UNDECIDED) left++;
            else if (lane == 0) state[first + j] = to;
        }
    }
    if (lane == 0 && left) atomicAdd(undecided, left);
}

// the same round for the hubs (list hubs[count], all of degree > HUB_DEG), one CTA each
__global__ void __launch_bounds__(HUB_TPB)
k_mis_round_hub(const uint32_t *__restrict__ hubs, uint32_t count, const uint32_t *__restrict__ indices,
                const uint32_t *__restrict__ adj, const uint32_t *__restrict__ pos, uint8_t *state,
                uint32_t *undecided) {
    for (uint32_t h = blockIdx.x; h < count; h += gridDim.x) {
        const uint32_t v = hubs[h];
        if (((volatile uint8_t *)state)[v] != UNDECIDED) continue;   // CTA-uniform: only this CTA writes it
        const uint32_t pv = pos[v], beg = indices[v], deg = indices[v + 1] - beg;
        int seed_seen = 0, open = 0;
        for (uint32_t i0 = 0; i0 < deg && !seed_seen; i0 += HUB_TPB) {
            bool s = false, u = false;
            const uint32_t i = i0 + threadIdx.x;
            if (i < deg) {
                const uint32_t w = adj[beg + i];
                if (pos[w] < pv) {
                    const uint8_t st = ((volatile uint8_t *)state)[w];
                    s = st == SEED;
                    u = st == UNDECIDED;
                }
            }
            seed_seen = __syncthreads_or(s);
            open = __syncthreads_or(u) || open;
        }
        if (threadIdx.x == 0) {
            if (seed_seen) state[v] = NONSEED;
            else if (!open) state[v] = SEED;
            else atomicAdd(undecided, 1u);
        }
        __syncthreads();
    }
}

struct SeedAt {
    const uint32_t *order;
    const uint8_t *state;
    __device__ uint32_t operator[](size_t i) const { return state[order[i]] == SEED; }
};

__global__ void k_seed_labels(uint32_t n, const uint32_t *__restrict__ pos, const uint8_t *__restrict__ state,
                              const uint32_t *__restrict__ seed_rank, uint32_t *labels) {
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x)
        if (state[v] == SEED) labels[v] = seed_rank[pos[v]];
}

// the earliest seed among a row's neighbours for a warp, its first 32 in w (INVALID: none)
__device__ __forceinline__ uint32_t first_seed(uint32_t w, uint32_t beg, uint32_t deg, const uint32_t *__restrict__ adj,
                                               const uint32_t *__restrict__ pos, const uint8_t *__restrict__ state) {
    const uint32_t lane = threadIdx.x & 31;
    uint32_t best_pos = INVALID, best = INVALID;
    for (uint32_t i0 = 0;;) {
        if (w != INVALID) {
            if (state[w] == SEED) {
                const uint32_t pw = pos[w];
                if (pw < best_pos) {
                    best_pos = pw;
                    best = w;
                }
            }
        }
        i0 += 32;
        if (i0 >= deg) break;
        w = i0 + lane < deg ? adj[beg + i0 + lane] : INVALID;
    }
    const uint32_t least = __reduce_min_sync(FULL, best_pos);
    return __shfl_sync(FULL, best, __ffs(__ballot_sync(FULL, best_pos == least)) - 1);
}

// a non-seed vertex takes the label of its earliest seed neighbour (it has one: a vertex
// becomes a non-seed by seeing a seed among its neighbours); units as in k_mis_round
__global__ void __launch_bounds__(TPB)
k_claim_labels(uint32_t n, uint32_t rows, WarpRows wr, const uint32_t *__restrict__ indices,
               const uint32_t *__restrict__ adj, const uint32_t *__restrict__ pos, const uint8_t *__restrict__ state,
               uint32_t *labels) {
    const uint32_t lane = threadIdx.x & 31, warps = (gridDim.x * blockDim.x) >> 5;
    const uint32_t groups = n / rows + (n % rows != 0);
    for (uint32_t unit = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; unit < wr.total + groups; unit += warps) {
        if (unit < wr.total) {
            const uint32_t v = wr[unit];
            if (state[v] != NONSEED) continue;
            const uint32_t beg = indices[v], deg = indices[v + 1] - beg;
            const uint32_t seed = first_seed(adj[beg + lane], beg, deg, adj, pos, state);
            if (lane == 0) labels[v] = seed == INVALID ? INVALID : labels[seed];
            continue;
        }
        const uint32_t mine = (unit - wr.total) * rows + lane;
        uint32_t my_beg = 0, my_deg = 0;
        bool look = lane < rows && mine < n && state[mine] == NONSEED;
        if (look) {
            my_beg = indices[mine];
            my_deg = indices[mine + 1] - my_beg;
            look = my_deg <= 32;
        }
        unsigned todo = __ballot_sync(FULL, look);
        uint32_t next_w = INVALID;
        if (todo) {
            const int j = __ffs(todo) - 1;
            const uint32_t b = __shfl_sync(FULL, my_beg, j), d = __shfl_sync(FULL, my_deg, j);
            if (lane < d) next_w = adj[b + lane];
        }
        uint32_t my_seed = INVALID;   // of the row of this lane
        while (todo) {
            const int j = __ffs(todo) - 1;
            todo &= todo - 1;
            const uint32_t beg = __shfl_sync(FULL, my_beg, j), deg = __shfl_sync(FULL, my_deg, j);
            const uint32_t w = next_w;
            next_w = INVALID;
            if (todo) {
                const int k = __ffs(todo) - 1;
                const uint32_t b = __shfl_sync(FULL, my_beg, k), d = __shfl_sync(FULL, my_deg, k);
                if (lane < d) next_w = adj[b + lane];
            }
            const uint32_t seed = first_seed(w, beg, deg, adj, pos, state);
            if (lane == (uint32_t)j) my_seed = seed;
        }
        if (look) labels[mine] = my_seed == INVALID ? INVALID : labels[my_seed];
    }
}

// the earliest seed neighbour of a non-seed hub, one CTA per hub
__global__ void __launch_bounds__(HUB_TPB)
k_claim_hub(const uint32_t *__restrict__ hubs, uint32_t count, const uint32_t *__restrict__ indices,
            const uint32_t *__restrict__ adj, const uint32_t *__restrict__ pos, const uint8_t *__restrict__ state,
            uint32_t *labels) {
    __shared__ unsigned long long s_best;
    for (uint32_t h = blockIdx.x; h < count; h += gridDim.x) {
        const uint32_t v = hubs[h];
        if (state[v] != NONSEED) continue;   // CTA-uniform
        if (threadIdx.x == 0) s_best = ~0ull;
        __syncthreads();
        const uint32_t beg = indices[v], deg = indices[v + 1] - beg;
        unsigned long long best = ~0ull;   // (position, vertex) of the earliest seed neighbour
        for (uint32_t i = threadIdx.x; i < deg; i += HUB_TPB) {
            const uint32_t w = adj[beg + i];
            if (state[w] == SEED) {
                const unsigned long long key = ((unsigned long long)pos[w] << 32) | w;
                best = key < best ? key : best;
            }
        }
        if (best != ~0ull) atomicMin(&s_best, best);
        __syncthreads();
        if (threadIdx.x == 0) labels[v] = labels[(uint32_t)s_best];
        __syncthreads();
    }
}

}  // namespace

void initial_partition(Ctx &c) {
    const Graph &g = c.g;
    cudaStream_t s = c.stream;
    const uint32_t n = g.n;
    c.num_comms = 0;
    if (n == 0) {
        c.b.h_comm_off.assign(c.b.G + 1, 0);
        CK(cudaMemsetAsync(c.b.comm_off, 0, 4 * (c.b.G + 1), s));
        c.has_labels = true;
        return;
    }
    PhaseScope ph(c, "partition");
    DevBuf<uint64_t> keys(n, s);
    DevBuf<uint32_t> order(n, s), pos(n, s), undecided(1, s);
    {   // no degree is above the bound of the highest class that has a vertex, or 2m
        uint32_t maxd = 2 * g.m;
        for (int k = DegreeClasses::K - 1; k >= 0 && !g.cls.count[k]; k--)
            if (k) maxd = std::min(maxd, DegreeClasses::upper[k - 1]);
        DevBuf<uint32_t> dkeys(n, s);
        k_order_keys<<<grid_for(n, TPB), TPB, 0, s>>>(n, g.indices, maxd, dkeys.get(), order.get());
        CK_LAUNCH("k_order_keys");
        radix_sort<uint32_t>(dkeys.get(), order.get(), n, 0, ceil_log2((uint64_t)maxd + 1), s);
    }
    k_cc_keys<<<grid_for(n, TPB), TPB, 0, s>>>(n, order.get(), g.indices, g.tri, keys.get());
    CK_LAUNCH("k_cc_keys");
    radix_sort<uint64_t>(keys.get(), order.get(), n, 0, 64, s);
    if (c.b.G > 1) {   // graph-major: each graph's order stays contiguous
        k_graph_keys<<<grid_for(n, TPB), TPB, 0, s>>>(n, order.get(), c.b.gid, keys.get());
        CK_LAUNCH("k_graph_keys");
        radix_sort<uint64_t>(keys.get(), order.get(), n, 0, ceil_log2(c.b.G), s);
        c.launches++;
    }
    keys.release();
    k_positions<<<grid_for(n, TPB), TPB, 0, s>>>(n, order.get(), pos.get());
    CK_LAUNCH("k_positions");
    c.launches += 3;

    DevBuf<uint8_t> state(n, s);
    CK(cudaMemsetAsync(state.get(), UNDECIDED, n, s));
    const uint32_t *hubs = g.cls.list[DegreeClasses::K - 1];   // degree > 4096 = HUB_DEG
    const uint32_t nhubs = g.cls.count[DegreeClasses::K - 1];
    const uint32_t rows = rows_per_warp(n);
    WarpRows wr{};
    for (int k = 0; k < WarpRows::K; k++)
        wr.set(k, g.cls.list[DegreeClasses::K - 2 - k], g.cls.count[DegreeClasses::K - 2 - k]);
    static_assert(DegreeClasses::upper[DegreeClasses::K - 2 - WarpRows::K] == 32, "rows of more than 32");
    const unsigned G = grid_for((((uint64_t)n + rows - 1) / rows + wr.total) * 32, TPB, 152 * 16);
    static_assert(DegreeClasses::upper[DegreeClasses::K - 2] == HUB_DEG, "hub class");
    // Rounds are queued four, then two at a time before the host looks at the undecided
    // count of the last one: a round too many finds nothing to do and costs less than a wait.
    for (uint64_t round = 0;;) {
        for (int k = round == 0 ? 4 : 2; k > 0; k--, round++) {
            CK(cudaMemsetAsync(undecided.get(), 0, 4, s));
            if (nhubs) {
                k_mis_round_hub<<<grid_for(nhubs, 1, 152 * 2), HUB_TPB, 0, s>>>(hubs, nhubs, g.indices, g.adj, pos.get(),
                                                                             state.get(), undecided.get());
                CK_LAUNCH("k_mis_round_hub");
                c.launches++;
            }
            k_mis_round<<<G, TPB, 0, s>>>(n, rows, wr, g.indices, g.adj, pos.get(), state.get(), undecided.get());
            CK_LAUNCH("k_mis_round");
            c.launches++;
        }
        uint32_t *left = c.host_u32 + HOST_PLAN;
        CK(cudaMemcpyAsync(left, undecided.get(), 4, cudaMemcpyDeviceToHost, s));
        CK(cudaStreamSynchronize(s));
        if (*left == 0) break;
        if (round > 4 * (uint64_t)n + 8) throw Error(SCD_ERR_TIMEOUT, "initial partition did not converge");
    }

    DevBuf<uint32_t> rank((size_t)n + 1, s);
    scan_exclusive<uint32_t>(SeedAt{order.get(), state.get()}, rank.get(), n, s);
    k_seed_labels<<<grid_for(n, TPB), TPB, 0, s>>>(n, pos.get(), state.get(), rank.get(), c.labels);
    CK_LAUNCH("k_seed_labels");
    k_claim_labels<<<G, TPB, 0, s>>>(n, rows, wr, g.indices, g.adj, pos.get(), state.get(), c.labels);
    CK_LAUNCH("k_claim_labels");
    if (nhubs) {
        k_claim_hub<<<grid_for(nhubs, 1, 152 * 2), HUB_TPB, 0, s>>>(hubs, nhubs, g.indices, g.adj, pos.get(),
                                                                 state.get(), c.labels);
        CK_LAUNCH("k_claim_hub");
        c.launches++;
    }
    c.launches += 4;
    k_comm_off<<<grid_for(c.b.G + 1, TPB), TPB, 0, s>>>(c.b.G, c.b.fin_off, rank.get(), c.b.comm_off);
    CK_LAUNCH("k_comm_off");
    c.b.h_comm_off.resize(c.b.G + 1);
    CK(cudaMemcpyAsync(c.b.h_comm_off.data(), c.b.comm_off, 4 * (c.b.G + 1), cudaMemcpyDeviceToHost, s));
    CK(cudaStreamSynchronize(s));
    c.num_comms = c.b.h_comm_off[c.b.G];
    c.cur = 0;
    collect_stats(c, c.labels, c.st[0]);
    CK(cudaMemcpyAsync(c.best, c.labels, (size_t)n * 4, cudaMemcpyDeviceToDevice, s));
    c.has_labels = true;
}

}  // namespace scd
