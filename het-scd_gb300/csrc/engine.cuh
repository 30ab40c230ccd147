// Engine state shared by the translation units of libscd_gb300.
//
// HBM layout of one resident graph (all 32-bit words, n vertices, m undirected
// edges, ids are degree-descending ranks as written by `convert`):
//   indices[n+1], adj[2m]       symmetric CSR, rows ascending (binary format)
//   tri[n], tri_deg[n]          2 x triangles per vertex, triangle degree
//   nlow[n]                     neighbours with a smaller id = the out-list of
//                               the degree orientation, a prefix of each row
// Partition state:
//   labels / labels_next / best [n]
//   stats[2] x {sizes, ext_edges, int_edges}[n]   (current / next)
//   slot_cnt[2m]                internal-triangle counters per out-slot
//   itri[n], itdeg[n]           internal triangles / triangle degree
//   wcc_part[], wcc_sum         fixed-order WCC reduction
#pragma once

#include <cstring>
#include <string>
#include <vector>

#include "primitives.cuh"

namespace scd {

// vertex lists by degree: (0,8], (8,16], (16,32], (32,256], (256,2048], (2048,8192], > 8192
struct DegreeClasses {
    static constexpr int K = 8;
    static constexpr uint32_t upper[K] = {8, 16, 32, 256, 1024, 2048, 4096, 0xffffffffu};
    uint32_t *list[K] = {};   // class 0 also holds the isolated vertices (degree 0)
    uint32_t count[K] = {};
};

// Rows longer than CHUNK cut into CHUNK-entry pieces: per-row kernels (statistics,
// internal degrees) take one warp per short row in id order and one warp per
// piece of a long row, so hub rows run alongside the rest instead of in a tail.
struct RowWork {
    static constexpr uint32_t CHUNK = 256;
    const uint32_t *llong = nullptr;       // vertices of degree > CHUNK
    const uint32_t *chunk_off = nullptr;   // first piece of each (nlong + 1 entries)
    uint32_t nlong = 0, nchunks = 0;
};

struct Graph {
    uint32_t n = 0, m = 0;
    uint32_t *indices = nullptr, *adj = nullptr, *nlow = nullptr;
    int32_t *tri = nullptr, *tri_deg = nullptr;
    double p_ext = 0.0;   // of graph 0 (the only graph of a plain context)
    // every entry (u, v) has its (v, u), rows ascend, no loops: always so after convert, checked
    // for a transferred graph
    bool symmetric = true;
    // no row lists an entry twice or out of order: also always so after convert, also checked
    bool distinct = true;
    // degree buckets of the improve kernels, built once per graph
    DegreeClasses cls;
    RowWork rows;
    uint64_t *big_table_off = nullptr;   // hash-table offsets of the last bucket
    uint64_t big_table_words = 0;
};

struct Stats {
    int32_t *sizes = nullptr, *ext = nullptr, *intl = nullptr;
};

// The graphs of a context.  A batch of G independent graphs is held as one
// block-diagonal union graph: graph g owns the vertex range
// [fin_off[g], fin_off[g+1]) and the label range [comm_off[g], comm_off[g+1]),
// so every kernel runs once over all graphs, while everything that is defined
// per graph (p_ext, the WCC and its summation order, the convergence test) is
// kept per graph.  A plain context is a batch with G = 1.
struct Batch {
    uint32_t G = 1;
    uint32_t *fin_off = nullptr;          // device, G+1
    std::vector<uint32_t> h_fin_off;      // host copy
    std::vector<uint32_t> h_m;            // undirected edges per graph
    uint32_t *gid = nullptr;              // device, n: graph of each vertex (nullptr if G == 1)
    double *p_ext = nullptr;              // device, G
    float2 *pe32 = nullptr;               // device, G: FP32 enclosure of p_ext
    std::vector<double> h_p_ext;
    uint32_t *comm_off = nullptr;         // device, G+1 (labels of the initial partition)
    std::vector<uint32_t> h_comm_off;
    uint32_t *blk_off = nullptr;          // device, G+1: WCC partial blocks of each graph
    uint32_t *blk_gid = nullptr;          // device, #blocks: graph of each WCC block
    uint32_t blocks = 0;
    double *wcc = nullptr;                // device, G: WCC of the current labels
    double *best_wcc = nullptr;           // device, G
    uint8_t *active = nullptr;            // device, G: still iterating
    uint8_t *improved = nullptr;          // device, G: last iteration beat the best
    int32_t *iters = nullptr;             // device, G
    uint32_t *n_active = nullptr;         // device, 1
};

// CUDA-event phase timers (active with SCD_FLAG_PROFILE)
struct PhaseTimers {
    struct Phase {
        double ms = 0;
        uint64_t count = 0;
    };
    std::vector<std::string> names;
    std::vector<Phase> phases;
    std::vector<std::pair<int, std::pair<cudaEvent_t, cudaEvent_t>>> pending;
    std::vector<cudaEvent_t> pool;
    int index(const char *name);
    cudaEvent_t get_event();
    void flush();   // waits for pending events and accumulates them
    void reset();
    void destroy();
};

// triangles.cu: oriented triangle counting (per out-slot counters)
struct Oriented {
    const uint32_t *beg;   // out-list of u starts at beg[u]
    const uint32_t *len;   // and has len[u] entries (sorted ascending by id)
    const uint32_t *adj;
    uint32_t n;
    // in-lists (the v with u in out(v)): iadj[ibeg[u], ibeg[u] + ilen[u]); without
    // ibeg, beg is the offset array of a symmetric CSR whose rows hold the
    // out-list first and the in-list after it
    const uint32_t *ibeg = nullptr, *ilen = nullptr, *iadj = nullptr;
    Spread at;   // where a vertex's triangle count lies in tcount
    __device__ __forceinline__ uint32_t in_beg(uint32_t u) const { return ibeg ? ibeg[u] : beg[u] + len[u]; }
    __device__ __forceinline__ uint32_t in_len(uint32_t u) const {
        return ibeg ? ilen[u] : beg[u + 1] - beg[u] - len[u];
    }
    __device__ __forceinline__ const uint32_t *in_adj() const { return ibeg ? iadj : adj; }
};
// The labelling that statistics and internal out-lists are made of (where only the graphs that
// stopped matter, labels is nullptr); with `active`, vertices of graphs of a batch that stopped
// iterating are skipped (their statistics and WCC are no longer read).
struct LabelFilter {
    const uint32_t *labels = nullptr;
    const uint32_t *gid = nullptr;
    const uint8_t *active = nullptr;
    __device__ __forceinline__ bool frozen(uint32_t v) const { return active && !active[gid[v]]; }
};
// The dense core of a skewed graph (tc_dense.cu): the vertices of degree > bound.  The
// triangles inside it, and those of two members and an outside vertex of a CTA bucket
// below them, are counted by row bitmaps.
struct DenseCore {
    uint32_t n = 0, bound = 0;
    DevBuf<uint32_t> verts, num;   // members ascending; number of each member (INVALID for the others)
    DevBuf<uint32_t> walk;         // out-degree of every vertex, 0 for members
    DevBuf<uint32_t> bits, sums;   // two bit matrices (the rows, the open bits); counts of the members' edges
    DevBuf<uint8_t> row_open;
};
// The vertices above the register groups' buckets by the length of their internal out-list,
// listed anew for every labelling by the pass that makes the internal lists: a community
// holds a few dozen of a hub's neighbours, so nearly all of them belong to a cheaper kernel
// than their whole out-list's. (The register groups, up to SMALL, find theirs themselves.)
// Measured, the CTA kernels of a step by whole out-lists -> by this list: R-MAT scale 22
// 650 -> 4-21 us, scale 20 210 -> 5 us; 96 planted graphs (register groups only) unchanged.
// Only where rows are distinct (Graph::distinct): of a repeated entry the register groups find
// the last place and their searches one, the table kernels' walks one for every item, so there a
// vertex stays with the kind of kernel that its whole out-list chooses.
struct InternalWork {
    static constexpr int K = 3;   // warp units, 128-thread CTA units, 256-thread CTA units
    static constexpr uint32_t SMALL = 32, MID = 64, CTA = 1024, LONGEST = 8192, CHUNK = 512;
    uint32_t *verts[K] = {}, *chunk[K] = {};   // chunk (CTA units only): 512 partners each
    uint32_t *count = nullptr;                 // K words
    // (out-lists above LONGEST keep k_tc_huge)
    // internal lists of up to this many entries are not listed (a centre of a triangle has two out-neighbours)
    static uint32_t above(bool distinct) { return distinct ? SMALL : 1u; }
};
// out-degree buckets and their work-unit offsets (built once per oriented graph)
// The out-lists above the register groups': a bucket for warp units, two for CTA units
// (1 and 2), one for the longest.
// Bucket k lists its out-list centres first (nfwd[k] of them) and, for the CTA
// buckets, then the in-list centres: a vertex b whose edges a -> b with
// d+(a) < d+(b) (b-centric edges, below) are counted from b's table.
struct TcPlan {
    static constexpr int K = 4;
    uint32_t *verts[K] = {};
    uint32_t *unit_off[K] = {};
    uint32_t nverts[K] = {};
    uint32_t nfwd[K] = {};
    uint32_t small_max = 0;   // longest out-list of the register groups
    uint32_t dir_lo = 0, dir_hi = 0, dir_amin = 0;   // b-centric iff d+(a) < d+(b),
                                                      // dir_lo < d+(b) <= dir_hi, d+(a) > dir_amin
    DevBuf<uint32_t> tmp[4];   // storage when the plan is temporary: the lists, the unit offsets
    DevBuf<uint32_t> owner[K]; // place in its list of every unit's vertex
    // Core map of the upper CTA bucket (tc_core_map): the vertices of degree >
    // cta_hi, numbered 0..core_n-1 in id order.  core_adj holds every out-list
    // in core numbers (core_n for a vertex outside the core), v's list at
    // core_adj[core_beg[v]..], each list starting on a 16-byte boundary and
    // padded with core_n to a multiple of 4 entries.  Every out-list of a centre
    // of that bucket lies in the core, so a bitmap of core_n bits holds it
    // exactly.  core_n == 0: no map (the hash-table kernels run); core_lcap:
    // the bucket's largest out-degree (rounded up to even).
    const uint32_t *core_adj = nullptr, *core_beg = nullptr;
    uint32_t core_n = 0, core_lcap = 0;
    uint32_t cta_lo = 0, cta_hi = 0;   // out-degree range (cta_lo, cta_hi] of the first CTA bucket
    DevBuf<uint32_t> core_buf, core_beg_buf;
    DenseCore dense;   // counted by bitmaps instead of walks (n == 0: none)
    const uint32_t *walk(const Oriented &o) const { return dense.n ? dense.walk.get() : o.len; }
};
struct Ctx;
// slots: entries of all out-lists (unused when owned)
// in_lists: also in-list centres (b-centric edges) in the CTA buckets
// core_from > 0: the upper CTA bucket starts at that out-degree (the core-bitmap
// kernel's split, for a plan that gets a core map) instead of tc_b1
void tc_plan(Ctx &c, const Oriented &o, uint64_t slots, TcPlan &plan, cudaStream_t s, bool owned, bool in_lists,
             uint32_t core_from = 0);
// builds the core map of the upper CTA bucket (from plan.cta_hi) for out-lists
// o.adj[0..slots) (symmetric degree of v = o.len[v] + o.in_len(v)); core_n: the
// core's size, lcap: the bucket's longest out-list (both counted beforehand)
void tc_core_map(Ctx &c, const Oriented &o, uint64_t slots, TcPlan &plan, uint32_t core_n, uint32_t lcap,
                 cudaStream_t s);
// tc_plan in two parts around a host read the caller shares with other reads: the
// bucket lists with their bounds (TC_LISTS + 1 device words), then, given the
// bounds on the host, the plan's pointers and (not owned: the WCC lists its units itself,
// InternalWork) the work-unit offsets
constexpr int TC_LISTS = TcPlan::K + 2;   // the two CTA buckets have an in-list part
void tc_plan_lists(Ctx &c, const Oriented &o, TcPlan &plan, uint32_t *lists, uint32_t *bounds, cudaStream_t s,
                   bool in_lists, uint32_t core_from);
void tc_plan_units(const Oriented &o, uint64_t slots, TcPlan &plan, uint32_t *lists, const uint32_t *host_bounds,
                   cudaStream_t s, bool owned);
// out-degree up to which the walks take a vertex by register groups or a warp
uint32_t tc_short_lists(const Ctx &c);
// tc_dense.cu.  pick (2 device words): members and degree bound of the dense core worth
// having for the sorted symmetric rows off/vals (INVALID holes), out-degrees olen and
// degrees deg; 0 members if none is
void tc_dense_pick(Ctx &c, const uint32_t *off, const uint32_t *vals, uint64_t entries, const uint32_t *olen,
                   const uint32_t *deg, uint32_t n, uint32_t *pick, cudaStream_t s);
// d.n == 0 if the device has no room for the bit matrices: the walks count everything then
void tc_dense_setup(Ctx &c, const Oriented &o, const uint32_t *deg, uint32_t members, uint32_t bound, DenseCore &d,
                    cudaStream_t s);
void tc_dense_count(Ctx &c, const Oriented &o, const TcPlan &plan, uint32_t *tcount, uint8_t *flag, uint32_t *ctr,
                    cudaStream_t s);
// the plan of a full count (preprocessing) over out-lists o.adj[0..slots) with in-list
// centres: the core split and its core map, or the hash kernels' split
void tc_plan_counting(Ctx &c, const Oriented &o, uint64_t slots, TcPlan &plan, cudaStream_t s);
// Sorts every row of a CSR (offsets off[nrows+1], values vals) ascending in place;
// with dedup, repeated values of a row become INVALID and udeg[r] receives the
// number of distinct values of row r.
void sort_rows(Ctx &c, const uint32_t *off, uint32_t nrows, uint32_t *vals, bool dedup, uint32_t *udeg,
               cudaStream_t s);
// tcount[o.at(v)] += triangles at v; flag[slot] = 1 for out-slots on a triangle.
// tcount and flag must be zeroed.  entries: of all out-lists.
void count_triangles(Ctx &c, const Oriented &o, uint64_t entries, const TcPlan &plan, uint32_t *tcount, uint8_t *flag,
                     cudaStream_t s);
// lists for the resident graph's WCC plan (InternalWork; in the memory of pin64 and civ), and the
// count of the internal out-lists o by that plan and those lists
void alloc_internal_work(Ctx &c);
void count_internal_triangles(Ctx &c, const Oriented &o, uint32_t *tcount, uint8_t *flag);
// times the triangle-counting bucket splits on the resident graph, keeps the fastest
double autotune_tc(Ctx &c, std::vector<std::string> *report);
// set kernel attributes (dynamic shared memory) once per device, outside any capture
void prepare_tc_kernels();
void prepare_improve_kernels();

constexpr int HOST_PLAN = 2, HOST_SUMS = 56, HOST_READ = 64, HOST_WORDS = 68;   // pinned words of a context (Ctx::host_u32)

struct Ctx;
// records [start, end) of a phase on the context's stream when profiling
struct PhaseScope {
    Ctx *c;
    int idx;
    cudaEvent_t start = nullptr;
    PhaseScope(Ctx &ctx, const char *name);
    ~PhaseScope();
};

struct ResidentSet;   // resident.cu: graphs that join and leave between iterations

struct Ctx {
    int device = 0;
    int work_group_size = 256;
    unsigned flags = 0;
    double alpha = 1.0;
    cudaStream_t stream = nullptr;
    cudaStream_t side = nullptr;
    cudaStream_t aux = nullptr;                        // improve: the hub kernel, or without hubs the longer rows', beside the other classes
    cudaEvent_t aux_fork = nullptr, aux_join = nullptr;
    std::string err;
    uint64_t launches = 0;
    uint32_t tc_small = 32, tc_b0 = 64, tc_b1 = 1024;   // triangle-counting bucket splits (autotuned)
    uint32_t tc_amin = 0;   // b-centric edges need d+(a) > tc_amin (autotuned; at most tc_small)

    Graph g;
    Batch b;
    bool has_graph = false;
    bool capturing = false;           // inside a CUDA-graph capture: no host syncs, no timers
    cudaEvent_t pext_ready = nullptr;  // p_ext (side stream) done
    bool pext_join_pending = false;    // the main stream has not waited for it yet
    bool pext_host_valid = false;      // b.h_p_ext / g.p_ext hold it

    // partition state
    uint32_t *labels = nullptr, *labels_next = nullptr, *best = nullptr;
    Stats st[2];
    int cur = 0;
    uint32_t num_comms = 0;
    bool has_labels = false;
    uint8_t *slot_flag = nullptr;     // internal-triangle flag per adjacency position
    uint32_t *itcount = nullptr;      // internal triangles per vertex
    int32_t *itdeg = nullptr;         // edges on an internal triangle per vertex
    uint32_t *int_len = nullptr;      // label-mode count: internal out-list lengths (n)
    uint32_t *int_adj = nullptr;      // and the internal out-lists at the CSR offsets (2m)
    TcPlan wplan;                     // triangle-counting plan of the resident graph
    InternalWork iwork;
    double *wcc_part = nullptr, *wcc_host = nullptr;
    uint32_t *host_u32 = nullptr;     // pinned words: the active-graph count of an iteration at 0, planning reads from HOST_PLAN on
    char *io_buf[2] = {};             // pinned pieces of a graph file on its way to the device
    cudaEvent_t io_done[2] = {};
    uint32_t *big_tables = nullptr;   // global hash tables of the last degree bucket
    double *pin64 = nullptr;          // per-community p_in of the current statistics
    int4 *civ = nullptr;              // size, external edges and the FP32 enclosure of p_in (bits)
    uint32_t *work_counter = nullptr; // dynamic work distribution

    ResidentSet *res = nullptr;       // set by scd_resident_init
    bool resident = false;            // every iteration skips the graphs that stopped

    PhaseTimers timers;
    BlockCache blocks;                // of the temporaries
    std::vector<void *> owned;        // device allocations freed with the graph
    uint64_t bytes = 0;

    // graph-lifetime device arrays: stream-ordered from the device's memory pool, which
    // keeps freed memory cached (release threshold raised at scd_create), so a new graph
    // reuses the previous one's memory without cudaMalloc/cudaFree synchronisation
    uint64_t mem_limit = 0;           // scd_set_memory_limit (0: none)

    template <typename T>
    T *alloc(size_t count) {
        void *p = nullptr;
        if (count == 0) count = 1;
        if (mem_limit && bytes + count * sizeof(T) > mem_limit)
            throw Error(SCD_ERR_OOM, "device memory limit of the context reached");
        CK(cudaMallocAsync(&p, count * sizeof(T), stream));
        owned.push_back(p);
        bytes += count * sizeof(T);
        return (T *)p;
    }
    void free_all();

    // one value from the device, waited for; through pinned words (a copy to pageable memory
    // is staged by the driver, 6 us more)
    template <typename T>
    T read(const T *dev) {
        static_assert(sizeof(T) <= 4 * (HOST_WORDS - HOST_READ), "pinned words");
        T v;
        CK(cudaMemcpyAsync(host_u32 + HOST_READ, dev, sizeof(T), cudaMemcpyDeviceToHost, stream));
        CK(cudaStreamSynchronize(stream));
        std::memcpy(&v, host_u32 + HOST_READ, sizeof(T));
        return v;
    }
};

// preprocess.cu
// rec_off (host, G+1 entries, nullable): records of graph g are [rec_off[g], rec_off[g+1]),
// each graph with its own vertex ids; the graphs become one block-diagonal union.
void convert_edges(Ctx &c, const uint32_t *pairs_dev, uint64_t count, const std::vector<uint64_t> *rec_off = nullptr);
// read_edges on the device: (min, max) records of the text in file order into out
uint64_t parse_edge_text(Ctx &c, const char *text, uint64_t bytes, DevBuf<uint32_t> &out);
// empty graph arrays of n vertices and m edges in place of the resident graph
void alloc_graph(Ctx &c, uint32_t n, uint32_t m);
void upload_graph(Ctx &c, uint32_t n, uint32_t m, const uint32_t *indices, const uint32_t *adj,
                  const int32_t *tri, const int32_t *tri_deg);
// nlow, p_ext, degree classes, partition buffers; transferred: the rows are a caller's
void finish_graph(Ctx &c, bool transferred);
// the derived structure of the union graph (see engine.cu); always_gid: a graph-id
// array even for one graph
void build_union_structure(Ctx &c, bool always_gid, bool check_symmetry);
// engine.cu: one refinement iteration of every running graph without host
// synchronisation (capturable); kernel nodes of a captured CUDA graph
void iterate_async(Ctx &c, double threshold, double *trace, int max_trace);
uint64_t kernel_nodes(cudaGraph_t gr);
// resident.cu
void resident_destroy(Ctx &c);


// partition.cu
void initial_partition(Ctx &c);

// refine.cu
void collect_stats(Ctx &c, const uint32_t *labels, Stats &st, bool frozen_graphs = false);
double compute_wcc(Ctx &c, const uint32_t *labels, const Stats &st);
// frozen_graphs: vertices of graphs whose loop has ended keep their labels
// clear (nullable): statistics to clear for the labels this call makes
void improve(Ctx &c, const uint32_t *labels, const Stats &st, uint32_t *next, bool frozen_graphs, Stats *clear);
// per-graph loop control after a WCC (src/main.cpp:68-81): iteration count, best WCC,
// convergence, whether the labels are the best yet; *n_active receives the graphs still
// running (active == nullptr: no step)
struct BatchStep {
    double *best;
    uint8_t *active, *improved;
    int32_t *iters;
    double threshold;
    uint32_t *n_active;
    double *trace;
    int max_trace;
};
// statistics (st cleared by improve) and WCC of an iteration's labels, and the step they decide
void launch_stats_wcc(Ctx &c, const uint32_t *labels, Stats &st, bool frozen_graphs, const BatchStep &step = BatchStep{});
double read_wcc(Ctx &c);   // waits for the WCC of graph 0
// per-graph WCC in c.b.wcc (device); frozen_graphs: skip the graphs of a batch that stopped iterating
// with_stats: also adds the labels' statistics to st
void launch_wcc(Ctx &c, const uint32_t *labels, const Stats &st, bool frozen_graphs = false, bool with_stats = false,
                const BatchStep &step = BatchStep{});
void compute_p_ext(Ctx &c);   // launches on the side stream
void join_p_ext(Ctx &c);      // main stream waits for p_ext (outside captures)
void host_p_ext(Ctx &c);      // host copies of p_ext (b.h_p_ext, g.p_ext)
void copy_improved(Ctx &c);   // best labels of the graphs whose last step improved them
void batch_reset(Ctx &c);   // best := current WCC, all non-empty graphs active

}  // namespace scd

// the opaque handle of the C ABI
struct scd_ctx {
    scd::Ctx c;
};
