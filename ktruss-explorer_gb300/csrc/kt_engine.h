// The device-resident engine: workspace layout in HBM and the internal stages.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <vector>

#include "kt_internal.h"

// Most blocks of the selector's statistics launch (its per-block partials buffer).
constexpr uint32_t kSelMaxBlocks = 1024;

struct kt_engine {
    int device = 0;
    int num_sms = 0;
    cudaStream_t stream = nullptr;
    cudaEvent_t ev_start = nullptr, ev_stop = nullptr, ev_built = nullptr, ev_counted = nullptr;
    cudaEvent_t ev_select = nullptr;  // after the build, before the selector's choice
    cudaEvent_t ev_copy[4] = {};      // host-buffer calls: around the input and output copies
    cudaEvent_t ev_peel0 = nullptr, ev_peel1 = nullptr;  // around the peel kernel launch
    cudaEvent_t ev_peeled = nullptr;  // decompositions: after the peel, before the per-entry output
    bool emit_timed = false;          // ev_peeled was recorded in this call
    bool peel_timed = false;
    uint64_t launches = 0;

    // Workspace arena: one allocation carved into the arrays below.
    void* arena = nullptr;
    size_t arena_bytes = 0;
    uint32_t cap_nodes = 0;
    uint64_t cap_entries = 0;

    // Sort buffers (2m entries): keys (src_rank << vb | dst_rank) and entry indices.
    uint64_t* key_a = nullptr;
    uint64_t* key_b = nullptr;
    uint32_t* val_a = nullptr;
    uint32_t* val_b = nullptr;
    // Per vertex (rank space unless noted).
    uint32_t* deg = nullptr;      // degree by original id
    uint32_t* rank = nullptr;     // original id -> rank
    uint32_t* s_ptr = nullptr;    // n+1: symmetric CSR row starts
    uint32_t* s_len = nullptr;    // n: live length of each symmetric row (after compaction)
    uint32_t* s_split = nullptr;  // n: first position of the row's higher-rank neighbours
    uint32_t* o_ptr = nullptr;    // n+1: oriented CSR row starts (edge id of a row's first edge)
    // Per symmetric entry (2m).
    uint32_t* s_col = nullptr;    // neighbour rank
    uint32_t* s_eid = nullptr;    // edge id of the entry
    uint32_t* sorted_entry = nullptr;  // input entry index at this sorted position (build only)
    uint32_t* entry_eid = nullptr;     // edge id of each input entry (outputs are gathered by it)
    // Per edge (m); edge id = position in the oriented CSR.
    uint32_t* o_col = nullptr;    // higher-rank endpoint
    uint32_t* o_fence = nullptr;  // o_fence[f] = o_col[32 f]: the first level of row searches
    uint32_t* e_src = nullptr;    // lower-rank endpoint
    uint32_t* sup = nullptr;      // support (alive triangles)
    uint32_t* rnd = nullptr;      // 0 while alive, else the peel round that removed it
    uint32_t* tr = nullptr;       // truss number (written at removal)
    uint32_t* q0 = nullptr;       // edges walked by whole blocks, by round parity
    uint32_t* q1 = nullptr;
    uint4* chunks0 = nullptr;     // peel work chunks, by round parity
    uint4* chunks1 = nullptr;
    uint32_t cap_chunks = 0;
    // Scratch of the one-pass scans and radix passes (kt_look.cuh): look-back words, digit counts
    // and tickets, cleared by begin_session; the current session's tag and count blocks in use.
    unsigned long long* look = nullptr;
    uint64_t look_cap = 0;
    uint32_t* digit_counts = nullptr;
    uint32_t look_tag = 0, look_count = 0;
    uint64_t look_limit_ns = 0;  // longest look-back wait of the session
    // Control block (device) and its pinned host mirror.
    uint32_t* ctrl = nullptr;
    uint32_t* h_ctrl = nullptr;
    // Per-round log: frontier size and level of each peel round.
    uint32_t* round_size = nullptr;
    uint32_t* round_level = nullptr;
    uint32_t* round_ns = nullptr;
    uint32_t cap_levels = 0;
    uint32_t* level_k = nullptr;      // per-level log (k, alive, start time, first frontier)
    uint32_t* level_alive = nullptr;
    uint32_t* level_ns = nullptr;
    uint32_t* level_front = nullptr;
    uint32_t cap_rounds = 0;
    // Staging for the host-buffer entry points.
    uint32_t* in_src = nullptr;
    uint32_t* in_dst = nullptr;
    uint32_t* out_u32 = nullptr;
    uint8_t* out_u8 = nullptr;
    uint32_t* aux = nullptr;       // batch staging: vertex offsets and per-graph k_max (own allocation)
    size_t aux_words = 0;
    uint32_t* tile_off = nullptr;  // tiled variant: first oriented position of each (vertex, column tile)
    size_t tile_off_words = 0;     //   (own allocation, made by the first tiled call)
    bool chained = false;  // the session's kernels start in their predecessors' tails (launch_chained)
    unsigned long long* ingest = nullptr;  // TSV ingest: outcome, tokens before each tile
    uint64_t ingest_words = 0;             //   (own allocation, made by the first ingest)
    uint2* lists = nullptr;        // triangle lists of a decomposition (own allocation, kt_lists.cu)
    uint64_t list_cap = 0;         //   entries it holds
    uint64_t list_limit = ~0ull;   //   bytes it may take (kt_engine_set_list_limit)
    uint64_t list_need = 0;        //   entries that the current call's lists need (0: it walks rows)
    bool lists_allowed = false;    //   kt_engine_create sets it; the allocation-free path never does

    // Current graph.
    uint32_t n = 0;
    uint64_t entries = 0;
    uint32_t m = 0;
    uint32_t vb = 1;  // bits per rank in sort keys

    kt_schedule sched{8, 32, 85, 50, 0};  // kernel schedule (kt_engine_set_schedule)
    kt_variant variant{KT_DIRECTED_BY_DEGREE, KT_FORMAT_COOCSR, KT_RECOUNT_ALL, 512, 8, 8};  // single-k calls
    bool orient_by_index = false;      // the next build orients by vertex id (KT_DIRECTED_BY_INDEX)
    bool by_index = false;             // the current graph is oriented by vertex id
    uint32_t variant_passes = 0;       // passes of the last undirected or tiled single-k call
    uint64_t wait_base_ns = 10ull * 1000 * 1000 * 1000;  // peel barrier wait limit: base ...
    uint64_t wait_ns_per_unit = 8;                        // ... plus per unit of covered work
    bool batch_call = false;           // the current call decomposes a batch of separate graphs
    kt_selector* selector = nullptr;   // learned schedule selector (kt_engine_set_selector)
    bool sched_on_device = false;      // this call's schedule is the selector's choice in ctrl[kPSched]
    uint32_t* sel_stats = nullptr;     // 16 u64: the selector's block ticket (word kTicket)
    uint64_t* sel_part = nullptr;      // per-block partial statistics (kSelMaxBlocks x 10 u64)
    float* sel_feat = nullptr;         // the 16 features
    uint32_t* sel_choice = nullptr;    // the selector's schedule index
    kt_stats stats{};
    int peel_mode = 0;          // 0 decomposition, 1 single-k peel, 2 k < 3, 3 single-k variant passes
    // Replay (kt_engine_replay): the last decomposition or single-k call on device buffers, and
    // its device pipeline as an instantiated CUDA graph once captured.  `trusted` marks a pipeline
    // run whose input already passed its checks: no host reads, no timing events (capturable).
    struct LastCall {
        int kind = 0;  // 0 none, 1 decomposition, 2 single-k truss
        const uint32_t* src = nullptr;
        const uint32_t* dst = nullptr;
        uint64_t entries = 0;
        uint32_t n = 0;
        uint32_t* truss = nullptr;
        uint32_t* k_max = nullptr;
        uint32_t k = 0;
        uint8_t* keep = nullptr;
        uint64_t list_need = 0;              // list buffer that the call needed (0: it walked rows)
    } last;
    cudaGraphExec_t replay = nullptr;
    bool replay_direct = false;      // the pipeline could not be captured: replays launch it directly
    uint64_t replay_launches = 0;    // kernel launches in one replay
    int replay_peel_mode = 0;
    bool trusted = false;
    bool replay_timing = false;      // last_ms of a replay is read when the stream has drained
    bool stats_ready = false;   // stats already read back from the device
    bool ctrl_fresh = false;    // h_ctrl holds the control block as the last call left it
};

namespace kt {

// Launch bookkeeping: every kernel launch of the engine goes through this.
inline void count_launch(kt_engine* e, uint64_t n = 1) { e->launches += n; }
int check_cuda(cudaError_t err, const char* what);
int check_launch(kt_engine* e, const char* what);

// Launches a kernel that begins with after_previous().  In a chained session it may start before its
// predecessor in the stream has finished, whose tail then hides the launch: building a graph of 15,000
// or 32,000 edges, 12 launches, takes 58 and 64 us instead of 81 and 87.
template <class... P, class... A>
int launch_chained(kt_engine* e, const char* what, void (*kernel)(P...), uint32_t blocks, int threads, int smem,
                   A&&... args) {
    cudaLaunchAttribute a;
    a.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    a.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c = {};
    c.gridDim = dim3(blocks);
    c.blockDim = dim3((unsigned)threads);
    c.dynamicSmemBytes = (size_t)smem;
    c.stream = e->stream;
    c.attrs = &a;
    c.numAttrs = e->chained ? 1 : 0;
    count_launch(e);
    return check_cuda(cudaLaunchKernelEx(&c, kernel, static_cast<P>(args)...), what);
}

int reserve(kt_engine* e, uint32_t max_nodes, uint64_t max_entries);
// kt_engine_replay bookkeeping (kt_engine.cu)
void drop_replay(kt_engine* e);
void remember(kt_engine* e, const kt_engine::LastCall& c);
void forget(kt_engine* e);
size_t carve(kt_engine* e, char* base, uint32_t n, uint64_t N, bool staging);

struct Look;  // kt_look.cuh

// kt_sort.cu.  Sorts of up to kSmallSort keys take small tiles (enough blocks for every SM).
constexpr uint64_t kSmallSort = 1u << 18;
constexpr uint64_t kSmallTile = 1024, kLargeTile = 6144;
constexpr uint32_t kCountWords = 32 * 256 + 64;  // digit count blocks and tickets of a session
inline uint64_t look_words(uint64_t keys) {
    return 256 * (keys <= kSmallSort ? (keys + kSmallTile - 1) / kSmallTile : (keys + kLargeTile - 1) / kLargeTile);
}
// A session clears the control block, deg[0, deg_words) and the look-back scratch for sorts of up to
// `words` (look_words) and sets the row marks to n; each launch that looks back takes a tag of it.
int begin_session(kt_engine* e, uint32_t n, uint32_t deg_words, uint64_t words, uint64_t keys);
Look next_look(kt_engine* e);
uint32_t* next_counts(kt_engine* e, unsigned passes);  // zeroed digit counts, 256 words a pass
int count_digits(kt_engine* e, const uint64_t* keys, uint64_t n, unsigned shift, unsigned passes, uint32_t* counts);
// Sorts keys by `passes` 8-bit digits from bit `shift` on, whose counts are in `counts`; ping-pongs
// between the a and b buffers and says in *result_in_b where the result is.  With value buffers the
// values are the keys' positions before the sort (not read, only written).
int radix_passes(kt_engine* e, uint64_t* key_a, uint32_t* val_a, uint64_t* key_b, uint32_t* val_b, uint64_t n,
                 unsigned shift, unsigned passes, const uint32_t* counts, int* result_in_b);

// kt_build.cu: relabel by degree, orient, sort, symmetric + oriented CSR, edge ids.  With `check` it
// waits and returns an input error as a status; without, the error stays in the control block, the
// kernels after the build return at once, and the caller reads it (input_status).
int build_graph(kt_engine* e, const uint32_t* d_src, const uint32_t* d_dst, uint64_t entries, uint32_t n,
                bool check);
int input_status(uint32_t err);
// Reads the control block back and waits for it; returns an input error or an expired wait.
int sync_and_check(kt_engine* e);

// Symmetric simple graph of an arbitrary entry list (directions merged, duplicates and self loops
// dropped): (lo, hi) pairs in sorted order, then the same pairs reversed; synchronous.
int symmetrize(kt_engine* e, const uint32_t* d_src, const uint32_t* d_dst, uint64_t entries, uint32_t n,
               uint32_t* d_src_out, uint32_t* d_dst_out, uint64_t capacity, uint64_t* num_out);

// Tiled COO/CSR of an entry list (the reference's tiled layout); synchronous.
int tiled_coocsr(kt_engine* e, const uint32_t* d_src, const uint32_t* d_dst, uint64_t entries, uint32_t n,
                 uint32_t tiles_per_dim, uint32_t* d_tile_src_ptr, uint32_t* d_src_out, uint32_t* d_dst_out);

// kt_support.cu: support of every edge (triangles through it) into e->sup.
// The credits lie in two arrays until merge_support (or the list peel's bounds) adds them up, and their
// sum into the control block's triangle counter, which the build cleared.
int count_support(kt_engine* e);
int merge_support(kt_engine* e, uint32_t limit);

int truss3(kt_engine* e);  // merge_support and the 3-truss: rnd 0 for the edges that stay

// Counts the edges left by a single-k call's first round again if that round removes `percent` or more
// of them (decided on the device; percent 0 in *out: never).  new_id: the edge's number among those
// left, or its top bit; count: their supports.
struct PrunedCount {
    uint32_t percent;
    const uint32_t* new_id;
    const uint32_t* count;
};
int recount_pruned(kt_engine* e, uint32_t limit, uint32_t percent, PrunedCount* out);
// Writes the triangle lists of the counted graph: list starts, and list ends (consumed).
int fill_lists(kt_engine* e, const uint64_t* tptr, uint64_t* ends);

// kt_peel.cu
int peel_decompose(kt_engine* e);
int peel_single_k(kt_engine* e, uint32_t k);
// kt_lists.cu: adds up the supports and decomposes from triangle lists where they apply (*done).
int peel_lists(kt_engine* e, bool* done);
// A list buffer for graphs of up to max_edges whose lists are made without reading the triangle count.
void reserve_small_lists(kt_engine* e, uint64_t max_edges);
void free_lists(kt_engine* e);
// cudaMalloc for the engine's other arrays: gives the list buffer back if there is no memory left.
cudaError_t alloc_device(kt_engine* e, void** p, size_t bytes);
int emit_truss_per_entry(kt_engine* e, uint32_t* d_out, uint32_t* d_k_max);
int emit_keep(kt_engine* e, uint8_t* d_keep);
int emit_graph_kmax(kt_engine* e, const uint32_t* d_src, const uint32_t* d_dst, const uint32_t* d_offsets,
                    uint32_t num_graphs, const uint32_t* d_truss, uint32_t* d_kmax);
// kt_selector.cu: graph statistics and features of the built graph into e->sel_feat (and, with
// d_params, the selector's schedule index into e->sel_choice and that schedule into
// ctrl[kPSched..]); select_schedule runs the attached selector on the device and marks the call's
// schedule as device-chosen (e->sched_on_device; the support count and the peel read it there).
int graph_features(kt_engine* e, const float* d_params);
int select_schedule(kt_engine* e);
// Reads the peel's control block and round log (stream must be drained); reports timeouts.
int finish_stats(kt_engine* e);
// Launches a grid barrier (kt_peel.cu), a barrier of the list peel (kt_lists.cu) or look-backs of a radix pass
// and of a scan (kt_sort.cu) that cannot complete and returns the status they report.
int barrier_timeout_probe(kt_engine* e, uint64_t timeout_ns);
int list_timeout_probe(kt_engine* e, uint64_t timeout_ns);
int look_timeout_probe(kt_engine* e, uint64_t timeout_ns);
// kt_variants.cu: single-k truss by count-and-delete passes (undirected capped counts; tiled
// counts); edge states in e->rnd, so emit_keep applies.  Synchronous (one read per pass).
int ktruss_undirected(kt_engine* e, uint32_t k, bool recount_all, uint32_t group);
int ktruss_tiled(kt_engine* e, uint32_t k, bool recount_all, bool capped);

}  // namespace kt
