// Edge support (triangle count per edge) on the degree-oriented CSR, and the triangle lists.
//
// Replaces count_triangles_kernel of the reference (kernel_ddc.cu:11-54): there one thread
// merges the two out-lists of its edge and issues three atomics per triangle.  Every triangle
// u < v < w (rank order) consists of the edges j = (u,v), x = (u,w) and y = (v,w).  Edge j's tail,
// o_col[j+1 .. o_ptr[u+1]), holds u's neighbours above v; the triangles of j are the tail's members
// that are also in v's row N+(v).  Two ways to test them, chosen by the middle vertex v:
//
// Vertex-centric (k_middle): vertices with at least kMidIn in-edges and a row of kMidOut to kMidRow
// entries.  A block hashes N+(v) into shared memory (column -> row position, in buckets of two, at most a
// quarter to a half full) and streams the tails of a range of v's in-edges (the lower half of v's
// symmetric row) through it: one or two shared-memory probes per entry instead of a binary search.  The
// tails of 256 in-edges at a time are laid end to end and dealt evenly over the warps, however
// different their lengths.  A triangle costs one global atomic (x); y is counted in shared memory and
// added once per item, j once per tail.
//
// Edge-centric (k_support): all other edges, G lanes each (the schedule's support_group).  The
// shorter of tail and row is walked, the longer binary-searched; x and y are credited with global
// atomics, j once per group.
//
// The lists are written by a second pass over the triangles (kFill), in list order of locality: eight-byte
// writes scattered over lists of many GB reach the DRAM in pieces of 32 bytes (R-MAT 20, 1.1 G entries:
// 18.0 ms with the edge-centric pass alone, 24.6 ms with the vertex-centric one; R-MAT 18 3.8 GB written for
// 1.8 GB of entries), so three kernels write what is next to each other:
//   k_middle  the entries of y for vertex-centric v: all in v's row.  An item's part of y's list was
//             claimed by the count, whose addition to `sup` returned where it starts (bases); all
//             other credits go to a second array (supx), so the claimed parts come first in a list;
//   k_rows    the entries of j and x for the same v and rows u of at least kRowMin entries: all in
//             u's row, after the claimed parts;
//   k_support everything else, with a global cursor that fills each list from its end.
//
// k_rows and k_support leave out edges in no triangle: K(2000, 2000) with a clique of 100 vertices, 4.0 M edges of
// which 3.8 M are in none, 2.9 -> 0.75 ms, a batch of 256 graphs 1.82 -> 1.67 (k_middle, which would gather the
// supports, does not: R-MAT 20 0.15 ms).
//
// Measured (GB300): count R-MAT 20 of 15 M edges 7.4 -> 3.5 ms, R-MAT 22 of 60 M edges 44.4 -> 18.6 ms
// (k_support alone -> with k_middle; 3.7 and 23.0 ms with eight lanes to a tail, half of whose stalls were
// waits for the longest tail).  k_middle issues in 84 % of the cycles, L1 70 % (bank conflicts of the
// probes), DRAM 5 %.  A filter of the row's columns in front of the table: 3.9-4.2 ms; lookups queued up
// to full warps, by binary search in the row: 5.0 ms.  Fill 18.0 -> 13.0 ms and 114 -> 76 ms, its DRAM
// writes on R-MAT 18 3.8 -> 2.1 GB.  It is no longer bound by memory (R-MAT 19, 4.5 GB of entries): k_middle
// issues in 48 % of the cycles, between loads (long scoreboard 8.4 of 24 stall cycles an instruction) and the
// barriers of a batch (5.5), with DRAM at 18 % and L2 at 42 % (each entry is a 32-byte sector there); k_rows is
// bound by its instructions, 75 %.

#include <algorithm>

#include "kt_engine.h"
#include "kt_look.cuh"

namespace kt {

namespace {

constexpr int kThreads = 256;

constexpr int kMidThreads = 256;
constexpr uint32_t kMidSlots = 4096;           // hash slots (32 KB with positions and counters: 6 blocks an SM)
constexpr uint32_t kMidRow = kMidSlots / 2;    // longest row that is hashed
// A vertex is vertex-centric with at least kMidIn in-edges and kMidOut row entries: with fewer, a
// table serves too few probes, or the search it replaces is short.  R-MAT 22 count 18.6 ms at 64
// in-edges, 18.7 at 32, 19.3 at 96 (R-MAT 16: 0.18, 0.19, 0.21 ms); a batch of 256 graphs, whose hubs
// have short rows, 1.01 ms at 32 row entries, 1.07 at 16.
constexpr uint32_t kMidIn = 64;
constexpr uint32_t kMidOut = 32;
constexpr uint32_t kMidItemIn = 256;           // in-edges per work item (more for longer rows)
// Rows of kRowMin entries or more get a block of the fill: R-MAT 22 76.4 ms at 128, 79.8 at 64, 79.9
// at 256; whole warps stream their rows (half warps: 81.0).
constexpr uint32_t kRowMin = 128;
// A row is streamed through the table unless it is this many times longer than the tail that could
// be searched in it instead (R-MAT 22: 76.4 ms at 6, 77.6 at 3, 78.8 at 12, 82.0 streaming always).
constexpr uint32_t kRowFactor = 6;
// With support group 0, at least kAllIn in-edges and row entries: R-MAT 20 count 3.65 ms (4.27 from one on, 3.72
// from 8), a batch of shorter rows, Watts-Strogatz of 4 M edges, 0.25 ms (1.69, 0.80), a path of 200,000 vertices
// 0.02 ms (0.48; a block a vertex).
constexpr uint32_t kAllIn = 16;
// A tail much longer than v's row costs more than the search of the row in it: the in-edges whose tail is more
// than kMidTail times v's row stay edge-centric.  K(2000, 2000) with a clique of 100 vertices, count 2.19 ms (2.11
// edge-centric, 5.20 without the limit; 2.21 at 2, 2.40 at 8, 3.79 at 16); R-MAT 20 3.83 (3.88 without).  By vertex id,
// where a hub's row can be any length, R-MAT 20, hubs first, 43.4 ms (46.4, 52.5; 44.7 at 2, 45.3 at 16), ids
// shuffled 32.7 (38.9, 35.5); graphs of fewer than kMidMinById edges and 128 neighbours a vertex, or than 16 a
// vertex, stay edge-centric altogether: R-MAT 15 0.52 ms (0.70), of edge factor 28 1.15 (1.39), R-MAT 18 of edge
// factor 4 0.94 (1.07); above, R-MAT 16 1.22 (1.21), shuffled 1.05 (0.96), G(2000, 0.3) 0.80 (0.45).
constexpr uint32_t kMidTail = 4;
constexpr uint32_t kMidMinById = 3u << 18;
// Smaller graphs are counted edge by edge: the plan and the extra launches cost more than they save
// (R-MAT 14 with 220,000 edges counts in 0.05 ms).
constexpr uint32_t kMidMinEdges = 1u << 18;
constexpr uint32_t kPruneMin = 1u << 19, kPruneEarly = 1u << 20;  // edges (see recount_pruned)
constexpr uint32_t kEmpty = 0xffffffffu;
// words of a plan (kMidPlan, kPrunePlan), zero since the build: items, bases, count cursor, fill cursor
constexpr uint32_t kPlanBases = 1, kPlanCursor = 2;

struct Graph {
    const uint32_t* ctrl;
    const uint32_t* __restrict__ o_ptr;
    const uint32_t* __restrict__ o_col;
    const uint32_t* __restrict__ e_src;
    const uint32_t* __restrict__ s_ptr;
    const uint32_t* __restrict__ s_split;
    const uint32_t* __restrict__ s_col;
    const uint32_t* __restrict__ s_eid;
    uint32_t n, m;
    uint32_t mid_in;   // vertices with this many in-edges are vertex-centric (0: none) ...
    uint32_t mid_out;  // ... if their row has this many entries
    uint32_t plan;     // first control word of the plan
    // The edges left by a first round (recount_pruned): o_ptr, o_col and e_src are theirs, m is the
    // edges of the whole graph, which s_ptr .. s_eid describe; new_id[j] is what became of edge j.
    uint32_t percent;
    const uint32_t* __restrict__ new_id;
};

// The round and level logs (kt_peel.cu).
struct PeelLog {
    uint32_t *round_size, *round_level, *round_ns, cap_rounds;
    uint32_t *level_k, *level_alive, *level_ns, *level_front, cap_levels;
};

// Where counts go, and what the fill reads.
struct Credits {
    uint32_t* sup;                      // count: credits of y by vertex-centric items, claimed
    uint32_t* supx;                     // count: all other credits
    uint32_t* ycount;                   // fill: length of the part of each list that the items claimed
    uint32_t* bases;                    // per item and row position: start of y's entries
    const uint64_t* __restrict__ tptr;  // fill: list starts
    unsigned long long* cur;            // fill: end of the free part of each list
    uint2* tri;                         // fill: the lists
};

__device__ __forceinline__ bool vertex_centric(const Graph& g, uint32_t v, uint32_t row) {
    return g.mid_in != 0 && row >= g.mid_out && row <= kMidRow && g.s_split[v] - g.s_ptr[v] >= g.mid_in;
}

constexpr uint32_t kGone = 0x80000000u;  // in new_id: removed (the low bits number the edges left before it)

// Nothing to do: the input was refused, or the first round is the peel's (kPruned).
template <bool kPruned>
__device__ __forceinline__ bool skip(const Graph& g) {
    return failed(g.ctrl) || (kPruned && !pruned_first(g.ctrl, g.m, g.percent));
}

// Whether the triangles of an in-edge of v are found at v: its tail has `tail` entries.
__device__ __forceinline__ bool at_middle(const Graph& g, uint32_t v, uint32_t row, uint32_t tail) {
    return vertex_centric(g, v, row) && tail <= kMidTail * row;  // (rows of at most kMidRow)
}

// Rows long enough for a row block of the fill (k_rows).
__device__ __forceinline__ bool row_block(uint32_t row) { return row >= kRowMin && row <= kMidRow; }

template <int G, bool kFill, bool kPruned = false>
__device__ __forceinline__ void edge_body(const Graph& g, const Credits& c) {
    const uint32_t lane = lane_id();
    const uint32_t glane = lane & (G - 1);
    const uint32_t gmask = (G == 32) ? kFullMask : (((1u << G) - 1) << (lane & ~(uint32_t)(G - 1)));
    const uint64_t gid = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) / G;
    const uint64_t ngroups = ((uint64_t)gridDim.x * blockDim.x) / G;
    const uint32_t m = kPruned ? __ldcg(g.ctrl + kPruneLeft) : g.m;
    for (uint64_t j64 = gid; j64 < m; j64 += ngroups) {
        const uint32_t j = (uint32_t)j64;
        const uint32_t u = g.e_src[j], v = g.o_col[j];
        const uint32_t a0 = j + 1, a1 = g.o_ptr[u + 1];
        const uint32_t b0 = g.o_ptr[v], b1 = g.o_ptr[v + 1];
        const uint32_t na = a1 - a0, nb = b1 - b0;
        if (!na || !nb || (kFill && !c.sup[j])) continue;  // the same for the whole group
        const bool middle = at_middle(g, v, nb, na);
        if (middle && (!kFill || row_block(a1 - g.o_ptr[u]))) continue;
        uint32_t cnt = 0;
        // iterate the shorter list, search the longer
        const bool iter_a = na <= nb;
        const uint32_t i0 = iter_a ? a0 : b0, ni = iter_a ? na : nb;
        const uint32_t s0 = iter_a ? b0 : a0, ns = iter_a ? nb : na;
        for (uint32_t t0 = 0; t0 < ni; t0 += G) {
            const uint32_t t = t0 + glane;
            bool hit = false;
            uint32_t x = 0, y = 0;
            if (t < ni) {
                x = i0 + t;
                const uint32_t w = g.o_col[x];
                const uint32_t idx = lower_bound_u32(g.o_col + s0, ns, w);
                y = s0 + idx;
                hit = idx < ns && g.o_col[y] == w;
            }
            if (!kFill) {
                if (hit) {
                    ++cnt;
                    atomicAdd(&c.supx[x], 1u);
                    atomicAdd(&c.supx[y], 1u);
                }
            } else {
                const uint32_t hits = __ballot_sync(gmask, hit) & gmask;
                if (hits) {
                    const uint32_t first = __ffs(hits) - 1;
                    unsigned long long own = 0;
                    if (lane == first) own = atomicAdd(&c.cur[j], 0ull - __popc(hits));
                    own = __shfl_sync(gmask, own, first);
                    if (hit) {
                        // walked and searched list in (u's row, v's row) or the other way round
                        const uint32_t ex = iter_a ? x : y, ey = iter_a ? y : x;
                        c.tri[own - 1 - __popc(hits & lanemask_lt())] = make_uint2(x, y);
                        c.tri[atomicAdd(&c.cur[ex], ~0ull) - 1] = make_uint2(j, ey);
                        if (!middle) c.tri[atomicAdd(&c.cur[ey], ~0ull) - 1] = make_uint2(j, ex);
                    }
                }
            }
        }
        if (!kFill) {
            __syncwarp(gmask);
#pragma unroll
            for (int o = G / 2; o > 0; o >>= 1) cnt += __shfl_xor_sync(gmask, cnt, o);
            if (glane == 0 && cnt) atomicAdd(&c.supx[j], cnt);
        }
    }
}

template <int G, bool kFill, bool kPruned = false>
__global__ void __launch_bounds__(kThreads) k_support(Graph g, Credits c) {
    after_previous();
    if (skip<kPruned>(g)) return;
    edge_body<G, kFill, kPruned>(g, c);
}

// The same count with the lane group read from the control block, where the learned selector's
// inference kernel wrote its choice: the schedule is chosen on the device, with no host read.
__global__ void __launch_bounds__(kThreads) k_support_chosen(Graph g, Credits c, const uint32_t* __restrict__ sched) {
    if (failed(g.ctrl)) return;
    switch (sched[0]) {
        case 4: edge_body<4, false>(g, c); break;
        case 16: edge_body<16, false>(g, c); break;
        case 32: edge_body<32, false>(g, c); break;
        default: edge_body<8, false>(g, c); break;
    }
}

// Work items {v, first in-edge, end in-edge, first word of bases} of the vertex-centric vertices.
// An item takes at least as many in-edges as v's row has entries, so all items together have at
// most 2m words of bases.  Also lists the rows of the fill's row blocks.
template <bool kPruned>
__global__ void k_middle_plan(Graph g, uint4* __restrict__ items, uint32_t* __restrict__ rows,
                              uint32_t* __restrict__ ctrl) {
    if (skip<kPruned>(g)) return;
    const uint32_t v = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t row = v < g.n ? g.o_ptr[v + 1] - g.o_ptr[v] : 0u;
    const uint32_t listed = kPruned ? 0u : __ballot_sync(kFullMask, row_block(row));
    if (listed) {
        uint32_t base = 0;
        if (lane_id() == 0) base = atomicAdd(ctrl + kRowItems, __popc(listed));
        base = __shfl_sync(kFullMask, base, 0);
        if (row_block(row)) rows[base + __popc(listed & lanemask_lt())] = v;
    }
    if (v >= g.n) return;
    const uint32_t a = g.s_ptr[v], indeg = g.s_split[v] - a;
    if (!row || !indeg || !vertex_centric(g, v, row)) return;
    const uint32_t step = max(kMidItemIn, (row + kMidItemIn - 1) / kMidItemIn * kMidItemIn);
    const uint32_t count = (indeg + step - 1) / step;
    const uint32_t i0 = atomicAdd(ctrl + g.plan, count), w0 = atomicAdd(ctrl + g.plan + kPlanBases, count * row);
    for (uint32_t i = 0; i < count; ++i)
        items[i0 + i] = make_uint4(v, a + i * step, a + min(indeg, (i + 1) * step), w0 + i * row);
}

template <bool kFill, bool kPruned = false>
__global__ void __launch_bounds__(kMidThreads, 1536 / kMidThreads) k_middle(Graph g, Credits c, const uint4* __restrict__ items,
                                                           uint32_t* __restrict__ ctrl) {
    __shared__ uint2 key[kMidSlots / 2];  // buckets of two, filled in order
    __shared__ uint16_t at[kMidSlots];
    __shared__ uint32_t cnt[kMidRow];  // count: triangles of y; fill: next list entry of y
    __shared__ uint32_t s_item;
    // a batch of in-edges, one a thread: tail entries before its tail, its tail's start less these, and
    // its triangles (count) or edge id (fill)
    __shared__ uint32_t before[kMidThreads + 1], start[kMidThreads], tag[kMidThreads], wsum[kMidThreads / 32];
    const uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
    const uint32_t n_items = skip<kPruned>(g) ? 0u : ctrl[g.plan];
    for (;;) {
        if (threadIdx.x == 0) s_item = atomicAdd(ctrl + g.plan + kPlanCursor + (kFill ? 1 : 0), 1u);
        __syncthreads();
        const uint32_t it = s_item;
        if (it >= n_items) return;
        const uint4 d = items[it];
        const uint32_t r0 = g.o_ptr[d.x], row = g.o_ptr[d.x + 1] - r0;
        uint32_t bits = 5;  // at least four slots an entry, as far as the table goes
        while (bits < 11 && (1u << bits) < 2 * row) ++bits;
        const uint32_t mask = (1u << bits) - 1, shift = 32 - bits;
        for (uint32_t i = threadIdx.x; i <= mask; i += kMidThreads) key[i] = make_uint2(kEmpty, kEmpty);
        // the fill counts list entries from the start of the row's lists (or, should they hold 2^32
        // entries or more, from the start of each list)
        uint64_t row_at = 0;
        bool wide = false;
        if (kFill) {
            row_at = c.tptr[r0];
            wide = c.tptr[r0 + row] - row_at >= 0xffffffffull;
        }
        for (uint32_t i = threadIdx.x; i < row; i += kMidThreads)
            cnt[i] = !kFill ? 0u : c.bases[d.w + i] + (wide ? 0u : (uint32_t)(c.tptr[r0 + i] - row_at));
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < row; i += kMidThreads) {
            const uint32_t w = g.o_col[r0 + i];
            uint32_t h = (w * 0x9E3779B1u) >> shift;
            for (;; h = (h + 1) & mask) {
                if (atomicCAS(&key[h].x, kEmpty, w) == kEmpty) {
                    at[2 * h] = (uint16_t)i;
                    break;
                }
                if (atomicCAS(&key[h].y, kEmpty, w) == kEmpty) {
                    at[2 * h + 1] = (uint16_t)i;
                    break;
                }
            }
        }
        for (uint32_t p0 = d.y; p0 < d.z; p0 += kMidThreads) {
            const uint32_t p = p0 + threadIdx.x;
            uint32_t j = 0, len = 0;
            if (p < d.z) {
                j = g.s_eid[p];
                if (kPruned) j = g.new_id[j];
                if (!kPruned || !(j & kGone)) len = g.o_ptr[g.s_col[p] + 1] - (j + 1);  // (else no tail)
                if (len > kMidTail * row) len = 0;  // k_support's
            }
            uint32_t incl = len;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t t = __shfl_up_sync(kFullMask, incl, o);
                if (lane >= (uint32_t)o) incl += t;
            }
            if (lane == 31) wsum[warp] = incl;
            __syncthreads();  // (for the table too)
            uint32_t total = 0, at0 = incl - len;
#pragma unroll
            for (int q = 0; q < kMidThreads / 32; ++q) {
                const uint32_t t = wsum[q];
                at0 += q < (int)warp ? t : 0u;
                total += t;
            }
            before[threadIdx.x] = at0;
            start[threadIdx.x] = j + 1 - at0;
            tag[threadIdx.x] = kFill ? j : 0u;
            if (threadIdx.x == 0) before[kMidThreads] = total;
            __syncthreads();
            // the warps share the entries of all tails evenly
            const uint32_t share = (total + kMidThreads - 1) / kMidThreads * 32;
            const uint32_t end = min(total, (warp + 1) * share);
            uint32_t t = warp * share + lane;
            if (t < end) {
                uint32_t own = 0;  // the last tail that starts at or before entry t
#pragma unroll
                for (uint32_t b = kMidThreads / 2; b > 0; b >>= 1)
                    if (before[own + b] <= t) own += b;
                uint32_t next = before[own + 1], off = start[own], found = 0;
                uint32_t j_own = kFill ? tag[own] : 0u;
                uint32_t x = t + off, w = g.o_col[x];
                while (t < end) {
                    const uint32_t x_now = x, w_now = w, j_now = j_own;
                    uint32_t* const tag_now = &tag[own];
                    const bool moves = t + 32 >= next;
                    t += 32;
                    if (t < end) {
                        if (moves) {
                            do next = before[++own + 1];
                            while (t >= next);
                            off = start[own];
                            if (kFill) j_own = tag[own];
                        }
                        x = t + off;
                        w = g.o_col[x];
                    }
                    uint32_t h = (w_now * 0x9E3779B1u) >> shift;
                    uint2 k = key[h];
                    while (k.x != w_now && k.y != w_now && k.y != kEmpty) k = key[h = (h + 1) & mask];
                    if (k.x == w_now || k.y == w_now) {
                        const uint32_t pos = at[2 * h + (k.y == w_now)];
                        if (!kFill) {
                            ++found;
                            atomicAdd(&cnt[pos], 1u);
                            atomicAdd(&c.supx[x_now], 1u);
                        } else {
                            c.tri[(wide ? __ldg(c.tptr + r0 + pos) : row_at) + atomicAdd(&cnt[pos], 1u)] =
                                make_uint2(j_now, x_now);
                        }
                    }
                    if (!kFill && moves && found) {
                        atomicAdd(tag_now, found);
                        found = 0;
                    }
                }
                if (!kFill && found) atomicAdd(&tag[own], found);
            }
            __syncthreads();
            if (!kFill && tag[threadIdx.x]) atomicAdd(&c.supx[j], tag[threadIdx.x]);
        }
        if (!kFill)
            for (uint32_t i = threadIdx.x; i < row; i += kMidThreads)
                if (cnt[i]) {
                    if (kPruned) atomicAdd(&c.supx[r0 + i], cnt[i]);
                    else c.bases[d.w + i] = atomicAdd(&c.sup[r0 + i], cnt[i]);
                }
    }
}

// The fill's row blocks: for the rows u of kRowMin entries or more, the list entries of j and x of
// the triangles whose middle vertex is vertex-centric (their y entries are k_middle's).  Both lie
// in u's own row, so a block with the row hashed into shared memory and a cursor per row position
// writes them without global atomics, into lists that are next to each other.  Warps stream the rows
// N+(v) through the table - or, where v's row is much longer than u's tail above v, search the tail's
// entries in it.
// Bound: instructions, issue active 75 % (R-MAT 19; DRAM 17 %, L2 36 %).
__global__ void __launch_bounds__(kMidThreads, 6) k_rows(Graph g, Credits c, const uint32_t* __restrict__ rows,
                                                         uint32_t* __restrict__ ctrl) {
    __shared__ uint2 key[kMidSlots / 2];  // (as in k_middle)
    __shared__ uint16_t at[kMidSlots];
    __shared__ uint32_t cur[kMidRow];  // next list entry, from the start of the row's lists
    __shared__ uint32_t s_row;
    constexpr uint32_t kWarps = kMidThreads / 32;
    const uint32_t lane = lane_id(), warp = threadIdx.x >> 5, n_rows = failed(ctrl) ? 0u : ctrl[kRowItems];
    for (;;) {
        if (threadIdx.x == 0) {
            const uint32_t t = atomicAdd(ctrl + kRowCursor, 1u);
            s_row = t < n_rows ? rows[t] : kEmpty;
        }
        __syncthreads();
        const uint32_t u = s_row;
        if (u == kEmpty) return;
        const uint32_t r0 = g.o_ptr[u], row = g.o_ptr[u + 1] - r0;
        uint32_t bits = 5;
        while (bits < 11 && (1u << bits) < 2 * row) ++bits;
        const uint32_t mask = (1u << bits) - 1, shift = 32 - bits;
        const uint64_t row_at = c.tptr[r0];
        const bool wide = c.tptr[r0 + row] - row_at >= 0xffffffffull;
        for (uint32_t i = threadIdx.x; i <= mask; i += kMidThreads) key[i] = make_uint2(kEmpty, kEmpty);
        for (uint32_t i = threadIdx.x; i < row; i += kMidThreads)
            cur[i] = c.ycount[r0 + i] + (wide ? 0u : (uint32_t)(c.tptr[r0 + i] - row_at));
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < row; i += kMidThreads) {
            const uint32_t w = g.o_col[r0 + i];
            uint32_t h = (w * 0x9E3779B1u) >> shift;
            for (;; h = (h + 1) & mask) {
                if (atomicCAS(&key[h].x, kEmpty, w) == kEmpty) {
                    at[2 * h] = (uint16_t)i;
                    break;
                }
                if (atomicCAS(&key[h].y, kEmpty, w) == kEmpty) {
                    at[2 * h + 1] = (uint16_t)i;
                    break;
                }
            }
        }
        __syncthreads();
        // positions warp, warp + kWarps, ...: the lanes load the rows of the next 32 together
        for (uint32_t i0 = warp; i0 + 1 < row; i0 += kWarps * 32) {
            uint32_t lb0 = 0, lb1 = 0;
            const uint32_t mine = i0 + lane * kWarps;
            if (mine + 1 < row) {
                const uint32_t v = g.o_col[r0 + mine];
                lb0 = g.o_ptr[v];
                lb1 = g.o_ptr[v + 1];
                if (lb0 != lb1 && (!at_middle(g, v, lb1 - lb0, row - 1 - mine) || !c.sup[r0 + mine])) lb1 = lb0;
            }
            for (int l = 0; l < 32; ++l) {
                const uint32_t i = i0 + l * kWarps, tail = row - 1 - i;
                const uint32_t b0 = __shfl_sync(kFullMask, lb0, l), b1 = __shfl_sync(kFullMask, lb1, l);
                if (b0 == b1) continue;
                const bool stream = b1 - b0 <= kRowFactor * tail;
                const uint32_t p0 = stream ? b0 : r0 + i + 1, p1 = stream ? b1 : r0 + row;
                uint32_t w_next = p0 + lane < p1 ? g.o_col[p0 + lane] : kEmpty;
                for (uint32_t q0 = p0; q0 < p1; q0 += 32) {
                    const uint32_t p = q0 + lane, w = w_next;
                    w_next = p + 32 < p1 ? g.o_col[p + 32] : kEmpty;
                    uint32_t pos = kEmpty, y = p;  // x = r0 + pos
                    if (w != kEmpty) {
                        if (stream) {
                            uint32_t h = (w * 0x9E3779B1u) >> shift;
                            uint2 k = key[h];
                            while (k.x != w && k.y != w && k.y != kEmpty) k = key[h = (h + 1) & mask];
                            if (k.x == w || k.y == w) pos = at[2 * h + (k.y == w)];
                        } else {
                            y = b0 + lower_bound_u32(g.o_col + b0, b1 - b0, w);
                            if (y < b1 && g.o_col[y] == w) pos = p - r0;
                        }
                    }
                    const uint32_t hits = __ballot_sync(kFullMask, pos != kEmpty);
                    if (hits) {
                        const uint32_t first = __ffs(hits) - 1;
                        uint32_t own = 0;
                        if (lane == first) own = atomicAdd(&cur[i], __popc(hits));
                        own = __shfl_sync(kFullMask, own, first);
                        if (pos != kEmpty) {
                            c.tri[(wide ? __ldg(c.tptr + r0 + i) : row_at) + own + __popc(hits & lanemask_lt())] =
                                make_uint2(r0 + pos, y);
                            c.tri[(wide ? __ldg(c.tptr + r0 + pos) : row_at) + atomicAdd(&cur[pos], 1u)] =
                                make_uint2(r0 + i, y);
                        }
                    }
                }
            }
        }
        __syncthreads();
    }
}

// sup += supx, what it was into ycount, the sum of all supports (three per triangle), and the number of
// supports below `limit` (a single-k call's first frontier).
template <bool kChained>
__global__ void k_merge_support(uint32_t* __restrict__ sup, const uint32_t* __restrict__ supx,
                                uint32_t* __restrict__ ycount, uint32_t m, uint32_t limit, uint32_t* __restrict__ ctrl) {
    if (kChained) after_previous(sup, supx, ycount, ctrl);
    if (failed(ctrl)) return;
    uint64_t s = 0;
    uint32_t low = 0;
    for (uint64_t j = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; j < m; j += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t y = sup[j], v = y + supx[j];
        ycount[j] = y;
        sup[j] = v;
        s += v;
        low += v < limit;
    }
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(kFullMask, s, o);
    if (lane_id() == 0 && s)
        atomicAdd(reinterpret_cast<unsigned long long*>(ctrl + kCtrlTriLo), (unsigned long long)s);
    low = __reduce_add_sync(kFullMask, low);
    if (lane_id() == 0 && low) atomicAdd(ctrl + kPruneFront, low);
}

// The triangle 3-truss from the counted supports, in one pass: an edge in no triangle goes, which takes
// no other edge's triangles, so there is one round at most.  rnd (it holds the second half of the
// credits, supx) gets 1 for the edges that go and 0 for the others.  The last block writes the statistics
// that the peel kernel would have left.
// Bound: memory, 12 bytes an edge, and for small graphs its own latency.  R-MAT 20 (15 M edges)
// 0.024 ms, 7.4 TB/s as the supports lie in L2 (merging the credits and the peel kernel's one round: 0.70 ms).
template <bool kChained>
__global__ void __launch_bounds__(kThreads) k_truss3(uint32_t* __restrict__ sup, uint32_t* __restrict__ rnd,
                                                     uint32_t m, PeelLog log, uint32_t* __restrict__ ctrl) {
    if (kChained) after_previous(sup, rnd, ctrl);
    __shared__ unsigned long long s_sum;
    __shared__ uint32_t s_low;
    if (__syncthreads_or(failed(ctrl))) return;
    if (threadIdx.x == 0) s_sum = s_low = 0;
    __syncthreads();
    uint64_t s = 0;
    uint32_t low = 0;
    const uint64_t step = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t q = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; 4 * q < m; q += step) {
        if (4 * q + 4 <= m) {
            uint4 a = reinterpret_cast<uint4*>(sup)[q];
            const uint4 b = reinterpret_cast<uint4*>(rnd)[q];
            a.x += b.x, a.y += b.y, a.z += b.z, a.w += b.w;
            const uint4 r = make_uint4(a.x == 0, a.y == 0, a.z == 0, a.w == 0);
            reinterpret_cast<uint4*>(rnd)[q] = r;
            s += (uint64_t)a.x + a.y + a.z + a.w;
            low += r.x + r.y + r.z + r.w;
        } else {
            for (uint64_t j = 4 * q; j < m; ++j) {
                const uint32_t v = sup[j] + rnd[j];
                rnd[j] = v == 0;
                s += v;
                low += v == 0;
            }
        }
    }
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(kFullMask, s, o);
    low = __reduce_add_sync(kFullMask, low);
    if (lane_id() == 0) {
        atomicAdd(&s_sum, (unsigned long long)s);
        atomicAdd(&s_low, low);
    }
    __syncthreads();
    if (threadIdx.x != 0) return;
    atomicAdd(reinterpret_cast<unsigned long long*>(ctrl + kCtrlTriLo), s_sum);
    atomicAdd(ctrl + kPruneFront, s_low);
    __threadfence();
    if (atomicAdd(ctrl + kPruneLeft, 1u) != gridDim.x - 1) return;
    const uint32_t front = atomicAdd(ctrl + kPruneFront, 0u);
    ctrl[kPRounds] = front != 0;
    ctrl[kPLevels] = 1;
    if (front && log.cap_rounds > 1) {
        log.round_size[1] = front;
        log.round_level[1] = 3;
        log.round_ns[1] = 0;
    }
    if (log.cap_levels) {
        log.level_k[0] = 3;
        log.level_alive[0] = m;
        log.level_ns[0] = 0;
        log.level_front[0] = front;
    }
}

// A single-k call's first round that removes many of the edges (pruned_first): the edges left are
// numbered in order (new_id) and their oriented CSR is written next to the old one, so that the
// kernels of the support count can count them again ...
__global__ void __launch_bounds__(kFlagThreads) k_prune(Graph whole, const uint32_t* __restrict__ sup, uint32_t limit,
                                                        uint32_t percent, uint32_t* __restrict__ new_id,
                                                        uint32_t* __restrict__ o_col, uint32_t* __restrict__ e_src,
                                                        uint32_t* __restrict__ count, Look L) {
    __shared__ FlagSmem S;
    if (__syncthreads_or(failed(L.ctrl) || !pruned_first(L.ctrl, whole.m, percent))) return;
    const uint32_t tile = look_tile(L, &S.tile);
    if (tile == kNoTile) return;
    const uint64_t j0 = (uint64_t)tile * kFlagTile + threadIdx.x;
    const uint32_t warp = threadIdx.x >> 5, m = whole.m;
    if (j0 == 0) *reinterpret_cast<unsigned long long*>(L.ctrl + kPruneT0) = global_ns();
    uint32_t left = 0;  // bit s: the edge of step s is left
#pragma unroll
    for (uint32_t s = 0; s < kFlagSteps; ++s) {
        const uint64_t j = j0 + s * kFlagThreads;
        left |= (uint32_t)(j < m && sup[j] >= limit) << s;
    }
#pragma unroll
    for (uint32_t s = 0; s < kFlagSteps; ++s) {
        const uint32_t b = __ballot_sync(kFullMask, left >> s & 1u);
        if (lane_id() == 0) S.before[s * kFlagWarps + warp] = __popc(b);
    }
    __syncthreads();
    flag_sums(S, L, tile);
#pragma unroll
    for (uint32_t s = 0; s < kFlagSteps; ++s) {
        const uint64_t j = j0 + s * kFlagThreads;
        const bool f = left >> s & 1u;
        const uint32_t id = (uint32_t)S.prefix + S.before[s * kFlagWarps + warp] +
                            __popc(__ballot_sync(kFullMask, f) & lanemask_lt());
        if (j >= m) continue;
        new_id[j] = f ? id : id | kGone;
        if (f) {
            o_col[id] = whole.o_col[j];
            e_src[id] = whole.e_src[j];
            count[id] = 0;
        }
        if (j == m - 1) L.ctrl[kPruneLeft] = id + f;
    }
}

// ... and the starts of their rows.
__global__ void k_prune_rows(Graph whole, uint32_t percent, const uint32_t* __restrict__ new_id,
                             uint32_t* __restrict__ o_ptr) {
    const uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r > whole.n || failed(whole.ctrl) || !pruned_first(whole.ctrl, whole.m, percent)) return;
    const uint32_t j = whole.o_ptr[r];
    o_ptr[r] = j < whole.m ? new_id[j] & ~kGone : whole.ctrl[kPruneLeft];
}

Graph graph_of(const kt_engine* e) {
    // the choice must be the same in the count and in the fill of one call
    const bool hash_all = !e->sched_on_device && e->sched.support_group == 0;
    const uint64_t m = e->m, n = e->n;
    const bool pays = m >= kMidMinEdges && (!e->by_index || (m >= 8 * n && (m >= kMidMinById || m >= 64 * n)));
    const uint32_t mid_in = hash_all ? kAllIn : pays ? kMidIn : 0u, mid_out = hash_all ? kAllIn : kMidOut;
    return Graph{e->ctrl, e->o_ptr, e->o_col, e->e_src, e->s_ptr, e->s_split, e->s_col, e->s_eid, e->n, e->m, mid_in, mid_out,
                 kMidPlan, 0, nullptr};
}

// The items lie in the first chunk buffer, the claims in the second, the rows in the first queue:
// all free until the peel.
uint4* items_of(const kt_engine* e) { return e->chunks0; }
uint32_t* rows_of(const kt_engine* e) { return e->q0; }
Credits credits_of(const kt_engine* e) {
    return Credits{e->sup, e->rnd, e->tr, reinterpret_cast<uint32_t*>(e->chunks1), nullptr, nullptr, nullptr};
}

template <bool kFill, bool kPruned = false>
int launch_middle(kt_engine* e, const Graph& g, const Credits& c) {
    int rc, per_sm = 0;
    if ((rc = check_cuda(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_middle<kFill, kPruned>, kMidThreads, 0),
                         "occupancy of k_middle")))
        return rc;
    if (per_sm < 1) return fail(KT_ERR_CUDA, "k_middle cannot be resident");
    k_middle<kFill, kPruned><<<(uint32_t)(e->num_sms * per_sm), kMidThreads, 0, e->stream>>>(g, c, items_of(e), e->ctrl);
    count_launch(e);
    return check_launch(e, "k_middle");
}

uint32_t edge_blocks(const kt_engine* e, uint32_t G) {
    return (uint32_t)std::min<uint64_t>(((uint64_t)e->m * G + kThreads - 1) / kThreads, (uint64_t)e->num_sms * 16);
}

}  // namespace

int count_support(kt_engine* e) {
    if (e->m == 0) return KT_OK;
    int rc;
    const Graph g = graph_of(e);
    const Credits c = credits_of(e);  // cleared by the build
    if (g.mid_in) {
        k_middle_plan<false><<<(e->n + kThreads - 1) / kThreads, kThreads, 0, e->stream>>>(g, items_of(e), rows_of(e),
                                                                                    e->ctrl);
        count_launch(e);
        if ((rc = check_launch(e, "k_middle_plan")) || (rc = launch_middle<false>(e, g, c))) return rc;
    }
    if (e->sched_on_device) {
        // any group the selector may choose (4, 8 or 16 lanes per edge) fits this grid
        k_support_chosen<<<edge_blocks(e, 16), kThreads, 0, e->stream>>>(g, c, e->ctrl + kPSched);
        count_launch(e);
        return check_launch(e, "k_support_chosen");
    }
    const uint32_t G = e->sched.support_group ? e->sched.support_group : 8;
    const uint32_t blocks = edge_blocks(e, G);
    switch (G) {
        case 4: rc = launch_chained(e, "k_support", k_support<4, false>, blocks, kThreads, 0, g, c); break;
        case 16: rc = launch_chained(e, "k_support", k_support<16, false>, blocks, kThreads, 0, g, c); break;
        case 32: rc = launch_chained(e, "k_support", k_support<32, false>, blocks, kThreads, 0, g, c); break;
        default: rc = launch_chained(e, "k_support", k_support<8, false>, blocks, kThreads, 0, g, c); break;
    }
    return rc;
}

int merge_support(kt_engine* e, uint32_t limit) {
    return launch_chained(e, "k_merge_support", e->chained ? k_merge_support<true> : k_merge_support<false>,
                          (uint32_t)e->num_sms * 4, kThreads, 0, e->sup, e->rnd, e->tr, e->m, limit, e->ctrl);
}

int truss3(kt_engine* e) {
    const PeelLog log{e->round_size, e->round_level, e->round_ns, e->cap_rounds,
                      e->level_k, e->level_alive, e->level_ns, e->level_front, e->cap_levels};
    const uint32_t blocks =
        (uint32_t)std::min<uint64_t>(((uint64_t)e->m + 4 * kThreads - 1) / (4 * kThreads), (uint64_t)e->num_sms * 8);
    return launch_chained(e, "k_truss3", e->chained ? k_truss3<true> : k_truss3<false>, blocks, kThreads, 0, e->sup,
                          e->rnd, e->m, log, e->ctrl);
}

// The first round of a single-k call whose frontier (supports below `limit`) is a recount round: the
// peel kernel's recount searches every surviving edge's rows among the removed entries; here the edges
// left are packed and counted like a graph of their own.  All kernels return at once when the
// frontier is smaller.
// Measured: R-MAT 18 (3.7 M edges), k = 32, the first round 2.4 ms walked, 2.0 recounted by the peel
// kernel, 0.53 here (the call 4.81 -> 2.88 ms); R-MAT 20, k = 32: 10.8 -> 2.4 ms; G(40000) with 6 M edges,
// k = 5: 16.7 walked, 0.86 here.
// The line lies at 7/10 of the schedule's recount share, as this recount costs less than the peel's: a
// frontier of 30-32 % of an R-MAT graph's edges takes 3.9 ms walked and 3.7 here (15 M edges), 0.80 and
// 0.81 (3.7 M); 26 %: 2.8 and 3.9, 0.55 and 0.88; 41 %: 7.5 and 3.5, 1.2 and 0.73.  Below 2^20 edges it is the
// share itself (400,000 edges: 40 % 0.10 and 0.14 ms, 48 % 0.135 and 0.125), and below 2^19 the peel's: the five
// launches that return cost a call 0.02 ms, 4 % of one on 400,000 edges whose frontier is smaller.  By vertex id,
// where the count itself costs ten times as much, it is the share too: R-MAT 21 of 12 M edges, k = 5, 48 % 5.4 ms
// walked and 12.5 here; R-MAT 20, k = 20, 53 % 25.7 walked, 58.6 recounted by the peel kernel, 20.9 here.
// The peel finds new ids in e->tr and the new counts in key_b (3 m words on); the sort keys are free
// after the build.
int recount_pruned(kt_engine* e, uint32_t limit, uint32_t percent, PrunedCount* out) {
    *out = PrunedCount{0, nullptr, nullptr};
    if (percent == 0 || e->m < kPruneMin || e->sched_on_device) return KT_OK;
    if (e->m >= kPruneEarly && !e->by_index) percent = std::max(1u, percent * 7 / 10);
    int rc;
    const Graph whole = graph_of(e);
    uint32_t* o_ptr = reinterpret_cast<uint32_t*>(e->key_a);  // n + 1 words of 2 max(n, entries)
    uint32_t* o_col = reinterpret_cast<uint32_t*>(e->key_b);  // 3 m words of 4 m
    uint32_t *e_src = o_col + e->m, *count = e_src + e->m, *new_id = e->tr;
    const uint32_t tiles = (e->m + kFlagTile - 1) / kFlagTile;
    k_prune<<<tiles, kFlagThreads, 0, e->stream>>>(whole, e->sup, limit, percent, new_id, o_col, e_src, count,
                                                   next_look(e));
    count_launch(e);
    if ((rc = check_launch(e, "k_prune"))) return rc;
    k_prune_rows<<<(uint32_t)(((uint64_t)e->n + kThreads) / kThreads), kThreads, 0, e->stream>>>(whole, percent, new_id, o_ptr);
    count_launch(e);
    if ((rc = check_launch(e, "k_prune_rows"))) return rc;
    Graph g = whole;
    g.o_ptr = o_ptr;
    g.o_col = o_col;
    g.e_src = e_src;
    g.plan = kPrunePlan;
    g.percent = percent;
    g.new_id = new_id;
    Credits c = credits_of(e);
    c.sup = c.supx = count;
    k_middle_plan<true><<<(e->n + kThreads - 1) / kThreads, kThreads, 0, e->stream>>>(g, items_of(e), nullptr, e->ctrl);
    count_launch(e);
    if ((rc = check_launch(e, "k_middle_plan")) || (rc = launch_middle<false, true>(e, g, c))) return rc;
    rc = launch_chained(e, "k_support", k_support<8, false, true>, edge_blocks(e, 8), kThreads, 0, g, c);
    *out = PrunedCount{percent, new_id, count};
    return rc;
}

int fill_lists(kt_engine* e, const uint64_t* tptr, uint64_t* ends) {
    int rc;
    const Graph g = graph_of(e);
    Credits c = credits_of(e);
    c.tptr = tptr;
    c.cur = reinterpret_cast<unsigned long long*>(ends);
    c.tri = e->lists;
    if (g.mid_in) {
        if ((rc = launch_middle<true>(e, g, c))) return rc;
        k_rows<<<(uint32_t)e->num_sms * 6, kMidThreads, 0, e->stream>>>(g, c, rows_of(e), e->ctrl);
        count_launch(e);
        if ((rc = check_launch(e, "k_rows"))) return rc;
    }
    return launch_chained(e, "k_support", k_support<8, true>, edge_blocks(e, 8), kThreads, 0, g, c);
}

}  // namespace kt
