// Device-side graph build: the GB300 replacement for the reference's relabel and COO->CSR
// conversion (sortByDegree graph.cu:152-185, undirected2directedCOO graph.cu:194-237,
// coo2coocsrOnDevice graph.cu:435-478).  The reference sorts vertices on the CPU and sorts
// every adjacency list on the CPU between two PCIe copies; here everything stays in HBM:
//
//   1. degree histogram of the input entries (with id, self-loop checks);
//   2. vertex rank = position in ascending (degree, id) order: a stable radix sort of the ids by the
//      digits of their degrees; ranks, row lengths and row starts in one scan (k_rank_rows);
//   3. every entry becomes the key (rank[src] << vb | rank[dst]) carrying its entry index;
//      one radix sort of the 2m keys yields the symmetric CSR with rows sorted by rank;
//   4. each row splits at its own rank: the part above it is the row of the degree-oriented
//      CSR (edge id = position in the oriented array), numbered by a scan of the sorted entries
//      that writes both CSRs at once (k_csr); the part below gets its edge id by a binary search in
//      the neighbour's oriented row, which also proves the input symmetric (k_entry_eid).
//
// Scans and radix passes are one kernel each (kt_look.cuh).  A small graph's build is bound by its
// launches: G(4096, 16/4095) takes 12 instead of 43, chained, 0.064 ms instead of 0.238; R-MAT 16 0.20 instead of
// 0.42 ms, R-MAT 20 2.53 instead of 3.05 ms (the sort's five passes 1.3 ms of it).
//
// Layout in HBM (n vertices, m undirected edges, all uint32):
//   s_ptr[n+1], s_len[n], s_split[n]   symmetric rows (lower ranks, then higher ranks)
//   s_col[2m], s_eid[2m]               neighbour rank and edge id per symmetric entry
//   o_ptr[n+1], o_col[m], e_src[m]     oriented CSR/COO; edge id = index
//   sorted_entry[2m]                   input entry index of each symmetric entry

#include <algorithm>

#include "kt_engine.h"
#include "kt_look.cuh"

namespace kt {

namespace {

constexpr int kThreads = 256;
constexpr uint32_t kBigRow = 2048;  // rows this long are compacted by a whole block
constexpr uint32_t kTinyRow = 8;    // rows this short are compacted by one thread

inline uint32_t grid_for(uint64_t n, int threads = kThreads) {
    uint64_t b = (n + threads - 1) / threads;
    return (uint32_t)(b == 0 ? 1 : b);
}

// Degree histogram with per-warp aggregation: lanes holding the same source add once (inputs
// listed row by row put a hub's many entries in the same warps).
template <bool kChained>
__global__ void k_degree(const uint32_t* __restrict__ src, const uint32_t* __restrict__ dst, uint64_t entries,
                         uint32_t n, uint32_t* __restrict__ deg, uint32_t* __restrict__ ctrl) {
    if (kChained) after_previous(src, dst, deg, ctrl);
    uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t err = 0, s = 0xffffffffu;
    if (i < entries) {
        s = src[i];
        const uint32_t d = dst[i];
        if (s >= n || d >= n) {
            err = kErrBadVertex;
            s = 0xffffffffu;
        } else if (s == d) {
            err = kErrSelfLoop;
        }
    }
    const uint32_t peers = __match_any_sync(kFullMask, s);
    if (s != 0xffffffffu && lane_id() == (uint32_t)(__ffs(peers) - 1)) atomicAdd(&deg[s], __popc(peers));
    err = __reduce_or_sync(kFullMask, err);
    if (err && lane_id() == 0) atomicOr(&ctrl[kCtrlError], err);
}

// Rank keys (degree << vb | id), listed by id: the sort is stable, so it needs the degree's digits
// only.  A simple graph's degrees are below n; a degree that is not (the input has duplicates and
// will be refused) is sorted by its low digits.
template <bool kChained>
__global__ void __launch_bounds__(kThreads) k_rank_keys(const uint32_t* __restrict__ deg, uint32_t n, unsigned vb,
                                                        unsigned passes, uint64_t* __restrict__ keys,
                                                        uint32_t* __restrict__ counts) {
    if (kChained) after_previous(deg, keys, counts);
    __shared__ uint32_t h[4 * 256];
    digit_counts_clear(h, passes);
    for (uint64_t v0 = (uint64_t)blockIdx.x * kThreads; v0 < n; v0 += (uint64_t)gridDim.x * kThreads) {
        const uint64_t v = v0 + threadIdx.x;
        const uint64_t d = v < n ? deg[v] : 0u;
        if (v < n) keys[v] = d << vb | v;
        digit_counts_add(h, d, v < n, passes);
    }
    digit_counts_flush(h, passes, counts);
}

// Ranks and row starts in one pass over the sorted rank keys: rank[v] = sorted position p (or v, when
// orienting by vertex id, KT_DIRECTED_BY_INDEX, graph.cu:194-207 without the relabel of
// kernel.cu:13-20), row lengths, and their exclusive scan.  Empty rows get their split and oriented
// start here (by degree they come first), the marks of the first long and first not tiny row too.
template <bool kByIndex, bool kChained>
__global__ void __launch_bounds__(kScanThreads) k_rank_rows(const uint64_t* __restrict__ sorted,
                                                            const uint32_t* __restrict__ deg, uint32_t n, unsigned vb,
                                                            uint32_t* __restrict__ rank, uint32_t* __restrict__ s_len,
                                                            uint32_t* __restrict__ s_ptr,
                                                            uint32_t* __restrict__ s_split,
                                                            uint32_t* __restrict__ o_ptr, Look L) {
    if (kChained) after_previous(sorted, deg, rank, s_len, s_ptr, s_split, o_ptr);
    __shared__ uint64_t ws[33], s_prefix;
    __shared__ uint32_t s_tile;
    const uint32_t tile = look_tile(L, &s_tile);
    if (tile == kNoTile) return;
    const uint64_t p0 = (uint64_t)tile * kScanTile + (uint64_t)threadIdx.x * kScanItems;
    const uint64_t mask = (1ull << vb) - 1;
    uint32_t len[kScanItems];
    uint64_t sum = 0;
    uint32_t before = !kByIndex && p0 > 0 && p0 < n ? (uint32_t)(sorted[p0 - 1] >> vb) : 0u;
#pragma unroll
    for (uint32_t i = 0; i < kScanItems; ++i) {
        const uint64_t p = p0 + i;
        len[i] = 0;
        if (p < n) {
            const uint64_t key = kByIndex ? (uint64_t)deg[p] << vb | p : sorted[p];
            len[i] = (uint32_t)(key >> vb);
            rank[key & mask] = (uint32_t)p;
            s_len[p] = len[i];
            if (!kByIndex) {  // (by vertex id rows are in no order of length: no marks)
                if (len[i] >= kBigRow && (p == 0 || before < kBigRow)) L.ctrl[kCtrlBigRow] = (uint32_t)p;
                if (len[i] > kTinyRow && (p == 0 || before <= kTinyRow)) L.ctrl[kCtrlTinyRow] = (uint32_t)p;
                before = len[i];
            }
        }
        sum += len[i];
    }
    uint64_t end;
    uint64_t at = tile_scan<uint64_t>(L, tile, sum, ws, &s_prefix, &end);
#pragma unroll
    for (uint32_t i = 0; i < kScanItems; ++i) {
        const uint64_t p = p0 + i;
        if (p < n) {
            s_ptr[p] = (uint32_t)at;
            if (len[i] == 0) {
                s_split[p] = (uint32_t)at;
                if (!kByIndex) o_ptr[p] = 0;
            }
            if (p == n - 1) {
                s_ptr[n] = (uint32_t)(at + len[i]);
                if (len[i] == 0 && at == 0) o_ptr[n] = 0;  // no entries at all
            }
        }
        at += len[i];
    }
}

// Entry keys (rank of the source << vb | rank of the destination) and their digit counts.  An id >= n
// (already flagged by k_degree; the call fails) is read as vertex 0, so that
// every kernel up to that check indexes inside its arrays.
template <bool kChained>
__global__ void __launch_bounds__(kThreads) k_edge_keys(const uint32_t* __restrict__ src,
                                                        const uint32_t* __restrict__ dst, uint64_t entries, uint32_t n,
                                                        const uint32_t* __restrict__ rank, unsigned vb, unsigned passes,
                                                        uint64_t* __restrict__ keys, uint32_t* __restrict__ counts,
                                                        const uint32_t* __restrict__ ctrl) {
    if (kChained) after_previous(src, dst, rank, keys, counts, ctrl);
    __shared__ uint32_t h[kMaxDigitPasses * 256];
    if (__syncthreads_or(timed_out(ctrl))) return;
    digit_counts_clear(h, passes);
    for (uint64_t i0 = (uint64_t)blockIdx.x * kThreads; i0 < entries; i0 += (uint64_t)gridDim.x * kThreads) {
        const uint64_t i = i0 + threadIdx.x;
        uint64_t key = 0;
        if (i < entries) {
            const uint32_t s = src[i], d = dst[i];
            key = ((uint64_t)rank[s < n ? s : 0] << vb) | rank[d < n ? d : 0];
            keys[i] = key;
        }
        digit_counts_add(h, key, i < entries, passes);
    }
    digit_counts_flush(h, passes, counts);
}

// A tile's sorted keys in shared memory, key[1] on, with the one before it (~0 in front of the first) and the
// one after it (past the last entry: ~0, then 0).  Ends with a __syncthreads.  Kept here over the look-back instead
// of in registers, 2,048 threads fit an SM: k_csr over 30 M keys 0.235 -> 0.195 ms.
__device__ __forceinline__ void stage_keys(uint64_t* key, const uint64_t* __restrict__ keys, uint64_t entries,
                                           uint32_t tile) {
    const uint64_t t0 = (uint64_t)tile * kFlagTile;
#pragma unroll
    for (uint32_t s = 0; s < kFlagSteps; ++s) {
        const uint32_t i = s * kFlagThreads + threadIdx.x;
        key[1 + i] = t0 + i < entries ? keys[t0 + i] : t0 + i == entries ? ~0ull : 0ull;
    }
    if (threadIdx.x == 0) {
        key[0] = t0 > 0 ? keys[t0 - 1] : ~0ull;
        key[1 + kFlagTile] = t0 + kFlagTile < entries ? keys[t0 + kFlagTile] : ~0ull;
    }
    __syncthreads();
}

// One pass over the sorted entry keys builds both CSRs: columns, the duplicate check, where each
// row's higher-rank part starts, and - by a scan of the higher-rank entries - their oriented
// positions, which are the edge ids.  A row's oriented start is the scan at its first entry.
template <bool kChained>
__global__ void __launch_bounds__(kFlagThreads, 4) k_csr(const uint64_t* __restrict__ keys, uint64_t entries, unsigned vb,
                                                      uint32_t n, uint32_t m, uint32_t* __restrict__ s_col,
                                                      uint32_t* __restrict__ s_eid, uint32_t* __restrict__ s_split,
                                                      uint32_t* __restrict__ o_ptr, uint32_t* __restrict__ o_col,
                                                      uint32_t* __restrict__ e_src, uint32_t* __restrict__ fence,
                                                      Look L) {
    if (kChained) after_previous(keys, s_col, s_eid, s_split, o_ptr, o_col, e_src, fence);
    __shared__ FlagSmem S;
    __shared__ uint64_t key[kFlagTile + 2];  // the tile's, one before and one after
    const uint32_t tile = look_tile(L, &S.tile);
    if (tile == kNoTile) return;
    const uint64_t p0 = (uint64_t)tile * kFlagTile + threadIdx.x;
    const uint64_t mask = (1ull << vb) - 1;
    const uint32_t warp = threadIdx.x >> 5;
    uint32_t fwd = 0;  // bit s: the entry of step s is a higher-rank one
    stage_keys(key, keys, entries, tile);
#pragma unroll
    for (uint32_t s = 0; s < kFlagSteps; ++s) {
        const uint64_t k = key[1 + s * kFlagThreads + threadIdx.x];
        const bool f = (uint32_t)(k & mask) > (uint32_t)(k >> vb);
        fwd |= (uint32_t)f << s;
        const uint32_t b = __ballot_sync(kFullMask, f);
        if (lane_id() == 0) S.before[s * kFlagWarps + warp] = __popc(b);
    }
    __syncthreads();
    flag_sums(S, L, tile);
    uint32_t err = 0;
#pragma unroll
    for (uint32_t s = 0; s < kFlagSteps; ++s) {
        const uint64_t p = p0 + s * kFlagThreads;
        const bool f = fwd >> s & 1u;
        const uint64_t j = S.prefix + S.before[s * kFlagWarps + warp] +
                           __popc(__ballot_sync(kFullMask, f) & lanemask_lt());
        if (p < entries) {
            const uint64_t* const at = key + 1 + s * kFlagThreads + threadIdx.x;
            const uint64_t k = *at, prev = at[-1], next = at[1];
            const uint32_t row = (uint32_t)(k >> vb), col = (uint32_t)(k & mask);
            const bool first = p == 0 || (uint32_t)(prev >> vb) != row;
            const bool last = p + 1 == entries || (uint32_t)(next >> vb) != row;
            s_col[p] = col;
            if (p > 0 && prev == k) err |= kErrDuplicate;
            if (first) o_ptr[row] = (uint32_t)(j < m ? j : m);
            if (f) {
                if (first || (uint32_t)(prev & mask) < row) s_split[row] = (uint32_t)p;
                if (j < m) {
                    o_col[j] = col;
                    e_src[j] = row;
                    s_eid[p] = (uint32_t)j;
                    if ((j & 31) == 0) fence[j >> 5] = col;  // every 32nd oriented column
                }
            } else if (last) {
                s_split[row] = (uint32_t)p + 1;
            }
            if (p + 1 == entries) {
                const uint64_t end = j + f;
                o_ptr[n] = (uint32_t)(end < m ? end : m);
                if (end != m) err |= kErrAsymmetric;
            }
        }
    }
    err = __reduce_or_sync(kFullMask, err);
    if (err && lane_id() == 0) atomicOr(&L.ctrl[kCtrlError], err);
}

// Oriented starts of empty rows when orienting by vertex id (by degree they come first, at 0): the
// start of the next row that has entries.
__global__ void k_empty_rows(const uint64_t* __restrict__ keys, uint64_t entries, unsigned vb, uint32_t n,
                             const uint32_t* __restrict__ s_ptr, const uint32_t* __restrict__ s_len,
                             uint32_t* __restrict__ o_ptr, const uint32_t* __restrict__ ctrl) {
    after_previous(keys, s_ptr, s_len, o_ptr, ctrl);
    const uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n || s_len[r] || timed_out(ctrl)) return;
    const uint32_t p = s_ptr[r];
    o_ptr[r] = p < entries ? o_ptr[(uint32_t)(keys[p] >> vb)] : o_ptr[n];
}

// Edge ids of all entries: higher-rank entries have theirs; lower-rank entries (row r, column c < r)
// take the id of edge (c, r) from c's oriented row.  Written per sorted entry (compacted while
// peeling) and per input entry (outputs are gathered by it).  An input that is not symmetric has
// entries whose edge is not there: flagged.  The supports are cleared on the way.
template <bool kChained>
__global__ void __launch_bounds__(kThreads) k_entry_eid(const uint64_t* __restrict__ keys, uint64_t entries, unsigned vb,
                                                        uint32_t m, const uint32_t* __restrict__ o_ptr,
                                                        const uint32_t* __restrict__ o_col,
                                                        const uint32_t* __restrict__ fence,
                                                        const uint32_t* __restrict__ sorted_entry,
                                                        uint32_t* __restrict__ s_eid, uint32_t* __restrict__ entry_eid,
                                                        uint32_t* __restrict__ sup, uint32_t* __restrict__ supx,
                                                        uint32_t* __restrict__ ctrl) {
    if (kChained) after_previous(keys, o_ptr, o_col, fence, sorted_entry, s_eid, entry_eid, sup, supx, ctrl);
    const uint64_t p = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (__any_sync(kFullMask, timed_out(ctrl))) return;
    uint32_t err = 0;
    if (p < m) sup[p] = supx[p] = 0;
    if (p < entries) {
        const uint64_t key = keys[p];
        const uint32_t row = (uint32_t)(key >> vb), col = (uint32_t)(key & ((1ull << vb) - 1));
        uint32_t eid = 0;
        if (col > row) {
            eid = s_eid[p];
        } else {
            const uint32_t lo = o_ptr[col], hi = o_ptr[col + 1];
            uint32_t idx = 0xffffffffu;
            if (col < row && lo <= hi && hi <= m) {
                idx = fenced_lower_bound(o_col, fence, lo, hi, row);
                if (idx >= hi || o_col[idx] != row) idx = 0xffffffffu;
            }
            if (idx != 0xffffffffu) eid = idx;
            else err = kErrAsymmetric;
            s_eid[p] = eid;
        }
        entry_eid[sorted_entry[p]] = eid;
    }
    err = __reduce_or_sync(kFullMask, err);
    if (err && lane_id() == 0) atomicOr(&ctrl[kCtrlError], err);
}

// Blocks of a kernel that makes sort keys: four keys a thread at least, at most eight blocks an SM
// (each adds its digit counts to the global ones).
uint32_t key_blocks(const kt_engine* e, uint64_t keys) {
    return (uint32_t)std::min<uint64_t>((keys + 4 * kThreads - 1) / (4 * kThreads), (uint64_t)e->num_sms * 8);
}

unsigned bits_for(uint64_t n) {
    unsigned b = 1;
    while (b < 64 && (1ull << b) < n) ++b;
    return b;
}

}  // namespace

int input_status(uint32_t err) {
    if (err & kErrBadVertex) return fail(KT_ERR_INVALID_ARG, "an entry names a vertex id >= num_nodes");
    if (err & kErrSelfLoop) return fail(KT_ERR_SELF_LOOP, "Edges from a vertex to itself are not allowed!");
    if (err & kErrDuplicate) return fail(KT_ERR_NOT_SYMMETRIC, "duplicate entry in the input edge list");
    if (err & kErrAsymmetric) return fail(KT_ERR_NOT_SYMMETRIC, "entry (u,v) without its reverse (v,u)");
    if (err & kErrTimeout) return fail(KT_ERR_TIMEOUT, "a bounded device wait expired");
    return KT_OK;
}

// Synchronizes and converts the device error word into a status.
int sync_and_check(kt_engine* e) {
    int rc = check_cuda(cudaMemcpyAsync(e->h_ctrl, e->ctrl, sizeof(uint32_t) * kCtrlWords, cudaMemcpyDeviceToHost,
                                        e->stream), "read control block");
    if (rc) return rc;
    rc = check_cuda(cudaStreamSynchronize(e->stream), "build synchronize");
    if (rc) return rc;
    return input_status(e->h_ctrl[kCtrlError]);
}

namespace {

// Tiled COO/CSR (coo2tiledcoocsr, graph.cu:641-706): key = row << vb | dst with row =
// (src / ts * T + dst / ts) * ts + src % ts; the entry index rides along as the value.
__global__ void k_tile_keys(const uint32_t* __restrict__ src, const uint32_t* __restrict__ dst, uint64_t entries,
                            uint32_t n, uint32_t T, uint32_t ts, unsigned vb, uint64_t* __restrict__ keys,
                            uint32_t* __restrict__ ctrl) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t err = 0;
    if (i < entries) {
        const uint32_t s = src[i], d = dst[i];
        if (s >= n || d >= n) {
            err = kErrBadVertex;
            keys[i] = 0;
        } else {
            const uint64_t row = ((uint64_t)(s / ts) * T + d / ts) * ts + s % ts;
            keys[i] = (row << vb) | d;
        }
    }
    err = __reduce_or_sync(kFullMask, err);
    if (err && lane_id() == 0) atomicOr(&ctrl[kCtrlError], err);
}

// Sorted keys back to entries: the source from the row, the destination from the key.  (An input error is read
// only behind this kernel and the next, which write nothing then.)
__global__ void k_tile_entries(const uint64_t* __restrict__ keys, uint64_t entries, uint32_t T, uint32_t ts,
                               unsigned vb, uint32_t* __restrict__ src_out, uint32_t* __restrict__ dst_out,
                               const uint32_t* __restrict__ ctrl) {
    const uint64_t p = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p < entries && !failed(ctrl)) {
        const uint64_t key = keys[p];
        const uint64_t row = key >> vb;
        const uint64_t tile = row / ts;  // src tile * T + dst tile
        src_out[p] = (uint32_t)((tile / T) * ts + row % ts);
        dst_out[p] = (uint32_t)(key & ((1ull << vb) - 1));
    }
}

// tile_src_ptr[r] = first sorted position whose row is >= r (rows + 1 offsets).
__global__ void k_tile_ptr(const uint64_t* __restrict__ keys, uint64_t entries, unsigned vb, uint64_t rows,
                           uint32_t* __restrict__ ptr, const uint32_t* __restrict__ ctrl) {
    const uint64_t r = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (r > rows || failed(ctrl)) return;
    uint64_t lo = 0, len = entries;
    while (len > 0) {
        const uint64_t half = len >> 1;
        if ((keys[lo + half] >> vb) < r) {
            lo += half + 1;
            len -= half + 1;
        } else {
            len = half;
        }
    }
    ptr[r] = (uint32_t)lo;
}

// Symmetrize and deduplicate: entry i becomes the undirected key (min << vb | max); ids >= n
// set kErrBadVertex (key 0, a self loop, dropped).
__global__ void __launch_bounds__(kThreads) k_canon_keys(const uint32_t* __restrict__ src,
                                                         const uint32_t* __restrict__ dst, uint64_t entries, uint32_t n,
                                                         unsigned vb, unsigned passes, uint64_t* __restrict__ keys,
                                                         uint32_t* __restrict__ counts, uint32_t* __restrict__ ctrl) {
    after_previous(src, dst, keys, counts, ctrl);
    __shared__ uint32_t h[kMaxDigitPasses * 256];
    digit_counts_clear(h, passes);
    uint32_t err = 0;
    for (uint64_t i0 = (uint64_t)blockIdx.x * kThreads; i0 < entries; i0 += (uint64_t)gridDim.x * kThreads) {
        const uint64_t i = i0 + threadIdx.x;
        uint64_t key = 0;
        if (i < entries) {
            const uint32_t s = src[i], d = dst[i];
            if (s >= n || d >= n) err = kErrBadVertex;
            else key = ((uint64_t)(s < d ? s : d) << vb) | (s < d ? d : s);
            keys[i] = key;
        }
        digit_counts_add(h, key, i < entries, passes);
    }
    digit_counts_flush(h, passes, counts);
    err = __reduce_or_sync(kFullMask, err);
    if (err && lane_id() == 0) atomicOr(&ctrl[kCtrlError], err);
}

// The first copy of each sorted key that is not a self loop.
__device__ __forceinline__ bool canon_first(const uint64_t* __restrict__ keys, uint64_t entries, unsigned vb,
                                            uint64_t p, uint64_t* key) {
    if (p >= entries) return false;
    *key = keys[p];
    return (*key >> vb) != (*key & ((1ull << vb) - 1)) && (p == 0 || keys[p - 1] != *key);
}

// Unique edges, into the control block.  (16.8 M keys: 37 us, and k_canon_emit, which numbers them by
// look-back, 119; with the look-back here, where the tiles finish almost together, 83 and 90.)
__global__ void __launch_bounds__(kFlagThreads) k_canon_count(const uint64_t* __restrict__ keys, uint64_t entries,
                                                              unsigned vb, uint32_t* __restrict__ ctrl) {
    after_previous(keys, ctrl);
    __shared__ uint32_t s_count;
    if (threadIdx.x == 0) s_count = 0;
    if (__syncthreads_or(timed_out(ctrl))) return;
    uint32_t count = 0;
    for (uint64_t p0 = (uint64_t)blockIdx.x * kFlagTile + threadIdx.x; p0 < entries;
         p0 += (uint64_t)gridDim.x * kFlagTile) {
#pragma unroll
        for (uint32_t s = 0; s < kFlagSteps; ++s) {
            uint64_t key;
            count += canon_first(keys, entries, vb, p0 + s * kFlagThreads, &key);
        }
    }
    count = __reduce_add_sync(kFullMask, count);
    if (lane_id() == 0 && count) atomicAdd(&s_count, count);
    __syncthreads();
    if (threadIdx.x == 0 && s_count) atomicAdd(ctrl + kCtrlTriLo, s_count);
}

// Unique edge j goes to j as (lo, hi) and to u + j as (hi, lo), where u is their number; nothing is
// written unless all 2u entries fit.
__global__ void __launch_bounds__(kFlagThreads, 4) k_canon_emit(const uint64_t* __restrict__ keys, uint64_t entries,
                                                             unsigned vb, uint64_t capacity,
                                                             uint32_t* __restrict__ src_out,
                                                             uint32_t* __restrict__ dst_out, Look L) {
    after_previous(keys, src_out, dst_out);
    __shared__ FlagSmem S;
    __shared__ uint64_t key[kFlagTile + 2];
    const uint64_t u = L.ctrl[kCtrlTriLo];
    if (__syncthreads_or(2 * u > capacity)) return;
    const uint32_t tile = look_tile(L, &S.tile);
    if (tile == kNoTile) return;
    const uint32_t warp = threadIdx.x >> 5;
    const uint64_t mask = (1ull << vb) - 1;
    uint32_t first = 0;
    stage_keys(key, keys, entries, tile);
#pragma unroll
    for (uint32_t s = 0; s < kFlagSteps; ++s) {
        const uint32_t i = s * kFlagThreads + threadIdx.x;
        const uint64_t k = key[1 + i];
        const bool f = (uint64_t)tile * kFlagTile + i < entries && k != key[i] && (k >> vb) != (k & mask);
        first |= (uint32_t)f << s;
        const uint32_t b = __ballot_sync(kFullMask, f);
        if (lane_id() == 0) S.before[s * kFlagWarps + warp] = __popc(b);
    }
    __syncthreads();
    flag_sums(S, L, tile);
#pragma unroll
    for (uint32_t s = 0; s < kFlagSteps; ++s) {
        const bool f = first >> s & 1u;
        const uint64_t j =
            S.prefix + S.before[s * kFlagWarps + warp] + __popc(__ballot_sync(kFullMask, f) & lanemask_lt());
        if (f) {
            const uint64_t k = key[1 + s * kFlagThreads + threadIdx.x];
            const uint32_t lo = (uint32_t)(k >> vb), hi = (uint32_t)(k & mask);
            src_out[j] = lo;
            dst_out[j] = hi;
            src_out[u + j] = hi;
            dst_out[u + j] = lo;
        }
    }
}

}  // namespace

int symmetrize(kt_engine* e, const uint32_t* d_src, const uint32_t* d_dst, uint64_t entries, uint32_t n,
               uint32_t* d_src_out, uint32_t* d_dst_out, uint64_t capacity, uint64_t* num_out) {
    *num_out = 0;
    if (entries >= 0xffffffffull) return fail(KT_ERR_TOO_LARGE, "more than 2^32-2 entries");
    if (entries && n == 0) return fail(KT_ERR_INVALID_ARG, "entries given for a graph with 0 vertices");
    if (entries == 0) return KT_OK;
    int rc;
    if ((n > e->cap_nodes || entries > e->cap_entries) &&
        (rc = reserve(e, n > e->cap_nodes ? n : e->cap_nodes, entries > e->cap_entries ? entries : e->cap_entries)))
        return rc;
    const unsigned vb = bits_for(n > 1 ? n : 2), passes = (2 * vb + 7) / 8;
    if ((rc = begin_session(e, n, 0, look_words(entries), entries))) return rc;
    uint32_t* counts = next_counts(e, passes);
    if ((rc = launch_chained(e, "k_canon_keys", k_canon_keys, key_blocks(e, entries), kThreads, 0, d_src, d_dst,
                             entries, n, vb, passes, e->key_a, counts, e->ctrl))) return rc;
    int in_b = 0;
    if ((rc = radix_passes(e, e->key_a, nullptr, e->key_b, nullptr, entries, 0, passes, counts, &in_b))) return rc;
    const uint64_t* keys = in_b ? e->key_b : e->key_a;
    const uint32_t tiles = ceil_div(entries, kFlagTile);
    if ((rc = launch_chained(e, "k_canon_count", k_canon_count, std::min(tiles, (uint32_t)e->num_sms * 4), kFlagThreads,
                             0, keys, entries, vb, e->ctrl))) return rc;
    if ((rc = launch_chained(e, "k_canon_emit", k_canon_emit, tiles, kFlagThreads, 0, keys, entries, vb, capacity,
                             d_src_out, d_dst_out, next_look(e))) || (rc = sync_and_check(e))) return rc;
    const uint32_t u = e->h_ctrl[kCtrlTriLo];
    *num_out = 2ull * u;
    if (2ull * u > capacity)
        return fail(KT_ERR_CAPACITY, "symmetrized graph has %llu entries, capacity %llu", 2ull * u,
                    (unsigned long long)capacity);
    return KT_OK;
}

int tiled_coocsr(kt_engine* e, const uint32_t* d_src, const uint32_t* d_dst, uint64_t entries, uint32_t n,
                 uint32_t tiles_per_dim, uint32_t* d_tile_src_ptr, uint32_t* d_src_out, uint32_t* d_dst_out) {
    if (tiles_per_dim == 0 || n == 0) return fail(KT_ERR_INVALID_ARG, "tiled layout needs tiles_per_dim >= 1 and n >= 1");
    if (entries >= 0xffffffffull) return fail(KT_ERR_TOO_LARGE, "more than 2^32-2 entries");
    const uint32_t T = tiles_per_dim;
    const uint32_t ts = (uint32_t)(((uint64_t)n + T - 1) / T);
    const uint64_t rows = (uint64_t)T * T * ts;
    const unsigned vb = bits_for(n > 1 ? n : 2);
    const unsigned rb = bits_for(rows + 1);
    if (rb + vb > 64) return fail(KT_ERR_TOO_LARGE, "tiles_per_dim %u too large for %u vertices", T, n);
    int rc;
    if ((n > e->cap_nodes || entries > e->cap_entries) &&
        (rc = reserve(e, n > e->cap_nodes ? n : e->cap_nodes, entries > e->cap_entries ? entries : e->cap_entries)))
        return rc;
    cudaStream_t st = e->stream;
    if ((rc = begin_session(e, n, 0, look_words(entries), entries))) return rc;
    int in_b = 0;
    if (entries) {
        k_tile_keys<<<grid_for(entries), kThreads, 0, st>>>(d_src, d_dst, entries, n, T, ts, vb, e->key_a, e->ctrl);
        count_launch(e);
        if ((rc = check_launch(e, "k_tile_keys"))) return rc;
        const unsigned passes = (rb + vb + 7) / 8;
        uint32_t* counts = next_counts(e, passes);
        if ((rc = count_digits(e, e->key_a, entries, 0, passes, counts)) ||
            (rc = radix_passes(e, e->key_a, nullptr, e->key_b, nullptr, entries, 0, passes, counts, &in_b)))
            return rc;
        k_tile_entries<<<grid_for(entries), kThreads, 0, st>>>(in_b ? e->key_b : e->key_a, entries, T, ts, vb,
                                                              d_src_out, d_dst_out, e->ctrl);
        count_launch(e);
        if ((rc = check_launch(e, "k_tile_entries"))) return rc;
    }
    k_tile_ptr<<<grid_for(rows + 1), kThreads, 0, st>>>(in_b ? e->key_b : e->key_a, entries, vb, rows, d_tile_src_ptr,
                                                       e->ctrl);
    count_launch(e);
    if ((rc = check_launch(e, "k_tile_ptr"))) return rc;
    return sync_and_check(e);
}

int build_graph(kt_engine* e, const uint32_t* d_src, const uint32_t* d_dst, uint64_t entries, uint32_t n,
                bool check) {
    if (entries & 1) return fail(KT_ERR_NOT_SYMMETRIC, "odd number of entries (%llu): every edge needs both directions",
                                 (unsigned long long)entries);
    if (entries >= 0xffffffffull) return fail(KT_ERR_TOO_LARGE, "more than 2^32-2 entries");
    // (an engine that has done nothing, or whose reservation failed, has no workspace: the session's kernels
    // write to it for an empty graph too)
    if (n > e->cap_nodes || entries > e->cap_entries || !e->look) {
        int rc = reserve(e, n > e->cap_nodes ? n : e->cap_nodes, entries > e->cap_entries ? entries : e->cap_entries);
        if (rc) return rc;
    }
    e->n = n;
    e->entries = entries;
    e->m = (uint32_t)(entries / 2);
    e->by_index = e->orient_by_index;
    e->sched_on_device = false;  // a call with a selector sets it after the build
    e->vb = bits_for(n > 1 ? n : 2);
    const unsigned vb = e->vb;
    int rc = begin_session(e, n, n, std::max(look_words(n), look_words(entries)), entries);
    if (rc) return rc;
    if (n == 0) return entries ? fail(KT_ERR_INVALID_ARG, "entries given for a graph with 0 vertices") : KT_OK;

    // 1. degrees (and id / self-loop checks)
    if (entries) {
        if ((rc = launch_chained(e, "k_degree", e->chained ? k_degree<true> : k_degree<false>, grid_for(entries),
                                 kThreads, 0, d_src, d_dst, entries, n, e->deg, e->ctrl))) return rc;
    }
    // (input errors are read back once, after the build: every kernel up to its end indexes inside its
    // arrays whatever the input, and the kernels after it return at once when the error word is set)

    // 2. ranks - ascending (degree, id), or the ids themselves when orienting by index - and the row
    // starts of the symmetric CSR (row r holds the neighbours of the rank-r vertex)
    int in_b = 0;
    if (e->orient_by_index) {
        rc = launch_chained(e, "k_rank_rows", e->chained ? k_rank_rows<true, true> : k_rank_rows<true, false>,
                            ceil_div(n, kScanTile), kScanThreads, 0, nullptr, e->deg, n, vb, e->rank, e->s_len,
                            e->s_ptr, e->s_split, e->o_ptr, next_look(e));
    } else {
        const unsigned passes = (vb + 7) / 8;
        uint32_t* counts = next_counts(e, passes);
        if ((rc = launch_chained(e, "k_rank_keys", e->chained ? k_rank_keys<true> : k_rank_keys<false>,
                                 key_blocks(e, n), kThreads, 0, e->deg, n, vb, passes, e->key_a, counts)) ||
            (rc = radix_passes(e, e->key_a, nullptr, e->key_b, nullptr, n, vb, passes, counts, &in_b)))
            return rc;
        rc = launch_chained(e, "k_rank_rows", e->chained ? k_rank_rows<false, true> : k_rank_rows<false, false>,
                            ceil_div(n, kScanTile), kScanThreads, 0, in_b ? e->key_b : e->key_a, e->deg, n, vb,
                            e->rank, e->s_len, e->s_ptr, e->s_split, e->o_ptr, next_look(e));
    }
    if (rc) return rc;

    // 3. sort entries by (rank[src], rank[dst]); 4. both CSRs and the edge ids
    if (entries) {
        const unsigned passes = (2 * vb + 7) / 8;
        uint32_t* counts = next_counts(e, passes);
        if ((rc = launch_chained(e, "k_edge_keys", e->chained ? k_edge_keys<true> : k_edge_keys<false>,
                                 key_blocks(e, entries), kThreads, 0, d_src, d_dst, entries, n, e->rank, vb, passes,
                                 e->key_a, counts, e->ctrl))) return rc;
        if ((rc = radix_passes(e, e->key_a, e->val_a, e->key_b, e->val_b, entries, 0, passes, counts, &in_b))) return rc;
        const uint64_t* keys = in_b ? e->key_b : e->key_a;
        e->sorted_entry = in_b ? e->val_b : e->val_a;
        e->entry_eid = in_b ? e->val_a : e->val_b;  // the sort's other value buffer is free now
        if ((rc = launch_chained(e, "k_csr", e->chained ? k_csr<true> : k_csr<false>, ceil_div(entries, kFlagTile),
                                 kFlagThreads, 0, keys, entries, vb, n, e->m, e->s_col, e->s_eid, e->s_split,
                                 e->o_ptr, e->o_col, e->e_src, e->o_fence, next_look(e)))) return rc;
        if (e->orient_by_index) {
            if ((rc = launch_chained(e, "k_empty_rows", k_empty_rows, grid_for(n), kThreads, 0, keys, entries, vb, n,
                                     e->s_ptr, e->s_len, e->o_ptr, e->ctrl))) return rc;
        }
        if ((rc = launch_chained(e, "k_entry_eid", e->chained ? k_entry_eid<true> : k_entry_eid<false>,
                                 grid_for(entries), kThreads, 0, keys, entries, vb, e->m, e->o_ptr, e->o_col,
                                 e->o_fence, e->sorted_entry, e->s_eid, e->entry_eid, e->sup, e->rnd, e->ctrl))) return rc;
    }
    return check && !e->trusted ? sync_and_check(e) : KT_OK;
}

}  // namespace kt
