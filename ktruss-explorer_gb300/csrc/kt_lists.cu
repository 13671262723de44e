// Peeling from triangle lists: the full decomposition of graphs whose triangles fit in HBM.
//
// The row-walking peel (kt_peel.cu) finds the triangles of a removed edge again, by a search in an
// oriented row for every entry of its shorter row: about twelve dependent or scattered loads per
// entry, three quarters of which find no triangle.  Here every triangle is found once more after
// the support count and written down: edge e's list tri[tptr[e] .. tptr[e+1]) holds, for each of
// its sup(e) triangles, the ids of the other two edges.  Removing e then streams its list
// (coalesced, eight bytes a triangle) and gathers two state bytes per triangle - no rows, no
// searches, no row compaction.
//
// Levels, rounds, ownership and results are those of kt_peel.cu: level k removes, in synchronous
// rounds, the alive edges with support < k-2; a triangle destroyed in a round is charged by its
// removed edge with the smallest id to each surviving edge.
//
// Edge states are bytes: 0 alive, 255 removed long ago, else the stamp 1 + r % 254 of the round r
// that removes (or removed) the edge.  A byte array is a quarter of the 32-bit round stamps of the
// walking peel, so its random gathers stay in L2 up to R-MAT 22.  Before a stamp could come round
// again, old stamps are swept to 255 (one pass over the bytes every 250 rounds).
//
// A round is one phase and one grid barrier:
//   1. warps take chunks (descriptors of up to 32 list entries) of the round's frontier; a decrement
//      that takes an edge from k-2 to k-3 appends it to the block's queue in shared memory;
//   2. the block flushes its queue: every queued edge is stamped, gets its truss number, and its
//      list is cut into chunks for the next round (one global atomic per 32 edges);
//   3. the barrier's arrival adds the block's queued edges to the arrival word, so the poll that
//      ends the wait also delivers the size of the next frontier.
//
// Bound by latency: a round of up to 512 frontier edges takes 5 us (8.5 us when walking rows: barrier,
// chunk, row entry, stamp, search, stamp, decrement, two pushes one after the other), larger ones by
// the two gathers an entry.  Measured against the walking peel (GB300, peel kernel / writing the
// lists included / whole decomposition): R-MAT 20 of 15 M edges 61.0 -> 22.8 / 40.8 / 71.5 -> 51.4 ms,
// R-MAT 22 of 60 M edges 246 -> 86 / 200 / 303 -> 257 ms, R-MAT 16 9.2 -> 5.1 / 5.6 / 10.1 -> 6.4 ms, a
// Watts-Strogatz graph of 10 M edges 13.8 -> 2.6 / 4.0 / 17.2 -> 6.9 ms, a batch of 256 graphs (18 M
// edges) 17.1 -> 4.3 / 5.9 / 22.4 -> 10.9 ms (the lists are written faster since, kt_support.cu).

#include <algorithm>

#include "kt_device.cuh"
#include "kt_engine.h"

namespace kt {

namespace {

constexpr int kListThreads = 1024;        // one block per SM
constexpr uint32_t kDead = 0xffffffffu;   // support of a removed edge (late decrements keep the top bit)
constexpr uint32_t kQueue = 4096;         // edges a block queues in shared memory per round
constexpr uint32_t kStampPeriod = 254;    // round stamps 1..254
constexpr uint32_t kOld = 255;            // state of edges removed before the last sweep
constexpr uint32_t kChunk = 32;           // list entries per chunk

// Control words of this kernel (beyond the words it shares with the walking peel).
constexpr uint32_t kLBar = 88;    // u64 [2]: arrivals << 32 | edges queued, by barrier parity
constexpr uint32_t kLSlot = 96;   // [4] x {u64 chunks, u32 overflowed edges, u32 minimum support}
constexpr uint32_t kLMinId = 112; // [4] smallest alive edge id of a level scan
static_assert(kLMinId + 4 <= kCtrlWords, "control block holds the list peel's words");

struct ListParams {
    const uint2* __restrict__ tri;       // per list entry: the triangle's other two edges
    const uint64_t* __restrict__ tptr;   // m+1: list starts
    uint32_t* sup;
    uint8_t* st;
    uint32_t* tr;
    uint4* ch[2];      // chunks {edge, list position (lo, hi), entries}, by frontier parity
    uint32_t cap_chunks;
    uint32_t* big[2];  // edges whose chunks did not fit, by frontier parity
    uint32_t* ctrl;
    uint32_t* round_size;
    uint32_t* round_level;
    uint32_t* round_ns;
    uint32_t* level_k;
    uint32_t* level_alive;
    uint32_t* level_ns;
    uint32_t* level_front;
    uint32_t cap_rounds, cap_levels, m;
    uint64_t wait_base_ns, wait_ns_per_unit;
};

__device__ __forceinline__ uint32_t stamp_of(uint32_t r) { return 1u + r % kStampPeriod; }

// What a barrier delivers: the next frontier's edges, chunks and overflowed edges, and a level
// scan's minimum support and smallest alive id.
struct Front {
    uint32_t edges, chunks, big, min_sup, min_id;
};

struct ListShared {
    uint32_t queue[kQueue];
    uint32_t queued;              // edges queued since the last barrier (may exceed kQueue)
    uint32_t bar_edges[2];        // the arrival words' edge sums when they last completed
    uint32_t bar_arrivals[2];     // ... and their arrivals
    Front front;
    uint32_t ok;
    uint32_t min_sup, min_id;     // a level scan's block minima
    unsigned long long walk;      // list entries queued (a statistic)
    unsigned long long ns[9];     // block 0: phase clock
};

// Stamps the edges of a warp's lanes for the next round and cuts their lists into chunks.  All 32
// lanes call it together; `slot` is the ring slot of the barrier that closes the current phase.
__device__ __forceinline__ void push_lists(const ListParams& P, ListShared& S, uint32_t e, bool take, uint32_t rr,
                                           uint32_t k, uint32_t slot, uint32_t parity) {
    uint64_t t0 = 0;
    uint32_t len = 0;
    if (take) {
        P.st[e] = (uint8_t)stamp_of(rr);
        P.tr[e] = k - 1;
        P.sup[e] = kDead;
        // an edge removed at level 3 has no triangle left whose other edges are alive or in its round
        if (k != 3) {
            t0 = __ldg(P.tptr + e);
            len = (uint32_t)(__ldg(P.tptr + e + 1) - t0);
        }
    }
    const uint32_t nch = (len + kChunk - 1) / kChunk;
    const uint32_t lane = lane_id();
    uint32_t incl = nch;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(kFullMask, incl, o);
        if (lane >= (uint32_t)o) incl += t;
    }
    const uint32_t total = __shfl_sync(kFullMask, incl, 31);
    if (total == 0) return;
    const uint32_t walked = __reduce_add_sync(kFullMask, len);
    unsigned long long cb = 0;
    if (lane == 0) {
        cb = atomicAdd(reinterpret_cast<unsigned long long*>(P.ctrl + kLSlot + 4 * slot), (unsigned long long)total);
        atomicAdd(&S.walk, (unsigned long long)walked);
    }
    cb = __shfl_sync(kFullMask, cb, 0);
    uint4* ch = P.ch[parity];
    if (cb + total <= P.cap_chunks) {
        // lanes write the chunks in turn, whichever lane's edge they belong to
        const uint32_t lo = (uint32_t)t0, hi = (uint32_t)(t0 >> 32);
        for (uint32_t i0 = 0; i0 < total; i0 += 32) {
            const uint32_t i = i0 + lane;
            uint32_t own = 0;  // the number of inclusive prefixes <= i
#pragma unroll
            for (uint32_t s = 16; s > 0; s >>= 1) {
                const uint32_t v = __shfl_sync(kFullMask, incl, own + s - 1);
                if (v <= i) own += s;
            }
            own &= 31u;
            const uint32_t oe = __shfl_sync(kFullMask, e, own), ol = __shfl_sync(kFullMask, len, own);
            const uint32_t oi = __shfl_sync(kFullMask, incl, own), on = __shfl_sync(kFullMask, nch, own);
            const uint64_t op = (uint64_t)__shfl_sync(kFullMask, hi, own) << 32 | __shfl_sync(kFullMask, lo, own);
            if (i < total) {
                const uint32_t off = (i - (oi - on)) * kChunk;
                const uint64_t p = op + off;
                ch[cb + i] = make_uint4(oe, (uint32_t)p, (uint32_t)(p >> 32), min(kChunk, ol - off));
            }
        }
    } else {
        const uint64_t stop = cb + total < P.cap_chunks ? cb + total : P.cap_chunks;
        for (uint64_t i = cb + lane; i < stop; i += 32) ch[i] = make_uint4(0, 0, 0, 0);
        const bool mine = len != 0;
        const uint32_t mb = __ballot_sync(kFullMask, mine);
        uint32_t bb = 0;
        if (lane == 0) bb = atomicAdd(P.ctrl + kLSlot + 4 * slot + 2, __popc(mb));
        bb = __shfl_sync(kFullMask, bb, 0);
        if (mine) P.big[parity][bb + __popc(mb & lanemask_lt())] = e;
    }
}

// Queues the taken edges of a warp in the block's queue (a full queue: straight to chunks).
__device__ __forceinline__ void enqueue(const ListParams& P, ListShared& S, uint32_t e, bool take, uint32_t rr,
                                        uint32_t k, uint32_t slot, uint32_t parity) {
    const uint32_t mt = __ballot_sync(kFullMask, take);
    if (!mt) return;
    uint32_t base = 0;
    if (lane_id() == 0) base = atomicAdd(&S.queued, __popc(mt));
    base = __shfl_sync(kFullMask, base, 0);
    const uint32_t pos = base + __popc(mt & lanemask_lt());
    const bool fits = pos < kQueue;
    if (take && fits) S.queue[pos] = e;
    if (base + __popc(mt) > kQueue) push_lists(P, S, e, take && !fits, rr, k, slot, parity);
}

// The block's queue becomes chunks of the next round.  Called by the whole block after a
// __syncthreads that follows the last enqueue.
__device__ __forceinline__ void flush(const ListParams& P, ListShared& S, uint32_t rr, uint32_t k, uint32_t slot,
                                      uint32_t parity) {
    const uint32_t n = min(S.queued, kQueue);
    for (uint32_t b = threadIdx.x & ~31u; b < n; b += blockDim.x) {
        const uint32_t i = b + lane_id();
        push_lists(P, S, i < n ? S.queue[i] : 0u, i < n, rr, k, slot, parity);
    }
}

// Grid barrier `epoch` (counted from 0): the block's queued edges are added to the arrival word of
// the epoch's parity together with its arrival.  Two words, so that a word read after its barrier
// completed stays still until every block has read it and arrived at the next barrier.  Bounded
// like grid_barrier.  Delivers the phase's frontier in S.front.
__device__ __forceinline__ bool list_barrier(const ListParams& P, ListShared& S, uint32_t epoch, uint64_t wait_ns) {
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long* word = reinterpret_cast<unsigned long long*>(P.ctrl + kLBar) + (epoch & 1);
        const unsigned long long add = 1ull << 32 | S.queued;
        const uint32_t target = S.bar_arrivals[epoch & 1] + gridDim.x;
        unsigned long long v = atom_add_acq_rel_u64(word, add) + add;
        uint32_t ok = 1;
        if ((uint32_t)(v >> 32) != target) {
            const uint64_t t0 = global_ns();
            uint32_t spins = 0;
            while ((uint32_t)((v = ld_acquire_u64(word)) >> 32) != target) {
                if ((++spins & 31u) == 0) {
                    if (ld_acquire(P.ctrl + kCtrlError) & kErrTimeout) { ok = 0; break; }
                    if (global_ns() - t0 > wait_ns) {
                        atomicOr(P.ctrl + kCtrlError, kErrTimeout);
                        ok = 0;
                        break;
                    }
                    if (spins > 256) __nanosleep(64);
                }
            }
        }
        const uint4 s = __ldcg(reinterpret_cast<const uint4*>(P.ctrl + kLSlot) + (epoch & 3));
        S.front.min_id = __ldcg(P.ctrl + kLMinId + (epoch & 3));
        S.front.edges = (uint32_t)v - S.bar_edges[epoch & 1];
        S.front.chunks = (uint32_t)min((unsigned long long)s.y << 32 | s.x, (unsigned long long)P.cap_chunks);
        S.front.big = s.z;
        S.front.min_sup = s.w;
        S.bar_edges[epoch & 1] = (uint32_t)v;
        S.bar_arrivals[epoch & 1] = target;
        S.queued = 0;
        S.ok = ok;
    }
    __syncthreads();
    return S.ok != 0;
}

// One list entry (f, g) of the edge e removed in round r: returns which of the two lose a support
// and reach k-3.  States seen: 0 alive, `nxt` alive but queued for the next round (its support no
// longer matters), `cur` removed in this round, anything else removed earlier.
__device__ __forceinline__ void destroy(const ListParams& P, uint32_t e, uint2 t, bool act, uint32_t cur, uint32_t nxt,
                                        uint32_t km2, bool* qf, bool* qg) {
    *qf = *qg = false;
    if (act) {
        const uint32_t sf = __ldcg(P.st + t.x), sg = __ldcg(P.st + t.y);
        const bool okf = sf == 0 || sf == nxt || (sf == cur && e < t.x);
        const bool okg = sg == 0 || sg == nxt || (sg == cur && e < t.y);
        if (okf && okg) {
            uint32_t of = 0, og = 0;
            if (sf == 0) of = atomicSub(&P.sup[t.x], 1u);
            if (sg == 0) og = atomicSub(&P.sup[t.y], 1u);
            *qf = of == km2;
            *qg = og == km2;
        }
    }
}

// The chunks [0, C) of round r, taken by warps gw, gw + nw, ... of nw.
__device__ __forceinline__ void run_chunks(const ListParams& P, ListShared& S, const uint4* __restrict__ ch, uint32_t C,
                                           uint32_t gw, uint32_t nw, uint32_t r, uint32_t k, uint32_t slot,
                                           uint32_t parity) {
    const uint32_t lane = lane_id(), cur = stamp_of(r), nxt = stamp_of(r + 1), km2 = k - 2;
    bool qf, qg;
    if (C <= 4 * nw) {
        // few chunks: one at a time, for the shortest chain
        for (uint32_t c = gw; c < C; c += nw) {
            const uint4 d = __ldcg(ch + c);
            const bool act = lane < d.w;
            uint2 t = make_uint2(0, 0);
            if (act) t = __ldcs(P.tri + ((uint64_t)d.z << 32 | d.y) + lane);
            destroy(P, d.x, t, act, cur, nxt, km2, &qf, &qg);
            enqueue(P, S, t.x, qf, r + 1, k, slot, parity);
            enqueue(P, S, t.y, qg, r + 1, k, slot, parity);
        }
        return;
    }
    // many chunks: 32 (or the warp's share) at a time, their entries flattened over the lanes, the
    // next step's entries loaded before the current step's are used
    const uint32_t D = min(32u, (C + nw - 1) / nw);
    for (uint64_t c0 = (uint64_t)gw * D; c0 < C; c0 += (uint64_t)nw * D) {
        uint4 d = make_uint4(0, 0, 0, 0);
        if (lane < D && c0 + lane < C) d = __ldcg(ch + c0 + lane);
        uint32_t incl = d.w;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(kFullMask, incl, o);
            if (lane >= (uint32_t)o) incl += t;
        }
        const uint32_t total = __shfl_sync(kFullMask, incl, 31);
        // position of flattened entry i of chunk `own`: p_own + i with p_own = start - prefix
        const uint64_t p0 = ((uint64_t)d.z << 32 | d.y) - (incl - d.w);
        const uint32_t plo = (uint32_t)p0, phi = (uint32_t)(p0 >> 32);
        uint32_t e_next = 0;
        uint2 t_next = make_uint2(0, 0);
        bool a_next = false;
        auto fetch = [&](uint32_t i) {
            uint32_t own = 0;
#pragma unroll
            for (uint32_t s = 16; s > 0; s >>= 1) {
                const uint32_t v = __shfl_sync(kFullMask, incl, own + s - 1);
                if (v <= i) own += s;
            }
            own &= 31u;
            e_next = __shfl_sync(kFullMask, d.x, own);
            const uint64_t p = ((uint64_t)__shfl_sync(kFullMask, phi, own) << 32 | __shfl_sync(kFullMask, plo, own)) + i;
            a_next = i < total;
            if (a_next) t_next = __ldcs(P.tri + p);
        };
        fetch(lane);
        for (uint32_t i0 = 0; i0 < total; i0 += 32) {
            const uint32_t e = e_next;
            const uint2 t = t_next;
            const bool act = a_next;
            if (i0 + 32 < total) fetch(i0 + 32 + lane);
            destroy(P, e, t, act, cur, nxt, km2, &qf, &qg);
            enqueue(P, S, t.x, qf, r + 1, k, slot, parity);
            enqueue(P, S, t.y, qg, r + 1, k, slot, parity);
        }
    }
}

__global__ void __launch_bounds__(kListThreads, 1) k_peel_lists(ListParams P) {
    __shared__ ListShared S;
    uint32_t* ctrl = P.ctrl;
    const uint32_t lane = lane_id();
    const uint32_t tid = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t nthreads = gridDim.x * blockDim.x;
    const uint32_t gwarp = tid >> 5, nwarps = nthreads >> 5;
    // the clock and the logs belong to a thread that is not the barrier's
    const bool scribe = blockIdx.x == 0 && threadIdx.x == blockDim.x - 1;
    if (threadIdx.x == 0) {
        S.queued = 0;
        S.bar_edges[0] = S.bar_edges[1] = S.bar_arrivals[0] = S.bar_arrivals[1] = 0;
        S.min_sup = S.min_id = kDead;
        S.walk = 0;
    }
    if (scribe) {
        for (int i = 0; i < 6; ++i) S.ns[i] = 0;
        S.ns[6] = global_ns();
    }
    __syncthreads();
    // ring slot s of the phase that barrier `epoch` closes is s = epoch & 3; slot (epoch + 2) & 3
    // is cleared meanwhile (its last readers arrived at barrier epoch - 1)
    auto clear_slot = [&](uint32_t epoch) {
        if (scribe) {
            *reinterpret_cast<uint4*>(ctrl + kLSlot + 4 * (epoch & 3)) = make_uint4(0, 0, 0, kDead);
            ctrl[kLMinId + (epoch & 3)] = kDead;
        }
    };
    auto phase = [&](int kind) {
        if (scribe) {
            const unsigned long long now = global_ns();
            S.ns[kind] += now - S.ns[6];
            S.ns[6] = now;
        }
    };
    const uint64_t phase_wait = P.wait_base_ns + P.wait_ns_per_unit * 2ull * P.m;
    uint32_t epoch = 0, parity = 0;  // parity: the chunk buffer the next frontier is written to
    clear_slot(1);
    clear_slot(2);
    {
        uint4* st4 = reinterpret_cast<uint4*>(P.st);
        const uint64_t n16 = ((uint64_t)P.m + 15) / 16;
        for (uint64_t i = tid; i < n16; i += nthreads) st4[i] = make_uint4(0, 0, 0, 0);
    }
    if (!list_barrier(P, S, epoch, phase_wait)) return;
    phase(0);
    ++epoch;

    uint32_t r = 0, level = 0, k_last = 2, live = P.m, start = 0, swept = 0;
    while (live) {
        if (scribe) S.ns[7] = S.ns[6];
        // level start: stream the supports (removed edges have the top bit) from the smallest id
        // alive at the last scan; collect the frontier of level k_last+1 and the minimum support
        uint32_t k = k_last + 1;
        clear_slot(epoch + 2);
        {
            uint32_t mn = kDead, mid = kDead;
            const uint4* sup4 = reinterpret_cast<const uint4*>(P.sup);
            const uint64_t m4 = ((uint64_t)P.m + 3) / 4;
            constexpr int kScan = 2;  // 16-byte loads in flight per lane
            for (uint64_t i0 = (start >> 2) + tid - lane; i0 < m4; i0 += (uint64_t)nthreads * kScan) {
                uint4 q4[kScan];
#pragma unroll
                for (int u = 0; u < kScan; ++u) {
                    const uint64_t i = i0 + (uint64_t)u * nthreads + lane;
                    q4[u] = i < m4 ? __ldcg(sup4 + i) : make_uint4(kDead, kDead, kDead, kDead);
                }
#pragma unroll
                for (int u = 0; u < kScan; ++u) {
                    const uint64_t i = i0 + (uint64_t)u * nthreads + lane;
                    const uint32_t sv[4] = {q4[u].x, q4[u].y, q4[u].z, q4[u].w};
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        const uint64_t j = 4 * i + c;
                        const uint32_t sj = j < P.m ? sv[c] : kDead;
                        if (sj < 0x80000000u) {
                            mn = min(mn, sj);
                            mid = min(mid, (uint32_t)j);
                        }
                        enqueue(P, S, (uint32_t)j, sj <= k - 3, r + 1, k, epoch & 3, parity);
                    }
                }
            }
            mn = __reduce_min_sync(kFullMask, mn);
            mid = __reduce_min_sync(kFullMask, mid);
            if (lane == 0 && mid != kDead) {
                atomicMin(&S.min_sup, mn);
                atomicMin(&S.min_id, mid);
            }
            __syncthreads();
            if (threadIdx.x == 0 && S.min_id != kDead) {
                atomicMin(ctrl + kLSlot + 4 * (epoch & 3) + 3, S.min_sup);
                atomicMin(ctrl + kLMinId + (epoch & 3), S.min_id);
                S.min_sup = S.min_id = kDead;
            }
            flush(P, S, r + 1, k, epoch & 3, parity);
        }
        if (!list_barrier(P, S, epoch, phase_wait)) return;
        phase(1);
        ++epoch;
        start = S.front.min_id;
        if (S.front.min_sup + 3 != k) {
            // level k_last+1 is empty: the next non-empty level is the minimum support + 3
            k = S.front.min_sup + 3;
            clear_slot(epoch + 2);
            for (uint64_t j0 = start + tid - lane; j0 < P.m; j0 += nthreads) {
                const uint64_t j = j0 + lane;
                const uint32_t sj = j < P.m ? __ldcg(P.sup + j) : kDead;
                enqueue(P, S, (uint32_t)j, sj <= k - 3, r + 1, k, epoch & 3, parity);
            }
            __syncthreads();
            flush(P, S, r + 1, k, epoch & 3, parity);
            if (!list_barrier(P, S, epoch, phase_wait)) return;
            phase(2);
            ++epoch;
        }
        uint32_t E = S.front.edges, C = S.front.chunks, B = S.front.big;
        if (E == 0 || E > live) {
            if (scribe) atomicOr(ctrl + kCtrlError, kErrRunaway);
            return;
        }
        if (scribe && level < P.cap_levels) {
            P.level_k[level] = k;
            P.level_alive[level] = live;
            P.level_ns[level] = (uint32_t)(S.ns[6] - S.ns[7]);
            P.level_front[level] = E;
        }
        while (E) {
            ++r;
            const bool log = scribe && r < P.cap_rounds;
            if (log) {
                P.round_size[r] = E;
                P.round_level[r] = k;
                S.ns[8] = S.ns[6];
            }
            const uint32_t from = parity;
            if (E == live || (C == 0 && B == 0)) {
                // nothing left to decrement, or nothing to walk: the round is done
                live -= E;
                if (log) P.round_ns[r] = 0;
                parity ^= 1;
                break;
            }
            parity ^= 1;
            if (r + 2 - swept >= kStampPeriod - 1) {
                // old stamps become 255 before they could be taken for this or the next round's
                const uint32_t keep = stamp_of(r);
                clear_slot(epoch + 2);
                for (uint64_t i = tid; i < P.m; i += nthreads) {
                    const uint32_t s = __ldcg(P.st + i);
                    if (s != 0 && s != keep && s != kOld) P.st[i] = (uint8_t)kOld;
                }
                if (!list_barrier(P, S, epoch, phase_wait)) return;
                phase(4);
                ++epoch;
                swept = r - 1;
            }
            clear_slot(epoch + 2);
            const uint64_t round_wait =
                P.wait_base_ns + P.wait_ns_per_unit * ((uint64_t)C * kChunk + (B ? 2ull * P.m : 0ull));
            run_chunks(P, S, P.ch[from], C, gwarp, nwarps, r, k, epoch & 3, parity);
            // edges whose chunks did not fit the buffer: one warp per edge
            for (uint32_t i = gwarp; i < B; i += nwarps) {
                const uint32_t e = __ldcg(P.big[from] + i);
                const uint64_t t0 = P.tptr[e], t1 = P.tptr[e + 1];
                const uint32_t cur = stamp_of(r), nxt = stamp_of(r + 1);
                for (uint64_t p0 = t0; p0 < t1; p0 += 32) {
                    const bool act = p0 + lane < t1;
                    uint2 t = make_uint2(0, 0);
                    if (act) t = __ldcs(P.tri + p0 + lane);
                    bool qf, qg;
                    destroy(P, e, t, act, cur, nxt, k - 2, &qf, &qg);
                    enqueue(P, S, t.x, qf, r + 1, k, epoch & 3, parity);
                    enqueue(P, S, t.y, qg, r + 1, k, epoch & 3, parity);
                }
            }
            __syncthreads();
            flush(P, S, r + 1, k, epoch & 3, parity);
            if (!list_barrier(P, S, epoch, round_wait)) return;
            phase(5);
            ++epoch;
            if (log) P.round_ns[r] = (uint32_t)(S.ns[6] - S.ns[8]);
            live -= E;
            E = S.front.edges;
            C = S.front.chunks;
            B = S.front.big;
        }
        ++level;
        k_last = k;
    }
    __syncthreads();
    if (threadIdx.x == 0 && S.walk) atomicAdd(reinterpret_cast<unsigned long long*>(ctrl + kPWalk), S.walk);
    if (scribe) {
        ctrl[kPKmax] = k_last - 1;
        ctrl[kPRounds] = r;
        ctrl[kPLevels] = level;
        ctrl[kPCompactions] = 0;
        for (int i = 0; i < 6; ++i) {
            ctrl[kPPhaseNs + 2 * i] = (uint32_t)S.ns[i];
            ctrl[kPPhaseNs + 2 * i + 1] = (uint32_t)(S.ns[i] >> 32);
        }
    }
}

}  // namespace

// Most list entries per edge on average (three per triangle) with which the lists are made.  Denser
// graphs spend more on writing the lists than the walks cost them, the more so as their last rounds
// remove most edges at once, which a recount round of the walking peel gets for little.  Whole
// decomposition, lists / walks: R-MAT 16 of edge factor 16 (52 entries an edge) 6.3 / 10.0 ms,
// G(3000, 0.2) (120) 5.2 / 8.6 ms, R-MAT 14 of edge factor 64 (134) 8.7 / 13.0 ms; past the line
// R-MAT 18 of edge factor 64 (261) 139 / 126 ms, R-MAT 16 of edge factor 128 (334) 72 / 66 ms,
// R-MAT 18 of edge factor 128 (480) 450 / 322 ms.
#ifndef KT_LIST_PER_EDGE
#define KT_LIST_PER_EDGE 192
#endif
constexpr uint64_t kMaxListPerEdge = KT_LIST_PER_EDGE;

// Whether the current graph's decomposition takes triangle lists; reads the triangle count (the
// supports must be counted and summed on e->stream) and sizes the list buffer.
int prepare_lists(kt_engine* e, bool* use) {
    *use = false;
    if (!e->lists_allowed || e->m == 0) return KT_OK;
    int rc;
    uint64_t total = e->last.list_entries;  // a trusted run repeats a call that counted them
    if (!e->trusted) {
        if ((rc = check_cuda(cudaMemcpyAsync(e->h_ctrl + kCtrlTriLo, e->ctrl + kCtrlTriLo, sizeof(uint64_t),
                                             cudaMemcpyDeviceToHost, e->stream), "read triangle count")) ||
            (rc = check_cuda(cudaStreamSynchronize(e->stream), "synchronize")))
            return rc;
        total = (uint64_t)e->h_ctrl[kCtrlTriHi] << 32 | e->h_ctrl[kCtrlTriLo];
        e->list_entries = total;
    }
    if (total > kMaxListPerEdge * e->m) return KT_OK;
    if (total > e->list_cap) {
        if (e->trusted) return KT_OK;
        const uint64_t want = std::max<uint64_t>(total + total / 16, 1u << 20);
        if ((rc = check_cuda(cudaStreamSynchronize(e->stream), "synchronize before resize"))) return rc;
        drop_replay(e);
        if (e->lists) cudaFree(e->lists);
        e->lists = nullptr;
        e->list_cap = 0;
        size_t free_bytes = 0, all_bytes = 0;
        if ((rc = check_cuda(cudaMemGetInfo(&free_bytes, &all_bytes), "free device memory"))) return rc;
        if (want * sizeof(uint2) > free_bytes / 2) return KT_OK;  // the rows are walked instead
        void* p = nullptr;
        if (cudaMalloc(&p, want * sizeof(uint2)) != cudaSuccess) {
            (void)cudaGetLastError();
            return KT_OK;
        }
        e->lists = static_cast<uint2*>(p);
        e->list_cap = want;
    }
    *use = true;
    return KT_OK;
}

// Builds the lists of the current graph and peels it from them.
int peel_lists(kt_engine* e) {
    int rc;
    const uint32_t m = e->m;
    // the sort's key buffers are free after the build: list starts, and ends for the fill
    uint64_t* tptr = e->key_a;
    uint64_t* ends = e->key_b;
    if ((rc = scan_offsets(e, e->sup, (uint64_t)m, tptr, ends)) || (rc = fill_lists(e, tptr, ends))) return rc;
    ListParams P;
    P.tri = e->lists;
    P.tptr = tptr;
    P.sup = e->sup;
    P.st = reinterpret_cast<uint8_t*>(e->rnd);
    P.tr = e->tr;
    P.ch[0] = e->chunks0;
    P.ch[1] = e->chunks1;
    P.cap_chunks = e->cap_chunks;
    P.big[0] = e->q0;
    P.big[1] = e->q1;
    P.ctrl = e->ctrl;
    P.round_size = e->round_size;
    P.round_level = e->round_level;
    P.round_ns = e->round_ns;
    P.level_k = e->level_k;
    P.level_alive = e->level_alive;
    P.level_ns = e->level_ns;
    P.level_front = e->level_front;
    P.cap_rounds = e->cap_rounds;
    P.cap_levels = e->cap_levels;
    P.m = m;
    P.wait_base_ns = e->wait_base_ns;
    P.wait_ns_per_unit = e->wait_ns_per_unit;
    void* args[] = {&P};
    const bool timed = e->ev_peel0 && e->ev_peel1 && !e->trusted;
    if (timed && (rc = check_cuda(cudaEventRecord(e->ev_peel0, e->stream), "record event"))) return rc;
    rc = check_cuda(cudaLaunchCooperativeKernel((const void*)k_peel_lists, dim3((unsigned)e->num_sms),
                                                dim3((unsigned)kListThreads), args, 0, e->stream),
                    "cooperative launch of k_peel_lists");
    count_launch(e);
    if (rc || !timed) return rc;
    e->peel_timed = true;
    return check_cuda(cudaEventRecord(e->ev_peel1, e->stream), "record event");
}

}  // namespace kt
