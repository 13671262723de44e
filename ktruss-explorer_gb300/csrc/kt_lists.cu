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
//      that takes an edge from k-2 to k-3 stamps it, writes its truss number and appends it to the
//      block's queue in shared memory;
//   2. the block flushes its queue: the edges' lists are cut into chunks for the next round, in a
//      buffer that all blocks share;
//   3. the barrier's arrival adds the block's queued edges to the arrival word, next to which lies
//      the count of chunks, so the 16-byte poll that ends the wait also delivers the size of the
//      next frontier.
//
// Bound: small rounds by one chain - chunk, entries, states, decrements, queue, claim of the next
// chunks, barrier - of about 8,000 cycles (3.6 us; 8.5 us when walking rows), large ones by the
// gathers in flight.  Measured against the walking peel (GB300, peel kernel / whole decomposition when
// the lists came in): R-MAT 20 of 15 M edges 61.0 -> 22.8 / 71.5 -> 51.4 ms, R-MAT 22 of 60 M edges
// 246 -> 86 / 303 -> 257 ms, R-MAT 16 9.2 -> 5.1 / 10.1 -> 6.4 ms, a Watts-Strogatz graph of 10 M edges
// 13.8 -> 2.6 / 17.2 -> 6.9 ms, a batch of 256 graphs (18 M edges) 17.1 -> 4.3 / 22.4 -> 10.9 ms (the lists
// are written faster since, kt_support.cu).  Chunks dealt to the blocks in turn, the frontier's size
// delivered by the barrier's own poll, list bounds loaded while the decrements are under way, entries
// prefetched across the barrier and four entries a lane under way in large rounds: peel kernel on
// R-MAT 20 22.4 -> 18.3 ms, R-MAT 22 83.4 -> 67.8, R-MAT 16 4.7 -> 4.0, Watts-Strogatz 2.5 -> 2.2, the batch
// 4.2 -> 3.5.

#include <algorithm>

#include "kt_engine.h"
#include "kt_list_rule.h"
#include "kt_look.cuh"

namespace kt {

namespace {

constexpr int kListThreads = 1024;        // one block per SM
constexpr uint32_t kDead = 0xffffffffu;   // support of a removed edge (late decrements keep the top bit)
constexpr uint32_t kQueue = 4096;         // edges a block queues in shared memory per round
constexpr uint32_t kStampPeriod = 254;    // round stamps 1..254
constexpr uint32_t kOld = 255;            // state of edges removed before the last sweep
constexpr uint32_t kChunk = 32;           // list entries per chunk
constexpr uint32_t kAhead = 1024;         // queue entries whose list bounds may be loaded ahead
constexpr uint32_t kNotLoaded = 0xffffffffu;
constexpr uint32_t kPrefetch = 1u << 16;  // chunks of a frontier whose entries are prefetched to L2 (16 MB):
                                          // R-MAT 20 peel kernel 20.9 -> 20.3 ms

// A barrier slot of the ring at kLRing: {u64 arrivals << 32 | edges queued, u64 global chunks, overflowed
// edges, minimum support, smallest alive edge id, unused}.
constexpr uint32_t kLChunks = 2, kLBig = 4, kLMin = 5, kLMinId = 6;
static_assert(kLMinId < kLSlotWords && kLSlotWords == 8, "a slot is two 16-byte words");

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
    uint64_t start[kAhead];       // list start and length of the first queue entries, where loaded
    uint32_t len[kAhead];
    uint32_t queued;              // edges queued since the last barrier (may exceed kQueue)
    Front front;
    uint32_t ok;
    uint32_t min_sup, min_id;     // a level scan's block minima
    uint32_t walk;                // list entries queued in the level, and before it (a statistic)
    unsigned long long walked;
    unsigned long long ns[9];     // block 0: phase clock
};

// List bounds of edge e.  An edge removed at level 3 has no triangle left whose other edges are
// alive or in its round: nothing to walk.
__device__ __forceinline__ void list_of(const ListParams& P, uint32_t e, bool take, uint32_t k, uint64_t* t0,
                                        uint32_t* len) {
    *t0 = 0;
    *len = 0;
    if (take && k != 3) {
        *t0 = __ldg(P.tptr + e);
        *len = (uint32_t)(__ldg(P.tptr + e + 1) - *t0);
    }
}

// Removes a warp's edges in round rr - stamp, truss number - and cuts their lists (len entries from
// t0 on; kNotLoaded: still to be looked up) into chunks of the next frontier.  All 32 lanes call it
// together; `slot` is the ring slot of the barrier that closes the current phase.
__device__ __forceinline__ void push_lists(const ListParams& P, ListShared& S, uint32_t e, bool take, uint64_t t0,
                                           uint32_t len, uint32_t rr, uint32_t k, uint32_t slot, uint32_t parity) {
    if (take) {
        P.st[e] = (uint8_t)stamp_of(rr);
        P.tr[e] = k - 1;
        P.sup[e] = kDead;
    }
    if (len == kNotLoaded) list_of(P, e, take, k, &t0, &len);
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
        cb = atomicAdd(reinterpret_cast<unsigned long long*>(P.ctrl + kLRing + kLSlotWords * slot + kLChunks),
                       (unsigned long long)total);
        atomicAdd(&S.walk, walked);
    }
    cb = __shfl_sync(kFullMask, cb, 0);
    uint4* ch = P.ch[parity];
    if (cb + total > P.cap_chunks) {
        // the claimed slots stay empty; the edges go to the overflow queue
        const uint64_t stop = cb + total < P.cap_chunks ? cb + total : P.cap_chunks;
#pragma unroll 1
        for (uint64_t i = cb + lane; i < stop; i += 32) ch[i] = make_uint4(0, 0, 0, 0);
        const bool mine = nch != 0;
        const uint32_t mb = __ballot_sync(kFullMask, mine);
        uint32_t bb = 0;
        if (lane == 0) bb = atomicAdd(P.ctrl + kLRing + kLSlotWords * slot + kLBig, __popc(mb));
        bb = __shfl_sync(kFullMask, bb, 0);
        if (mine) P.big[parity][bb + __popc(mb & lanemask_lt())] = e;
        return;
    }
    // lanes write the chunks in turn, whichever lane's edge they belong to
    const uint32_t lo = (uint32_t)t0, hi = (uint32_t)(t0 >> 32);
#pragma unroll 1
    for (uint32_t i0 = 0; i0 < total; i0 += 32) {
        const uint32_t i = i0 + lane;
        uint32_t at = 0;  // the number of inclusive prefixes <= i
#pragma unroll
        for (uint32_t s = 16; s > 0; s >>= 1) {
            const uint32_t v = __shfl_sync(kFullMask, incl, at + s - 1);
            if (v <= i) at += s;
        }
        at &= 31u;
        const uint32_t oe = __shfl_sync(kFullMask, e, at), ol = __shfl_sync(kFullMask, len, at);
        const uint32_t oi = __shfl_sync(kFullMask, incl, at), on = __shfl_sync(kFullMask, nch, at);
        const uint64_t op = (uint64_t)__shfl_sync(kFullMask, hi, at) << 32 | __shfl_sync(kFullMask, lo, at);
        if (i < total) {
            const uint32_t off = (i - (oi - on)) * kChunk;
            const uint64_t p = op + off;
            const uint32_t cnt = min(kChunk, ol - off);
            ch[cb + i] = make_uint4(oe, (uint32_t)p, (uint32_t)(p >> 32), cnt);
            if (cb < kPrefetch) {  // on their way while the blocks meet at the barrier
                asm volatile("prefetch.global.L2 [%0];" ::"l"(P.tri + p));
                if (cnt > 16) asm volatile("prefetch.global.L2 [%0];" ::"l"(P.tri + p + 16));
            }
        }
    }
}

// The rare push of edges that did not fit the queue, kept out of the callers' code.
__device__ __noinline__ void push_overflow(const ListParams& P, ListShared& S, uint32_t e, bool take, uint32_t rr,
                                           uint32_t k, uint32_t slot, uint32_t parity) {
    push_lists(P, S, e, take, 0, take ? kNotLoaded : 0u, rr, k, slot, parity);
}

// Queues the taken edges of a warp, to be removed in round rr, in the block's queue (a full queue:
// straight to chunks).
__device__ __forceinline__ void enqueue(const ListParams& P, ListShared& S, uint32_t e, bool take, uint32_t rr,
                                        uint32_t k, uint32_t slot, uint32_t parity) {
    const uint32_t mt = __ballot_sync(kFullMask, take);
    if (!mt) return;
    uint32_t base = 0;
    if (lane_id() == 0) base = atomicAdd(&S.queued, __popc(mt));
    base = __shfl_sync(kFullMask, base, 0);
    const uint32_t pos = base + __popc(mt & lanemask_lt());
    if (take && pos < kQueue) {
        S.queue[pos] = e;
        if (pos < kAhead) S.len[pos] = kNotLoaded;
    }
    if (base + __popc(mt) > kQueue) push_overflow(P, S, e, take && pos >= kQueue, rr, k, slot, parity);
}

// The same for two edges a lane, with the list bounds of the first kAhead queue entries.
__device__ __forceinline__ void enqueue_two(const ListParams& P, ListShared& S, uint2 e, bool qf, bool qg, uint32_t rr,
                                            uint32_t k, uint32_t slot, uint32_t parity, uint64_t f0, uint32_t flen,
                                            uint64_t g0, uint32_t glen) {
    const uint32_t mf = __ballot_sync(kFullMask, qf), mg = __ballot_sync(kFullMask, qg);
    if (!(mf | mg)) return;
    uint32_t base = 0;
    if (lane_id() == 0) base = atomicAdd(&S.queued, __popc(mf) + __popc(mg));
    base = __shfl_sync(kFullMask, base, 0);
    const uint32_t pf = base + __popc(mf & lanemask_lt()), pg = base + __popc(mf) + __popc(mg & lanemask_lt());
    if (qf && pf < kQueue) {
        S.queue[pf] = e.x;
        if (pf < kAhead) {
            S.start[pf] = f0;
            S.len[pf] = flen;
        }
    }
    if (qg && pg < kQueue) {
        S.queue[pg] = e.y;
        if (pg < kAhead) {
            S.start[pg] = g0;
            S.len[pg] = glen;
        }
    }
    if (base + __popc(mf) + __popc(mg) > kQueue) {
        push_overflow(P, S, e.x, qf && pf >= kQueue, rr, k, slot, parity);
        push_overflow(P, S, e.y, qg && pg >= kQueue, rr, k, slot, parity);
    }
}

// The block's queue becomes chunks of the next round.  Called by the whole block after a
// __syncthreads that follows the last enqueue.
__device__ __forceinline__ void flush(const ListParams& P, ListShared& S, uint32_t rr, uint32_t k, uint32_t slot,
                                      uint32_t parity) {
    const uint32_t n = min(S.queued, kQueue);
#pragma unroll 1
    for (uint32_t b = threadIdx.x & ~31u; b < n; b += blockDim.x) {
        const uint32_t i = b + lane_id();
        uint32_t e = 0, len = 0;
        uint64_t t0 = 0;
        if (i < n) {
            e = S.queue[i];
            len = i < kAhead ? S.len[i] : kNotLoaded;
            if (i < kAhead) t0 = S.start[i];
        }
        push_lists(P, S, e, i < n, t0, len, rr, k, slot, parity);
    }
}

// Grid barrier `epoch` (counted from 0) on ring slot epoch & 3, which was zero when the epoch
// began: the block's queued edges are added to the slot's first word together with its arrival.
// Bounded like grid_barrier (`units`: the work it covers).  Delivers the phase's frontier in S.front (kScan: and
// the minima).  kAbsent: blocks that never arrive (the self-test's).
template <bool kScan, uint32_t kAbsent = 0>
__device__ __forceinline__ bool list_barrier(const ListParams& P, ListShared& S, uint32_t epoch, uint64_t units) {
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t* slot = P.ctrl + kLRing + kLSlotWords * (epoch & 3);
        asm volatile("red.release.gpu.global.add.u64 [%0], %1;" ::"l"(slot), "l"(1ull << 32 | S.queued) : "memory");
        uint64_t bar, chunks, t0 = 0;
        uint32_t ok = 1, spins = 0;
        for (;;) {
            // one 16-byte access: the count of chunks is final once every block has arrived
            asm volatile(
                "{\n\t.reg .b128 q;\n\tld.acquire.gpu.global.b128 q, [%2];\n\tmov.b128 {%0, %1}, q;\n\t}"
                : "=l"(bar), "=l"(chunks)
                : "l"(slot)
                : "memory");
            if ((uint32_t)(bar >> 32) == gridDim.x + kAbsent) break;
            if ((++spins & 31u) == 0) {
                if (spins == 32) t0 = global_ns();
                if (ld_acquire(P.ctrl + kCtrlError) & kErrTimeout) { ok = 0; break; }
                if (global_ns() - t0 > P.wait_base_ns + P.wait_ns_per_unit * units) {
                    atomicOr(P.ctrl + kCtrlError, kErrTimeout);
                    ok = 0;
                    break;
                }
                if (spins > 256) __nanosleep(64);
            }
        }
        S.front.edges = (uint32_t)bar;
        S.front.chunks = (uint32_t)min(chunks, (uint64_t)P.cap_chunks);
        S.front.big = chunks > P.cap_chunks ? __ldcg(slot + kLBig) : 0u;
        if (kScan) {
            S.front.min_sup = __ldcg(slot + kLMin);
            S.front.min_id = __ldcg(slot + kLMinId);
        }
        S.queued = 0;
        S.ok = ok;
    }
    __syncthreads();
    return S.ok != 0;
}

// N list entries t = (f, g) a lane of edges e removed in round r: the two edges that survive it lose
// a support; those that reach k-3 are removed in the next round.  States seen: 0 alive, `nxt` alive
// but queued for the next round (its support no longer matters), `cur` removed in this round,
// anything else removed earlier.  With kAheadLoads the list bounds of f and g are loaded while their
// decrements are under way (for rounds bound by latency).
template <int N, bool kAheadLoads>
__device__ __forceinline__ void destroy(const ListParams& P, ListShared& S, const uint32_t (&e)[N], const uint2 (&t)[N],
                                        const bool (&act)[N], uint32_t cur, uint32_t nxt, uint32_t r, uint32_t k,
                                        uint32_t slot, uint32_t parity) {
    uint32_t sf[N], sg[N];
#pragma unroll
    for (int i = 0; i < N; ++i) {
        sf[i] = act[i] ? __ldcg(P.st + t[i].x) : kOld;
        sg[i] = act[i] ? __ldcg(P.st + t[i].y) : kOld;
    }
    uint32_t of[N], og[N];
    uint64_t f0[N], f1[N], g0[N], g1[N];
#pragma unroll
    for (int i = 0; i < N; ++i) {
        of[i] = og[i] = 0;
        f0[i] = g0[i] = 0;
        f1[i] = g1[i] = kNotLoaded;
        const bool okf = sf[i] == 0 || sf[i] == nxt || (sf[i] == cur && e[i] < t[i].x);
        const bool okg = sg[i] == 0 || sg[i] == nxt || (sg[i] == cur && e[i] < t[i].y);
        if (okf && okg) {
            if (sf[i] == 0) {
                of[i] = atomicSub(&P.sup[t[i].x], 1u);
                if (kAheadLoads) {
                    f0[i] = __ldg(P.tptr + t[i].x);
                    f1[i] = __ldg(P.tptr + t[i].x + 1);
                }
            }
            if (sg[i] == 0) {
                og[i] = atomicSub(&P.sup[t[i].y], 1u);
                if (kAheadLoads) {
                    g0[i] = __ldg(P.tptr + t[i].y);
                    g1[i] = __ldg(P.tptr + t[i].y + 1);
                }
            }
        }
    }
#pragma unroll
    for (int i = 0; i < N; ++i)
        enqueue_two(P, S, t[i], of[i] == k - 2, og[i] == k - 2, r + 1, k, slot, parity, f0[i],
                    (uint32_t)(f1[i] - f0[i]), g0[i], (uint32_t)(g1[i] - g0[i]));
}

// N of the chunks c, c + step, ... < C a warp at once.
template <int N>
__device__ __forceinline__ void whole_chunks(const ListParams& P, ListShared& S, const uint4* __restrict__ ch,
                                             uint32_t C, uint32_t first, uint32_t step, uint32_t cur, uint32_t nxt,
                                             uint32_t r, uint32_t k, uint32_t slot, uint32_t parity) {
    const uint32_t lane = lane_id();
#pragma unroll 1
    for (uint32_t c = first; c < C; c += N * step) {
        uint4 d[N];
        uint32_t e[N];
        uint2 t[N];
        bool act[N];
#pragma unroll
        for (int i = 0; i < N; ++i)
            d[i] = i == 0 || c + i * step < C ? __ldcg(ch + c + i * step) : make_uint4(0, 0, 0, 0);
#pragma unroll
        for (int i = 0; i < N; ++i) {
            e[i] = d[i].x;
            act[i] = lane < d[i].w;
            t[i] = make_uint2(0, 0);
            if (act[i]) t[i] = __ldcs(P.tri + ((uint64_t)d[i].z << 32 | d[i].y) + lane);
        }
        destroy<N, true>(P, S, e, t, act, cur, nxt, r, k, slot, parity);
    }
}

// The chunks [0, C) of round r, taken by warps gw, gw + nw, ... of nw.
__device__ __forceinline__ void run_chunks(const ListParams& P, ListShared& S, const uint4* __restrict__ ch, uint32_t C,
                                           uint32_t gw, uint32_t nw, uint32_t r, uint32_t k, uint32_t slot,
                                           uint32_t parity) {
    const uint32_t lane = lane_id(), cur = stamp_of(r), nxt = stamp_of(r + 1);
    if (C <= nw) {
        // a chunk a warp: the shortest chain
        whole_chunks<1>(P, S, ch, C, gw, nw, cur, nxt, r, k, slot, parity);
        return;
    }
    if (C <= 4 * nw) {
        whole_chunks<2>(P, S, ch, C, gw, nw, cur, nxt, r, k, slot, parity);
        return;
    }
    // many chunks: 32 (or the warp's share) at a time, their entries flattened over the lanes, kFlat
    // entries a lane under way at once (R-MAT 22 peel kernel: 84.7 ms with one, 74.7 with two, 67.8
    // with four, 69.4 with eight, which spills)
    constexpr int kFlat = 4;
    const uint32_t D = min(32u, (C + nw - 1) / nw);
#pragma unroll 1
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
#pragma unroll 1
        for (uint32_t i0 = 0; i0 < total; i0 += 32 * kFlat) {
            uint32_t e[kFlat];
            uint2 t[kFlat];
            bool act[kFlat];
#pragma unroll
            for (int q = 0; q < kFlat; ++q) {
                const uint32_t i = i0 + 32 * q + lane;
                uint32_t own = 0;
#pragma unroll
                for (uint32_t s = 16; s > 0; s >>= 1) {
                    const uint32_t v = __shfl_sync(kFullMask, incl, own + s - 1);
                    if (v <= i) own += s;
                }
                own &= 31u;
                e[q] = __shfl_sync(kFullMask, d.x, own);
                const uint64_t p =
                    ((uint64_t)__shfl_sync(kFullMask, phi, own) << 32 | __shfl_sync(kFullMask, plo, own)) + i;
                act[q] = i < total;
                t[q] = make_uint2(0, 0);
                if (act[q]) t[q] = __ldcs(P.tri + p);
            }
            destroy<kFlat, false>(P, S, e, t, act, cur, nxt, r, k, slot, parity);
        }
    }
}

__global__ void __launch_bounds__(kListThreads, 1) k_peel_lists(const __grid_constant__ ListParams P) {
    __shared__ ListShared S;
    uint32_t* ctrl = P.ctrl;
    if (__syncthreads_or(failed(ctrl))) return;  // the same for all blocks: set, if at all, by earlier kernels
    const uint32_t lane = lane_id();
    const uint32_t tid = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t nthreads = gridDim.x * blockDim.x;
    // chunks go to the blocks in turn: few chunks do not crowd on few SMs (R-MAT 16: peel kernel
    // 4.96 -> 4.29 ms)
    const uint32_t nwarps = nthreads >> 5, gwarp = (threadIdx.x >> 5) * gridDim.x + blockIdx.x;
    // the clock and the logs belong to a thread that is not the barrier's
    const bool scribe = blockIdx.x == 0 && threadIdx.x == blockDim.x - 1;
    if (threadIdx.x == 0) {
        S.queued = 0;
        S.min_sup = S.min_id = kDead;
        S.walk = 0;
        S.walked = 0;
    }
    if (scribe) {
        for (int i = 0; i < 6; ++i) S.ns[i] = 0;
        S.ns[6] = global_ns();
    }
    __syncthreads();
    // the phase that barrier `epoch` closes uses ring slot epoch & 3; slot (epoch + 2) & 3 is cleared
    // meanwhile (its last readers arrived at barrier epoch - 1)
    auto clear_slot = [&](uint32_t epoch) {
        if (scribe) {
            uint4* slot = reinterpret_cast<uint4*>(ctrl + kLRing + kLSlotWords * (epoch & 3));
            slot[0] = make_uint4(0, 0, 0, 0);
            slot[1] = make_uint4(0, kDead, kDead, 0);
        }
    };
    auto phase = [&](int kind) {
        if (scribe) {
            const unsigned long long now = global_ns();
            S.ns[kind] += now - S.ns[6];
            S.ns[6] = now;
        }
    };
    const uint64_t phase_units = 2ull * P.m;  // work that a level phase's barrier covers
    uint32_t epoch = 0, parity = 0;  // parity: the chunk buffer the next frontier is written to
    clear_slot(1);
    clear_slot(2);
    {
        uint4* st4 = reinterpret_cast<uint4*>(P.st);
        const uint64_t n16 = ((uint64_t)P.m + 15) / 16;
#pragma unroll 1
        for (uint64_t i = tid; i < n16; i += nthreads) st4[i] = make_uint4(0, 0, 0, 0);
    }
    if (!list_barrier<false>(P, S, epoch, phase_units)) return;
    phase(0);
    ++epoch;

    uint32_t r = 0, level = 0, k_last = 2, live = P.m, start = 0, swept = 0;
    while (live) {
        if (scribe) S.ns[7] = S.ns[6];
        if (threadIdx.x == 0) {
            S.walked += S.walk;
            S.walk = 0;
        }
        // level start: stream the supports (removed edges have the top bit) from the smallest id
        // alive at the last scan; collect the frontier of level k_last+1 and the minimum support
        uint32_t k = k_last + 1;
        clear_slot(epoch + 2);
        {
            uint32_t mn = kDead, mid = kDead;
            const uint4* sup4 = reinterpret_cast<const uint4*>(P.sup);
            const uint64_t m4 = ((uint64_t)P.m + 3) / 4;
            constexpr int kScan = 2;  // 16-byte loads in flight per lane
#pragma unroll 1
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
                    uint32_t sv[4] = {q4[u].x, q4[u].y, q4[u].z, q4[u].w};
                    bool low = false;
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        const uint64_t j = 4 * i + c;
                        if (j >= P.m) sv[c] = kDead;
                        if (sv[c] < 0x80000000u) {
                            mn = min(mn, sv[c]);
                            mid = min(mid, (uint32_t)j);
                        }
                        low = low || sv[c] <= k - 3;
                    }
                    if (!__any_sync(kFullMask, low)) continue;
#pragma unroll 1
                    for (uint32_t c = 0; c < 4; ++c) {
                        const uint32_t sj = c == 0 ? sv[0] : c == 1 ? sv[1] : c == 2 ? sv[2] : sv[3];
                        enqueue(P, S, (uint32_t)(4 * i) + c, sj <= k - 3, r + 1, k, epoch & 3, parity);
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
                uint32_t* slot = ctrl + kLRing + kLSlotWords * (epoch & 3);
                atomicMin(slot + kLMin, S.min_sup);
                atomicMin(slot + kLMinId, S.min_id);
                S.min_sup = S.min_id = kDead;
            }
            flush(P, S, r + 1, k, epoch & 3, parity);
        }
        if (!list_barrier<true>(P, S, epoch, phase_units)) return;
        phase(1);
        ++epoch;
        start = S.front.min_id;
        if (S.front.min_sup + 3 != k) {
            // level k_last+1 is empty: the next non-empty level is the minimum support + 3
            k = S.front.min_sup + 3;
            clear_slot(epoch + 2);
#pragma unroll 1
            for (uint64_t j0 = start + tid - lane; j0 < P.m; j0 += nthreads) {
                const uint64_t j = j0 + lane;
                const uint32_t sj = j < P.m ? __ldcg(P.sup + j) : kDead;
                enqueue(P, S, (uint32_t)j, sj <= k - 3, r + 1, k, epoch & 3, parity);
            }
            __syncthreads();
            flush(P, S, r + 1, k, epoch & 3, parity);
            if (!list_barrier<false>(P, S, epoch, phase_units)) return;
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
            if (E == live || k == 3) {
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
#pragma unroll 1
                for (uint64_t i = tid; i < P.m; i += nthreads) {
                    const uint32_t s = __ldcg(P.st + i);
                    if (s != 0 && s != keep && s != kOld) P.st[i] = (uint8_t)kOld;
                }
                if (!list_barrier<false>(P, S, epoch, phase_units)) return;
                phase(4);
                ++epoch;
                swept = r - 1;
            }
            clear_slot(epoch + 2);
            run_chunks(P, S, P.ch[from], C, gwarp, nwarps, r, k, epoch & 3, parity);
            // edges whose chunks did not fit the buffer: one warp per edge
#pragma unroll 1
            for (uint32_t i = gwarp; i < B; i += nwarps) {
                const uint32_t e = __ldcg(P.big[from] + i);
                const uint64_t t0 = P.tptr[e], t1 = P.tptr[e + 1];
#pragma unroll 1
                for (uint64_t p0 = t0; p0 < t1; p0 += 32) {
                    const uint32_t ea[1] = {e};
                    const bool act[1] = {p0 + lane < t1};
                    const uint2 t[1] = {act[0] ? __ldcs(P.tri + p0 + lane) : make_uint2(0, 0)};
                    destroy<1, false>(P, S, ea, t, act, stamp_of(r), stamp_of(r + 1), r, k, epoch & 3, parity);
                }
            }
            __syncthreads();
            flush(P, S, r + 1, k, epoch & 3, parity);
            if (!list_barrier<false>(P, S, epoch, (uint64_t)C * kChunk + (B ? phase_units : 0ull))) return;
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
    if (threadIdx.x == 0 && S.walked + S.walk)
        atomicAdd(reinterpret_cast<unsigned long long*>(ctrl + kPWalk), S.walked + S.walk);
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

// Self-test: a barrier that one block never reaches; *passed counts the blocks that got past it.
__global__ void k_list_barrier_probe(const __grid_constant__ ListParams P, uint32_t* passed) {
    __shared__ ListShared S;
    if (threadIdx.x == 0) S.queued = 0;
    __syncthreads();
    if (list_barrier<false, 1>(P, S, 0, 0) && threadIdx.x == 0) atomicAdd(passed, 1u);
}

// sup += supx, what it was into ycount (the claimed part of each list), list starts (tptr[m] is the
// total, three per triangle) and ends.  With rows (symmetric row lengths), also the entries of edges most
// of whose endpoint's neighbours are common ones, near-cliques, the edges in triangles and their least
// support (walks_rows).  More than `cap` entries, what the buffer of a call holds that does not wait for the
// total, are an error: nothing is written to it.  Two blocks an SM: with one, R-MAT 20 takes 0.04 ms more.
template <bool kChained>
__global__ void __launch_bounds__(kScanThreads, 2) k_list_bounds(uint32_t* __restrict__ sup,
                                                                 const uint32_t* __restrict__ supx,
                                                                 uint32_t* __restrict__ ycount, uint32_t m,
                                                                 uint64_t* __restrict__ tptr,
                                                                 uint64_t* __restrict__ ends,
                                                                 const uint32_t* __restrict__ rows,
                                                                 const uint32_t* __restrict__ e_src,
                                                                 const uint32_t* __restrict__ o_col, uint64_t cap,
                                                                 Look L) {
    if (kChained) after_previous(sup, supx, ycount, tptr, ends, rows, e_src, o_col);
    __shared__ uint64_t ws[33], s_prefix;
    __shared__ uint32_t s_tile, s_with, s_least;
    if (threadIdx.x == 0) {
        s_with = 0;
        s_least = ~0u;
    }
    if (__syncthreads_or(failed(L.ctrl))) return;
    const uint32_t tile = look_tile(L, &s_tile);
    if (tile == kNoTile) return;
    const uint64_t j0 = (uint64_t)tile * kScanTile + (uint64_t)threadIdx.x * kScanItems;
    uint32_t y[kScanItems], v[kScanItems];
    const bool whole = j0 + kScanItems <= m;
    if (whole) {
        const uint4 a = *reinterpret_cast<const uint4*>(sup + j0), b = *reinterpret_cast<const uint4*>(supx + j0);
        y[0] = a.x, y[1] = a.y, y[2] = a.z, y[3] = a.w;
        v[0] = a.x + b.x, v[1] = a.y + b.y, v[2] = a.z + b.z, v[3] = a.w + b.w;
        *reinterpret_cast<uint4*>(ycount + j0) = a;
        *reinterpret_cast<uint4*>(sup + j0) = make_uint4(v[0], v[1], v[2], v[3]);
    } else {
#pragma unroll
        for (uint32_t i = 0; i < kScanItems; ++i) {
            y[i] = v[i] = 0;
            if (j0 + i < m) {
                y[i] = sup[j0 + i];
                v[i] = y[i] + supx[j0 + i];
                ycount[j0 + i] = y[i];
                sup[j0 + i] = v[i];
            }
        }
    }
    static_assert(kScanItems == 4, "four supports a thread");
    uint64_t end;
    uint64_t at = tile_scan<uint64_t>(L, tile, (uint64_t)v[0] + v[1] + v[2] + v[3], ws, &s_prefix, &end), local = 0;
#pragma unroll
    for (uint32_t i = 0; i < kScanItems; ++i) {
        if (j0 + i < m) {
            tptr[j0 + i] = at;
            at += v[i];
            ends[j0 + i] = at;
            if (rows && 16 * (uint64_t)(v[i] + 1) >= 15 * (uint64_t)min(rows[e_src[j0 + i]], rows[o_col[j0 + i]]))
                local += v[i];
            if (j0 + i == m - 1) {
                tptr[m] = at;
                L.ctrl[kCtrlTriLo] = (uint32_t)at;
                L.ctrl[kCtrlTriHi] = (uint32_t)(at >> 32);
                if (at > cap) atomicOr(&L.ctrl[kCtrlError], kErrListSpace);
            }
        }
    }
    if (!rows) return;
    uint32_t with = 0, least = ~0u;
#pragma unroll
    for (uint32_t i = 0; i < kScanItems; ++i) {
        with += v[i] != 0;
        least = v[i] ? min(least, v[i]) : least;
    }
    with = __reduce_add_sync(kFullMask, with);
    least = __reduce_min_sync(kFullMask, least);
    if (lane_id() == 0) {
        atomicAdd(&s_with, with);
        atomicMin(&s_least, least);
    }
    __syncthreads();
    if (threadIdx.x == 0 && s_with) {
        atomicAdd(L.ctrl + kListWith, s_with);
        atomicMax(L.ctrl + kListLeast, ~s_least);
    }
    for (int o = 16; o > 0; o >>= 1) local += __shfl_xor_sync(kFullMask, local, o);
    if (lane_id() == 0 && local)
        atomicAdd(reinterpret_cast<unsigned long long*>(L.ctrl + kListLocal), (unsigned long long)local);
}

}  // namespace

namespace {

bool grow_lists(kt_engine* e, uint64_t entries) {
    free_lists(e);
    void* p = nullptr;
    if (cudaMalloc(&p, entries * sizeof(uint2)) != cudaSuccess) {
        (void)cudaGetLastError();
        return false;
    }
    e->lists = static_cast<uint2*>(p);
    e->list_cap = entries;
    return true;
}

// Whether the current graph takes lists: reads its triangle count and sizes the list buffer.
int want_lists(kt_engine* e, bool* use) {
    *use = false;
    int rc;
    if ((rc = sync_and_check(e))) return rc;
    const uint64_t total = (uint64_t)e->h_ctrl[kCtrlTriHi] << 32 | e->h_ctrl[kCtrlTriLo];
    const uint64_t local = (uint64_t)e->h_ctrl[kListLocal + 1] << 32 | e->h_ctrl[kListLocal];
    if (walks_rows(e->m, e->h_ctrl[kListWith], total, local, ~e->h_ctrl[kListLeast])) return KT_OK;
    const uint64_t need = std::max<uint64_t>(total, 1);
    if (need > e->list_cap) {
        const uint64_t want = buffer_entries(total, e->list_limit);
        if (want == 0) return KT_OK;  // walk rows instead
        size_t free_bytes = 0, all_bytes = 0;
        if ((rc = check_cuda(cudaMemGetInfo(&free_bytes, &all_bytes), "free device memory"))) return rc;
        if (want * sizeof(uint2) > (free_bytes + e->list_cap * sizeof(uint2)) / 2) return KT_OK;
        if (!grow_lists(e, want)) return KT_OK;
    }
    e->list_need = need;
    *use = true;
    return KT_OK;
}

}  // namespace

void free_lists(kt_engine* e) {
    if (!e->lists) return;
    drop_replay(e);  // a captured pipeline may point to them
    cudaFree(e->lists);  // (waits for the device)
    e->lists = nullptr;
    e->list_cap = 0;
}

void reserve_small_lists(kt_engine* e, uint64_t max_edges) {
    const uint64_t want = most_entries(std::min<uint64_t>(max_edges, kSmallLists));
    if (e->lists_allowed && want > e->list_cap && want <= e->list_limit / sizeof(uint2)) grow_lists(e, want);
}

cudaError_t alloc_device(kt_engine* e, void** p, size_t bytes) {
    cudaError_t err = cudaMalloc(p, bytes);
    if (err != cudaErrorMemoryAllocation || !e->lists) return err;
    (void)cudaGetLastError();
    free_lists(e);
    return cudaMalloc(p, bytes);
}

int peel_lists(kt_engine* e, bool* done) {
    int rc;
    const uint32_t m = e->m;
    // the sort's key buffers are free after the build: list starts, and ends for the fill
    uint64_t* tptr = e->key_a;
    uint64_t* ends = e->key_b;
    // a repeated call does what the call did; a small graph's lists fit whatever it is: neither waits
    const bool small = !e->trusted && small_lists(m, e->list_cap);
    if (e->trusted) e->list_need = repeat_lists(e->last.list_need, e->list_cap) ? e->last.list_need : 0;
    else e->list_need = small ? most_entries(m) : 0;
    *done = e->list_need != 0;
    if ((rc = launch_chained(e, "k_list_bounds", e->chained ? k_list_bounds<true> : k_list_bounds<false>,
                             ceil_div(m, kScanTile), kScanThreads, 0, e->sup, e->rnd, e->tr, m, tptr, ends,
                             e->trusted || small ? nullptr : e->s_len, e->e_src, e->o_col,
                             *done ? e->list_cap : ~0ull, next_look(e))) ||
        (!e->trusted && !small && (rc = want_lists(e, done))) || !*done || (rc = fill_lists(e, tptr, ends)))
        return rc;
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

int list_timeout_probe(kt_engine* e, uint64_t timeout_ns) {
    e->ctrl_fresh = false;
    int rc = check_cuda(cudaMemsetAsync(e->ctrl, 0, sizeof(uint32_t) * kCtrlWords, e->stream), "clear control block");
    if (rc) return rc;
    ListParams P{};
    P.ctrl = e->ctrl;
    P.wait_base_ns = timeout_ns;
    uint32_t* passed = e->ctrl + kPRounds;
    void* args[] = {&P, &passed};
    if ((rc = check_cuda(cudaLaunchCooperativeKernel((const void*)k_list_barrier_probe, dim3(2), dim3(32), args, 0,
                                                     e->stream), "cooperative launch of k_list_barrier_probe")))
        return rc;
    count_launch(e);
    rc = sync_and_check(e);
    if (rc != KT_ERR_TIMEOUT || e->h_ctrl[kPRounds])
        return rc && rc != KT_ERR_TIMEOUT ? rc : fail(KT_ERR_INTERNAL, "list barrier probe: the wait did not expire");
    return fail(KT_ERR_TIMEOUT, "list barrier probe: wait expired as intended");
}

}  // namespace kt
