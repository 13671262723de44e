// A stable LSD radix sort for the CSR build, one kernel a digit.
//
// It replaces the per-row CPU quicksort of the reference build (graph.cu:462-476 "Sort outgoing
// edges ... on CPU").  Every digit's histogram is counted by the kernel that makes the keys (or by
// k_digit_counts), so a pass reads the keys once: a tile counts its digits and publishes the counts, then
// ranks its keys by warp ballots, arranges itself in digit order in shared memory, learns where its
// digits' runs start from its predecessors (decoupled look-back, one word a digit), and writes runs of
// consecutive positions.  The first pass can make the values (entry indices) itself.
//
// Bound: the serial chain of a tile (ticket, loads, counts, ranks, look-back, runs) at half occupancy, 64
// registers, issue active 47 % - and for small inputs the launches.  A pass over 30 M keys with values
// takes 0.255 ms, 2.8 TB/s of keys and values (0.31 ms when the counts were published after the ranks
// and a tile's places were added up from three tables; histogram, scan and scatter kernels: 0.33 ms); a
// pass over 64,000 entries is one launch instead of four.

#include <algorithm>
#include <utility>
#include <vector>

#include "kt_engine.h"
#include "kt_look.cuh"

namespace kt {

namespace {

constexpr int kDigits = 256;
// Large tiles: 512 threads of 12 keys, two blocks an SM.  Build of R-MAT 20 / symmetrize of 16.8 M edges:
// 2.61 / 0.96 ms with 12 keys, 2.63 / 0.97 with 10, 2.67 / 1.00 with 8, 2.68 / 1.02 with 14; three blocks of 6
// keys 2.66 / 1.04, 256 threads of 8 keys 2.75 / 1.12.
constexpr int kLargeThreads = 512, kLargeItems = (int)kLargeTile / kLargeThreads;
constexpr int kSmallThreads = 256, kSmallItems = (int)kSmallTile / kSmallThreads;

// Digit counts of all passes for keys that are there already.
__global__ void __launch_bounds__(256) k_digit_counts(const uint64_t* __restrict__ keys, uint64_t n, unsigned shift,
                                                      unsigned passes, uint32_t* __restrict__ counts) {
    after_previous(keys, counts);
    __shared__ uint32_t h[kMaxDigitPasses * kDigits];
    digit_counts_clear(h, passes);
    for (uint64_t i0 = (uint64_t)blockIdx.x * blockDim.x; i0 < n; i0 += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t i = i0 + threadIdx.x;
        digit_counts_add(h, i < n ? keys[i] >> shift : 0, i < n, passes);
    }
    digit_counts_flush(h, passes, counts);
}

// Shared memory of a pass, by tile shape.
template <int kThreads, int kItems>
struct PassSmem {
    uint32_t wh[kThreads / 32][kDigits];  // per warp: keys of each digit, then the place of the next one in the tile
    uint64_t key[kThreads * kItems];
    uint32_t val[kThreads * kItems];
    uint32_t goff[kDigits];  // where the tile's run of each digit goes, less its start in the tile
    uint32_t ws[2][kDigits / 32];
    uint32_t tile, ok;
};

template <int kThreads, int kItems, bool kVals>
__global__ void __launch_bounds__(kThreads, 1024 / kThreads) k_radix_pass(const uint64_t* __restrict__ kin,
                                                         const uint32_t* __restrict__ vin,
                                                         uint64_t* __restrict__ kout, uint32_t* __restrict__ vout,
                                                         uint64_t n, unsigned shift,
                                                         const uint32_t* __restrict__ counts, Look L) {
    if (kThreads * kItems == (int)kSmallTile) after_previous(kin, vin, kout, vout, counts);
    extern __shared__ __align__(16) unsigned char raw[];
    PassSmem<kThreads, kItems>& S = *reinterpret_cast<PassSmem<kThreads, kItems>*>(raw);
    constexpr int kWarps = kThreads / 32;
    static_assert(kThreads >= kDigits, "the first kDigits threads own one digit each");
    const uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
    const bool owner = threadIdx.x < (uint32_t)kDigits;  // of digit threadIdx.x (whole warps)
    for (uint32_t i = threadIdx.x; i < kWarps * kDigits; i += kThreads) (&S.wh[0][0])[i] = 0;
    if (threadIdx.x == 0) S.ok = 1;
    const uint32_t tile = look_tile(L, &S.tile);
    if (tile == kNoTile) return;
    const uint64_t tbase = (uint64_t)tile * (kThreads * kItems);
    const uint32_t left = (uint32_t)min((uint64_t)(kThreads * kItems), n - tbase);  // keys of the tile
    const uint32_t p0 = warp * (32 * kItems) + lane;  // this lane's first one
    uint64_t key[kItems];
#pragma unroll
    for (int s = 0; s < kItems; ++s) {
        const uint32_t p = p0 + (uint32_t)s * 32;
        key[s] = p < left ? kin[tbase + p] : 0ull;
    }
    // the counts first: the tile's successors wait for them, not for its ranks
#pragma unroll
    for (int s = 0; s < kItems; ++s)
        if (p0 + (uint32_t)s * 32 < left) atomicAdd(&S.wh[warp][(uint32_t)(key[s] >> shift) & 255u], 1u);
    __syncthreads();
    uint32_t count = 0, all = 0;  // keys of digit threadIdx.x in the tile, and in all tiles
    uint32_t x = 0, y = 0;
    if (owner) {
#pragma unroll
        for (int w = 0; w < kWarps; ++w) count += S.wh[w][threadIdx.x];
        all = counts[threadIdx.x];
        st_relaxed_u64(L.words + (uint64_t)tile * kDigits + threadIdx.x,
                       look_word(tile ? kLookAggregate : kLookInclusive, L.tag, count));
        // exclusive scans over the digits: starts in the tile and in the output
        x = count;
        y = all;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t a = __shfl_up_sync(kFullMask, x, o), b = __shfl_up_sync(kFullMask, y, o);
            if (lane >= (uint32_t)o) {
                x += a;
                y += b;
            }
        }
        if (lane == 31) {
            S.ws[0][warp] = x;
            S.ws[1][warp] = y;
        }
    }
    __syncthreads();
    uint32_t start = 0, toff = 0;
    if (owner) {
        uint32_t bx = 0, by = 0;
#pragma unroll
        for (int w = 0; w < kDigits / 32; ++w) {
            bx += w < (int)warp ? S.ws[0][w] : 0u;
            by += w < (int)warp ? S.ws[1][w] : 0u;
        }
        toff = bx + x - count;
        start = by + y - all;
        uint32_t run = toff;
#pragma unroll
        for (int w = 0; w < kWarps; ++w) {
            const uint32_t c = S.wh[w][threadIdx.x];
            S.wh[w][threadIdx.x] = run;
            run += c;
        }
    }
    __syncthreads();
    // the leader of each set of equal digits claims its places, four steps at a time, without waiting for
    // the atomics' results in between (all twelve at once spill: symmetrize 0.93 ms, 0.90 in fours)
    static_assert(kItems % 4 == 0, "steps in groups of four");
    uint32_t rk[kItems];
#pragma unroll
    for (int s0 = 0; s0 < kItems; s0 += 4) {
        uint32_t first[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int s = s0 + q;
            const bool valid = p0 + (uint32_t)s * 32 < left;
            const uint32_t d = valid ? ((uint32_t)(key[s] >> shift) & 255u) : 256u;
            // lanes with the same digit, bit by bit (match.any instead of the eight ballots made the
            // warps wait on its result: short-scoreboard stalls 11 against 2 cycles an instruction)
            uint32_t peers = __ballot_sync(kFullMask, valid);
            peers = valid ? peers : 0u;
#pragma unroll
            for (int b = 0; b < 8; ++b) {
                const uint32_t ones = __ballot_sync(kFullMask, d >> b & 1u);
                peers &= (d >> b & 1u) ? ones : ~ones;
            }
            const uint32_t leader = __ffs(peers) - 1;
            first[q] = 0;
            if (valid && lane == leader) first[q] = atomicAdd(&S.wh[warp][d], __popc(peers));
            __syncwarp();
            rk[s] = leader << 8 | __popc(peers & lanemask_lt());
        }
#pragma unroll
        for (int q = 0; q < 4; ++q)
            rk[s0 + q] = __shfl_sync(kFullMask, first[q], rk[s0 + q] >> 8) + (rk[s0 + q] & 255u);
    }
#pragma unroll
    for (int s = 0; s < kItems; ++s) {
        const uint32_t p = p0 + (uint32_t)s * 32;
        if (p < left) {
            S.key[rk[s]] = key[s];
            if (kVals) S.val[rk[s]] = vin ? vin[tbase + p] : (uint32_t)tbase + p;
        }
    }
    // the owners look back, four predecessors at a time
    if (owner) {
        uint64_t prefix = 0;
        if (tile) {
            LookWait wait;
            int64_t t = (int64_t)tile - 1;
            bool done = false;
            while (!done) {
                unsigned long long w[4];
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    w[q] = t - q >= 0 ? ld_relaxed_u64(L.words + (uint64_t)(t - q) * kDigits + threadIdx.x)
                                      : look_word(kLookInclusive, L.tag, 0);
                int used = 0;
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    if (!done && used == q && look_valid(w[q], L.tag)) {
                        prefix += (uint64_t)w[q] & kLookValue;
                        done = (w[q] >> 62) == kLookInclusive;
                        ++used;
                    }
                }
                t -= used;
                if (!done && used == 0 && !wait.again(L)) {
                    S.ok = 0;
                    break;
                }
            }
            st_relaxed_u64(L.words + (uint64_t)tile * kDigits + threadIdx.x,
                           look_word(kLookInclusive, L.tag, prefix + count));
        }
        S.goff[threadIdx.x] = start + (uint32_t)prefix - toff;
    }
    __syncthreads();
    if (!S.ok) return;
    for (uint32_t i = threadIdx.x; i < left; i += kThreads) {
        const uint64_t k = S.key[i];
        const uint64_t pos = S.goff[(uint32_t)(k >> shift) & 255u] + i;  // modulo 2^32
        if ((uint32_t)pos < n) {
            kout[(uint32_t)pos] = k;
            if (kVals) vout[(uint32_t)pos] = S.val[i];
        }
    }
}

// Starts a session: clears the control block (if asked to), the degrees, the look-back words and
// the digit counts and tickets; the row marks start at n.
__global__ void k_session(uint32_t* __restrict__ ctrl, uint32_t ctrl_words, uint32_t n, uint32_t* __restrict__ deg,
                          uint32_t deg_words, uint4* __restrict__ words, uint64_t quads, uint32_t* __restrict__ counts,
                          uint32_t count_words) {
    after_previous(ctrl, deg, words, counts);
    const uint64_t tid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x, step = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i = tid; i < ctrl_words; i += step) ctrl[i] = i == kCtrlBigRow || i == kCtrlTinyRow ? n : 0u;
    for (uint64_t i = tid; i < deg_words; i += step) deg[i] = 0;
    for (uint64_t i = tid; i < quads; i += step) words[i] = make_uint4(0, 0, 0, 0);
    for (uint64_t i = tid; i < count_words; i += step) counts[i] = 0;
}

// Self-test: takes a tile's number without running it, so that the next tile's look-back runs out.
__global__ void k_drop_tile(Look L) { atomicAdd(L.tickets + L.tag, 1u); }

// Self-test: one block's look-back as in a scan.
__global__ void k_look_probe(Look L, uint32_t* __restrict__ prefix) {
    __shared__ uint32_t s_tile;
    const uint32_t tile = look_tile(L, &s_tile);
    if (tile == kNoTile) return;
    const uint64_t p = look_back(L, tile, 1);
    if (threadIdx.x == 0) *prefix = (uint32_t)p;
}

template <int kThreads, int kItems, bool kVals>
int launch_pass(kt_engine* e, const uint64_t* kin, const uint32_t* vin, uint64_t* kout, uint32_t* vout, uint64_t n,
                unsigned shift, const uint32_t* counts, const Look& L) {
    const int smem = (int)sizeof(PassSmem<kThreads, kItems>);
    int rc = KT_OK;
    if (smem > 48 * 1024)
        rc = check_cuda(cudaFuncSetAttribute(k_radix_pass<kThreads, kItems, kVals>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize, smem),
                        "shared memory of k_radix_pass");
    if (rc) return rc;
    const uint64_t tiles = (n + kThreads * kItems - 1) / (kThreads * kItems);
    if (kThreads * kItems == (int)kSmallTile)
        return launch_chained(e, "k_radix_pass", k_radix_pass<kThreads, kItems, kVals>, (uint32_t)tiles, kThreads, smem,
                              kin, vin, kout, vout, n, shift, counts, L);
    k_radix_pass<kThreads, kItems, kVals><<<(uint32_t)tiles, kThreads, smem, e->stream>>>(kin, vin, kout, vout, n, shift,
                                                                                         counts, L);
    count_launch(e);
    return check_launch(e, "k_radix_pass");
}

}  // namespace

int begin_session(kt_engine* e, uint32_t n, uint32_t deg_words, uint64_t words, uint64_t keys) {
    // Small graphs: their kernels are no longer than a launch takes (R-MAT of 2^20 vertices gains nothing, and
    // the pointers that a chained kernel launders cost its build 8 %).  Not on a caller's own stream.
    e->chained = e->lists_allowed && keys <= kSmallSort && n <= kSmallSort;
    if (!e->look || words > e->look_cap) return fail(KT_ERR_INTERNAL, "look-back scratch too small");
    e->look_tag = e->look_count = 0;
    e->look_limit_ns = e->wait_base_ns + e->wait_ns_per_unit * std::max<uint64_t>(keys, n);
    e->ctrl_fresh = false;
    const uint64_t work = std::max<uint64_t>(words / 2, std::max<uint32_t>(deg_words, kCountWords));
    const uint32_t blocks = (uint32_t)std::min<uint64_t>((work + 255) / 256, (uint64_t)e->num_sms * 8);
    return launch_chained(e, "k_session", k_session, blocks, 256, 0, e->ctrl, kCtrlWords, n, e->deg, deg_words,
                          reinterpret_cast<uint4*>(e->look), words / 2, e->digit_counts, kCountWords);
}

Look next_look(kt_engine* e) {
    ++e->look_tag;
    return Look{e->look, e->digit_counts + kLookTags * 256, e->ctrl, e->look_tag, e->look_limit_ns};
}

uint32_t* next_counts(kt_engine* e, unsigned passes) {
    uint32_t* c = e->digit_counts + 256 * e->look_count;
    e->look_count += passes;
    return c;
}

int count_digits(kt_engine* e, const uint64_t* keys, uint64_t n, unsigned shift, unsigned passes, uint32_t* counts) {
    const uint32_t blocks = (uint32_t)std::min<uint64_t>((n + 1023) / 1024, (uint64_t)e->num_sms * 8);
    return launch_chained(e, "k_digit_counts", k_digit_counts, blocks, 256, 0, keys, n, shift, passes, counts);
}

int radix_passes(kt_engine* e, uint64_t* key_a, uint32_t* val_a, uint64_t* key_b, uint32_t* val_b, uint64_t n,
                 unsigned shift, unsigned passes, const uint32_t* counts, int* result_in_b) {
    *result_in_b = 0;
    uint64_t *kin = key_a, *kout = key_b;
    uint32_t *vin = nullptr, *vout = val_b;  // the first pass numbers the keys
    for (unsigned p = 0; p < passes; ++p) {
        const Look L = next_look(e);
        int rc;
        if (n <= kSmallSort)
            rc = val_a ? launch_pass<kSmallThreads, kSmallItems, true>(e, kin, vin, kout, vout, n, shift + 8 * p, counts + 256 * p, L)
                       : launch_pass<kSmallThreads, kSmallItems, false>(e, kin, vin, kout, vout, n, shift + 8 * p, counts + 256 * p, L);
        else
            rc = val_a ? launch_pass<kLargeThreads, kLargeItems, true>(e, kin, vin, kout, vout, n, shift + 8 * p, counts + 256 * p, L)
                       : launch_pass<kLargeThreads, kLargeItems, false>(e, kin, vin, kout, vout, n, shift + 8 * p, counts + 256 * p, L);
        if (rc) return rc;
        std::swap(kin, kout);
        if (val_a) {
            vin = vout;
            vout = vin == val_b ? val_a : val_b;
        }
        *result_in_b ^= 1;
    }
    return KT_OK;
}

int look_timeout_probe(kt_engine* e, uint64_t timeout_ns) {
    constexpr uint64_t kKeys = 2 * kSmallTile;
    int rc;
    if ((!e->look || e->cap_entries < kKeys) &&
        (rc = reserve(e, e->cap_nodes, std::max<uint64_t>(e->cap_entries, kKeys))))
        return rc;
    std::vector<uint64_t> out(kKeys);
    for (int scan = 0; scan < 2; ++scan) {
        if ((rc = begin_session(e, 0, 0, look_words(kKeys), kKeys))) return rc;
        e->look_limit_ns = timeout_ns;
        if ((rc = check_cuda(cudaMemsetAsync(e->key_a, 0, kKeys * 8, e->stream), "clear keys")) ||
            (rc = check_cuda(cudaMemsetAsync(e->key_b, 0xff, kKeys * 8, e->stream), "mark keys")))
            return rc;
        // tile 1 waits for a tile 0 that nobody runs, with every other kernel of the session behind it
        const Look L = next_look(e);
        k_drop_tile<<<1, 1, 0, e->stream>>>(L);
        if (scan)
            k_look_probe<<<1, 32, 0, e->stream>>>(L, reinterpret_cast<uint32_t*>(e->key_a));
        else
            k_radix_pass<kSmallThreads, kSmallItems, false>
                <<<1, kSmallThreads, (int)sizeof(PassSmem<kSmallThreads, kSmallItems>), e->stream>>>(
                    e->key_a, nullptr, e->key_b, nullptr, kKeys, 0, next_counts(e, 1), L);
        count_launch(e, 2);
        int in_b = 0;
        if ((rc = check_launch(e, "look-back probe")) ||
            (rc = radix_passes(e, e->key_a, nullptr, e->key_b, nullptr, kKeys, 0, 1, next_counts(e, 1), &in_b)) ||
            (rc = check_cuda(cudaMemcpyAsync(out.data(), e->key_b, kKeys * 8, cudaMemcpyDeviceToHost, e->stream),
                             "read keys")))
            return rc;
        rc = sync_and_check(e);
        if (rc != KT_ERR_TIMEOUT) return rc ? rc : fail(KT_ERR_INTERNAL, "look-back probe: the wait did not expire");
        for (const uint64_t k : out)
            if (k != ~0ull) return fail(KT_ERR_INTERNAL, "look-back probe: keys written after the wait expired");
    }
    return fail(KT_ERR_TIMEOUT, "look-back probe: waits expired as intended");
}

}  // namespace kt
