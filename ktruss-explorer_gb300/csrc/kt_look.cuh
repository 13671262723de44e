// Decoupled look-back: the device side of the one-pass scans and radix passes of the CSR build.
//
// A kernel's tiles take numbers from a ticket, so a tile's predecessors are always running or done.
// Each tile publishes its aggregate, adds up its predecessors' words backwards until it meets an
// inclusive one, and publishes its own inclusive prefix.  A word is flag << 62 | tag << 56 | value:
// every launch of a session has a tag of its own, so the words of earlier launches need no clearing.
// Every wait is bounded: past the session's limit (kt_engine_set_wait_limit) it sets kErrTimeout and gives
// up, and every kernel that would index by what such a launch left behind returns at once when it sees that bit.
#pragma once

#include "kt_device.cuh"

namespace kt {

constexpr uint64_t kLookValue = (1ull << 56) - 1;
constexpr uint32_t kLookTags = 32;  // launches of one session
enum : uint64_t { kLookAggregate = 1, kLookInclusive = 2 };

struct Look {
    unsigned long long* words;
    uint32_t* tickets;  // one per tag
    uint32_t* ctrl;
    uint32_t tag;
    uint64_t limit_ns;
};

__device__ __forceinline__ unsigned long long ld_relaxed_u64(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ void st_relaxed_u64(unsigned long long* p, unsigned long long v) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

__device__ __forceinline__ unsigned long long look_word(uint64_t flag, uint32_t tag, uint64_t value) {
    return flag << 62 | (unsigned long long)tag << 56 | value;
}

__device__ __forceinline__ bool look_valid(unsigned long long w, uint32_t tag) {
    return (w >> 62) != 0 && ((uint32_t)(w >> 56) & 63u) == tag;
}

__device__ __forceinline__ bool timed_out(const uint32_t* ctrl) { return __ldca(ctrl + kCtrlError) & kErrTimeout; }

// A waiting thread's bound: false when the wait should be given up.
struct LookWait {
    uint32_t spins = 0;
    uint64_t t0 = 0;
    __device__ __forceinline__ bool again(const Look& L) {
        if ((++spins & 63u) == 0) {
            if (spins == 64) t0 = global_ns();
            if (ld_acquire(L.ctrl + kCtrlError) & kErrTimeout) return false;
            if (global_ns() - t0 > L.limit_ns) {
                atomicOr(L.ctrl + kCtrlError, kErrTimeout);
                return false;
            }
        }
        return true;
    }
};

// The next tile's number, for the whole block; kNoTile when an earlier wait was given up.
constexpr uint32_t kNoTile = 0xffffffffu;

__device__ __forceinline__ uint32_t look_tile(const Look& L, uint32_t* s_tile) {
    if (threadIdx.x == 0) *s_tile = timed_out(L.ctrl) ? kNoTile : atomicAdd(L.tickets + L.tag, 1u);
    __syncthreads();
    return *s_tile;
}

// Exclusive prefix of `aggregate` over the tiles before `tile`, for all 32 lanes of one warp
// (`aggregate` the same in all of them).
__device__ __forceinline__ uint64_t look_back(const Look& L, uint32_t tile, uint64_t aggregate) {
    const uint32_t lane = lane_id();
    if (lane == 0)
        st_relaxed_u64(L.words + tile, look_word(tile ? kLookAggregate : kLookInclusive, L.tag, aggregate));
    if (tile == 0) return 0;
    uint64_t prefix = 0;
    LookWait wait;
    for (int64_t base = (int64_t)tile - 1; base >= 0;) {
        const int64_t t = base - lane;
        const unsigned long long w = t >= 0 ? ld_relaxed_u64(L.words + t) : look_word(kLookInclusive, L.tag, 0);
        const uint32_t valid = __ballot_sync(kFullMask, look_valid(w, L.tag));
        const uint32_t incl = __ballot_sync(kFullMask, look_valid(w, L.tag) && (w >> 62) == kLookInclusive);
        const uint32_t first = incl ? __ffs(incl) - 1 : 31;  // the last word to add
        if ((~valid & (0xffffffffu >> (31 - first))) != 0) {
            if (!__all_sync(kFullMask, wait.again(L))) break;
            continue;
        }
        uint64_t v = lane <= first ? (uint64_t)w & kLookValue : 0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFullMask, v, o);
        prefix += v;
        if (incl) break;
        base -= 32;
    }
    if (lane == 0) st_relaxed_u64(L.words + tile, look_word(kLookInclusive, L.tag, prefix + aggregate));
    return prefix;
}

// Block-wide exclusive scan of one value per thread (every thread calls it); *total is the sum.
template <class T>
__device__ __forceinline__ T block_exclusive_scan(T v, T* warp_sums, T* total) {
    const uint32_t lane = lane_id(), warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    T x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        T y = __shfl_up_sync(kFullMask, x, o);
        if (lane >= (uint32_t)o) x += y;
    }
    if (lane == 31) warp_sums[warp] = x;
    __syncthreads();
    if (warp == 0) {
        T w = lane < nwarps ? warp_sums[lane] : T(0);
        T s = w;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            T y = __shfl_up_sync(kFullMask, s, o);
            if (lane >= (uint32_t)o) s += y;
        }
        if (lane < nwarps) warp_sums[lane] = s - w;
        if (lane == 31) warp_sums[32] = s;
    }
    __syncthreads();
    T r = warp_sums[warp] + x - v;
    *total = warp_sums[32];
    __syncthreads();
    return r;
}

// The block's tile in a one-pass exclusive scan over tiles: `v` per thread -> its global prefix;
// *total is the inclusive prefix of the tile's end.
template <class T>
__device__ __forceinline__ uint64_t tile_scan(const Look& L, uint32_t tile, T v, T* warp_sums, uint64_t* s_prefix,
                                              uint64_t* end) {
    T total;
    const T r = block_exclusive_scan<T>(v, warp_sums, &total);
    if (threadIdx.x < 32) {
        const uint64_t p = look_back(L, tile, (uint64_t)total);
        if (threadIdx.x == 0) *s_prefix = p;
    }
    __syncthreads();
    *end = *s_prefix + (uint64_t)total;
    return *s_prefix + (uint64_t)r;
}

// Digit counts of up to kMaxDigitPasses 8-bit digits, gathered per block in h[passes * 256].
constexpr unsigned kMaxDigitPasses = 8;

__device__ __forceinline__ void digit_counts_clear(uint32_t* h, unsigned passes) {
    for (uint32_t i = threadIdx.x; i < passes * 256; i += blockDim.x) h[i] = 0;
    __syncthreads();
}

// All 32 lanes of a warp call it together.  Sorted inputs give a warp the same high digits: one
// addition for all of its lanes instead of 32 on the same word.
__device__ __forceinline__ void digit_counts_add(uint32_t* h, uint64_t key, bool valid, unsigned passes) {
    const uint32_t act = __ballot_sync(kFullMask, valid);
    if (!act) return;
    for (unsigned p = 0; p < passes; ++p) {
        const uint32_t d = (uint32_t)(key >> (8 * p)) & 255u;
        const uint32_t d0 = __shfl_sync(kFullMask, d, __ffs(act) - 1);
        if (__all_sync(kFullMask, !valid || d == d0)) {
            if (lane_id() == 0) atomicAdd(h + 256 * p + d0, __popc(act));
        } else if (valid) {
            atomicAdd(h + 256 * p + d, 1u);
        }
    }
}

__device__ __forceinline__ void digit_counts_flush(const uint32_t* h, unsigned passes, uint32_t* counts) {
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < passes * 256; i += blockDim.x)
        if (h[i]) atomicAdd(counts + i, h[i]);
}

// A tile of kFlagTile entries, taken kFlagThreads at a time (coalesced), whose flagged entries are
// numbered in order: the block gives each step's warp ballots, then every flagged entry's number is
// flag_number.
constexpr uint32_t kFlagThreads = 512, kFlagSteps = 8, kFlagTile = kFlagThreads * kFlagSteps;
constexpr uint32_t kFlagWarps = kFlagThreads / 32;

struct FlagSmem {
    uint32_t before[kFlagSteps * kFlagWarps];  // flagged entries before each step's warp, in the tile
    uint64_t prefix;
    uint32_t tile, total;
};

// Turns the counts in S.before into exclusive sums (after a __syncthreads by the caller; ends with
// one).  The tile's prefix over all tiles comes from its predecessors.
__device__ __forceinline__ void flag_sums(FlagSmem& S, const Look& L, uint32_t tile) {
    constexpr uint32_t kPer = kFlagSteps * kFlagWarps / 32;
    const uint32_t lane = lane_id();
    if (threadIdx.x < 32) {
        uint32_t c[kPer], sum = 0;
#pragma unroll
        for (uint32_t i = 0; i < kPer; ++i) {
            c[i] = S.before[lane * kPer + i];
            sum += c[i];
        }
        uint32_t incl = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(kFullMask, incl, o);
            if (lane >= (uint32_t)o) incl += t;
        }
        uint32_t at = incl - sum;
#pragma unroll
        for (uint32_t i = 0; i < kPer; ++i) {
            S.before[lane * kPer + i] = at;
            at += c[i];
        }
        const uint32_t total = __shfl_sync(kFullMask, incl, 31);
        const uint64_t p = look_back(L, tile, total);
        if (lane == 0) {
            S.prefix = p;
            S.total = total;
        }
    }
    __syncthreads();
}

constexpr uint32_t kScanThreads = 1024;
constexpr uint32_t kScanItems = 4;
constexpr uint32_t kScanTile = kScanThreads * kScanItems;

}  // namespace kt
