// Device-side TSV ingest: the graph file parsed in HBM instead of by fscanf on the host.
//
// Replaces createCOOFromFile (graph.cu:37-79), which reads "dst src x" triples of unsigned
// decimal numbers separated by any whitespace, 1-based ids, x ignored, rejecting self loops.
// The text is taken in units of 16 bytes, one a thread and step, in registers: bit masks say which
// bytes are digits and where tokens start (a digit that follows a non-digit).  Pass 1 counts the tokens
// of every 16 KB tile and flags bytes that are neither digits nor whitespace; one block turns the counts
// into token numbers.  Pass 2 - which returns at once if the text was refused or holds more entries
// than the caller's buffers - parses the ids, four digits at a time: token t is field t % 3 of entry
// t / 3, converted to 0-based; a number of more than 10 digits or above 2^32-1, an id of 0 and a self
// loop are errors, and the largest id is the vertex count.  Pass 3 looks for self loops among the
// entries that tiles share.  The host reads the outcome once.  Errors carry the position of the first
// offending byte or entry, and the call returns the same statuses as the host reader (KT_ERR_IO,
// KT_ERR_SELF_LOOP) plus KT_ERR_CAPACITY when the output buffers are too small.
//
// Bound: instructions a byte (the text is read twice, the entries are written once): pass 2 issues at
// 79 % of the rate with memory at 16 %.  Measured on 101.6 MB of text with 7.4 M entries: the call 137 us,
// of it the passes 29, 8, 75 and 4 (a byte a thread and step, with a digit loop a token, a pass to
// convert the entries, and allocations and a host scan of the tile counts in each call: 1,159 us; one
// token after the other by the thread that holds its unit: 249 us).

#include <cerrno>
#include <cstdio>
#include <cstring>

#include "kt_device.cuh"
#include "kt_engine.h"

namespace kt {

namespace {

constexpr int kIngestThreads = 256, kIngestWarps = kIngestThreads / 32;
constexpr uint32_t kUnits = 4;                              // 16-byte units a thread
constexpr uint32_t kTileUnits = kUnits * kIngestThreads;    // units a tile, kIngestThreads at a time
constexpr uint32_t kTileBytes = kTileUnits * 16;
constexpr uint32_t kTileTokens = kTileBytes / 2;            // at most: a token and a space are two bytes
constexpr int kScanThreads = 1024;
constexpr uint32_t kScanItems = 8;  // tiles a thread of the scan, each step
constexpr uint32_t kMaxDigits = 10;

// The outcome words (u64) at the start of the ingest scratch: positions of the first errors (all
// ones: none), the complement of the largest id, the tokens.
enum : uint32_t { kErrChar = 0, kErrOverflow = 1, kErrZero = 2, kErrLoop = 3, kMaxId = 4, kTokens = 5, kOutcome = 6 };

// Bytes of w that are not digits: 0x80 in each.
__device__ __forceinline__ uint32_t non_digits(uint32_t w) {
    const uint32_t x = (w ^ 0x30303030u) & 0x7f7f7f7fu;  // 0..9 for digits
    return (x + 0x76767676u | w) & 0x80808080u;
}

// Bytes of w that are neither a space nor a tab, newline or carriage return: 0x80 in each.
__device__ __forceinline__ uint32_t non_spaces(uint32_t w) {
    const uint32_t low = w & 0x7f7f7f7fu;
    const uint32_t all = ((low ^ 0x20202020u) + 0x7f7f7f7fu) & ((low ^ 0x09090909u) + 0x7f7f7f7fu) &
                         ((low ^ 0x0a0a0a0au) + 0x7f7f7f7fu) & ((low ^ 0x0d0d0d0du) + 0x7f7f7f7fu);
    return (all | w) & 0x80808080u;
}

// 0x80 marks of four words as 16 bits, first byte lowest.  (The product brings a word's four marks to
// bits 28-31; no two of its terms meet.)
__device__ __forceinline__ uint32_t mark_bits(const uint32_t (&m)[4]) {
    uint32_t r = 0;
#pragma unroll
    for (int i = 3; i >= 0; --i) r = __funnelshift_l(m[i] * 0x00204081u, r, 4);
    return r;
}

// Unit u of the text: 16 bytes, spaces past its end.
__device__ __forceinline__ uint4 load_unit(const unsigned char* __restrict__ text, uint64_t bytes, uint64_t u) {
    const uint64_t at = u * 16;
    if (at + 16 <= bytes && (reinterpret_cast<uintptr_t>(text) & 15) == 0)
        return __ldg(reinterpret_cast<const uint4*>(text + at));
    uint32_t w[4];
    for (int i = 0; i < 4; ++i) {
        w[i] = 0;
        for (int b = 0; b < 4; ++b) {
            const uint64_t p = at + 4 * i + b;
            w[i] |= (uint32_t)(p < bytes ? text[p] : ' ') << (8 * b);
        }
    }
    return make_uint4(w[0], w[1], w[2], w[3]);
}

__device__ __forceinline__ uint4 unit_or_blank(const unsigned char* __restrict__ text, uint64_t bytes, uint64_t u) {
    return u * 16 < bytes ? load_unit(text, bytes, u)
                          : make_uint4(0x20202020u, 0x20202020u, 0x20202020u, 0x20202020u);
}

// Which bytes of unit u start a token, from the marks of its bytes that are not digits.
__device__ __forceinline__ uint32_t token_starts(const unsigned char* __restrict__ text, uint64_t u, uint32_t digits) {
    // whether the byte before the unit is a digit: from the lane before, or from memory
    uint32_t before = __shfl_up_sync(kFullMask, digits >> 15, 1);
    if (lane_id() == 0) {
        const unsigned char c = u > 0 && digits ? text[u * 16 - 1] : ' ';
        before = c >= '0' && c <= '9';
    }
    return digits & ~(digits << 1 | before);
}

__device__ __forceinline__ uint32_t inclusive_scan(uint32_t v) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(kFullMask, v, o);
        if (lane_id() >= (uint32_t)o) v += t;
    }
    return v;
}

// Pass 1: tokens of each tile, and the first byte that is neither a digit nor whitespace.
__global__ void __launch_bounds__(kIngestThreads) k_tsv_count(const unsigned char* __restrict__ text, uint64_t bytes,
                                                              unsigned long long* __restrict__ tile_tokens,
                                                              unsigned long long* __restrict__ out) {
    __shared__ uint32_t wsum[kIngestWarps];
    uint32_t count = 0;
    uint64_t bad = ~0ull;
    uint4 q[kUnits];
    const uint64_t u0 = (uint64_t)blockIdx.x * kTileUnits + threadIdx.x;
#pragma unroll
    for (uint32_t s = 0; s < kUnits; ++s) q[s] = unit_or_blank(text, bytes, u0 + s * kIngestThreads);
#pragma unroll
    for (uint32_t s = 0; s < kUnits; ++s) {
        const uint64_t u = u0 + s * kIngestThreads;
        const uint32_t w[4] = {q[s].x, q[s].y, q[s].z, q[s].w};
        uint32_t other[4], wrong = 0;
#pragma unroll
        for (int i = 0; i < 4; ++i) other[i] = non_digits(w[i]);
        count += __popc(token_starts(text, u, ~mark_bits(other) & 0xffffu));
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            other[i] &= non_spaces(w[i]);
            wrong |= other[i];
        }
        if (wrong) bad = min(bad, u * 16 + __ffs(mark_bits(other)) - 1);
    }
    if (bad != ~0ull) atomicMin(out + kErrChar, (unsigned long long)bad);  // rare: one atomic per offending thread
    count = __reduce_add_sync(kFullMask, count);
    if (lane_id() == 0) wsum[threadIdx.x >> 5] = count;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t total = 0;
#pragma unroll
        for (int w = 0; w < kIngestWarps; ++w) total += wsum[w];
        tile_tokens[blockIdx.x] = total;
    }
}

// Tokens before each tile, and all of them.  One block: a tile in 16 KB of text is one word here, and
// look-back in the counting pass, whose tiles finish almost together, cost more (63 us against 37 + 7).
__global__ void __launch_bounds__(kScanThreads) k_tsv_offsets(unsigned long long* __restrict__ tile_tokens,
                                                              uint64_t tiles, unsigned long long* __restrict__ out) {
    __shared__ uint32_t wsum[kScanThreads / 32];
    const uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
    uint64_t base = 0;
    for (uint64_t t0 = 0; t0 < tiles; t0 += kScanThreads * kScanItems) {
        const uint64_t first = t0 + threadIdx.x * kScanItems;
        uint32_t c[kScanItems], sum = 0;
#pragma unroll
        for (uint32_t i = 0; i < kScanItems; ++i) {
            c[i] = first + i < tiles ? (uint32_t)tile_tokens[first + i] : 0u;
            sum += c[i];
        }
        const uint32_t incl = inclusive_scan(sum);
        if (lane == 31) wsum[warp] = incl;
        __syncthreads();
        static_assert(kScanThreads == 1024, "one lane per warp");
        const uint32_t ws = wsum[lane];
        const uint32_t wincl = inclusive_scan(ws);
        uint64_t at = base + __shfl_sync(kFullMask, wincl - ws, warp) + incl - sum;
        base += __shfl_sync(kFullMask, wincl, 31);
#pragma unroll
        for (uint32_t i = 0; i < kScanItems; ++i) {
            if (first + i < tiles) tile_tokens[first + i] = at;
            at += c[i];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) out[kTokens] = base;
}

// Entries of an accepted text, ~0 otherwise.
__device__ __forceinline__ uint64_t accepted(const unsigned long long* __restrict__ out, uint64_t capacity) {
    const uint64_t tokens = out[kTokens];
    const bool ok = out[kErrChar] == ~0ull && tokens % 3 == 0 && tokens / 3 <= capacity && tokens / 3 < 0xffffffffull;
    return ok ? tokens / 3 : ~0ull;
}

// Four digit values, most significant in the lowest byte, as a number.
__device__ __forceinline__ uint32_t four_digits(uint32_t d) {
    const uint32_t pairs = d * 10 + (d >> 8) & 0x00ff00ffu;  // two numbers below 100
    return __dp2a_lo(pairs, 100u | 1u << 8, 0u);
}

// The digits of the token that starts at byte `at` of the tile, kMaxDigits + 1 at most.
__device__ __forceinline__ uint32_t token_length(const uint16_t* digits, uint32_t at) {
    const uint32_t u = at >> 4;
    const uint32_t run = ((uint32_t)digits[u + 1] << 16 | digits[u]) >> (at & 15);
    return __ffs(~run | 1u << (kMaxDigits + 1)) - 1;
}

// The number at byte `at` of the tile; ~0 if it does not fit 32 bits.
__device__ __forceinline__ uint64_t token_value(const uint32_t* words, const uint16_t* digits, uint32_t at) {
    const uint32_t len = token_length(digits, at), w = at >> 2, sh = 8 * at;  // (funnel shifts take 5 bits)
    const uint32_t b = words[w + 1], c = words[w + 2];
    uint64_t d = (uint64_t)__funnelshift_r(b, c, sh) << 32 | __funnelshift_r(words[w], b, sh);
    if (len < 8) d <<= 64 - 8 * len;  // the first eight digits, right-aligned; digit values below
    const uint32_t v = four_digits((uint32_t)d & 0x0f0f0f0fu) * 10000u + four_digits((uint32_t)(d >> 32) & 0x0f0f0f0fu);
    if (len <= 8) return v;
    if (len > kMaxDigits) return ~0ull;
    const uint32_t x = __funnelshift_r(c, words[w + 3], sh);
    const uint64_t nine = (uint64_t)v * 10 + (x & 0xfu);
    const uint64_t ten = len == 9 ? nine : nine * 10 + (x >> 8 & 0xfu);
    return ten > 0xffffffffull ? ~0ull : ten;
}

// Pass 2: number the tokens in file order and parse them into the entry fields.  The tile's tokens are
// numbered first - each token's position in the text, in shared memory - so that every lane parses one
// and neighbours write neighbouring places.
__global__ void __launch_bounds__(kIngestThreads) k_tsv_parse(const unsigned char* __restrict__ text, uint64_t bytes,
                                                              const unsigned long long* __restrict__ tile_tokens,
                                                              uint64_t capacity, uint32_t* __restrict__ dst,
                                                              uint32_t* __restrict__ src,
                                                              unsigned long long* __restrict__ out) {
    __shared__ __align__(16) uint32_t words[kTileUnits * 4 + 8];  // the tile, and 32 bytes more
    __shared__ uint16_t digits[kTileUnits + 2];
    __shared__ uint16_t at_token[kTileTokens + 4];
    __shared__ uint32_t before[kUnits * kIngestWarps];
    __shared__ uint32_t s_max, s_tokens;
    if (threadIdx.x == 0) s_max = 0;
    if (__syncthreads_or(accepted(out, capacity) == ~0ull)) return;
    const uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
    const uint64_t unit0 = (uint64_t)blockIdx.x * kTileUnits, base = tile_tokens[blockIdx.x];
    uint4 q[kUnits];
    uint32_t starts[kUnits], rank[kUnits];  // token starts, and tokens of the warp before this lane
#pragma unroll
    for (uint32_t s = 0; s < kUnits; ++s) q[s] = unit_or_blank(text, bytes, unit0 + s * kIngestThreads + threadIdx.x);
    if (threadIdx.x < 2) {
        const uint4 x = unit_or_blank(text, bytes, unit0 + kTileUnits + threadIdx.x);
        const uint32_t other[4] = {non_digits(x.x), non_digits(x.y), non_digits(x.z), non_digits(x.w)};
        reinterpret_cast<uint4*>(words)[kTileUnits + threadIdx.x] = x;
        digits[kTileUnits + threadIdx.x] = (uint16_t)~mark_bits(other);
    }
#pragma unroll
    for (uint32_t s = 0; s < kUnits; ++s) {
        const uint32_t u = s * kIngestThreads + threadIdx.x;
        const uint32_t other[4] = {non_digits(q[s].x), non_digits(q[s].y), non_digits(q[s].z), non_digits(q[s].w)};
        const uint32_t mine = ~mark_bits(other) & 0xffffu;
        reinterpret_cast<uint4*>(words)[u] = q[s];
        digits[u] = (uint16_t)mine;
        starts[s] = token_starts(text, unit0 + u, mine);
    }
    // two steps a scan: a warp's tokens of a step are 256 at most
#pragma unroll
    for (uint32_t s = 0; s < kUnits; s += 2) {
        const uint32_t c = __popc(starts[s]) | __popc(starts[s + 1]) << 16, incl = inclusive_scan(c);
        rank[s] = incl - c & 0xffffu;
        rank[s + 1] = incl - c >> 16;
        if (lane == 31) {
            before[s * kIngestWarps + warp] = incl & 0xffffu;
            before[(s + 1) * kIngestWarps + warp] = incl >> 16;
        }
    }
    __syncthreads();
    static_assert(kUnits * kIngestWarps == 32, "one lane per warp and step");
    if (warp == 0) {
        const uint32_t c = before[lane], incl = inclusive_scan(c);
        before[lane] = incl - c;
        if (lane == 31) s_tokens = incl;
    }
    __syncthreads();
    const uint64_t e0 = base / 3;
    const uint32_t r = (uint32_t)(base - 3 * e0);  // the field of the tile's first token
#pragma unroll
    for (uint32_t s = 0; s < kUnits; ++s) {
        uint16_t* p = at_token + r + before[s * kIngestWarps + warp] + rank[s];
        const uint32_t at = (s * kIngestThreads + threadIdx.x) * 16;
        for (uint32_t left = starts[s]; left; left &= left - 1) *p++ = (uint16_t)(at + __ffs(left) - 1);
    }
    __syncthreads();
    // One entry a lane: tokens r to end - 1 are this tile's, the first and last entry may be shared.
    const uint32_t end = r + s_tokens;
    uint32_t mx = 0;
    for (uint32_t k = threadIdx.x; 3 * k < end; k += kIngestThreads) {
        const uint32_t t = 3 * k;
        const bool a_here = t >= r, b_here = t + 1 >= r && t + 1 < end, c_here = t + 2 >= r && t + 2 < end;
        const uint64_t e = e0 + k;
        uint64_t a = ~0ull, b = ~0ull;
        if (a_here) {
            a = token_value(words, digits, at_token[t]);
            if (a <= 0xffffffffull) dst[e] = (uint32_t)a - 1;
        }
        if (b_here) {
            b = token_value(words, digits, at_token[t + 1]);
            if (b <= 0xffffffffull) src[e] = (uint32_t)b - 1;
        }
        // the third field is not kept, but it is a number of 32 bits: looked at if the next token is so far
        const bool c_long = c_here && (t + 3 >= end || at_token[t + 3] - at_token[t + 2] > kMaxDigits);
        const bool c_bad = c_long && token_value(words, digits, at_token[t + 2]) == ~0ull;
        const bool a_bad = a_here && a == ~0ull, b_bad = b_here && b == ~0ull;
        const uint32_t good_a = (uint32_t)(a == ~0ull ? 0 : a), good_b = (uint32_t)(b == ~0ull ? 0 : b);
        mx = max(mx, max(good_a, good_b));
        const bool zero = a == 0 || b == 0, loop = a == b && a != ~0ull && !zero;  // (k_tsv_loops: shared entries)
        if (a_bad || b_bad || c_bad) {
            const uint32_t at = at_token[a_bad ? t : b_bad ? t + 1 : t + 2];
            atomicMin(out + kErrOverflow, (unsigned long long)(unit0 * 16 + at));
        }
        if (zero) atomicMin(out + kErrZero, (unsigned long long)e);
        if (loop) atomicMin(out + kErrLoop, (unsigned long long)e);
    }
    mx = __reduce_max_sync(kFullMask, mx);
    if (lane == 0 && mx) atomicMax(&s_max, mx);
    __syncthreads();
    if (threadIdx.x == 0 && s_max) atomicMin(out + kMaxId, ~(unsigned long long)s_max);
}

// Pass 3: self loops among the entries that a tile's start cuts (an id of 0 reads ~0 and is flagged already).
__global__ void k_tsv_loops(const uint32_t* __restrict__ dst, const uint32_t* __restrict__ src, uint64_t capacity,
                            const unsigned long long* __restrict__ tile_tokens, uint64_t tiles,
                            unsigned long long* __restrict__ out) {
    const uint64_t entries = accepted(out, capacity), i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (entries == ~0ull || i >= tiles) return;
    const uint64_t base = tile_tokens[i], e = base / 3;
    if (base % 3 == 0 || e >= entries) return;
    const uint32_t a = dst[e];
    if (a == src[e] && a != 0xffffffffu) atomicMin(out + kErrLoop, (unsigned long long)e);
}

}  // namespace

int parse_tsv(kt_engine* e, const char* d_text, uint64_t bytes, uint32_t* d_src, uint32_t* d_dst, uint64_t capacity,
              uint64_t* num_entries, uint32_t* num_nodes) {
    *num_entries = 0;
    *num_nodes = 0;
    if (bytes == 0) return KT_OK;
    const unsigned char* text = reinterpret_cast<const unsigned char*>(d_text);
    const uint64_t tiles = (bytes + kTileBytes - 1) / kTileBytes;
    if (tiles > 0x7fffffffull) return fail(KT_ERR_TOO_LARGE, "text of %llu bytes is too large", (unsigned long long)bytes);
    int rc;
    // the engine keeps the scratch: the outcome, and the tokens before each tile (a two-thousandth of the text)
    const uint64_t words = kOutcome + tiles;
    if (words > e->ingest_words) {
        if ((rc = check_cuda(cudaStreamSynchronize(e->stream), "synchronize"))) return rc;
        if (e->ingest) cudaFree(e->ingest);
        e->ingest = nullptr;
        e->ingest_words = 0;
        if ((rc = check_cuda(alloc_device(e, (void**)&e->ingest, sizeof(unsigned long long) * words),
                             "allocate ingest scratch")))
            return rc;
        e->ingest_words = words;
    }
    unsigned long long* out = e->ingest;
    unsigned long long* tile_tokens = out + kOutcome;
    const bool outputs = d_src && d_dst;  // without buffers the text is only counted
    if ((rc = check_cuda(cudaMemsetAsync(out, 0xff, sizeof(unsigned long long) * kOutcome, e->stream), "clear")))
        return rc;
    k_tsv_count<<<(uint32_t)tiles, kIngestThreads, 0, e->stream>>>(text, bytes, tile_tokens, out);
    count_launch(e);
    if ((rc = check_launch(e, "k_tsv_count"))) return rc;
    k_tsv_offsets<<<1, kScanThreads, 0, e->stream>>>(tile_tokens, tiles, out);
    count_launch(e);
    if ((rc = check_launch(e, "k_tsv_offsets"))) return rc;
    if (outputs) {
        k_tsv_parse<<<(uint32_t)tiles, kIngestThreads, 0, e->stream>>>(text, bytes, tile_tokens, capacity, d_dst, d_src, out);
        count_launch(e);
        if ((rc = check_launch(e, "k_tsv_parse"))) return rc;
        k_tsv_loops<<<(uint32_t)((tiles + 255) / 256), 256, 0, e->stream>>>(d_dst, d_src, capacity, tile_tokens, tiles,
                                                                         out);
        count_launch(e);
        if ((rc = check_launch(e, "k_tsv_loops"))) return rc;
    }
    const unsigned long long* res = reinterpret_cast<unsigned long long*>(e->h_ctrl);
    e->ctrl_fresh = false;
    if ((rc = check_cuda(cudaMemcpyAsync(e->h_ctrl, out, sizeof(unsigned long long) * kOutcome, cudaMemcpyDeviceToHost,
                                         e->stream), "read the outcome")) ||
        (rc = check_cuda(cudaStreamSynchronize(e->stream), "synchronize")))
        return rc;
    if (res[kErrChar] != ~0ull)
        return fail(KT_ERR_IO, "byte %llu is neither a digit nor whitespace", (unsigned long long)res[kErrChar]);
    const unsigned long long tokens = res[kTokens];
    if (tokens % 3 != 0)
        return fail(KT_ERR_IO, "entry %llu is not a 'dst src x' triple", (unsigned long long)(tokens / 3 + 1));
    const uint64_t entries = tokens / 3;
    if (entries >= 0xffffffffull) return fail(KT_ERR_TOO_LARGE, "more than 2^32-2 entries");
    if (entries > capacity)
        return fail(KT_ERR_CAPACITY, "the text holds %llu entries, the output buffers %llu",
                    (unsigned long long)entries, (unsigned long long)capacity);
    if (entries && !outputs) return fail(KT_ERR_INVALID_ARG, "null output buffer");
    if (res[kErrOverflow] != ~0ull)
        return fail(KT_ERR_IO, "the number at byte %llu does not fit 32 bits", (unsigned long long)res[kErrOverflow]);
    const unsigned long long zero = res[kErrZero], loop = res[kErrLoop];
    if (zero != ~0ull && zero < loop)
        return fail(KT_ERR_IO, "entry %llu has a 0 vertex id (ids are 1-based)", zero + 1);
    if (loop != ~0ull)
        return fail(KT_ERR_SELF_LOOP, "entry %llu: Edges from a vertex to itself are not allowed!", loop + 1);
    *num_entries = entries;
    *num_nodes = (uint32_t)~res[kMaxId];
    return KT_OK;
}

}  // namespace kt

using kt::check_cuda;
using kt::fail;

extern "C" {

int kt_engine_parse_tsv(kt_engine* e, const char* d_text, uint64_t bytes, uint32_t* d_src, uint32_t* d_dst,
                        uint64_t capacity, uint64_t* num_entries, uint32_t* num_nodes) {
    kt::clear_error();
    if (!e || !num_entries || !num_nodes || (bytes && !d_text))
        return fail(KT_ERR_INVALID_ARG, "kt_engine_parse_tsv: null argument");
    int rc = check_cuda(cudaSetDevice(e->device), "cudaSetDevice");
    if (rc) return rc;
    return kt::parse_tsv(e, d_text, bytes, d_src, d_dst, capacity, num_entries, num_nodes);
}

int kt_engine_read_tsv(kt_engine* e, const char* path, uint32_t* d_src, uint32_t* d_dst, uint64_t capacity,
                       uint64_t* num_entries, uint32_t* num_nodes) {
    kt::clear_error();
    if (!e || !path || !num_entries || !num_nodes) return fail(KT_ERR_INVALID_ARG, "kt_engine_read_tsv: null argument");
    FILE* fp = fopen(path, "rb");
    if (!fp) return fail(KT_ERR_IO, "cannot open %s: %s", path, strerror(errno));
    fseek(fp, 0, SEEK_END);
    const long sz = ftell(fp);
    fseek(fp, 0, SEEK_SET);
    if (sz < 0) {
        fclose(fp);
        return fail(KT_ERR_IO, "cannot size %s", path);
    }
    int rc = check_cuda(cudaSetDevice(e->device), "cudaSetDevice");
    char* h = nullptr;
    char* d = nullptr;
    if (!rc && sz > 0) {
        if (!(rc = check_cuda(cudaMallocHost(&h, (size_t)sz), "allocate pinned staging")) &&
            !(rc = check_cuda(kt::alloc_device(e, (void**)&d, (size_t)sz), "allocate device text"))) {
            if (fread(h, 1, (size_t)sz, fp) != (size_t)sz) rc = fail(KT_ERR_IO, "short read on %s", path);
            if (!rc) rc = check_cuda(cudaMemcpyAsync(d, h, (size_t)sz, cudaMemcpyHostToDevice, e->stream), "H2D");
        }
    }
    fclose(fp);
    if (!rc) rc = kt::parse_tsv(e, d, (uint64_t)sz, d_src, d_dst, capacity, num_entries, num_nodes);
    if (d) cudaFree(d);
    if (h) cudaFreeHost(h);
    return rc;
}

}  // extern "C"
