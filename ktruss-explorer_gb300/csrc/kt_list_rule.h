// Host side of the triangle lists' buffer: what it holds and which calls may use it (kt_lists.cu).  No
// CUDA in here, so that its tests run anywhere.
#pragma once

#include <cmath>
#include <cstdint>

namespace kt {

// Graphs of up to this many edges take lists whatever their density: m edges have at most
// (sqrt(2) / 3) m^1.5 triangles, so a buffer of 8.4 M entries (67 MB) holds their lists and the call
// need not wait for the triangle count.
constexpr uint32_t kSmallLists = 1u << 15;

// At least three times the triangles that m edges can form.
inline uint64_t most_entries(uint64_t m) { return (uint64_t)(1.41422 * (double)m * std::sqrt((double)m)) + 64; }

// Whether a buffer of `cap` entries holds the lists of any graph of m edges, uncounted.
inline bool small_lists(uint64_t m, uint64_t cap) { return m <= kSmallLists && most_entries(m) <= cap; }

// Entries of a buffer for lists of `total` entries: a sixteenth more, so that graphs of about a size do not
// grow it again and again, or the entries alone where `limit` bytes hold no more; 0 if not even these fit.
inline uint64_t buffer_entries(uint64_t total, uint64_t limit) {
    const uint64_t need = total ? total : 1, want = need + need / 16;
    return want <= limit / 8 ? want : need <= limit / 8 ? need : 0;
}

// Whether a repeated call takes lists again: the call itself did, with a buffer of `need` entries (0: it
// walked rows), and the buffer is still that large.  It may not be: a larger reservation that found no
// memory leaves none.
inline bool repeat_lists(uint64_t need, uint64_t cap) { return need != 0 && need <= cap; }

}  // namespace kt
