// Which decompositions peel from triangle lists (kt_lists.cu), and what their buffer holds.  No CUDA in
// here, so that the tests of these rules run anywhere.
#pragma once

#include <cmath>
#include <cstdint>

namespace kt {

// Most list entries per edge on average (three per triangle) with which the lists are made: writing them
// costs more than the walks in denser graphs.  Whole decomposition, lists / walks: R-MAT 16 of edge
// factor 16 (52 entries an edge) 5.3 / 9.8 ms, G(3000, 0.2) (120) 3.7 / 7.9, R-MAT 18 of edge factor 64
// (261) 88 / 116, R-MAT 16 of edge factor 128 (334) 50 / 62, G(3000, 0.4) (479) 18.6 / 20.3, R-MAT 18 of
// edge factor 128 (480) 255 / 291.  Past the line it is no longer the density that decides but how many edges
// go in one round, which a recount gets for little: G(8000, 0.3) (719) 186 / 201, but G(3000, 0.5) (749)
// 34 / 20 and G(3000, 0.9) (2,429) 203 / 38.
constexpr uint64_t kMaxListPerEdge = 512;

// Near-cliques go in a few rounds that remove most edges at once, which a recount round of the walking
// peel gets for little.  A graph of kCliqueEdges edges with kCliqueEntries or more entries an edge walks
// if more than three quarters of them belong to edges with 15/16 or more of their shorter row in
// triangles: disjoint cliques of 100 vertices 2.1 / 0.65 ms, of 400 10.7 / 1.5 ms, G(200000, 16/n) with
// cliques of 300-500 vertices 4.8 / 3.8 ms; cliques of 20 (18 entries an edge) 0.53 / 0.44 ms, cliques of 50
// with a tenth of the edges rewired (35; not near-cliques) 1.6 / 2.6 ms.
constexpr uint64_t kCliqueEntries = 32;
constexpr uint32_t kCliqueEdges = 1u << 18;

// With fewer edges it is the lists' entries that cost, 9 us a million more than the walks of a near-clique,
// and the rest of the graph that the walks pay for, 2 us a thousand entries more than the lists: such a
// graph walks from kCliqueTotal entries on if at most one in kCliqueRest is outside near-cliques.
// Cliques of 500 vertices, two of them (124 M entries) 1.57 / 0.52 ms, of 400, two (64 M) 0.87 / 0.35, of 200,
// six (24 M) 0.41 / 0.24; below the line of 100, 26 (13 M) 0.29 / 0.22.  (At 17 M entries the lists take
// what a decomposition took that knew only walks and built its graph in 0.15 ms more: 0.37.)  Beside an
// R-MAT graph of 26,000 edges (0.4 M entries): cliques of 200, five 1.14 / 1.79, of 400, two 1.65 / 1.87.
constexpr uint64_t kCliqueTotal = 1u << 24, kCliqueRest = 256;

// A graph of kEvenPerEdge or more entries an edge whose least support is four fifths or more of the mean goes
// in a few rounds too.  G(400, 0.9) (323 entries an edge, 0.87 of the mean) 0.65 / 0.58 ms, G(700, 0.7) (343, 0.84)
// 1.62 / 1.48, G(700, 0.84) (494, 0.90) 2.47 / 1.85, G(900, 0.6) (323, 0.81) 2.33 / 2.16; with fewer entries
// G(600, 0.7) (293) 1.29 / 1.46, G(724, 0.66) (314) 1.63 / 1.71; where supports differ, of Barabasi-Albert graphs
// of 700 vertices (493, 0.45) 12.2 / 21.6, of geometric ones (348, 0.41) 5.7 / 10.3, of cliques of 500 with a tenth
// of the edges rewired (391, 0.03) 3.1 / 3.9.  (Between 2^18 and 2^19 edges it would be the same: G(900, 0.75)
// 3.2 / 2.0, G(1200, 0.65) 5.1 / 3.6.)
constexpr uint64_t kEvenPerEdge = 320;
// Edges in no triangle go first and cost either way nothing: evenness is that of the others, which also walk past
// kMaxListPerEdge entries an edge of theirs if the least support is two thirds of the mean.  K(4000, 2500) with
// a clique of 600 vertices (143 entries an edge, 867 an edge in triangles, 0.69 of the mean) 35 / 19 ms, a tree of
// 4 M edges beside a clique of 600 (26, 598, 1) 2.9 / 2.3, beside G(1500, 0.7) (121, 734, 0.86) 11.5 / 10.4, beside
// G(3000, 0.5) (269, 749, 0.8) 33 / 35; uneven: beside a Barabasi-Albert graph of 3,000 vertices (299, 874) 95 / 150,
// beside a geometric one of 4,000 (177, 590) 39 / 59.

// Whether a graph of m edges, `with` of them in triangles, and `total` list entries walks its rows; `local` of the
// entries are near-cliques' and `least` is the least support but 0.
inline bool walks_rows(uint64_t m, uint64_t with, uint64_t total, uint64_t local, uint32_t least) {
    if (total / kMaxListPerEdge > m) return true;
    if (total / kMaxListPerEdge > with && least * with >= total / 3 * 2) return true;
    if (m >= kCliqueEdges) return total >= kCliqueEntries * m && local > total / 4 * 3;
    if (total >= kCliqueTotal && total - local <= total / kCliqueRest) return true;
    return total / kEvenPerEdge > with && least * with >= total / 5 * 4;
}

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
