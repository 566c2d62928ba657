// Verlet list rows for pairs of atoms: layout (builder, statistics and export: dsmd_rows.cuh).
//
// Two neighbouring atoms share one row. Owned atoms are sorted by cell, x fastest, so consecutive slots of a cell row (a
// run of x cells at one y, z) are neighbours in space (mean distance about one atom spacing); the union of their two
// neighbourhoods is 1.3 times one of them for a Lennard-Jones liquid (cutoff + skin 2.8 sigma) and 1.2 times for water
// (12 A). A row for two atoms therefore holds 0.65 entries per atom instead of one per partner: the force kernel gathers
// 0.65 times the partner positions (its bound: the L1 unit, 13 wavefronts per 32 random 16-byte gathers) and the list
// is 0.65 times as long. Entries that lie inside the list radius of one of the two atoms only are tested by both; the
// cutoff test of the force kernel discards them.
//
// Units. Four consecutive atoms of one cell row form a quad (two pairs), the unit of the builder; quads never reach
// across a cell row. Quad numbers follow from slots by arithmetic (quad_base), so no prefix sum is needed; a cell row
// leaves at most one quad number unused (its word stays kNoQuad).
//   quad[q]  = first slot * 4 + (atoms - 1); row of pair p = 2 q + h (h = 0, 1).
//
// Entries lie in chunks of four (one 16-byte word), 32 rows interleaved, so that a warp with a row per lane reads 512
// consecutive bytes: entry k of row p at ((p >> 5) * stride + (k & ~3)) * 32 + (p & 31) * 4 + (k & 3) (row_base + row_offset).
//   Long rows (ORDER 2) are shared by four lanes at least, and have the entries of a group of 16 in the order in which four lanes
// take them: entry 4 j + l of the group is word j of chunk l. So four lanes gather four consecutive entries at a time, which as a
// rule are neighbours in memory (a run of x cells is a run of slots): 2 to 3 lines of the L1 for four gathers instead of 4.
// Ewald force kernel, 648,000 water atoms, rows of 550 entries: 0.97 ms (1.12 with a row per lane, 1.06 with four lanes and this order
// alone; eight lanes 0.99). Rows of 100 (Lennard-Jones) do not pay for more than one lane: 0.36 ms at 4,000,000 atoms, 0.38 with two.
//   Owned partners come first, [0, row_int[p]); ghosts follow from the next group (4 << ORDER entries) on and end at row_end[p];
//   groups are filled up with an atom that the search found outside the list radius of both atoms, so that the force kernel
//   need not count, or, where the search had met none by then, with the row's own first atom, whose r^2 = 0 makes the force
//   kernel count after all (a row for which no such atom turned up is marked kRowCareful and is counted from the start).
//   The two atoms themselves are not listed. Partners that one of them excludes are kept apart, from the row's last place
//   downwards, marked kExclFirst / kExclSecond: the main loop of the force kernel has no flags to look at.
//   row_special[p] = owned excluded partners | ghosts << kRowCountBits | kRowCareful | kRowOwnExcluded (the two atoms exclude
//   each other).
#pragma once

#include "dsmd_force.cuh"

namespace {

using dsmd::RowArrays;

constexpr unsigned kExclFirst = 0x80000000u, kExclSecond = 0x40000000u;
constexpr unsigned kIndexMask = 0x3FFFFFFFu;
constexpr unsigned kNoQuad = 0xFFFFFFFFu;
constexpr int kLongOrder = 2;   // order of the entries of long rows
constexpr int kRowCountBits = 15, kRowCountMask = (1 << kRowCountBits) - 1;
constexpr unsigned kRowCareful = 0x40000000u, kRowOwnExcluded = 0x80000000u;

__host__ __device__ inline int quad_base(int first_slot, int row) { return (first_slot + 3 * row + 3) >> 2; }

// Words of a row: where it starts, and entry k's place from there.
template <int ORDER>
__host__ __device__ inline size_t row_base(unsigned pair, int stride) {
    constexpr unsigned rows = 32u >> ORDER;
    return static_cast<size_t>(pair / rows) * stride * rows + (pair % rows) * (4u << ORDER);
}
template <int ORDER>
__host__ __device__ inline int row_offset(int k) {   // k / group * 128 + k % lanes * 4 + k / lanes % 4, for k >= 0
    static_assert(ORDER == 0 || ORDER == 2, "the orders in use");
    return ORDER == 0 ? k * 32 - (k & 3) * 31 : 8 * k - 31 * ((k >> 2) & 3) - 4 * (k & 3);
}
// The next multiple of a group of entries.
template <int ORDER>
__host__ __device__ inline int whole_groups(int k) {
    constexpr int group = 4 << ORDER;
    return (k + group - 1) & -group;
}

// First atom and number of atoms (0, 1, 2) of a pair.
__device__ __forceinline__ int pair_atoms(const unsigned* quad, int pair, int& first) {
    const unsigned w = quad[pair >> 1];
    first = static_cast<int>(w >> 2) + 2 * (pair & 1);
    return w == kNoQuad ? 0 : min(max(static_cast<int>(w & 3u) + 1 - 2 * (pair & 1), 0), 2);
}

}  // namespace
