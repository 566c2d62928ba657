// Verlet list rows (dsmd_row_layout.cuh): builder, statistics and export. Included by dsmd_core.cu.
#pragma once

#include "dsmd_row_layout.cuh"

namespace {

constexpr int kBuildThreads = 128;

struct QuadArgs {
    int nx, ny, rows, n_owned;
    unsigned* quad;
    volatile unsigned long long* layer_start;   // pinned host memory, see below
    unsigned tag;
};

// The quads of cell row `row` (a warp): the numbers between two rows' bases that no atoms fill are kNoQuad.
// layer_start: first slot of every z layer of cells, and the end, by which a caller cuts the sorted
// atoms into slabs; with `tag` in the same word, so that the host sees of each whether it has arrived.
__device__ __forceinline__ void row_quads(const QuadArgs& a, int row, const int* cell_start) {
    const int lane = threadIdx.x & 31;
    if (row >= a.rows) return;
    const int begin = min(cell_start[static_cast<size_t>(row) * a.nx], a.n_owned);
    const int end = row + 1 < a.rows ? min(cell_start[static_cast<size_t>(row + 1) * a.nx], a.n_owned) : a.n_owned;
    const int q0 = row == 0 ? 0 : quad_base(begin, row), q1 = quad_base(end, row + 1);
    const int q_first = quad_base(begin, row);
    const unsigned long long tagged = static_cast<unsigned long long>(a.tag) << 32;
    if (lane == 0 && row % a.ny == 0) a.layer_start[row / a.ny] = tagged | static_cast<unsigned>(begin);
    if (lane == 0 && row + 1 == a.rows) a.layer_start[a.rows / a.ny] = tagged | static_cast<unsigned>(end);
    for (int q = q0 + lane; q < q1; q += 32) {
        const int s = begin + 4 * (q - q_first);
        a.quad[q] = (q >= q_first && s < end) ? static_cast<unsigned>(s) * 4u + static_cast<unsigned>(min(end - s, 4) - 1) : kNoQuad;
    }
}

// Behind the scan of a sort: atoms into the cells' lists (the first place_blocks blocks), quads (the others).
__global__ void k_place(int place_blocks, int first, int end, const unsigned* key, const int* arrival,
                        const int* cell_start, int* __restrict__ list, int cells, int* __restrict__ cell_count, QuadArgs quads) {
    if (!dsmd::after_previous()) return;
    const int block = static_cast<int>(blockIdx.x) - place_blocks;
    if (block < 0) dsmd::cell_place(blockIdx.x * blockDim.x + threadIdx.x, place_blocks * blockDim.x, first, end, key, arrival, cell_start, list, cells, cell_count);
    else row_quads(quads, (block * static_cast<int>(blockDim.x) + static_cast<int>(threadIdx.x)) >> 5, cell_start);
}

struct ExclusionTable {
    const int* offsets;    // [n_global + 1] by global id, or null
    const int* partners;   // sorted per atom
    int n_global;          // ids at or beyond this have no exclusions
};

// Squared distance of the nearest images in fp64, rounded as the plain expression dx*dx + dy*dy + dz*dz rounds (no FMA
// contraction). The number of box lengths is taken with the reciprocal of the length: it can differ from a division's only where
// two images are half a box away, beyond the list radius both.
__device__ __forceinline__ double list_distance2(const Grid& g, const double (&pi)[3], const double (&pj)[3]) {
    double d[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        d[a] = pi[a] - pj[a];
        if (g.wrap[a]) d[a] -= g.box[a] * rint(d[a] * g.inv_len[a]);
    }
    return __dadd_rn(__dadd_rn(__dmul_rn(d[0], d[0]), __dmul_rn(d[1], d[1])), __dmul_rn(d[2], d[2]));
}

// The search of one quad by one warp. Each lane takes one cell row of the stencil and works out the x window that the
// four atoms' list spheres cut out of it (the union of their chords, rounded outwards to x cells). A scan over the lanes
// numbers the candidates of all rows consecutively, the lanes write their rows' slots into shared memory under those
// numbers, and the warp walks them 32 at a time: a position per lane, tested against the four atoms, hits of a pair
// packed behind each other by ballot.
// What bounds it: instruction issue; 8 to 9 rounds of 32 candidates per quad of a Lennard-Jones liquid (130 of the 250
// candidates lie inside the list radius of one of the four atoms), about 60 for water. A thread-per-atom walk of the same
// windows spent 340 warp instructions per atom at 20 of 32 active lanes. In small systems the reads of a round: they are under way
// a round ahead. Rebuild of 4,000,000 Lennard-Jones atoms 1.79 ms, of 1,048,575 of the mixture 0.585, of 648,000 of water 1.83, of
// 3,993 0.069 (without reading ahead 1.80, 0.595, 1.88, 0.073; thread per atom: 2.58, 1.02, 5.97 ms). Blocks per SM: eight with
// exclusions (seven 1.89 ms for water), seven without (eight 0.603 ms for the mixture).
constexpr int kCandidates = 512;   // candidates numbered at a time (per warp, in shared memory)

struct QuadSearch {
    int x, y, z;            // the first atom (fixed-point)
    F2 off[2][3];           // offsets of the four atoms from it, negated: {atom 0, atom 1}, {atom 2, atom 3}
    float hi_band;
    int first;              // first slot
    unsigned *row0, *row1;  // rows of the two pairs
    int stride;
    int count0, count1;
    unsigned special0, special1;   // row_special so far (owned excluded partners)
    int far0, far1;                // a slot outside both atoms' list radius, or -1
    int n_atoms;
};

// The ids an atom excludes lie in [lo, lo + span] (an id that no atom carries where it excludes none).
struct ExcludedRange {
    int lo[4];
    unsigned span[4];
};

// NEAR: the quad is compact against the box, so that the image of a candidate nearest to the first atom is the nearest
// to all four: one fixed-point difference and conversion per candidate, the other atoms by their float offsets from the
// first. Otherwise every atom takes its own fixed-point difference (exact for any placement).
template <bool NEAR, bool EXCL, int ORDER>
__device__ __forceinline__ void test_candidates(const Grid& g, QuadSearch& q, int n, const int* s_slot,
                                                const int4* pq, const int* gid, const ExclusionTable& excl,
                                                const ExcludedRange& s_excluded) {
    const int lane = threadIdx.x & 31;
    const unsigned lt_mask = (1u << lane) - 1u;
    const unsigned own_first = static_cast<unsigned>(min(q.n_atoms, 2)), own_second = static_cast<unsigned>(max(q.n_atoms - 2, 0));
    // the next round's candidate is on its way while this one is tested, and its slot a round before that (__ldca: ordinary loads, but
    // the compiler need not keep their order with the stores of rows; 1.79 ms at 4,000,000 atoms, 1.83 with the order kept)
    int s_next = lane < n ? s_slot[lane] : q.first;
    int4 c_next = __ldca(&pq[s_next]);
    int g_next = EXCL ? __ldca(&gid[s_next]) : 0;
    int s_after = lane + 32 < n ? s_slot[lane + 32] : q.first;
    for (int t = lane; t - lane < n; t += 32) {
        const bool valid = t < n;
        const int s = s_next, gj = g_next;
        const int4 c = c_next;
        s_next = s_after;
        c_next = __ldca(&pq[s_next]);
        if (EXCL) g_next = __ldca(&gid[s_next]);
        s_after = t + 64 < n ? s_slot[t + 64] : q.first;
        float r[4];
        if (NEAR) {
            const F2 rx = both(dsmd::fixed_delta(c.x, q.x, g.scale[0]));
            const F2 ry = both(dsmd::fixed_delta(c.y, q.y, g.scale[1]));
            const F2 rz = both(dsmd::fixed_delta(c.z, q.z, g.scale[2]));
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const F2 dx = add(rx, q.off[h][0]), dy = add(ry, q.off[h][1]), dz = add(rz, q.off[h][2]);
                parts(fma(dz, dz, fma(dy, dy, mul(dx, dx))), r[2 * h], r[2 * h + 1]);
            }
        } else {
#pragma unroll
            for (int m = 0; m < 4; ++m) {
                const int4 atom = __ldca(&pq[q.first + min(m, q.n_atoms - 1)]);
                const float dx = dsmd::fixed_delta(c.x, atom.x, g.scale[0]);
                const float dy = dsmd::fixed_delta(c.y, atom.y, g.scale[1]);
                const float dz = dsmd::fixed_delta(c.z, atom.z, g.scale[2]);
                r[m] = dx * dx + dy * dy + dz * dz;
            }
        }
        const float limit = valid ? q.hi_band : -1.0f;
        bool hit0 = fminf(r[0], r[1]) < limit, hit1 = fminf(r[2], r[3]) < limit;
        if (q.far0 < 0 || q.far1 < 0) {   // as a rule found in the first round
            const unsigned f0 = __ballot_sync(0xFFFFFFFFu, valid && !hit0), f1 = __ballot_sync(0xFFFFFFFFu, valid && !hit1);
            if (f0) q.far0 = __shfl_sync(0xFFFFFFFFu, s, __ffs(f0) - 1);
            if (f1) q.far1 = __shfl_sync(0xFFFFFFFFu, s, __ffs(f1) - 1);
        }
        // the two atoms of a pair are no partners of its row
        const unsigned own = static_cast<unsigned>(s - q.first);
        const bool own0 = own < own_first, own1 = own - 2u < own_second;
        if (EXCL) {
            // a candidate inside the range of ids that one of the four atoms excludes (molecules are numbered together: few
            // are) is looked up in the atom's table row; the row's end holds those that are excluded for one of its atoms
            const int4 lo = *reinterpret_cast<const int4*>(s_excluded.lo);
            const uint4 span = *reinterpret_cast<const uint4*>(s_excluded.span);
            const bool look = static_cast<unsigned>(gj - lo.x) <= span.x || static_cast<unsigned>(gj - lo.y) <= span.y ||
                              static_cast<unsigned>(gj - lo.z) <= span.z || static_cast<unsigned>(gj - lo.w) <= span.w;
            if (__any_sync(0xFFFFFFFFu, look && (hit0 || hit1))) {
                unsigned flags0 = 0, flags1 = 0;
#pragma unroll 1
                for (int m = 0; m < q.n_atoms; ++m) {
                    if (look && static_cast<unsigned>(gj - s_excluded.lo[m]) <= s_excluded.span[m]) {
                        const int g_m = gid[q.first + m], end = excl.offsets[g_m + 1];
                        for (int e = excl.offsets[g_m]; e < end; ++e)
                            if (excl.partners[e] == gj) {
                                if (m < 2) flags0 |= m == 0 ? kExclFirst : kExclSecond;
                                else flags1 |= m == 2 ? kExclFirst : kExclSecond;
                            }
                    }
                }
                const unsigned x0 = __ballot_sync(0xFFFFFFFFu, hit0 && flags0), x1 = __ballot_sync(0xFFFFFFFFu, hit1 && flags1);
                const int p0 = static_cast<int>((q.special0 & kRowCountMask) + __popc(x0 & lt_mask));
                const int p1 = static_cast<int>((q.special1 & kRowCountMask) + __popc(x1 & lt_mask));
                if (hit0 && flags0 && p0 < q.stride) q.row0[row_offset<ORDER>(q.stride - 1 - p0)] = static_cast<unsigned>(s) | flags0;
                if (hit1 && flags1 && p1 < q.stride) q.row1[row_offset<ORDER>(q.stride - 1 - p1)] = static_cast<unsigned>(s) | flags1;
                q.special0 += __popc(x0);
                q.special1 += __popc(x1);
                if (__any_sync(0xFFFFFFFFu, hit0 && flags0 && own0)) q.special0 |= kRowOwnExcluded;
                if (__any_sync(0xFFFFFFFFu, hit1 && flags1 && own1)) q.special1 |= kRowOwnExcluded;
                hit0 = hit0 && !flags0;
                hit1 = hit1 && !flags1;
            }
        }
        hit0 = hit0 && !own0;
        hit1 = hit1 && !own1;
        const unsigned m0 = __ballot_sync(0xFFFFFFFFu, hit0), m1 = __ballot_sync(0xFFFFFFFFu, hit1);
        const int k0 = q.count0 + __popc(m0 & lt_mask), k1 = q.count1 + __popc(m1 & lt_mask);
        if (hit0 && k0 < q.stride) q.row0[row_offset<ORDER>(k0)] = static_cast<unsigned>(s);
        if (hit1 && k1 < q.stride) q.row1[row_offset<ORDER>(k1)] = static_cast<unsigned>(s);
        q.count0 += __popc(m0);
        q.count1 += __popc(m1);
    }
}

template <bool EXCL, int ORDER>
__global__ void __launch_bounds__(kBuildThreads, EXCL ? 8 : 7)
k_build_rows(Grid g, int n_owned, int n_total, int n_quads, const int4* pq, const int* gid,
             ExclusionTable excl, const int* cell_start, const int* ghost_near_lo,
             const int* ghost_near_hi, RowArrays out, int* __restrict__ boundary_pairs, Status* st) {
    if (!dsmd::after_previous()) return;
    __shared__ int s_slots[kBuildThreads / 32][kCandidates];
    __shared__ __align__(16) ExcludedRange s_ranges[EXCL ? kBuildThreads / 32 : 1];
    const int quad = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (quad >= n_quads) return;
    int* slots = s_slots[threadIdx.x >> 5];
    const unsigned word = out.quad[quad];
    if (word == kNoQuad) {
        if (lane < 2) out.row_end[2 * quad + lane] = out.row_int[2 * quad + lane] = 0;
        if (lane < 2) out.row_special[2 * quad + lane] = 0u;
        return;
    }
    QuadSearch q;
    q.first = static_cast<int>(word >> 2);
    const int n_atoms = static_cast<int>(word & 3u) + 1;
    float off[4][3];
    bool compact = true;
    const int4 home = pq[q.first];
    q.x = home.x;
    q.y = home.y;
    q.z = home.z;
#pragma unroll
    for (int m = 0; m < 4; ++m) {
        const int4 atom = pq[q.first + min(m, n_atoms - 1)];   // a missing atom: a copy of the last one
        off[m][0] = dsmd::fixed_delta(atom.x, home.x, g.scale[0]);
        off[m][1] = dsmd::fixed_delta(atom.y, home.y, g.scale[1]);
        off[m][2] = dsmd::fixed_delta(atom.z, home.z, g.scale[2]);
        // how far the quad may spread for the nearest image of a candidate to be the same for all four atoms (wrapping
        // axes), and for the rounding band to hold
        compact = compact && fabsf(off[m][0]) <= g.quad_spread[0] && fabsf(off[m][1]) <= g.quad_spread[1] &&
                  fabsf(off[m][2]) <= g.quad_spread[2];
    }
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int a = 0; a < 3; ++a) q.off[h][a] = f2(-off[2 * h][a], -off[2 * h + 1][a]);
    // a pair inside the rounding band is listed whether or not it lies inside the list radius (the export decides in fp64)
    q.hi_band = g.r2_list + g.band_rows;
    q.stride = out.stride;
    q.row0 = out.rows + row_base<ORDER>(2 * quad, out.stride);
    q.row1 = q.row0 + (4 << ORDER);   // the rows of a quad are neighbours
    q.count0 = q.count1 = 0;
    q.special0 = q.special1 = 0u;
    q.far0 = q.far1 = -1;
    q.n_atoms = n_atoms;
    ExcludedRange& s_excluded = s_ranges[EXCL ? threadIdx.x >> 5 : 0];
    if (EXCL && lane < 4) {
        int lo = static_cast<int>(0x80000000u);   // no atom carries this id
        unsigned span = 0u;
        const int g_m = gid[q.first + min(lane, n_atoms - 1)];
        if (lane < n_atoms && g_m >= 0 && g_m < excl.n_global) {
            const int b = excl.offsets[g_m], e = excl.offsets[g_m + 1];
            if (e > b) {
                lo = excl.partners[b];
                span = static_cast<unsigned>(excl.partners[e - 1] - lo);
            }
        }
        s_excluded.lo[lane] = lo;
        s_excluded.span[lane] = span;
    }

    // this lane's cell row, (dy, dz) from the home row, and its x window in cells
    const int S = g.stencil, side = 2 * S + 1;
    const int lane_z = S == 2 ? (lane * 13) >> 6 : (lane * 11) >> 5;   // lane / 5, lane / 3
    const int dz = lane_z - S, dy = lane - lane_z * side - S;
    // places of the first atom on the three axes, in cells (float: good to 3e-4 of a cell)
    const float at_x = __uint2float_rn(static_cast<unsigned>(home.x)) * g.cells_per_unit[0];
    const float at_y = __uint2float_rn(static_cast<unsigned>(home.y)) * g.cells_per_unit[1];
    const float at_z = __uint2float_rn(static_cast<unsigned>(home.z)) * g.cells_per_unit[2];
    const int cy0 = static_cast<int>(dsmd::cell_of(static_cast<unsigned>(home.y), g.wrap[1], g.nc[1]));
    const int cz0 = static_cast<int>(dsmd::cell_of(static_cast<unsigned>(home.z), g.wrap[2], g.nc[2]));
    const float to_y = static_cast<float>(cy0 + dy) - at_y, to_z = static_cast<float>(cz0 + dz) - at_z;   // lower face of the row
    int yc = cy0 + dy, zc = cz0 + dz;
    bool open = lane < side * side;
    if (g.wrap[1]) { if (yc < 0) yc += g.nc[1]; else if (yc >= g.nc[1]) yc -= g.nc[1]; }
    else if (yc < 0 || yc >= g.nc[1]) open = false;
    if (g.wrap[2]) { if (zc < 0) zc += g.nc[2]; else if (zc >= g.nc[2]) zc -= g.nc[2]; }
    else if (zc < 0 || zc >= g.nc[2]) open = false;
    // the chord of each atom's sphere at the row's distance from it (g.r_pad carries 1e-4 of slack, far more than the
    // approximate square root gives away; 1e-3 of a cell covers the rounding of the places)
    const float reach2 = g.r_pad * g.r_pad;
    float lo = 3.0e38f, hi = -3.0e38f;
#pragma unroll
    for (int m = 0; m < 4; ++m) {
        const float y0 = to_y * g.cellw[1] - off[m][1], z0 = to_z * g.cellw[2] - off[m][2];   // from the atom to the lower face
        const float gy = fmaxf(fmaxf(y0, -y0 - g.cellw[1]) - 1e-3f * g.cellw[1], 0.f);
        const float gz = fmaxf(fmaxf(z0, -z0 - g.cellw[2]) - 1e-3f * g.cellw[2], 0.f);
        const float chord2 = reach2 - gy * gy - gz * gz;
        if (chord2 > 0.f) {
            const float hw = fminf(chord2 * rsqrt_approx(chord2), g.x_reach);
            lo = fminf(lo, off[m][0] - hw);
            hi = fmaxf(hi, off[m][0] + hw);
        }
    }
    open = open && lo <= hi;
    int a0 = 0, b0 = -1, a1 = 0, b1 = -1;   // x cells [a0, b0] and, across the periodic boundary, [a1, b1]
    if (open) {
        const int c_lo = __float2int_rd(at_x + lo * g.cells_per_length - 2e-3f), c_hi = __float2int_rd(at_x + hi * g.cells_per_length + 2e-3f);
        if (!g.wrap[0]) {
            a0 = max(c_lo, 0);
            b0 = min(c_hi, g.nc[0] - 1);
        } else if (c_hi - c_lo >= g.nc[0] - 1) {
            b0 = g.nc[0] - 1;   // the window is as long as the box
        } else {
            a0 = c_lo < 0 ? c_lo + g.nc[0] : (c_lo >= g.nc[0] ? c_lo - g.nc[0] : c_lo);
            b0 = c_hi < 0 ? c_hi + g.nc[0] : (c_hi >= g.nc[0] ? c_hi - g.nc[0] : c_hi);
            if (b0 < a0) {   // in ascending slots: the part at the lower end of the box first
                a1 = a0;
                b1 = g.nc[0] - 1;
                a0 = 0;
            }
        }
    }
    // the ghost pass only for quads whose x windows reach an x cell with ghosts in one of the rows they search (on an
    // axis that wraps the window may come round the box: any ghost in those rows counts)
    int n_seg = 1;
    if (n_total > n_owned) {
        const int row_yz = cz0 * g.nc[1] + cy0;
        const int near_lo = ghost_near_lo[row_yz], near_hi = ghost_near_hi[row_yz];
        const int reach_cells = static_cast<int>(g.x_reach / g.cellw[0]) + 2;
        int c_min = g.nc[0], c_max = -1;   // x cells of the atoms
        for (int m = 0; m < n_atoms; ++m) {
            const int cx = static_cast<int>(dsmd::cell_of(static_cast<unsigned>(pq[q.first + m].x), g.wrap[0], g.nc[0]));
            c_min = min(c_min, cx);
            c_max = max(c_max, cx);
        }
        if (g.wrap[0] ? (near_lo > 0 || near_hi < g.nc[0]) : (c_min - reach_cells < near_lo || c_max + reach_cells >= near_hi))
            n_seg = 2;
    }
    int interior0 = 0, interior1 = 0;
    unsigned interior_special0 = 0u, interior_special1 = 0u;
    for (int seg = 0; seg < n_seg; ++seg) {
        const int row = seg * g.ncells + (zc * g.nc[1] + yc) * g.nc[0];
        int s0 = 0, len0 = 0, s1 = 0, len1 = 0;
        if (b0 >= a0) { s0 = cell_start[row + a0]; len0 = cell_start[row + b0 + 1] - s0; }
        if (b1 >= a1) { s1 = cell_start[row + a1]; len1 = cell_start[row + b1 + 1] - s1; }
        const int len = len0 + len1;
        int incl = len;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xFFFFFFFFu, incl, o);
            if (lane >= o) incl += v;
        }
        const int total = __shfl_sync(0xFFFFFFFFu, incl, 31), begin = incl - len;
        for (int base = 0; base < total; base += kCandidates) {
            __syncwarp();
            // this row's share of the numbers [base, base + kCandidates): the first run, then (rare) the second
            int* to = slots + (begin - base);
            const int k0 = max(base - begin, 0), k1 = min(base + kCandidates - begin, len);
            const int first_end = min(k1, len0);
            int k = k0;
            for (; k + 3 < first_end; k += 4) {
                to[k] = s0 + k;
                to[k + 1] = s0 + k + 1;
                to[k + 2] = s0 + k + 2;
                to[k + 3] = s0 + k + 3;
            }
            if (k < first_end) to[k] = s0 + k;
            if (k + 1 < first_end) to[k + 1] = s0 + k + 1;
            if (k + 2 < first_end) to[k + 2] = s0 + k + 2;
            if (len1 > 0)
                for (k = max(k0, len0); k < k1; ++k) to[k] = s1 + (k - len0);
            __syncwarp();
            const int n = min(total - base, kCandidates);
            if (compact) test_candidates<true, EXCL, ORDER>(g, q, n, slots, pq, gid, excl, s_excluded);
            else test_candidates<false, EXCL, ORDER>(g, q, n, slots, pq, gid, excl, s_excluded);
        }
        if (n_atoms <= 2) { q.count1 = 0; q.special1 = 0u; }
        if (seg == 0) { interior0 = q.count0; interior1 = q.count1; interior_special0 = q.special0; interior_special1 = q.special1; }
        // Fill up the last group. Where the search has met no atom to fill it with, the row's own first atom does: the force kernel
        // sees r^2 = 0 and counts the row's entries (as it does from the start if no such atom turns up at all: kRowCareful).
        constexpr int group = 4 << ORDER;
        static_assert(2 * group <= 32, "a lane per place of the last group of either row");
        const bool second = lane >= group;
        const int c = second ? q.count1 : q.count0, far = second ? q.far1 : q.far0;
        const int k = c / group * group + lane % group;
        if (lane < 2 * group && k >= c && c % group && k < out.stride)
            (second ? q.row1 : q.row0)[row_offset<ORDER>(k)] = static_cast<unsigned>(far < 0 ? q.first + (second ? 2 : 0) : far);
        if (seg == 0 && n_seg == 2) {
            q.count0 = whole_groups<ORDER>(q.count0);
            q.count1 = whole_groups<ORDER>(q.count1);
        }
    }
    if (lane < 2) {
        const int interior = lane ? interior1 : interior0, count = lane ? q.count1 : q.count0;
        const unsigned special = lane ? q.special1 : q.special0, special_own = lane ? interior_special1 : interior_special0;
        const unsigned n_special = special & kRowCountMask, n_own = special_own & kRowCountMask;
        // a ghost pass without hits leaves the row as it was
        const bool ghosts = n_seg == 2 && count > whole_groups<ORDER>(interior);
        out.row_end[2 * quad + lane] = min(ghosts ? count : interior, out.stride);
        out.row_int[2 * quad + lane] = min(interior, out.stride);
        out.row_special[2 * quad + lane] = n_own | ((n_special - n_own) << kRowCountBits) | (special & kRowOwnExcluded) |
                                           ((lane ? q.far1 : q.far0) < 0 ? kRowCareful : 0u);
        const int need = whole_groups<ORDER>(count) + static_cast<int>(n_special);   // whole groups, and the ones apart behind them
        if (need > out.stride) atomicMax(&st->need_stride, static_cast<unsigned>(need));
        // pairs with a ghost partner, collected for the boundary pass of the force kernel (the order of the collection
        // does not matter: every pair's sums are its own threads')
        if (ghosts || n_special > n_own) boundary_pairs[atomicAdd(&st->boundary_pairs, 1u)] = 2 * quad + lane;
    }
}

// Members of the list proper, decided in fp64 on the reference positions of the last build (the builder lists every
// candidate inside the rounding band and, for an atom, its pair-mate's partners): counts per atom, or (WRITE) the
// directed pairs themselves, atom after atom in row order, from the atoms' first places on. stats: members, members with an
// owned partner, tests inside the rounding band.
// A warp per row, an entry per lane for both atoms, rows in turn. What bounds it: scattered reads of the partners' three doubles.
// 4,000,000 Lennard-Jones atoms: 2.7 ms to count, 2.7 to write (a thread per row 3.5 and 8.3); 3,993 of water 0.05 ms each (1.5).
constexpr int kMemberThreads = 256;
template <bool WRITE, int ORDER>
__global__ void __launch_bounds__(kMemberThreads) k_list_members(Grid g, int n_pairs, RowArrays in, const double* __restrict__ x,
                               const double* __restrict__ y, const double* __restrict__ z, unsigned long long* __restrict__ per_atom,
                               unsigned long long* __restrict__ stats, int* __restrict__ out_i, int* __restrict__ out_j,
                               unsigned char* __restrict__ out_flags) {
    const int lane = threadIdx.x & 31, warps = gridDim.x * (kMemberThreads / 32);
    const unsigned lt_mask = (1u << lane) - 1u;
    unsigned long long sums[3] = {0, 0, 0};   // members, interior, banded of this lane's entries
    for (int pair = (blockIdx.x * kMemberThreads + threadIdx.x) >> 5; pair < n_pairs; pair += warps) {
        int first = 0;
        const int atoms = pair_atoms(in.quad, pair, first);
        if (atoms == 0) continue;
        const int mid = in.row_int[pair], end = in.row_end[pair];
        const unsigned special = in.row_special[pair];
        const int special_own = special & kRowCountMask, special_all = special_own + ((special >> kRowCountBits) & kRowCountMask);
        const int total = end + special_all + (atoms > 1 && !(special & kRowOwnExcluded) ? 1 : 0);
        const unsigned* row = in.rows + row_base<ORDER>(static_cast<unsigned>(pair), in.stride);
        const int last = first + atoms - 1;
        const double at_atom[2][3] = {{x[first], y[first], z[first]}, {x[last], y[last], z[last]}};
        unsigned long long at[2] = {WRITE ? per_atom[first] : 0ull, WRITE && atoms > 1 ? per_atom[first + 1] : 0ull};
        for (int base = 0; base < total; base += 32) {
            const int k = base + lane, nth = k - end;   // the entries, then those at the row's end, then the pair's other atom
            const bool there = k < total && !(k >= mid && k < min(whole_groups<ORDER>(mid), end));
            const bool other = nth >= special_all;
            const bool owned = nth < 0 ? k < mid : (nth < special_own || other);
            const unsigned e = !there || other ? 0u : row[row_offset<ORDER>(nth < 0 ? k : in.stride - 1 - nth)];
            const int partner = static_cast<int>(e & kIndexMask);
            double pj[3] = {0.0, 0.0, 0.0};
            if (there && !other) { pj[0] = x[partner]; pj[1] = y[partner]; pj[2] = z[partner]; }
#pragma unroll
            for (int m = 0; m < 2; ++m) {
                if (m >= atoms) break;
                const int i = first + m, j = other ? first + 1 - m : partner;
                const double to[3] = {other ? at_atom[1 - m][0] : pj[0], other ? at_atom[1 - m][1] : pj[1], other ? at_atom[1 - m][2] : pj[2]};
                const double r2 = list_distance2(g, at_atom[m], to);
                const bool member = there && j != i && r2 < g.r2_list_d;
                const unsigned members = __ballot_sync(0xFFFFFFFFu, member);
                if (WRITE) {
                    if (member) {
                        const unsigned long long place = at[m] + __popc(members & lt_mask);
                        out_i[place] = i;
                        out_j[place] = j;
                        if (out_flags) out_flags[place] = (e & (m == 0 ? kExclFirst : kExclSecond)) ? 1 : 0;
                    }
                } else if (member) {
                    ++sums[0];
                    if (owned) ++sums[1];
                    if (g.r2_list_d - r2 < static_cast<double>(g.band_rows)) ++sums[2];
                }
                at[m] += __popc(members);
            }
        }
        if (!WRITE && lane < atoms) per_atom[first + lane] = lane ? at[1] : at[0];
    }
    if (!WRITE) {
        __shared__ unsigned long long s_sums[3];
        if (threadIdx.x < 3) s_sums[threadIdx.x] = 0;
        __syncthreads();
        for (int c = 0; c < 3; ++c) {
            for (int o = 16; o > 0; o >>= 1) sums[c] += __shfl_down_sync(0xFFFFFFFFu, sums[c], o);
            if (lane == 0 && sums[c]) atomicAdd(&s_sums[c], sums[c]);
        }
        __syncthreads();
        if (threadIdx.x < 3 && s_sums[threadIdx.x]) atomicAdd(&stats[threadIdx.x], s_sums[threadIdx.x]);
    }
}

}  // namespace
