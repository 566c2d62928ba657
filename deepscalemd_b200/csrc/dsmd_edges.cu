// Radius-graph edge builder for the machine-learned-potential backends (sm_100a).
//
// Semantics of the reference's EdgeBuilder::build (include/EdgeBuilder.cuh:12-59, src/EdgeBuilder.cu:233-334): every
// ordered pair (i, j), i != j, |r_j - r_i| < cutoff over the atoms given, no minimum image; optional periodic-image
// description (centres restricted to the real atoms, neighbour replaced by the atom it copies, per-edge shift) and
// optional receiver pruning. Output int64 [2, E] + double [E, 3].
//
// What is done differently: the neighbourhood search runs ONCE (the reference searches twice, to count and to fill),
// in fp32 with an fp64 re-decision inside the rounding band (so membership is that of an fp64 search), and leaves its hits
// in 32-atom slices and the start of every slice's edges; a second pass expands the slices into the interface arrays with
// fully coalesced stores, which is where the bytes are (40 B per edge).
// A second entry point emits the compact periodic form (int32 src/dst, int8 lattice shift, fp32 edge vector).

#include <cub/cub.cuh>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <limits>
#include <string>

#include "../../include/dsmd_b200.h"
#include "dsmd_cells.cuh"
#include "dsmd_common.cuh"
#include "dsmd_launch.cuh"
#include "dsmd_report.cuh"
#include "dsmd_scan.cuh"

using dsmd::Grid;

namespace {

constexpr int kThreads = 256;
constexpr int kSearchThreads = 128;
constexpr int kFillThreads = 128;

inline unsigned blocks_for(int64_t n, int threads) { return static_cast<unsigned>((n + threads - 1) / threads); }

struct EdgeStatus {
    unsigned int out_of_bounds;
    unsigned int need_stride;
    unsigned int outside_box;     // periodic form: an atom lies outside [0, box), wrap counts matter
    unsigned int ticket;
};

__global__ void k_edge_keys(Grid g, int n, const double* x, const double* y,
                            const double* z, unsigned* __restrict__ key, int* __restrict__ arrival,
                            int* __restrict__ cell_count, EdgeStatus* st) {
    if (!dsmd::after_previous()) return;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    unsigned bad = 0;
    const unsigned fx = dsmd::to_fixed(x[i], 0, g, bad);
    const unsigned fy = dsmd::to_fixed(y[i], 1, g, bad);
    const unsigned fz = dsmd::to_fixed(z[i], 2, g, bad);
    if (bad) atomicOr(&st->out_of_bounds, 1u);
    const unsigned cx = dsmd::cell_of(fx, g.wrap[0], g.nc[0]);
    const unsigned cy = dsmd::cell_of(fy, g.wrap[1], g.nc[1]);
    const unsigned cz = dsmd::cell_of(fz, g.wrap[2], g.nc[2]);
    const unsigned cell = (cz * g.nc[1] + cy) * g.nc[0] + cx;
    key[i] = cell;
    arrival[i] = atomicAdd(&cell_count[cell], 1);
}

// How many box lengths a coordinate lies from its wrapped place, consistent with to_fixed (which maps a coordinate that
// rounds up to the upper face onto the lower face of the next image).
__device__ __forceinline__ int wrap_count(double v, int axis, const Grid& g) {
    if (!g.wrap[axis]) return 0;
    const double u = (v - g.org[axis]) * g.inv_len[axis];
    if (!(u == u) || fabs(u) > 1.0e9) return 0;
    const double w = floor(u);
    return static_cast<int>(w) + (u - w >= 1.0 ? 1 : 0);
}

constexpr int kWrapBits = 10, kWrapBias = 1 << (kWrapBits - 1), kWrapMask = (1 << kWrapBits) - 1;

__device__ __forceinline__ int packed_wraps(int wx, int wy, int wz) {
    auto field = [](int w) { return min(max(w + kWrapBias, 0), kWrapMask); };
    return field(wx) | (field(wy) << kWrapBits) | (field(wz) << (2 * kWrapBits));
}

__device__ __forceinline__ int wrap_field(int packed, int axis) {
    return ((packed >> (axis * kWrapBits)) & kWrapMask) - kWrapBias;
}

constexpr int kPruned = static_cast<int>(0x80000000u);   // in the index of a sorted atom: no receiver (row 1: no neighbour)

// Distance of a fixed-point coordinate from the grid's origin.
__device__ __forceinline__ float place_of(int fixed, float scale) { return __uint2float_rn(static_cast<unsigned>(fixed)) * scale; }

// Sorted atoms in two forms, fixed-point and float (w = the caller's atom index, kPruned: not wanted as a neighbour), and
// their wrap counts (periodic form only). A thread takes the atom at its place of the cell lists.
__global__ void k_edge_gather(Grid g, int n, const unsigned* key, const int* list,
                              const int* cell_start, const double* x, const double* y,
                              const double* z, const unsigned char* neighbour_ok,
                              const int* owner, int4* __restrict__ pq, float4* __restrict__ pf, int* __restrict__ wraps,
                              EdgeStatus* st) {
    if (!dsmd::after_previous()) return;
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    const int a = list[t];
    const int s = dsmd::cell_slot(a, key[a], cell_start, list);
    unsigned bad = 0;
    const double px = x[a], py = y[a], pz = z[a];
    int4 p;
    p.x = static_cast<int>(dsmd::to_fixed(px, 0, g, bad));
    p.y = static_cast<int>(dsmd::to_fixed(py, 1, g, bad));
    p.z = static_cast<int>(dsmd::to_fixed(pz, 2, g, bad));
    p.w = a;
    if (neighbour_ok && !neighbour_ok[owner ? owner[a] : a]) p.w |= kPruned;
    pq[s] = p;
    pf[s] = make_float4(place_of(p.x, g.scale[0]), place_of(p.y, g.scale[1]), place_of(p.z, g.scale[2]), __int_as_float(p.w));
    if (wraps) {
        const int w = packed_wraps(wrap_count(px, 0, g), wrap_count(py, 1, g), wrap_count(pz, 2, g));
        wraps[s] = w;
        if (w != (kWrapBias | (kWrapBias << kWrapBits) | (kWrapBias << (2 * kWrapBits)))) st->outside_box = 1u;
    }
}

__global__ void k_edge_place(int n, const unsigned* key, const int* arrival, const int* cell_start,
                             int* __restrict__ list, int cells, int* __restrict__ cell_count) {
    if (!dsmd::after_previous()) return;
    dsmd::cell_place(blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x, 0, n, key, arrival, cell_start, list, cells, cell_count);
}

struct SearchArgs {
    int n, n_centers, stride;
    float band;                        // of the float form: |r2 - r2_list| below this is decided in fp64
    const int4* pq;
    const float4* pf;
    const double *x, *y, *z;
    const int* cell_start;
    const unsigned char* centre_ok;    // or null
    unsigned* rows;
    int* counts;                       // by sorted slot
    int* group_sum;                    // edges of the slots of one block
    long long* group_start;            // their exclusive sums, written by the last block
    EdgeStatus* st;
    dsmd::Mail* mail;                  // edges, out_of_bounds, need_stride, outside_box
    unsigned long long seq;
};

template <bool PERIODIC>
__device__ __forceinline__ bool within_fp64(const Grid& g, const SearchArgs& a, int ai, int aj) {
    double dx = a.x[aj] - a.x[ai], dy = a.y[aj] - a.y[ai], dz = a.z[aj] - a.z[ai];
    if (PERIODIC) {
        dx -= g.box[0] * rint(dx / g.box[0]);
        dy -= g.box[1] * rint(dy / g.box[1]);
        dz -= g.box[2] * rint(dz / g.box[2]);
    }
    const double r2 = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
    return r2 < g.r2_list_d;
}

// The end of a search: counts of the block's slots become the block's sum, and the block that finishes last turns the sums
// into starts and reports to the host. Saves a scan over the atoms and a copy of its end.
__device__ __forceinline__ void finish_search(const SearchArgs& a, int count) {
    __shared__ int warp_sum[kSearchThreads / 32];
    __shared__ long long carry;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int sum = min(count, a.stride), most = count;
    for (int o = 16; o > 0; o >>= 1) {
        sum += __shfl_down_sync(0xffffffffu, sum, o);
        most = max(most, __shfl_down_sync(0xffffffffu, most, o));
    }
    if (lane == 0) {
        warp_sum[w] = sum;
        if (most > a.stride) atomicMax(&a.st->need_stride, static_cast<unsigned>(most));
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        int total = 0;
        for (int k = 0; k < kSearchThreads / 32; ++k) total += warp_sum[k];
        a.group_sum[blockIdx.x] = total;
        carry = 0;
    }
    if (!dsmd::last_block(&a.st->ticket)) return;
    constexpr int kEach = 16;   // consecutive sums per thread and round
    for (unsigned base = 0; base < gridDim.x; base += kSearchThreads * kEach) {
        const unsigned first = base + threadIdx.x * kEach;
        int v[kEach], mine = 0;
#pragma unroll
        for (int k = 0; k < kEach; ++k) v[k] = first + k < gridDim.x ? __ldcg(&a.group_sum[first + k]) : 0;
#pragma unroll
        for (int k = 0; k < kEach; ++k) mine += v[k];
        int incl = mine;
        for (int o = 1; o < 32; o <<= 1) {
            const int up = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += up;
        }
        if (lane == 31) warp_sum[w] = incl;
        __syncthreads();
        long long at = carry + incl - mine;
        int all = 0;
        for (int k = 0; k < kSearchThreads / 32; ++k) {
            if (k < w) at += warp_sum[k];
            all += warp_sum[k];
        }
#pragma unroll
        for (int k = 0; k < kEach; ++k) {
            if (first + k < gridDim.x) a.group_start[first + k] = at;
            at += v[k];
        }
        __syncthreads();
        if (threadIdx.x == 0) carry += all;
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        const double out[4] = {static_cast<double>(carry), static_cast<double>(__ldcg(&a.st->out_of_bounds)),
                               static_cast<double>(__ldcg(&a.st->need_stride)), static_cast<double>(__ldcg(&a.st->outside_box))};
        *a.st = EdgeStatus{};   // for the next build; one that has to search again remembers the other words
        dsmd::post(a.mail, out, 4, a.seq);
    }
}

constexpr unsigned kUndecided = 0x80000000u;   // in a row: inside the rounding band
constexpr int kAtATime = 3;                    // candidates in flight per thread (0.535 ms per graph of 1,000,000; 0.54 to 0.57 ms with 2, 4, 6)

// One thread per sorted slot; hits go to the slot's column of its 32-atom slice: the neighbour's atom index, or, PERIODIC
// (all axes wrap), its sorted slot (the expansion reads the neighbour's position by slot).
//
// What bounds it: instruction issue. The loop over the candidates of a cell row does nothing but three subtractions, a sum
// of squares and a comparison on float places: the image of a cell row is known (the row's window crosses the boundary or
// not), so the atom's own place is shifted instead of taking nearest images of every candidate; hits inside the rounding
// band are marked and decided in fp64 afterwards. 1,000,000 atoms, 100 candidates and 26 hits each: 0.28 ms (0.35 ms before).
template <bool PERIODIC>
__global__ void __launch_bounds__(kSearchThreads) k_edge_search(Grid g, SearchArgs a) {
    if (!dsmd::after_previous()) return;
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    int count = 0;
    const int4 pi = a.pq[min(p, a.n - 1)];
    const int centre = pi.w & ~kPruned;
    if (p < a.n && centre < a.n_centers && !(a.centre_ok && !a.centre_ok[centre])) {
        unsigned* row_of_p = a.rows + (static_cast<size_t>(p >> 5) * a.stride) * 32 + (p & 31);
        const float fx = place_of(pi.x, g.scale[0]), fy = place_of(pi.y, g.scale[1]), fz = place_of(pi.z, g.scale[2]);
        const float len[3] = {static_cast<float>(g.box[0]), static_cast<float>(g.box[1]), static_cast<float>(g.box[2])};   // PERIODIC
        const float near2 = g.r2_list - a.band, far2 = g.r2_list + a.band;
        unsigned undecided = 0u;
        const int cx = static_cast<int>(dsmd::cell_of(static_cast<unsigned>(pi.x), g.wrap[0], g.nc[0]));
        const int cy = static_cast<int>(dsmd::cell_of(static_cast<unsigned>(pi.y), g.wrap[1], g.nc[1]));
        const int cz = static_cast<int>(dsmd::cell_of(static_cast<unsigned>(pi.z), g.wrap[2], g.nc[2]));
        const int S = g.stencil;
        for (int dz = -S; dz <= S; ++dz) {
            int zc = cz + dz;
            float sz = fz;   // the atom's place as the cell row sees it
            if (PERIODIC) {
                if (zc < 0) { zc += g.nc[2]; sz += len[2]; }
                else if (zc >= g.nc[2]) { zc -= g.nc[2]; sz -= len[2]; }
            } else if (zc < 0 || zc >= g.nc[2]) continue;
            for (int dy = -S; dy <= S; ++dy) {
                int yc = cy + dy;
                float sy = fy;
                if (PERIODIC) {
                    if (yc < 0) { yc += g.nc[1]; sy += len[1]; }
                    else if (yc >= g.nc[1]) { yc -= g.nc[1]; sy -= len[1]; }
                } else if (yc < 0 || yc >= g.nc[1]) continue;
                const int* row = a.cell_start + (zc * g.nc[1] + yc) * g.nc[0];
                dsmd::RowWindow win;
                if (!dsmd::row_window(g, pi, cy, cz, dy, dz, win)) continue;
                int s = row[win.a0], end = row[win.b0 + 1];
                float sx = fx;
                if (PERIODIC && win.b1 >= win.a1 && cx > win.b0) sx -= len[0];   // an atom near the upper face: the lower end first
                for (;;) {
                    for (; s < end; s += kAtATime) {   // loads first, and no branch but the stores'
                        float4 pj[kAtATime];
#pragma unroll
                        for (int u = 0; u < kAtATime; ++u) pj[u] = a.pf[min(s + u, end - 1)];
#pragma unroll
                        for (int u = 0; u < kAtATime; ++u) {
                            const float dx = pj[u].x - sx, ey = pj[u].y - sy, ez = pj[u].z - sz;
                            const float r2 = fmaf(dx, dx, fmaf(ey, ey, ez * ez));
                            const int w = __float_as_int(pj[u].w);
                            const bool hit = r2 < far2 && s + u != p && s + u < end && (PERIODIC || w >= 0);
                            const unsigned v = static_cast<unsigned>(PERIODIC ? s + u : w) | (r2 >= near2 ? kUndecided : 0u);
                            if (hit && count < a.stride) row_of_p[count * 32] = v;
                            undecided |= hit ? v : 0u;
                            count += hit ? 1 : 0;
                        }
                    }
                    if (!PERIODIC || win.b1 < win.a1) break;
                    s = row[win.a1];   // the part of the window at the other end of the box
                    end = row[win.b1 + 1];
                    sx = cx <= win.b0 ? fx + len[0] : fx;
                    win.b1 = win.a1 - 1;
                }
            }
        }
        if ((undecided & kUndecided) && count <= a.stride) {
            int kept = 0;
            for (int k = 0; k < count; ++k) {
                unsigned v = row_of_p[k * 32];
                if (v & kUndecided) {
                    v &= ~kUndecided;
                    if (!within_fp64<PERIODIC>(g, a, centre, PERIODIC ? a.pq[v].w & ~kPruned : static_cast<int>(v))) continue;
                }
                row_of_p[kept++ * 32] = v;
            }
            count = kept;
        }
    }
    if (p < a.n) a.counts[p] = min(count, a.stride);
    finish_search(a, count);
}

// Few atoms: a warp per atom. What bounds the form above there is the chain of dependent reads along one thread's candidates
// (40 us at 2,000 atoms), here the lanes take a cell row each, number the candidates of all rows (in the order of the other
// form), and test 32 at a time. Costs three times the instructions.
constexpr int kWarpSearchMost = 32768;   // atoms: whole builds of 10,000 take 90 us (99 us by thread), of 30,000 110 (113), of 60,000 144 (123)
constexpr int kWarpCandidates = 512;     // numbered at a time

template <bool PERIODIC>
__global__ void __launch_bounds__(kSearchThreads) k_edge_search_warp(Grid g, SearchArgs a) {
    if (!dsmd::after_previous()) return;
    __shared__ int s_slots[kSearchThreads / 32][kWarpCandidates];
    const int p = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    int* slots = s_slots[threadIdx.x >> 5];
    int count = 0;
    const int4 pi = a.pq[min(p, a.n - 1)];
    const int centre = pi.w & ~kPruned;
    if (p < a.n && centre < a.n_centers && !(a.centre_ok && !a.centre_ok[centre])) {
        unsigned* row_of_p = a.rows + (static_cast<size_t>(p >> 5) * a.stride) * 32 + (p & 31);
        const int S = g.stencil, side = 2 * S + 1;
        const int dz = lane / side - S, dy = lane % side - S;
        const int cy = static_cast<int>(dsmd::cell_of(static_cast<unsigned>(pi.y), g.wrap[1], g.nc[1]));
        const int cz = static_cast<int>(dsmd::cell_of(static_cast<unsigned>(pi.z), g.wrap[2], g.nc[2]));
        int yc = cy + dy, zc = cz + dz;
        bool open = lane < side * side;
        if (PERIODIC) {
            if (yc < 0) yc += g.nc[1]; else if (yc >= g.nc[1]) yc -= g.nc[1];
            if (zc < 0) zc += g.nc[2]; else if (zc >= g.nc[2]) zc -= g.nc[2];
        } else {
            open = open && yc >= 0 && yc < g.nc[1] && zc >= 0 && zc < g.nc[2];
        }
        dsmd::RowWindow win;
        open = open && dsmd::row_window(g, pi, cy, cz, dy, dz, win);
        int s0 = 0, s1 = 0, len0 = 0, len1 = 0;
        if (open) {
            const int* row = a.cell_start + (zc * g.nc[1] + yc) * g.nc[0];
            s0 = row[win.a0];
            len0 = row[win.b0 + 1] - s0;
            if (win.b1 >= win.a1) {
                s1 = row[win.a1];
                len1 = row[win.b1 + 1] - s1;
            }
        }
        const int len = len0 + len1;
        int incl = len;
        for (int o = 1; o < 32; o <<= 1) {
            const int up = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += up;
        }
        const int total = __shfl_sync(0xffffffffu, incl, 31), begin = incl - len;
        for (int base = 0; base < total; base += kWarpCandidates) {
            __syncwarp();
            const int k0 = max(base - begin, 0), k1 = min(base + kWarpCandidates - begin, len);
            for (int k = k0; k < k1; ++k) slots[begin + k - base] = k < len0 ? s0 + k : s1 + (k - len0);
            __syncwarp();
            const int n = min(total - base, kWarpCandidates);
            for (int t = lane; t - lane < n; t += 32) {
                const int s = t < n ? slots[t] : p;
                const int4 pj = a.pq[s];
                const float dx = dsmd::fixed_delta(pj.x, pi.x, g.scale[0]);
                const float ey = dsmd::fixed_delta(pj.y, pi.y, g.scale[1]);
                const float ez = dsmd::fixed_delta(pj.z, pi.z, g.scale[2]);
                const float r2 = dx * dx + ey * ey + ez * ez;
                bool hit = r2 < g.r2_list + g.band && s != p && pj.w >= 0;
                if (hit && r2 >= g.r2_list - g.band) hit = within_fp64<PERIODIC>(g, a, centre, pj.w);
                const unsigned hits = __ballot_sync(0xffffffffu, hit);
                const int k = count + __popc(hits & ((1u << lane) - 1u));
                if (hit && k < a.stride) row_of_p[k * 32] = static_cast<unsigned>(PERIODIC ? s : pj.w);
                count += __popc(hits);
            }
        }
    }
    if (p < a.n && lane == 0) a.counts[p] = min(count, a.stride);
    finish_search(a, lane == 0 ? count : 0);
}

// What the expansion of a 32-atom slice knows of its edges: a block takes the slice, lays its rows out in flat order in
// shared memory (rows lie 32 atoms side by side: read and transposed here, the rows come in full lines) and walks the flat
// order 32 edges at a time, aligned to multiples of 32 in the output, so that every array is written in whole sectors.
constexpr int kFlat = 1024;   // edges laid out at a time

struct FlatSlice {
    int entry[kFlat];
    unsigned char atom[kFlat];   // of the slice, 0 .. 31
    int prefix[33];
    long long start;
};

// Where the slice's edges start, and the prefix sums of its atoms' counts.
__device__ __forceinline__ void open_slice(FlatSlice& f, int n, int group_shift, const int* counts,
                                           const long long* group_start) {
    if (threadIdx.x < 32) {
        const int lane = threadIdx.x, p0 = blockIdx.x * 32, p = p0 + lane;
        const int cnt = p < n ? counts[p] : 0;
        int incl = cnt;
        for (int o = 1; o < 32; o <<= 1) {
            const int up = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += up;
        }
        f.prefix[lane + 1] = incl;
        if (lane == 0) f.prefix[0] = 0;
        // the atoms between the group's first and the slice's (groups of 2^group_shift atoms)
        int before = 0;
        for (int q = ((p0 >> group_shift) << group_shift) + lane; q < p0; q += 32) before += counts[q];
        for (int o = 16; o > 0; o >>= 1) before += __shfl_down_sync(0xffffffffu, before, o);
        if (lane == 0) f.start = group_start[p0 >> group_shift] + before;
    }
    __syncthreads();
}

// Flat positions [from, from + kFlat) of the slice.
__device__ __forceinline__ void lay_flat(FlatSlice& f, int from, int stride, const unsigned* rows) {
    const int lane = threadIdx.x & 31, begin = f.prefix[lane], cnt = f.prefix[lane + 1] - begin;
    const unsigned* slice = rows + static_cast<size_t>(blockIdx.x) * stride * 32 + lane;
    const int k1 = min(cnt, from + kFlat - begin);
    for (int k = threadIdx.x >> 5; k < k1; k += kFillThreads / 32) {
        const int at = begin + k - from;
        if (at < 0) continue;
        f.entry[at] = static_cast<int>(__ldcs(slice + static_cast<size_t>(k) * 32));
        f.atom[at] = static_cast<unsigned char>(lane);
    }
    __syncthreads();
}

// Interface form.
__global__ void __launch_bounds__(kFillThreads) k_edge_fill(int n, long long n_edges, int stride, int group_shift, const int4* pq,
                            const unsigned* rows, const int* counts,
                            const long long* group_start, int n_centers, const int* owner,
                            const double* shift_x, const double* shift_y,
                            const double* shift_z, long long* __restrict__ edges,
                            double* __restrict__ shift) {
    if (!dsmd::after_previous()) return;
    __shared__ FlatSlice f;
    __shared__ int centres[32];
    // the three shift components of 32 edges are 96 consecutive doubles of the output
    __shared__ double stage[kFillThreads / 32][96];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double* mine = stage[warp];
    if (warp == 1) centres[lane] = pq[min(blockIdx.x * 32 + lane, n - 1)].w & ~kPruned;
    open_slice(f, n, group_shift, counts, group_start);
    const int total = f.prefix[32];
    const int skip = static_cast<int>(f.start & 31);   // tiles are aligned in the output
    for (int from = 0; from < total; from += kFlat) {
        lay_flat(f, from, stride, rows);
        const int upto = min(total, from + kFlat);
        for (int t0 = ((from + skip) & ~31) - skip + 32 * warp; t0 < upto; t0 += kFillThreads) {
            const int t = t0 + lane;
            if (t >= from && t < upto) {
                const int nb = f.entry[t - from];
                const long long o = f.start + t;
                // the first n_centers atoms are real: they stand for themselves and carry no shift (EdgeBuilder::Images'
                // contract), so only image atoms cost the four scattered reads
                const bool image = owner && nb >= n_centers;
                __stcs(edges + o, static_cast<long long>(centres[f.atom[t - from]]));
                __stcs(edges + n_edges + o, static_cast<long long>(image ? owner[nb] : nb));
                if (shift) {
                    mine[3 * lane] = image ? shift_x[nb] : 0.0;
                    mine[3 * lane + 1] = image ? shift_y[nb] : 0.0;
                    mine[3 * lane + 2] = image ? shift_z[nb] : 0.0;
                }
            }
            if (shift) {
                __syncwarp();
                double* out = shift + 3 * (f.start + t0);
                const int q0 = 3 * max(from - t0, 0), q1 = 3 * min(32, upto - t0);
                for (int q = lane; q < q1; q += 32)
                    if (q >= q0) __stcs(out + q, mine[q]);
                __syncwarp();
            }
        }
        __syncthreads();
    }
}

// Compact periodic form: centres in cell order, the neighbours of a centre in the order of the search, as in the interface
// form. Rows hold neighbour slots, so positions and wrap counts are read where they lie whatever the caller's atom
// numbering. Displacements come from the fixed-point coordinates (resolution box / 2^32); the lattice shift refers to the
// caller's coordinates: x[dst] + shift * box - x[src] = vec. WRAPS: some atom lies outside the box.
// What bounds it: writing 23 bytes per edge (0.6 GB for 26 million edges: 0.09 ms at copy speed), then the gathers of the
// neighbours; 0.19 ms (0.28 ms before). 14 blocks per SM: registers for 14 cost nothing and hide the start of a slice.
template <bool WRAPS>
__global__ void __launch_bounds__(kFillThreads, 14) k_edge_fill_compact(
    Grid g, int n, int stride, int group_shift, const int4* pq, const int* wraps,
    const unsigned* rows, const int* counts, const long long* group_start,
    int* __restrict__ src, int* __restrict__ dst, signed char* __restrict__ shift, float* __restrict__ vec) {
    if (!dsmd::after_previous()) return;
    __shared__ FlatSlice f;
    __shared__ int4 centres[32];
    __shared__ int centre_wraps[32];
    // shift bytes and vector components of 32 edges are 96 consecutive bytes / floats of the output, written as words
    __shared__ __align__(16) float stage_vec[kFillThreads / 32][96];
    __shared__ __align__(16) signed char stage_shift[kFillThreads / 32][96];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float* my_vec = stage_vec[warp];
    signed char* my_shift = stage_shift[warp];
    if (warp == 1) {
        const int p = min(blockIdx.x * 32 + lane, n - 1);
        centres[lane] = pq[p];
        if (WRAPS) centre_wraps[lane] = wraps[p];
    }
    open_slice(f, n, group_shift, counts, group_start);
    const int total = f.prefix[32];
    const int skip = static_cast<int>(f.start & 31);   // tiles are aligned in the output
    const double unit[3] = {g.box[0] / 4294967296.0, g.box[1] / 4294967296.0, g.box[2] / 4294967296.0};
    for (int from = 0; from < total; from += kFlat) {
        lay_flat(f, from, stride, rows);
        const int upto = min(total, from + kFlat);
        int t0 = ((from + skip) & ~31) - skip + 32 * warp;
        // the next tile's neighbours are on their way while this one is written
        int4 pj_next{};
        int wj_next = 0;
        const auto fetch = [&](int t) {
            if (t < from || t >= upto) return;
            const int slot = f.entry[t - from];
            pj_next = pq[slot];
            if (WRAPS) wj_next = wraps[slot];
        };
        fetch(t0 + lane);
        for (; t0 < upto; t0 += kFillThreads) {
            const int t = t0 + lane;
            const int4 pj = pj_next;
            const int wj = wj_next;
            fetch(t + kFillThreads);
            if (t >= from && t < upto) {
                const int c = f.atom[t - from];
                const int4 pi = centres[c];
                const int wi = WRAPS ? centre_wraps[c] : 0;
                const long long o = f.start + t;
                const unsigned cj[3] = {static_cast<unsigned>(pj.x), static_cast<unsigned>(pj.y), static_cast<unsigned>(pj.z)};
                const unsigned ci[3] = {static_cast<unsigned>(pi.x), static_cast<unsigned>(pi.y), static_cast<unsigned>(pi.z)};
#pragma unroll
                for (int a = 0; a < 3; ++a) {
                    // the wrapped 32-bit difference is the nearest image; its sign against the order of the wrapped
                    // coordinates tells which image of the neighbour that is
                    const int nearest = static_cast<int>(cj[a] - ci[a]);
                    int image = (cj[a] < ci[a] ? 1 : 0) - (nearest < 0 ? 1 : 0);
                    if (WRAPS) image -= wrap_field(wj, a) - wrap_field(wi, a);
                    my_shift[3 * lane + a] = static_cast<signed char>(image);
                    my_vec[3 * lane + a] = static_cast<float>(static_cast<double>(nearest) * unit[a]);
                }
                __stcs(src + o, pi.w);
                __stcs(dst + o, pj.w);
            }
            __syncwarp();
            float* out_vec = vec + 3 * (f.start + t0);
            signed char* out_shift = shift + 3 * (f.start + t0);
            const int q0 = 3 * max(from - t0, 0), q1 = 3 * min(32, upto - t0);
            if (q0 == 0 && q1 == 96) {   // a whole tile
                if (lane < 24) {
                    __stcs(reinterpret_cast<float4*>(out_vec) + lane, reinterpret_cast<const float4*>(my_vec)[lane]);
                    __stcs(reinterpret_cast<int*>(out_shift) + lane, reinterpret_cast<const int*>(my_shift)[lane]);
                }
            } else {
                for (int q = lane; q < q1; q += 32)
                    if (q >= q0) {
                        out_vec[q] = my_vec[q];
                        out_shift[q] = my_shift[q];
                    }
            }
            __syncwarp();
        }
        __syncthreads();
    }
}

// Smallest and largest coordinate per axis, reported to the host: x, y, z least, x, y, z most. NaN coordinates do not count
// (they are found when the atoms are put into cells).
__global__ void __launch_bounds__(kThreads) k_edge_bounds(int n, const double* x, const double* y,
                                                          const double* z, double* __restrict__ partials, unsigned* ticket,
                                                          dsmd::Mail* mail, unsigned long long seq) {
    if (!dsmd::after_previous()) return;
    __shared__ double sh[kThreads / 32][6];
    const auto over_block = [&](double (&v)[6]) {
        for (int k = 0; k < 6; ++k)
            for (int o = 16; o > 0; o >>= 1) {
                const double u = __shfl_down_sync(0xffffffffu, v[k], o);
                v[k] = k < 3 ? fmin(v[k], u) : fmax(v[k], u);
            }
        if ((threadIdx.x & 31) == 0)
            for (int k = 0; k < 6; ++k) sh[threadIdx.x >> 5][k] = v[k];
        __syncthreads();
        for (int k = 0; k < 6; ++k)
            for (int w = 0; w < kThreads / 32; ++w) v[k] = k < 3 ? fmin(v[k], sh[w][k]) : fmax(v[k], sh[w][k]);
        __syncthreads();
    };
    const double inf = __longlong_as_double(0x7FF0000000000000ll);
    double v[6] = {inf, inf, inf, -inf, -inf, -inf};
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const double c[3] = {x[i], y[i], z[i]};
        for (int k = 0; k < 3; ++k) {
            v[k] = fmin(v[k], c[k]);
            v[3 + k] = fmax(v[3 + k], c[k]);
        }
    }
    over_block(v);
    if (threadIdx.x == 0)
        for (int k = 0; k < 6; ++k) partials[6 * blockIdx.x + k] = v[k];
    if (!dsmd::last_block(ticket)) return;
    for (unsigned b = threadIdx.x; b < gridDim.x; b += blockDim.x)
        for (int k = 0; k < 6; ++k) {
            const double u = __ldcg(&partials[6 * b + k]);
            v[k] = k < 3 ? fmin(v[k], u) : fmax(v[k], u);
        }
    over_block(v);
    if (threadIdx.x == 0) {
        *ticket = 0u;
        dsmd::post(mail, v, 6, seq);
    }
}

// ---- periodic image atoms, their forces folded back, receiver marking (the work of MLIPStep::prepare / add_forces /
// virial around the edge build, src/MLIPStep.cu:214-432) ----------------------------------------------------------------
//
// Semantics (what parity depends on): on an axis with images, a position is first wrapped into [from, from + period);
// the image with lattice shift (sx, sy, sz) != 0, |s_a| <= reach[a], exists when p_a + s_a period_a lies inside
// [keep_lo, keep_hi] on every axis with images; the images of an atom are numbered in the order sx, sy, sz ascending and
// stored consecutively, atom after atom, behind the wrapped atoms.
//
// Along one axis the admissible shifts of an atom are a handful of values, found once and kept as a bit mask (bit
// s + reach). The images of an atom are then the product of three bit sets minus the origin, so their count is a product
// of population counts, and the k-th image is decoded from k by division - which lets the writing kernel run one thread
// per OUTPUT slot (unit-stride stores of every output array) instead of one thread per atom with scattered stores.
struct ImageLattice {
    double period[3], from[3], keep_lo[3], keep_hi[3];
    int reach[3];
};

constexpr int kMaskBits = 17;   // shifts -8 .. 8

__device__ __forceinline__ double image_coord(double p, int s, double period) {
    return __dadd_rn(p, __dmul_rn(static_cast<double>(s), period));   // no contraction: rounds as p + s * period
}

__device__ __forceinline__ double wrapped_coord(const ImageLattice& L, int a, double v) {
    return L.reach[a] > 0 ? v - L.period[a] * floor((v - L.from[a]) / L.period[a]) : v;
}

__device__ __forceinline__ unsigned axis_mask(const ImageLattice& L, int a, double p) {
    const int r = L.reach[a];
    if (r == 0) return 1u;
    unsigned m = 0;
    for (int s = -r; s <= r; ++s) {
        const double q = image_coord(p, s, L.period[a]);
        if (!(q < L.keep_lo[a] || q > L.keep_hi[a])) m |= 1u << (s + r);
    }
    return m;
}

__device__ __forceinline__ int nth_set_bit(unsigned mask, int n) {
    int b = 0;
    for (;; ++b)
        if ((mask >> b) & 1u) {
            if (n == 0) break;
            --n;
        }
    return b;
}

// Per atom: the three shift masks packed into one word, and how many images that makes.
__global__ void k_image_masks(ImageLattice L, int n, const double* x, const double* y,
                              const double* z, unsigned long long* __restrict__ masks,
                              long long* __restrict__ counts) {
    if (!dsmd::after_previous()) return;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const unsigned mx = axis_mask(L, 0, wrapped_coord(L, 0, x[i]));
    const unsigned my = axis_mask(L, 1, wrapped_coord(L, 1, y[i]));
    const unsigned mz = axis_mask(L, 2, wrapped_coord(L, 2, z[i]));
    const bool self = ((mx >> L.reach[0]) & (my >> L.reach[1]) & (mz >> L.reach[2]) & 1u) != 0u;
    masks[i] = static_cast<unsigned long long>(mx) | (static_cast<unsigned long long>(my) << kMaskBits) |
               (static_cast<unsigned long long>(mz) << (2 * kMaskBits));
    counts[i] = static_cast<long long>(__popc(mx)) * __popc(my) * __popc(mz) - (self ? 1 : 0);
}

// Images of the whole system, reported to the host.
__global__ void k_image_total(int n, const long long* counts, const long long* first_image, dsmd::Mail* mail,
                              unsigned long long seq) {
    if (!dsmd::after_previous()) return;
    const double total[1] = {static_cast<double>(first_image[n - 1] + counts[n - 1])};
    dsmd::post(mail, total, 1, seq);
}

// One thread per output slot: slots [0, n) are the wrapped atoms, slot n + m is image number m of the whole system, which
// belongs to the last atom whose first image number is <= m.
__global__ void k_image_fill(ImageLattice L, int n, long long n_images, const double* x,
                             const double* y, const double* z, const int* type,
                             const unsigned long long* masks, const long long* first_image,
                             double* __restrict__ out_x, double* __restrict__ out_y, double* __restrict__ out_z,
                             int* __restrict__ out_type, int* __restrict__ out_owner, double* __restrict__ off_x,
                             double* __restrict__ off_y, double* __restrict__ off_z) {
    if (!dsmd::after_previous()) return;
    const long long t = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
    if (t >= n + n_images) return;
    int owner;
    int s[3] = {0, 0, 0};
    if (t < n) {
        owner = static_cast<int>(t);
    } else {
        const long long m = t - n;
        int lo = 0, hi = n;   // first_image is non-decreasing; atoms without images repeat their successor's value
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (first_image[mid] <= m) lo = mid; else hi = mid;
        }
        owner = lo;
        const unsigned long long w = masks[owner];
        const unsigned field = (1u << kMaskBits) - 1u;
        const unsigned mx = static_cast<unsigned>(w) & field, my = static_cast<unsigned>(w >> kMaskBits) & field,
                       mz = static_cast<unsigned>(w >> (2 * kMaskBits)) & field;
        const int ny = __popc(my), nz = __popc(mz);
        int k = static_cast<int>(m - first_image[owner]);
        if ((mx >> L.reach[0]) & (my >> L.reach[1]) & (mz >> L.reach[2]) & 1u) {
            // the origin sits in the product too: images at or behind its rank move up by one
            const int rank = (__popc(mx & ((1u << L.reach[0]) - 1u)) * ny + __popc(my & ((1u << L.reach[1]) - 1u))) * nz +
                             __popc(mz & ((1u << L.reach[2]) - 1u));
            if (k >= rank) ++k;
        }
        s[0] = nth_set_bit(mx, k / (ny * nz)) - L.reach[0];
        s[1] = nth_set_bit(my, (k / nz) % ny) - L.reach[1];
        s[2] = nth_set_bit(mz, k % nz) - L.reach[2];
    }
    const double px = wrapped_coord(L, 0, x[owner]), py = wrapped_coord(L, 1, y[owner]), pz = wrapped_coord(L, 2, z[owner]);
    const double qx = s[0] ? image_coord(px, s[0], L.period[0]) : px;
    const double qy = s[1] ? image_coord(py, s[1], L.period[1]) : py;
    const double qz = s[2] ? image_coord(pz, s[2], L.period[2]) : pz;
    out_x[t] = qx; out_y[t] = qy; out_z[t] = qz;
    out_type[t] = type ? type[owner] : 0;
    out_owner[t] = owner;
    off_x[t] = qx - px; off_y[t] = qy - py; off_z[t] = qz - pz;
}

// target[i] += f[i] + the forces on the images of atom i, added in slot order (MLIPStep::add_forces,
// src/MLIPStep.cu:108-124, 373-381), for the first n_out of the n atoms. with_images == 0: the images were edge shifts,
// not atoms the model saw, and carry no force.
__global__ void k_image_fold(int n_out, int n, int with_images, const double* fx,
                             const double* fy, const double* fz,
                             const long long* first_image, const long long* counts,
                             double* __restrict__ tx, double* __restrict__ ty, double* __restrict__ tz) {
    if (!dsmd::after_previous()) return;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_out) return;
    double sx = fx[i], sy = fy[i], sz = fz[i];
    if (with_images) {
        const long long begin = n + first_image[i], end = begin + counts[i];
        for (long long k = begin; k < end; ++k) {
            sx += fx[k];
            sy += fy[k];
            sz += fz[k];
        }
    }
    tx[i] += sx;
    ty[i] += sy;
    tz[i] += sz;
}

// Sum over atoms of r . F and of its three diagonal terms (MLIPStep::virial / virial_diag, src/MLIPStep.cu:126-148,
// 383-432): per-block sums in a fixed order, which the block that finishes last adds up in a fixed order and reports.
__global__ void __launch_bounds__(kThreads) k_virial(long long n, const double* x, const double* y,
                                                     const double* z, const double* fx,
                                                     const double* fy, const double* fz,
                                                     double* __restrict__ partials, unsigned* ticket, dsmd::Mail* mail, unsigned long long seq) {
    if (!dsmd::after_previous()) return;
    __shared__ double sh[kThreads / 32][3];
    const auto over_block = [&](double (&v)[3]) {   // the total in thread 0
        for (int a = 0; a < 3; ++a)
            for (int o = 16; o > 0; o >>= 1) v[a] += __shfl_down_sync(0xffffffffu, v[a], o);
        __syncthreads();
        if ((threadIdx.x & 31) == 0)
            for (int a = 0; a < 3; ++a) sh[threadIdx.x >> 5][a] = v[a];
        __syncthreads();
        if (threadIdx.x == 0)
            for (int a = 0; a < 3; ++a)
                for (int w = 1; w < kThreads / 32; ++w) v[a] += sh[w][a];
    };
    double v[3] = {0.0, 0.0, 0.0};
    for (long long p = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; p < n;
         p += static_cast<long long>(gridDim.x) * blockDim.x) {
        v[0] += x[p] * fx[p];
        v[1] += y[p] * fy[p];
        v[2] += z[p] * fz[p];
    }
    over_block(v);
    if (threadIdx.x == 0)
        for (int a = 0; a < 3; ++a) partials[3 * blockIdx.x + a] = v[a];
    if (!dsmd::last_block(ticket)) return;
    v[0] = v[1] = v[2] = 0.0;
    for (unsigned b = threadIdx.x; b < gridDim.x; b += blockDim.x)
        for (int a = 0; a < 3; ++a) v[a] += __ldcg(&partials[3 * b + a]);
    over_block(v);
    if (threadIdx.x == 0) {
        *ticket = 0u;
        const double out[4] = {v[0] + v[1] + v[2], v[0], v[1], v[2]};
        dsmd::post(mail, out, 4, seq);
    }
}

__global__ void k_mark_receivers(int n, const double* x, const double* y,
                                 const double* z, double lx, double ly, double lz, double hx, double hy,
                                 double hz, double reach2, unsigned char* __restrict__ ok) {
    if (!dsmd::after_previous()) return;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double dx = fmax(fmax(lx - x[i], x[i] - hx), 0.0);
    const double dy = fmax(fmax(ly - y[i], y[i] - hy), 0.0);
    const double dz = fmax(fmax(lz - z[i], z[i] - hz), 0.0);
    const double d2 = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
    ok[i] = d2 <= reach2 ? 1 : 0;   // a NaN position gives 0
}

template <class T>
bool grow(T*& ptr, size_t& capacity, size_t needed) {
    if (needed <= capacity) return true;
    const size_t grown = std::max(needed, capacity + capacity / 2);
    if (ptr) cudaFree(ptr);
    ptr = nullptr;
    capacity = 0;
    if (cudaMalloc(&ptr, grown * sizeof(T)) != cudaSuccess) return false;
    capacity = grown;
    return true;
}

}  // namespace

constexpr int kStatusWords = sizeof(EdgeStatus) / sizeof(int);
constexpr int kReduceBlocks = 592;   // 4 per SM of a B200: a fixed grid keeps the order of a sum the same for every n

struct dsmd_edges {
    int device = 0;
    std::string error;
    unsigned* key = nullptr;                size_t cap_key = 0;       // cell of an atom
    int* arrival = nullptr;                 size_t cap_arrival = 0;   // its place among the cell's atoms as they came
    int* list = nullptr;                    size_t cap_list = 0;      // the cells' atoms as they came
    int* cell_count = nullptr;              size_t cap_cell_count = 0;   // behind kStatusWords words of EdgeStatus
    bool counts_zero = false;               // counts and status are zero, as every search leaves them
    int* scan_sums = nullptr;               // [kScanBlocksMost]
    int4* pq = nullptr;                     size_t cap_pq = 0;
    float4* pf = nullptr;                   size_t cap_pf = 0;
    int* wraps = nullptr;                   size_t cap_wraps = 0;     // per sorted slot, periodic form
    int* cell_start = nullptr;              size_t cap_cells = 0;
    unsigned* rows = nullptr;               size_t cap_rows = 0;
    int* counts = nullptr;                  size_t cap_counts = 0;
    int* group_sum = nullptr;               size_t cap_group_sum = 0;
    long long* group_start = nullptr;       size_t cap_group_start = 0;
    int group_shift = 0;
    bool outside_box = false;
    unsigned char* temp = nullptr;          size_t cap_temp = 0;
    long long* edges = nullptr;             size_t cap_edges = 0;
    double* shift = nullptr;                size_t cap_shift = 0;
    int* c_src = nullptr;                   size_t cap_csrc = 0;
    int* c_dst = nullptr;                   size_t cap_cdst = 0;
    signed char* c_shift = nullptr;         size_t cap_cshift = 0;
    float* c_vec = nullptr;                 size_t cap_cvec = 0;
    // image atoms
    long long* img_counts = nullptr;        size_t cap_img_counts = 0;
    long long* img_offsets = nullptr;       size_t cap_img_offsets = 0;
    unsigned long long* img_masks = nullptr; size_t cap_img_masks = 0;
    int64_t n_img_src = 0;                  // atoms the last image build was given
    double* partials = nullptr;             // [6 * kReduceBlocks]
    unsigned* ticket = nullptr;             // blocks of a reduction that have finished
    dsmd::Mail* mail = nullptr;             // pinned: reports to the host
    unsigned long long seq = 0;
    double* ext[6] = {};                    size_t cap_ext[6] = {};     // x y z shift_x shift_y shift_z
    int* ext_type = nullptr;                size_t cap_ext_type = 0;
    int* ext_owner = nullptr;               size_t cap_ext_owner = 0;
    int64_t n_ext = 0;
    int stride = 0;
    int64_t n_edges = 0;
    bool have_shift = false;
    int64_t launches = 0;
};

namespace {

int efail(dsmd_edges* e, int code, const std::string& what) {
    e->error = what;
    return code;
}

#define EDGE_CUDA(e, call)                                                            \
    do {                                                                              \
        cudaError_t err_ = (call);                                                    \
        if (err_ != cudaSuccess) {                                                    \
            (e)->error = std::string(#call) + ": " + cudaGetErrorString(err_);        \
            return DSMD_ERR_CUDA;                                                     \
        }                                                                             \
    } while (0)

#define EDGE_ALLOC(e, ok)                                                             \
    do {                                                                              \
        if (!(ok)) return efail(e, DSMD_ERR_CUDA, "device allocation failed");        \
    } while (0)

// Grid over [lo, hi] (non-periodic) or [0, box) (periodic): cells at least cutoff / stencil wide, not more than about
// two cells per atom (a sparse box must not allocate a huge grid: src/EdgeBuilder.cu:50-61).
int edge_grid(dsmd_edges* e, Grid& g, const double lo[3], const double hi[3], bool periodic, double cutoff, int64_t n) {
    double max_scale = 0.0;
    double len[3];
    for (int a = 0; a < 3; ++a) {
        g.box[a] = periodic ? hi[a] : 0.0;
        if (periodic) {
            len[a] = hi[a];
            g.wrap[a] = 1;
            g.org[a] = 0.0;
            g.scale[a] = static_cast<float>(len[a] / 4294967296.0);
            max_scale = std::max(max_scale, len[a] / 4294967296.0);
        } else {
            // the upper face belongs to the box: stretch the mapped range by a hair so that hi maps below 1
            len[a] = std::max(hi[a] - lo[a], cutoff) * (1.0 + 1e-9);
            g.wrap[a] = 0;
            g.org[a] = lo[a];
            g.scale[a] = static_cast<float>(len[a] / 2147483648.0);
            max_scale = std::max(max_scale, len[a] / 2147483648.0);
        }
        g.inv_len[a] = 1.0 / len[a];
    }
    const long long max_cells = std::max<long long>(64, 2 * static_cast<long long>(n));
    // Half-width cells (25 cell rows around an atom) pay when a row holds a few atoms; in a sparse system the cost of
    // opening a row outweighs the tighter windows and 9 rows of full-width cells are faster (measured on 1,000,000
    // atoms at 0.05 / A^3, cutoff 5 A, 0.8 atoms per half-width cell: 0.79 ms against 0.89 ms per build).
    const double per_half_cell = static_cast<double>(n) / (len[0] * len[1] * len[2]) * (cutoff * cutoff * cutoff / 8.0);
    bool done = false;
    for (int stencil = per_half_cell >= 1.0 ? 2 : 1; stencil >= 1 && !done; --stencil) {
        double width = cutoff / stencil * (1.0 + 1e-6);
        for (int tries = 0; tries < 64; ++tries) {
            long long cells = 1;
            bool ok = true;
            for (int a = 0; a < 3; ++a) {
                int nc = std::max(1, static_cast<int>(std::floor(len[a] / width)));
                nc = std::min(nc, 1024);
                if (periodic && nc < 2 * stencil + 1) ok = false;
                g.nc[a] = nc;
                cells *= nc;
            }
            if (!ok) break;                       // box too small for this stencil: try the wider cells
            if (cells <= max_cells || stencil == 1) {
                if (cells > max_cells) { width *= 1.26; continue; }
                g.stencil = stencil;
                g.ncells = static_cast<int>(cells);
                done = true;
                break;
            }
            break;                                // too many half-width cells: fall back to full-width cells
        }
    }
    if (!done) return efail(e, DSMD_ERR_BOX_TOO_SMALL, "periodic box shorter than three cells of width cutoff");
    // finer cells along x: a cell row is a contiguous run of slots whatever the x cell width, and the search window
    // (rounded outwards to whole cells) is tighter
    g.x_reach = static_cast<float>(g.stencil * (len[0] / g.nc[0]) * 0.9999999);
    for (int refine = 4; refine > 1; refine >>= 1) {
        if (static_cast<long long>(g.nc[0]) * refine <= 4096 &&
            static_cast<long long>(g.ncells) * refine <= 4 * max_cells) {
            g.nc[0] *= refine;
            g.ncells *= refine;
            break;
        }
    }
    g.r2_list = static_cast<float>(cutoff * cutoff);
    g.r2_list_d = cutoff * cutoff;
    g.band = static_cast<float>(8.0 * cutoff * max_scale + 16.0 * cutoff * cutoff * 5.9604645e-8);
    double max_len = 0.0;
    for (int a = 0; a < 3; ++a) {
        g.cellw[a] = static_cast<float>(len[a] / g.nc[a]);
        max_len = std::max(max_len, len[a]);
    }
    g.r_pad = static_cast<float>(cutoff * (1.0 + 1e-4) + 8.0 * max_len * 1.2e-7);
    return DSMD_OK;
}

// Rounding band of the float form of the search: places carry up to 5 * 2^-24 of the box (two places, the box length added
// to one of them), and the sum of squares its roundings.
float float_band(const Grid& g, double cutoff) {
    double most = 0.0;
    for (int a = 0; a < 3; ++a) most = std::max(most, 1.0 / g.inv_len[a]);
    const double off = 5.0 * most * 5.9604645e-8 * 1.7320509;
    return static_cast<float>(static_cast<double>(g.band) + 2.0 * cutoff * off + off * off);
}

// bin, sort, gather, search (with row-overflow retry); returns the edge count.
template <bool PERIODIC>
int edge_search(dsmd_edges* e, const Grid& g, const double* d_x, const double* d_y, const double* d_z, int64_t n,
                int64_t n_centers, const int* d_owner, const unsigned char* d_ok, int row, double density_hint, double cutoff,
                int64_t* n_edges, cudaStream_t s) {
    const size_t un = static_cast<size_t>(n), table = static_cast<size_t>(g.ncells) + 1;
    const int in = static_cast<int>(n);
    const bool by_warp = n <= kWarpSearchMost;
    e->group_shift = by_warp ? 2 : 7;   // atoms per block of the search
    static_assert(kSearchThreads == 128, "group_shift");
    const unsigned groups = blocks_for(n, 1 << e->group_shift);
    EDGE_ALLOC(e, grow(e->key, e->cap_key, un));
    EDGE_ALLOC(e, grow(e->arrival, e->cap_arrival, un));
    EDGE_ALLOC(e, grow(e->list, e->cap_list, un));
    EDGE_ALLOC(e, grow(e->pq, e->cap_pq, un));
    EDGE_ALLOC(e, grow(e->pf, e->cap_pf, un));
    if (PERIODIC) EDGE_ALLOC(e, grow(e->wraps, e->cap_wraps, un));
    if (table + kStatusWords > e->cap_cell_count) e->counts_zero = false;
    EDGE_ALLOC(e, grow(e->cell_count, e->cap_cell_count, table + kStatusWords));
    EDGE_ALLOC(e, grow(e->cell_start, e->cap_cells, table));
    EDGE_ALLOC(e, grow(e->counts, e->cap_counts, un));
    EDGE_ALLOC(e, grow(e->group_sum, e->cap_group_sum, static_cast<size_t>(groups)));
    EDGE_ALLOC(e, grow(e->group_start, e->cap_group_start, static_cast<size_t>(groups)));
    int* const cell_count = e->cell_count + kStatusWords;
    EdgeStatus* const st = reinterpret_cast<EdgeStatus*>(e->cell_count);
    if (!e->counts_zero) EDGE_CUDA(e, cudaMemsetAsync(e->cell_count, 0, sizeof(int) * e->cap_cell_count, s));
    e->counts_zero = false;
    // (every launch is looked at before the next one is made: that one indexes with what it writes)
    dsmd::launch_next(k_edge_keys, blocks_for(n, kThreads), kThreads, 0, s, g, in, d_x, d_y, d_z, e->key, e->arrival, cell_count, st);
    EDGE_CUDA(e, cudaGetLastError());
    if (table <= static_cast<size_t>(dsmd::kScanMost)) {
        const int launched = dsmd::launch_cell_scan(static_cast<int>(table), 0, cell_count, e->scan_sums, e->cell_start, s);
        EDGE_CUDA(e, cudaGetLastError());
        e->launches += launched;
    } else {
        size_t scan_bytes = 0;
        cub::DeviceScan::ExclusiveSum(nullptr, scan_bytes, cell_count, e->cell_start, static_cast<int>(table), s);
        EDGE_ALLOC(e, grow(e->temp, e->cap_temp, scan_bytes));
        EDGE_CUDA(e, cub::DeviceScan::ExclusiveSum(e->temp, scan_bytes, cell_count, e->cell_start, static_cast<int>(table), s));
    }
    dsmd::launch_next(k_edge_place, blocks_for(n, kThreads), kThreads, 0, s, in, e->key, e->arrival, e->cell_start, e->list, static_cast<int>(table), cell_count);
    EDGE_CUDA(e, cudaGetLastError());
    dsmd::launch_next(k_edge_gather, blocks_for(n, kThreads), kThreads, 0, s, g, in, e->key, e->list, e->cell_start, d_x, d_y, d_z,
                      row == 1 ? d_ok : nullptr, d_owner, e->pq, e->pf, PERIODIC ? e->wraps : nullptr, st);
    EDGE_CUDA(e, cudaGetLastError());
    e->launches += 3;
    if (e->stride == 0) {
        const double expect = density_hint * 4.18879020479 * g.r2_list_d * std::sqrt(g.r2_list_d);
        e->stride = (std::max(16, static_cast<int>(expect * 1.5) + 16) + 3) & ~3;
    }
    for (int attempt = 0; attempt < 5; ++attempt) {
        const size_t slices = (un + 31) / 32;
        EDGE_ALLOC(e, grow(e->rows, e->cap_rows, slices * static_cast<size_t>(e->stride) * 32));
        const SearchArgs a{in, static_cast<int>(n_centers), e->stride, float_band(g, cutoff), e->pq, e->pf, d_x, d_y, d_z, e->cell_start,
                           row == 0 ? d_ok : nullptr, e->rows, e->counts, e->group_sum, e->group_start, st, e->mail, ++e->seq};
        if (by_warp) dsmd::launch_next(k_edge_search_warp<PERIODIC>, groups, kSearchThreads, 0, s, g, a);
        else dsmd::launch_next(k_edge_search<PERIODIC>, groups, kSearchThreads, 0, s, g, a);
        ++e->launches;
        EDGE_CUDA(e, cudaGetLastError());
        // the one wait of a build that does not overflow: edge count, bounds flag, row overflow
        EDGE_CUDA(e, dsmd::wait_report(e->mail, 4, e->seq, s));
        e->counts_zero = true;
        if (attempt == 0) e->outside_box = e->mail->value(3) != 0.0;
        if (e->mail->value(1) != 0.0)
            return efail(e, DSMD_ERR_OUT_OF_DOMAIN, "an atom lies outside the given box (or has a NaN position)");
        const int need = static_cast<int>(e->mail->value(2));
        if (need <= e->stride) {
            *n_edges = static_cast<int64_t>(e->mail->value(0));
            return DSMD_OK;
        }
        e->stride = (static_cast<int>(need * 1.2) + 8 + 3) & ~3;
    }
    return efail(e, DSMD_ERR_CAPACITY, "edge rows kept overflowing");
}

}  // namespace

extern "C" {

int dsmd_edges_create(int device, dsmd_edges** out) {
    if (!out) return DSMD_ERR_INVALID;
    int count = 0;
    if (cudaGetDeviceCount(&count) != cudaSuccess || device < 0 || device >= count) return DSMD_ERR_CUDA;
    dsmd_edges* e = new dsmd_edges();
    e->device = device;
    *out = e;
    EDGE_CUDA(e, cudaSetDevice(device));
    EDGE_CUDA(e, cudaMalloc(&e->partials, sizeof(double) * 6 * kReduceBlocks));
    EDGE_CUDA(e, cudaMalloc(&e->scan_sums, sizeof(int) * dsmd::kScanBlocksMost));
    EDGE_CUDA(e, cudaMalloc(&e->ticket, sizeof(unsigned)));
    EDGE_CUDA(e, cudaMemset(e->ticket, 0, sizeof(unsigned)));
    EDGE_CUDA(e, cudaMallocHost(&e->mail, sizeof(dsmd::Mail)));
    std::memset(e->mail, 0, sizeof(dsmd::Mail));
    return DSMD_OK;
}

void dsmd_edges_destroy(dsmd_edges* e) {
    if (!e) return;
    cudaSetDevice(e->device);
    cudaFree(e->key); cudaFree(e->arrival); cudaFree(e->list); cudaFree(e->cell_count); cudaFree(e->pf);
    cudaFree(e->pq); cudaFree(e->wraps); cudaFree(e->cell_start); cudaFree(e->rows); cudaFree(e->counts);
    cudaFree(e->group_sum); cudaFree(e->group_start); cudaFree(e->temp); cudaFree(e->edges); cudaFree(e->shift);
    cudaFree(e->c_src); cudaFree(e->c_dst); cudaFree(e->c_shift); cudaFree(e->c_vec); cudaFree(e->partials);
    cudaFree(e->ticket); cudaFree(e->scan_sums); cudaFree(e->img_counts); cudaFree(e->img_offsets); cudaFree(e->img_masks);
    if (e->mail) cudaFreeHost(e->mail);
    cudaFree(e->ext_type); cudaFree(e->ext_owner);
    for (int k = 0; k < 6; ++k) cudaFree(e->ext[k]);
    delete e;
}

const char* dsmd_edges_last_error(const dsmd_edges* e) { return e ? e->error.c_str() : "null edge builder"; }

int dsmd_edges_build(dsmd_edges* e, const double* d_x, const double* d_y, const double* d_z, int64_t n, double cutoff,
                     const double* lo, const double* hi, int64_t n_centers, const int32_t* d_owner,
                     const double* d_shift_x, const double* d_shift_y, const double* d_shift_z,
                     const unsigned char* d_receiver_ok, int row, int64_t* n_edges, void* stream) {
    if (!e || !n_edges) return DSMD_ERR_INVALID;
    *n_edges = 0;
    e->n_edges = 0;
    e->have_shift = false;
    if (!(cutoff > 0.0)) return efail(e, DSMD_ERR_INVALID, "cutoff must be positive");
    if (n < 0 || n >= std::numeric_limits<int32_t>::max() / 2) return efail(e, DSMD_ERR_INVALID, "atom count out of range");
    const bool images = d_owner != nullptr;
    if (images && (n_centers < 0 || n_centers > n || !d_shift_x || !d_shift_y || !d_shift_z))
        return efail(e, DSMD_ERR_INVALID, "invalid periodic image description");
    if (!images) n_centers = n;
    if (d_receiver_ok && row != 0 && row != 1) return efail(e, DSMD_ERR_INVALID, "invalid prune description");
    if (n <= 1) return DSMD_OK;
    if (!d_x || !d_y || !d_z) return DSMD_ERR_INVALID;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    EDGE_CUDA(e, cudaSetDevice(e->device));

    double box_lo[3], box_hi[3];
    if (lo && hi) {
        for (int a = 0; a < 3; ++a) { box_lo[a] = lo[a]; box_hi[a] = hi[a]; }
    } else {   // bounding box on the device: one extra wait
        dsmd::launch_next(k_edge_bounds, std::min<unsigned>(blocks_for(n, kThreads), kReduceBlocks), kThreads, 0, s, static_cast<int>(n), d_x, d_y, d_z, e->partials, e->ticket, e->mail, ++e->seq);
        ++e->launches;
        EDGE_CUDA(e, cudaGetLastError());
        EDGE_CUDA(e, dsmd::wait_report(e->mail, 6, e->seq, s));
        for (int a = 0; a < 3; ++a) { box_lo[a] = e->mail->value(a); box_hi[a] = e->mail->value(3 + a); }
    }
    for (int a = 0; a < 3; ++a)
        if (!(box_lo[a] <= box_hi[a]) || !std::isfinite(box_lo[a]) || !std::isfinite(box_hi[a]))
            return efail(e, DSMD_ERR_OUT_OF_DOMAIN, "invalid box or a non-finite position");

    Grid g{};
    { const int rc = edge_grid(e, g, box_lo, box_hi, false, cutoff, n); if (rc) return rc; }
    double volume = 1.0;
    for (int a = 0; a < 3; ++a) volume *= 1.0 / g.inv_len[a];
    int64_t E = 0;
    { const int rc = edge_search<false>(e, g, d_x, d_y, d_z, n, n_centers, d_owner, d_receiver_ok, row,
                                        static_cast<double>(n) / volume, cutoff, &E, s); if (rc) return rc; }
    e->n_edges = E;
    *n_edges = E;
    if (E == 0) return DSMD_OK;
    EDGE_ALLOC(e, grow(e->edges, e->cap_edges, 2 * static_cast<size_t>(E)));
    if (images) EDGE_ALLOC(e, grow(e->shift, e->cap_shift, 3 * static_cast<size_t>(E)));
    dsmd::launch_next(k_edge_fill, blocks_for(n, 32), kFillThreads, 0, s, static_cast<int>(n), E, e->stride, e->group_shift, e->pq, e->rows, e->counts,
                                                          e->group_start, static_cast<int>(n_centers), d_owner, d_shift_x,
                                                          d_shift_y, d_shift_z, e->edges, images ? e->shift : nullptr);
    ++e->launches;
    EDGE_CUDA(e, cudaGetLastError());
    e->have_shift = images;
    return DSMD_OK;
}

int dsmd_edges_result(const dsmd_edges* e, const int64_t** d_edge_index, const double** d_edge_shift, int64_t* n_edges) {
    if (!e) return DSMD_ERR_INVALID;
    if (d_edge_index) *d_edge_index = reinterpret_cast<const int64_t*>(e->edges);
    if (d_edge_shift) *d_edge_shift = e->have_shift ? e->shift : nullptr;
    if (n_edges) *n_edges = e->n_edges;
    return DSMD_OK;
}

int dsmd_edges_build_periodic(dsmd_edges* e, const double* d_x, const double* d_y, const double* d_z, int64_t n,
                              const double box[3], double cutoff, int64_t* n_edges, void* stream) {
    if (!e || !n_edges || !box) return DSMD_ERR_INVALID;
    *n_edges = 0;
    e->n_edges = 0;
    if (!(cutoff > 0.0)) return efail(e, DSMD_ERR_INVALID, "cutoff must be positive");
    if (n < 0 || n >= std::numeric_limits<int32_t>::max() / 2) return efail(e, DSMD_ERR_INVALID, "atom count out of range");
    for (int a = 0; a < 3; ++a)
        if (!(box[a] > 2.0 * cutoff)) return efail(e, DSMD_ERR_BOX_TOO_SMALL, "box must be longer than two cutoffs");
    if (n <= 1) return DSMD_OK;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    EDGE_CUDA(e, cudaSetDevice(e->device));
    Grid g{};
    const double zero[3] = {0.0, 0.0, 0.0};
    { const int rc = edge_grid(e, g, zero, box, true, cutoff, n); if (rc) return rc; }
    const double volume = box[0] * box[1] * box[2];
    int64_t E = 0;
    { const int rc = edge_search<true>(e, g, d_x, d_y, d_z, n, n, nullptr, nullptr, 1, static_cast<double>(n) / volume, cutoff, &E, s);
      if (rc) return rc; }
    e->n_edges = E;
    *n_edges = E;
    if (E == 0) return DSMD_OK;
    EDGE_ALLOC(e, grow(e->c_src, e->cap_csrc, static_cast<size_t>(E)));
    EDGE_ALLOC(e, grow(e->c_dst, e->cap_cdst, static_cast<size_t>(E)));
    EDGE_ALLOC(e, grow(e->c_shift, e->cap_cshift, 3 * static_cast<size_t>(E)));
    EDGE_ALLOC(e, grow(e->c_vec, e->cap_cvec, 3 * static_cast<size_t>(E)));
    const auto fill = e->outside_box ? k_edge_fill_compact<true> : k_edge_fill_compact<false>;
    dsmd::launch_next(fill, blocks_for(n, 32), kFillThreads, 0, s, g, static_cast<int>(n), e->stride, e->group_shift, e->pq, e->wraps, e->rows, e->counts,
                                                   e->group_start, e->c_src, e->c_dst, e->c_shift, e->c_vec);
    ++e->launches;
    EDGE_CUDA(e, cudaGetLastError());
    return DSMD_OK;
}

int dsmd_images_build(dsmd_edges* e, const double* d_x, const double* d_y, const double* d_z, const int32_t* d_type,
                      int64_t n, const double box[3], const double origin[3], const double region_lo[3],
                      const double region_hi[3], const int shells[3], int64_t* n_all, void* stream) {
    if (!e || !n_all || !box || !origin || !region_lo || !region_hi || !shells) return DSMD_ERR_INVALID;
    *n_all = 0;
    e->n_ext = 0;
    if (n < 0 || n >= std::numeric_limits<int32_t>::max() / 2) return efail(e, DSMD_ERR_INVALID, "atom count out of range");
    if (n == 0) return DSMD_OK;
    if (!d_x || !d_y || !d_z) return DSMD_ERR_INVALID;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    EDGE_CUDA(e, cudaSetDevice(e->device));
    ImageLattice lattice;
    for (int a = 0; a < 3; ++a) {
        if (shells[a] < 0 || shells[a] > 8) return efail(e, DSMD_ERR_INVALID, "image shells must be in 0 .. 8");
        if (shells[a] > 0 && !(box[a] > 0.0)) return efail(e, DSMD_ERR_INVALID, "box length must be positive on an image axis");
        lattice.period[a] = box[a];
        lattice.from[a] = origin[a];
        lattice.keep_lo[a] = region_lo[a];
        lattice.keep_hi[a] = region_hi[a];
        lattice.reach[a] = shells[a];
    }
    const size_t un = static_cast<size_t>(n);
    EDGE_ALLOC(e, grow(e->img_counts, e->cap_img_counts, un));
    EDGE_ALLOC(e, grow(e->img_offsets, e->cap_img_offsets, un));
    EDGE_ALLOC(e, grow(e->img_masks, e->cap_img_masks, un));
    size_t scan_bytes = 0;
    cub::DeviceScan::ExclusiveSum(nullptr, scan_bytes, e->img_counts, e->img_offsets, static_cast<int>(n), s);
    EDGE_ALLOC(e, grow(e->temp, e->cap_temp, scan_bytes));
    dsmd::launch_next(k_image_masks, blocks_for(n, kThreads), kThreads, 0, s, lattice, static_cast<int>(n), d_x, d_y, d_z, e->img_masks,
                                                              e->img_counts);
    EDGE_CUDA(e, cub::DeviceScan::ExclusiveSum(e->temp, scan_bytes, e->img_counts, e->img_offsets, static_cast<int>(n), s));
    // the image count comes to the host: the one synchronisation (MLIPStep::prepare does the same, src/MLIPStep.cu:254-255)
    dsmd::launch_next(k_image_total, 1, 1, 0, s, static_cast<int>(n), e->img_counts, e->img_offsets, e->mail, ++e->seq);
    EDGE_CUDA(e, cudaGetLastError());
    EDGE_CUDA(e, dsmd::wait_report(e->mail, 1, e->seq, s));
    const int64_t n_images = static_cast<int64_t>(e->mail->value(0));
    const int64_t total = n + n_images;
    if (total >= std::numeric_limits<int32_t>::max() / 2) return efail(e, DSMD_ERR_CAPACITY, "too many image atoms");
    for (int k = 0; k < 6; ++k) EDGE_ALLOC(e, grow(e->ext[k], e->cap_ext[k], static_cast<size_t>(total)));
    EDGE_ALLOC(e, grow(e->ext_type, e->cap_ext_type, static_cast<size_t>(total)));
    EDGE_ALLOC(e, grow(e->ext_owner, e->cap_ext_owner, static_cast<size_t>(total)));
    dsmd::launch_next(k_image_fill, blocks_for(total, kThreads), kThreads, 0, s, lattice, static_cast<int>(n), n_images, d_x, d_y, d_z, d_type,
                                                                 e->img_masks, e->img_offsets, e->ext[0], e->ext[1], e->ext[2],
                                                                 e->ext_type, e->ext_owner, e->ext[3], e->ext[4], e->ext[5]);
    e->launches += 3;
    EDGE_CUDA(e, cudaGetLastError());
    e->n_ext = total;
    e->n_img_src = n;
    *n_all = total;
    return DSMD_OK;
}

int dsmd_images_fold_forces(dsmd_edges* e, const double* d_fx, const double* d_fy, const double* d_fz, int64_t n_out,
                            int with_images, double* d_tx, double* d_ty, double* d_tz, void* stream) {
    if (!e || !d_fx || !d_fy || !d_fz || !d_tx || !d_ty || !d_tz) return DSMD_ERR_INVALID;
    if (e->n_img_src <= 0) return efail(e, DSMD_ERR_STATE, "no image atoms built");
    if (n_out < 0 || n_out > e->n_img_src) n_out = e->n_img_src;
    if (n_out == 0) return DSMD_OK;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    dsmd::launch_next(k_image_fold, blocks_for(n_out, kThreads), kThreads, 0, s, static_cast<int>(n_out), static_cast<int>(e->n_img_src),
                                                                 with_images, d_fx, d_fy, d_fz, e->img_offsets, e->img_counts,
                                                                 d_tx, d_ty, d_tz);
    ++e->launches;
    EDGE_CUDA(e, cudaGetLastError());
    return DSMD_OK;
}

int dsmd_virial_from_forces(dsmd_edges* e, const double* d_x, const double* d_y, const double* d_z, const double* d_fx,
                            const double* d_fy, const double* d_fz, int64_t n, double out[4], void* stream) {
    if (!e || !out || n < 0 || (n > 0 && (!d_x || !d_y || !d_z || !d_fx || !d_fy || !d_fz))) return DSMD_ERR_INVALID;
    out[0] = out[1] = out[2] = out[3] = 0.0;
    if (n == 0) return DSMD_OK;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    EDGE_CUDA(e, cudaSetDevice(e->device));
    const int blocks = static_cast<int>(std::min<int64_t>(kReduceBlocks, (n + kThreads - 1) / kThreads));
    dsmd::launch_next(k_virial, blocks, kThreads, 0, s, n, d_x, d_y, d_z, d_fx, d_fy, d_fz, e->partials, e->ticket, e->mail, ++e->seq);
    ++e->launches;
    EDGE_CUDA(e, cudaGetLastError());
    EDGE_CUDA(e, dsmd::wait_report(e->mail, 4, e->seq, s));
    for (int k = 0; k < 4; ++k) out[k] = e->mail->value(k);
    return DSMD_OK;
}

int dsmd_images_result(const dsmd_edges* e, const double** d_x, const double** d_y, const double** d_z,
                       const int32_t** d_type, const int32_t** d_owner, const double** d_shift_x, const double** d_shift_y,
                       const double** d_shift_z, int64_t* n_all) {
    if (!e) return DSMD_ERR_INVALID;
    if (d_x) *d_x = e->ext[0];
    if (d_y) *d_y = e->ext[1];
    if (d_z) *d_z = e->ext[2];
    if (d_type) *d_type = e->ext_type;
    if (d_owner) *d_owner = e->ext_owner;
    if (d_shift_x) *d_shift_x = e->ext[3];
    if (d_shift_y) *d_shift_y = e->ext[4];
    if (d_shift_z) *d_shift_z = e->ext[5];
    if (n_all) *n_all = e->n_ext;
    return DSMD_OK;
}

int dsmd_mark_receivers(dsmd_edges* e, const double* d_x, const double* d_y, const double* d_z, int64_t n,
                        const double lo[3], const double hi[3], double reach, unsigned char* d_ok, void* stream) {
    if (!e || !lo || !hi || n < 0 || (n > 0 && (!d_x || !d_y || !d_z || !d_ok))) return DSMD_ERR_INVALID;
    if (n == 0) return DSMD_OK;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    dsmd::launch_next(k_mark_receivers, blocks_for(n, kThreads), kThreads, 0, s, static_cast<int>(n), d_x, d_y, d_z, lo[0], lo[1], lo[2],
                                                                 hi[0], hi[1], hi[2], reach * reach, d_ok);
    ++e->launches;
    EDGE_CUDA(e, cudaGetLastError());
    return DSMD_OK;
}

int dsmd_edges_result_compact(const dsmd_edges* e, const int32_t** d_src, const int32_t** d_dst, const int8_t** d_shift,
                              const float** d_vec, int64_t* n_edges) {
    if (!e) return DSMD_ERR_INVALID;
    if (d_src) *d_src = e->c_src;
    if (d_dst) *d_dst = e->c_dst;
    if (d_shift) *d_shift = reinterpret_cast<const int8_t*>(e->c_shift);
    if (d_vec) *d_vec = e->c_vec;
    if (n_edges) *n_edges = e->n_edges;
    return DSMD_OK;
}

}  // extern "C"
