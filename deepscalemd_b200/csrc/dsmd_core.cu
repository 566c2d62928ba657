// The short-range nonbonded path on one B200 (sm_100a): cell binning and sort, Verlet list build with skin,
// LJ + real-space Ewald pair kernel, displacement check, velocity-Verlet halves, ghost pack/unpack, and the C ABI
// declared in include/dsmd_b200.h.
//
// Data layout in HBM (all arrays indexed by "slot"; owned atoms occupy [0, n_owned), ghosts [n_owned, n_total); both
// segments are sorted by cell, x fastest, at every list build):
//   x y z vx vy vz fx fy fz mass charge   double[capacity] each, two sets (the sort gathers from one into the other)
//   type gid                               int32[capacity], two sets
//   pq                                     int4[capacity]: fixed-point x, y, z and the type in w (what the kernels read)
//   qf                                     float[capacity]: charge (read only with Coulomb on)
//   xref yref zref                         double[capacity]: positions at the last build (displacement check, list export)
//   cell_start                             int32[2 * cells + 1]: first slot of every cell, owned cells then ghost cells
//   quad, rows, row_end, row_int           the Verlet list: one row per pair of neighbouring owned atoms (dsmd_rows.cuh)
//
// No tensor cores: the path is a gather over a sparse geometric neighbourhood, not a dense contraction.

#include <cub/cub.cuh>
#include <thrust/iterator/counting_iterator.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <string>
#include <vector>

#include "../../include/dsmd_b200.h"
#include "dsmd_cells.cuh"
#include "dsmd_common.cuh"
#include "dsmd_force.cuh"
#include "dsmd_launch.cuh"
#include "dsmd_report.cuh"
#include "dsmd_scan.cuh"
#include "dsmd_sums.cuh"
#include "ewald_table.hpp"

using dsmd::ForceArgs;
using dsmd::Grid;
using dsmd::Mail;
using dsmd::PairParams;
using dsmd::Status;
using dsmd::StepArgs;
using dsmd::kEwaldCopiesMost;
using dsmd::kEwaldFirst;
using dsmd::kFewTypes;
using dsmd::kOneType;
using dsmd::kPairBlocks;
using dsmd::kPairThreads;
using dsmd::post;

namespace {

constexpr int kThreads = 256;
constexpr int kDeviceSms = 148;                       // of a B200
// Lanes that keep them busy, below which a row gets twice as many: half of those that an SM holds of the plain force kernel (1,024)
// before rows are shared at all, a third where a row's set-up is paid by several lanes. Steps of 16,000, 32,000, 64,000, 90,000 and
// 130,000 Lennard-Jones atoms: 9.3, 11.3, 15.3, 17.7 and 22.0 us; with 512 throughout 9.6, 12.2, 15.1, 17.7 and 22.0, with 1,024 13.7, 15.7, 21.3,
// 23.7 and 27.6, with 256 9.3, 11.3, 14.8, 22.1 and 27.4. Of 30,000, 60,000 and 90,000 of the mixture: 13.0, 19.0 and 22.2; with 512 16.2, 22.3 and 22.3.
constexpr int64_t pair_lanes_wanted(int shift) { return kDeviceSms * (shift == 0 ? 512 : 352); }
constexpr int64_t kPairLanesWantedEwald = kDeviceSms * 768;   // one and a half rounds of one block of 512 each
// Threads of a launch up to which its last block reports the displacement check; beyond, a launch of its own does, and no block waits
// for its writes to arrive before it takes its ticket (one word for all) and makes room for the next. A step, us, with tickets and
// with the launch:
//   k_step, blocks of 64 (18,000 threads at 2,048 atoms, 26,000 at 2,916, 35,000 at 4,000): 1,372 atoms 7.2 and 7.7, 2,048 7.9 and 7.4,
//   2,916 7.7 and 8.1, 4,000 9.0 and 8.1, 5,324 9.9 and 8.8, 16,384 13.2 and 10.0, 32,000 15.4 and 11.3, 131,072 24.1 and 22.2, 256,000 41.7 and 38.6;
//   k_pack, a thread per atom, blocks of 256 (step with the force kernel): 8,788 12.0 and 12.8, 16,384 14.8 and 15.3, 23,328 19.2 and 19.0,
//   32,000 18.4 and 18.7, 55,296 23.7 and 22.4, 131,072 48.2 and 40.3, 256,000 73.3 and 68.5;
//   k_constrained, a thread per group, blocks of 128 (step of water): 1,728 groups 30.8 and 30.6, 13,824 98.2 and 98.1, 216,000 1,032 and 1,033.
// So the lines cross between 18,000 and 35,000 threads of the first and 23,000 and 55,000 of the second, and the third does not care. In
// blocks they lie further apart, 290 to 550 and 90 to 220: a block of 256 holds more back while it waits.
constexpr int64_t kTicketThreadsMost = 25000;
constexpr int kLongRow = 240;                         // entries (with the row's spare room): about 150 partners per atom
constexpr int64_t kRowsAlways = 4096;                 // cell rows that any system may have: 2 MB of list rows
constexpr int kXRefine = 4;    // x cells per cell width of the y and z axes (tighter row windows in the list build)
// Rows (of positions and of velocities together) up to which an upload goes through pinned memory of the context, so that it returns
// while what is queued in the stream is still at work. 1,000 atoms 25 us (by the runtime 40), 8,000 36 (35), 16,000 47 (46), 32,000 73
// (66); with velocities 1,000 31 (65), 8,000 47 (56), 16,000 72 (83).
constexpr int64_t kStageRows = 32768;
enum { kMailDisplacement = 0, kMailKinetic = 4, kMailScalars = 5, kMailBuild = 6, kMailSlots = 7 };   // report slots
constexpr unsigned kLinkBlocks = 64;      // blocks of kernels that read or write host memory: enough to fill the link
// Host-buffer calls: below kPipelineLeast atoms one pass with kernels that read and write the host's memory (131,072 atoms
// 0.18 ms, slabs 0.25; 262,144 atoms 0.37, slabs 0.36), above it four to eight slabs (1,000,000 atoms 0.86 ms with 4 or 6,
// 0.89 with 8, 1.0 with 12; 4,000,000 atoms 2.79, 2.66, 2.54 and 2.71 ms).
constexpr int kPipelineLeast = 250000, kSlabAtoms = 200000, kSlabs = 8;
constexpr int kNumReal = 11;   // x y z vx vy vz fx fy fz mass charge
constexpr double kCoulomb = 332.0636;

inline unsigned blocks_for(int64_t n, int threads) { return static_cast<unsigned>((n + threads - 1) / threads); }

// ---------------------------------------------------------------------------------------------------------------------
// kernels: binning, sort support, reorder
// ---------------------------------------------------------------------------------------------------------------------

struct RealArrays {
    double* p[kNumReal];
};

// This rank's brick on the axes that are split between ranks (drop != 0: atoms outside it are to be removed).
struct Brick {
    double lo[3], hi[3];
    int split[3];
    int drop;
};

// Cells are numbered [0, ncells) for owned atoms, [ncells, 2 ncells) for ghosts; atoms to be removed (only in a sort without
// ghosts) count as cell ncells, behind every other.
__global__ void k_cell_begin(int cells, int* __restrict__ cell_count, Status* st) {   // st: to be cleared as well, or null
    if (!dsmd::after_previous()) return;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < cells; k += gridDim.x * blockDim.x) cell_count[k] = 0;
    if (st && blockIdx.x == 0 && threadIdx.x == 0) *st = Status{};
}

__global__ void k_cell_keys(Grid g, Brick brick, int first, int n_owned, int n_total, const double* x,
                            const double* y, const double* z, unsigned* __restrict__ key,
                            int* __restrict__ arrival, int* __restrict__ cell_count, Status* st) {
    if (!dsmd::after_previous()) return;
    const int s = first + blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n_total) return;
    const double p[3] = {x[s], y[s], z[s]};
    unsigned bad = 0;
    const unsigned fx = dsmd::to_fixed(p[0], 0, g, bad);
    const unsigned fy = dsmd::to_fixed(p[1], 1, g, bad);
    const unsigned fz = dsmd::to_fixed(p[2], 2, g, bad);
    if (bad) atomicAdd(&st->sort_outside, 1u);
    const unsigned cx = dsmd::cell_of(fx, g.wrap[0], g.nc[0]);
    const unsigned cy = dsmd::cell_of(fy, g.wrap[1], g.nc[1]);
    const unsigned cz = dsmd::cell_of(fz, g.wrap[2], g.nc[2]);
    unsigned c = (cz * g.nc[1] + cy) * g.nc[0] + cx;
    if (s >= n_owned) c += g.ncells;
    if (brick.drop) {   // an atom that left the brick (the same comparisons as the migration's classifier) sorts last
        bool outside = false;
        for (int a = 0; a < 3; ++a)
            if (brick.split[a] && (p[a] < brick.lo[a] || p[a] >= brick.hi[a])) outside = true;
        if (outside) {
            c = static_cast<unsigned>(g.ncells);
            atomicAdd(&st->dropped, 1u);
        }
    }
    key[s] = c;
    arrival[s] = atomicAdd(&cell_count[c], 1);
}

// Gathers every particle array into sorted order, writes the fixed-point layout, the displacement reference and the
// ghost slot map. FORCES: the force arrays too (a loop that evaluates forces next does not need them). unranked: the cell of
// atoms that are about to be removed, any number of them in any order, or a number that no cell has.
template <bool FORCES>
__global__ void k_reorder(Grid g, int first, int n_owned, int n_total, unsigned unranked, const unsigned* key,
                          const int* list, const int* cell_start, RealArrays src, RealArrays dst, const int* type_src,
                          const int* gid_src, int* __restrict__ type_dst, int* __restrict__ gid_dst,
                          int4* __restrict__ pq, float* __restrict__ qf, double* __restrict__ xref,
                          double* __restrict__ yref, double* __restrict__ zref, int* __restrict__ ghost_slot) {
    if (!dsmd::after_previous()) return;
    const int t = first + blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n_total) return;
    const int from = list[t];
    const int s = key[from] == unranked ? t : dsmd::cell_slot(from, key[from], cell_start, list);
    double r[kNumReal];
#pragma unroll
    for (int f = 0; f < kNumReal; ++f)
        if (FORCES || f < DSMD_FX || f > DSMD_FZ) r[f] = src.p[f][from];
    const int ty = type_src[from], id = gid_src[from];   // (reads before the writes: for all the compiler knows it is the same memory)
#pragma unroll
    for (int f = 0; f < kNumReal; ++f)
        if (FORCES || f < DSMD_FX || f > DSMD_FZ) dst.p[f][s] = r[f];
    type_dst[s] = ty;
    gid_dst[s] = id;
    unsigned bad = 0;
    int4 p;
    p.x = static_cast<int>(dsmd::to_fixed(r[0], 0, g, bad));
    p.y = static_cast<int>(dsmd::to_fixed(r[1], 1, g, bad));
    p.z = static_cast<int>(dsmd::to_fixed(r[2], 2, g, bad));
    p.w = ty;
    pq[s] = p;
    qf[s] = static_cast<float>(r[10]);
    xref[s] = r[0];
    yref[s] = r[1];
    zref[s] = r[2];
    if (s >= n_owned) ghost_slot[from - n_owned] = s;
}

// ---------------------------------------------------------------------------------------------------------------------
// kernels: support of the list build
// ---------------------------------------------------------------------------------------------------------------------

// A ghost-only sort gathers the ghosts into the other buffer set; this brings them back, so that the owned atoms
// (already in place) need not be copied across: one thread per ghost, all per-atom arrays.
__global__ void k_copy_back(int first, int count, RealArrays from, RealArrays to, const int* type_from,
                            const int* gid_from, int* __restrict__ type_to, int* __restrict__ gid_to) {
    if (!dsmd::after_previous()) return;
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= count) return;
    const int s = first + t;
#pragma unroll
    for (int f = 0; f < kNumReal; ++f) to.p[f][s] = from.p[f][s];
    type_to[s] = type_from[s];
    gid_to[s] = gid_from[s];
}

__global__ void k_post_displacement(DisplacementReport r) {
    if (!dsmd::after_previous() || dsmd::gate_closed(r.st, r.gate2)) return;
    post_displacement(r);
}

// The end of a list build: its status goes to the host (atoms outside, dropped, need_stride, boundary_pairs), and the status words
// start again at zero, the displacement word with them; or, where the host is going to report an error, keep what it says.
// A build that failed, or has to be done again with longer rows, closes the gate of the launches queued behind it.
__global__ void k_build_done(Status* st, unsigned expect_dropped, unsigned stride, Mail* mail, unsigned long long seq) {
    if (!dsmd::after_previous()) return;
    const double out[4] = {static_cast<double>(st->sort_outside), static_cast<double>(st->dropped), static_cast<double>(st->need_stride),
                           static_cast<double>(st->boundary_pairs)};
    Status next{};
    if (st->sort_outside != 0u || st->dropped != expect_dropped) {
        next = *st;
        next.out_of_domain = next.sort_outside;
        next.max_disp2 = 0ull;
        next.constraint_failed = 0u;
    }
    if (st->sort_outside != 0u || st->dropped != expect_dropped || st->need_stride > stride) next.gate = __longlong_as_double(0x7FF0000000000000ll);
    *st = next;
    post(mail, out, 4, seq);
}

// Where the ghosts of a cell row sit: lo_end = one past the last x cell of the row's lower half that holds a ghost (0:
// none), hi_begin = the first x cell of its upper half that holds one (nc[0]: none). One warp per (y, z) row.
__global__ void k_ghost_row_extent(Grid g, const int* ghost_cell_start, int* __restrict__ lo_end,
                                   int* __restrict__ hi_begin) {
    if (!dsmd::after_previous()) return;
    const int row = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (row >= g.nc[1] * g.nc[2]) return;
    const int* cells = ghost_cell_start + static_cast<size_t>(row) * g.nc[0];
    const int half = g.nc[0] >> 1;
    int lo = 0, hi = g.nc[0];
    for (int c = lane; c < g.nc[0]; c += 32) {
        if (cells[c + 1] > cells[c]) {
            if (c < half) lo = max(lo, c + 1);
            else hi = min(hi, c);
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        lo = max(lo, __shfl_down_sync(0xffffffffu, lo, o));
        hi = min(hi, __shfl_down_sync(0xffffffffu, hi, o));
    }
    if (lane == 0) { lo_end[row] = lo; hi_begin[row] = hi; }
}

// The same over the rows a centre of row (yc, zc) searches (stencil reach in y and z, wrapping where the axis does): an
// owned atom whose x window stays inside [near_lo, near_hi) of its row cannot have a ghost partner and skips the ghost
// pass of the list build altogether.
__global__ void k_ghost_rows_near(Grid g, const int* lo_end, const int* hi_begin,
                                  int* __restrict__ near_lo, int* __restrict__ near_hi) {
    if (!dsmd::after_previous()) return;
    const int row = blockIdx.x * blockDim.x + threadIdx.x;
    if (row >= g.nc[1] * g.nc[2]) return;
    const int yc0 = row % g.nc[1], zc0 = row / g.nc[1];
    int lo = 0, hi = g.nc[0];
    for (int dz = -g.stencil; dz <= g.stencil; ++dz) {
        int zc = zc0 + dz;
        if (g.wrap[2]) zc = (zc + g.nc[2]) % g.nc[2];
        else if (zc < 0 || zc >= g.nc[2]) continue;
        for (int dy = -g.stencil; dy <= g.stencil; ++dy) {
            int yc = yc0 + dy;
            if (g.wrap[1]) yc = (yc + g.nc[1]) % g.nc[1];
            else if (yc < 0 || yc >= g.nc[1]) continue;
            lo = max(lo, lo_end[zc * g.nc[1] + yc]);
            hi = min(hi, hi_begin[zc * g.nc[1] + yc]);
        }
    }
    near_lo[row] = lo;
    near_hi[row] = hi;
}

// ---------------------------------------------------------------------------------------------------------------------
// kernels: per-step pack, displacement, integration
// ---------------------------------------------------------------------------------------------------------------------

// Positions out of pinned host memory into the context, and forces back: a kernel that reads or writes the host's memory moves
// three arrays at once and needs no copy engine: 3 us instead of three copies of 8 us each, 41 GB/s instead of 52.
__global__ void k_pull(int first, int count, const double* __restrict__ hx, const double* __restrict__ hy, const double* __restrict__ hz,
                       double* __restrict__ x, double* __restrict__ y, double* __restrict__ z) {
    for (int s = first + blockIdx.x * blockDim.x + threadIdx.x; s < first + count; s += gridDim.x * blockDim.x) {
        const double px = __ldcs(hx + s), py = __ldcs(hy + s), pz = __ldcs(hz + s);
        x[s] = px; y[s] = py; z[s] = pz;
    }
}

__global__ void k_push(int first, int count, const double* __restrict__ fx, const double* __restrict__ fy, const double* __restrict__ fz,
                       double* __restrict__ hx, double* __restrict__ hy, double* __restrict__ hz) {
    for (int s = first + blockIdx.x * blockDim.x + threadIdx.x; s < first + count; s += gridDim.x * blockDim.x) {
        hx[s] = fx[s]; hy[s] = fy[s]; hz[s] = fz[s];
    }
}

// Atoms that k_constrained takes through the step, by global id; ids the constraints do not reach up to are free.
struct ClusterMembers {
    const unsigned char* member;   // [n_global], or null: no atom
    int n_global;
    const int* gid;
    __device__ __forceinline__ bool has(int s) const {
        if (!member) return false;
        const int g = gid[s];
        return g >= 0 && g < n_global && member[g];
    }
};

__global__ void k_vv2(int n, double half_dt_c, double* __restrict__ vx, double* __restrict__ vy,
                      double* __restrict__ vz, const double* fx, const double* fy,
                      const double* fz, const double* mass, ClusterMembers skip) {
    if (!dsmd::after_previous()) return;
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n || skip.has(s)) return;
    const double a = half_dt_c / mass[s];
    vx[s] += a * fx[s];
    vy[s] += a * fy[s];
    vz[s] += a * fz[s];
}

// What an upload leaves out: zero velocities, forces and charges, unit masses, type 0, ids in order (null: given by the
// caller).
__global__ void k_upload_defaults(int n, RealArrays r, int* type, int* gid) {
    if (!dsmd::after_previous()) return;
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n) return;
#pragma unroll
    for (int f = 0; f < kNumReal; ++f)
        if (r.p[f]) r.p[f][s] = f == DSMD_MASS ? 1.0 : 0.0;
    if (type) type[s] = 0;
    if (gid) gid[s] = s;
}

// [n][3] rows, n words of them in each of three arrays (device memory, or pinned host memory), to three columns.
__global__ void k_split_rows(int n, const double* rows0, const double* rows1, const double* rows2,
                             double* __restrict__ x, double* __restrict__ y, double* __restrict__ z) {
    if (!dsmd::after_previous()) return;
    for (long long k = blockIdx.x * blockDim.x + threadIdx.x; k < 3ll * n; k += gridDim.x * blockDim.x) {
        const int s = static_cast<int>(k / 3), a = static_cast<int>(k - 3ll * s);
        (a == 0 ? x : (a == 1 ? y : z))[s] = k < n ? rows0[k] : (k < 2ll * n ? rows1[k - n] : rows2[k - 2ll * n]);
    }
}

// Thermostat step of the velocity-scaling kind (the reference's nose_hoover_thermostat_kernel,
// src/thermostat_kernels.cu:68-76): v *= factor.
__global__ void k_scale_velocities(int n, double factor, double* __restrict__ vx, double* __restrict__ vy,
                                   double* __restrict__ vz) {
    if (!dsmd::after_previous()) return;
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n) return;
    vx[s] *= factor;
    vy[s] *= factor;
    vz[s] *= factor;
}

__global__ void k_kinetic(int n, const double* vx, const double* vy,
                          const double* vz, const double* mass, double* partials, unsigned* ticket,
                          double* out, Mail* mail, unsigned long long seq) {
    if (!dsmd::after_previous()) return;
    double v[1] = {0.0};
    for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < n; s += gridDim.x * blockDim.x)
        v[0] += 0.5 * mass[s] * (vx[s] * vx[s] + vy[s] * vy[s] + vz[s] * vz[s]);
    sum_over_grid<1>(v, partials, ticket, out, false, mail, seq);
}

}  // namespace

#include "dsmd_constraints.cuh"
#include "dsmd_bonded.cuh"
#include "dsmd_f32x2.cuh"
#include "dsmd_rows.cuh"

namespace {

// INTEGRATE: kick and drift before the pack (v += kick_c f / m, x += dt v): the first velocity-Verlet half with
// kick_c = dt/2 (times the force-to-acceleration factor), or, with kick_c = dt, the second half of the previous step and
// the first half of this one in one pass (both use the same forces).
// BONDED: the forces of the bonded terms are not in the force arrays yet; the launches before are the force kernel and the bonded terms
// beside it, which write nothing but forces and have waited for all before them: the atoms' state is read while they end.
template <bool INTEGRATE, bool BONDED>
__global__ void k_pack(Grid g, int first, int count, int n_owned, double* __restrict__ x, double* __restrict__ y,
                       double* __restrict__ z, double* __restrict__ vx, double* __restrict__ vy,
                       double* __restrict__ vz, const double* fx, const double* fy,
                       const double* fz, const double* mass, const int* type,
                       const double* xref, const double* yref,
                       const double* zref, int4* __restrict__ pq, double dt, double kick_c,
                       ClusterMembers skip, BondedForces bonded, DisplacementReport report) {
    if (!BONDED && !dsmd::after_previous()) return;
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    const int s = first + t;
    double d2 = 0.0;
    double state[7] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};   // BONDED: x, y, z, kick_c / mass, vx, vy, vz
    BondedRange range{};
    if (BONDED) {   // while the forces before end
        if (t < count) {
            state[0] = x[s]; state[1] = y[s]; state[2] = z[s];
            state[3] = kick_c / mass[s];
            state[4] = vx[s]; state[5] = vy[s]; state[6] = vz[s];
            range = bonded_range(bonded, s);
        }
        if (!dsmd::after_previous()) return;
    }
    if (dsmd::gate_closed(report.st, report.gate2)) return;
    if (t < count && !skip.has(s)) {
        // (without INTEGRATE nothing is written there: __ldcg keeps the reads from the read-only path)
        double px = BONDED ? state[0] : __ldcg(x + s), py = BONDED ? state[1] : __ldcg(y + s), pz = BONDED ? state[2] : __ldcg(z + s);
        if (INTEGRATE) {
            const double a = BONDED ? state[3] : kick_c / mass[s];
            double f[3] = {0.0, 0.0, 0.0};
            if (BONDED) bonded_force(bonded, range, f);
            const double ux = (BONDED ? state[4] : vx[s]) + a * (fx[s] + f[0]), uy = (BONDED ? state[5] : vy[s]) + a * (fy[s] + f[1]),
                         uz = (BONDED ? state[6] : vz[s]) + a * (fz[s] + f[2]);
            vx[s] = ux; vy[s] = uy; vz[s] = uz;
            px += dt * ux; py += dt * uy; pz += dt * uz;
            x[s] = px; y[s] = py; z[s] = pz;
        }
        unsigned bad = 0;
        int4 p;
        p.x = static_cast<int>(dsmd::to_fixed(px, 0, g, bad));
        p.y = static_cast<int>(dsmd::to_fixed(py, 1, g, bad));
        p.z = static_cast<int>(dsmd::to_fixed(pz, 2, g, bad));
        p.w = type[s];
        pq[s] = p;
        if (bad) atomicAdd(&report.st->out_of_domain, 1u);
        if (s < n_owned) {
            const double ddx = px - xref[s], ddy = py - yref[s], ddz = pz - zref[s];
            d2 = ddx * ddx + ddy * ddy + ddz * ddz;
            // a position that is no number must not vanish in the block maximum (fmax drops NaN): it forces a rebuild,
            // and the rebuild reports the atom
            if (!(d2 == d2)) d2 = __longlong_as_double(0x7FF0000000000000ll);
        }
    }
    report_displacement(d2, report);
}

// ---------------------------------------------------------------------------------------------------------------------
// kernels: ghosts
// ---------------------------------------------------------------------------------------------------------------------

__global__ void k_halo_pack(int count, const int* __restrict__ index, const signed char* __restrict__ image,
                            const double* __restrict__ x, const double* __restrict__ y, const double* __restrict__ z,
                            double bx, double by, double bz, double* __restrict__ out) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= count) return;
    const int s = index[k];
    double sx = 0.0, sy = 0.0, sz = 0.0;
    if (image) {
        sx = image[3 * k] * bx;
        sy = image[3 * k + 1] * by;
        sz = image[3 * k + 2] * bz;
    }
    out[3 * k] = x[s] + sx;
    out[3 * k + 1] = y[s] + sy;
    out[3 * k + 2] = z[s] + sz;
}

__global__ void k_halo_unpack(Grid g, int first_ghost, int count, const double* __restrict__ in,
                              const int* __restrict__ ghost_slot, double* __restrict__ x, double* __restrict__ y,
                              double* __restrict__ z, const int* __restrict__ type, int4* __restrict__ pq, Status* st) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= count) return;
    const int s = ghost_slot[first_ghost + k];
    const double px = in[3 * k], py = in[3 * k + 1], pz = in[3 * k + 2];
    x[s] = px; y[s] = py; z[s] = pz;
    unsigned bad = 0;
    int4 p;
    p.x = static_cast<int>(dsmd::to_fixed(px, 0, g, bad));
    p.y = static_cast<int>(dsmd::to_fixed(py, 1, g, bad));
    p.z = static_cast<int>(dsmd::to_fixed(pz, 2, g, bad));
    p.w = type[s];
    pq[s] = p;
    if (bad) atomicAdd(&st->out_of_domain, 1u);
}

__global__ void k_halo_flag(int n_owned, const double* __restrict__ x, const double* __restrict__ y,
                            const double* __restrict__ z, double lx, double ly, double lz, double hx, double hy,
                            double hz, unsigned char* __restrict__ flag) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n_owned) return;
    const double px = x[s], py = y[s], pz = z[s];
    flag[s] = (px >= lx && px < hx && py >= ly && py < hy && pz >= lz && pz < hz) ? 1 : 0;
}

__global__ void k_halo_pack_records(int count, const int* __restrict__ index, RealArrays a,
                                    const int* __restrict__ type, const int* __restrict__ gid, double sx, double sy,
                                    double sz, double* __restrict__ real_out, int* __restrict__ int_out) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= count) return;
    const int s = index[k];
    double* o = real_out + 8 * static_cast<size_t>(k);
    o[0] = a.p[0][s] + sx; o[1] = a.p[1][s] + sy; o[2] = a.p[2][s] + sz;
    o[3] = a.p[3][s]; o[4] = a.p[4][s]; o[5] = a.p[5][s];
    o[6] = a.p[9][s]; o[7] = a.p[10][s];
    int_out[2 * k] = type[s];
    int_out[2 * k + 1] = gid[s];
}

__global__ void k_halo_append_records(int count, int first_slot, const double* __restrict__ real_in,
                                      const int* __restrict__ int_in, RealArrays a, int* __restrict__ type,
                                      int* __restrict__ gid) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= count) return;
    const int s = first_slot + k;
    const double* r = real_in + 8 * static_cast<size_t>(k);
    a.p[0][s] = r[0]; a.p[1][s] = r[1]; a.p[2][s] = r[2];
    a.p[3][s] = r[3]; a.p[4][s] = r[4]; a.p[5][s] = r[5];
    a.p[6][s] = 0.0; a.p[7][s] = 0.0; a.p[8][s] = 0.0;
    a.p[9][s] = r[6]; a.p[10][s] = r[7];
    type[s] = int_in[2 * k];
    gid[s] = int_in[2 * k + 1];
}

// Full records as one run of nine doubles per atom: x y z vx vy vz mass charge and the two int32 words (type, gid) in the
// ninth - one message per peer carries every field.
__global__ void k_halo_append_packed(int count, int first_slot, const double* __restrict__ rec, RealArrays a,
                                     int* __restrict__ type, int* __restrict__ gid) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= count) return;
    const int s = first_slot + k;
    const double* r = rec + 9 * static_cast<size_t>(k);
    a.p[0][s] = r[0]; a.p[1][s] = r[1]; a.p[2][s] = r[2];
    a.p[3][s] = r[3]; a.p[4][s] = r[4]; a.p[5][s] = r[5];
    a.p[6][s] = 0.0; a.p[7][s] = 0.0; a.p[8][s] = 0.0;
    a.p[9][s] = r[6]; a.p[10][s] = r[7];
    const long long words = __double_as_longlong(r[8]);
    type[s] = static_cast<int>(words & 0xFFFFFFFFll);
    gid[s] = static_cast<int>(words >> 32);
}

// Dependent-FMA-free throughput probe: 8 independent fp32 FMA chains per thread. The benchmark times it to get the
// fp32 CUDA-core peak of the device it runs on (the denominator of the pair kernel's compute roofline).
__global__ void __launch_bounds__(256) k_fma_probe(int iters, float seed, float* out) {
    float a0 = seed + threadIdx.x, a1 = a0 + 1.f, a2 = a0 + 2.f, a3 = a0 + 3.f, a4 = a0 + 4.f, a5 = a0 + 5.f,
          a6 = a0 + 6.f, a7 = a0 + 7.f;
    const float m = 0.999f, c = 0.001f;
#pragma unroll 4
    for (int k = 0; k < iters; ++k) {
        a0 = a0 * m + c; a1 = a1 * m + c; a2 = a2 * m + c; a3 = a3 * m + c;
        a4 = a4 * m + c; a5 = a5 * m + c; a6 = a6 * m + c; a7 = a7 * m + c;
    }
    const float sum = a0 + a1 + a2 + a3 + a4 + a5 + a6 + a7;
    if (sum == 12345.678f) out[0] = sum;   // never true: keeps the chains alive
}

}  // namespace

// ---------------------------------------------------------------------------------------------------------------------
// the context
// ---------------------------------------------------------------------------------------------------------------------

struct dsmd_ctx {
    int device = 0;
    int64_t capacity = 0;
    int64_t n_owned = 0, n_total = 0;
    std::string error;
    int64_t launches = 0;

    // box
    double box[3] = {0, 0, 0}, lo[3] = {0, 0, 0}, hi[3] = {0, 0, 0}, halo = 0.0;
    int periodic[3] = {1, 1, 1};
    bool box_set = false;
    // parameters
    int ntypes = 0;
    double cutoff = 0.0, skin = 0.0, switch_distance = -1.0;
    bool params_set = false;
    bool coulomb = false;
    double alpha = 0.0;
    int ewald_intervals = 0;
    Grid grid{};
    bool grid_valid = false;

    // device storage
    double* real[2][kNumReal] = {};
    int* type[2] = {};
    int* gid[2] = {};
    int cur = 0;
    int4* pq = nullptr;               // positions as the kernels read them; pq_next: where a fused step writes the next ones
    int4* pq_next = nullptr;
    float* qf = nullptr;
    double* ref[3] = {};
    unsigned* key = nullptr;       // cell of an atom, by the slot it came from
    int* arrival = nullptr;        // its place among the atoms of the cell as they came
    int* list = nullptr;           // the cells' atoms as they came
    int* cell_count = nullptr;
    bool counts_zero = false;      // the counts are zero, as every sort leaves them
    bool sort_words_zero = false;  // the status words that a sort counts in are zero, as every list build leaves them
    int* scan_sums = nullptr;      // [kScanBlocksMost]
    int* ghost_slot = nullptr;
    // the host-buffer force call as a pipeline (dsmd_forces_host): first slot of every z layer of cells as of the last
    // build, two copy streams, one event pair per piece
    unsigned long long* h_layer_start = nullptr;   // pinned, [nc_z + 1]: slot, and in the upper half the build's layer_tag
    unsigned layer_tag = 0;
    int layer_capacity = 0;
    cudaStream_t copy_in = nullptr, copy_out = nullptr;
    cudaEvent_t piece_up[16] = {}, piece_done[16] = {}, pipe_begin = nullptr, pipe_end = nullptr;
    int* boundary_pairs = nullptr;    // pairs with a ghost partner, as the last list build found them
    int64_t n_boundary = 0;
    float* type_charge = nullptr;     // [ntypes] charges by type (dsmd_set_type_charges), or null: per-atom charges
    int* cell_start = nullptr;
    int64_t cell_capacity = 0;
    int* ghost_rows = nullptr;        // [4 * rows]: lo_end, hi_begin per (y, z) row, then the same over the rows searched
    int64_t ghost_rows_capacity = 0;
    // list rows (dsmd_rows.cuh)
    unsigned* quad = nullptr;
    int* row_end = nullptr;
    int* row_int = nullptr;
    unsigned* row_special = nullptr;
    int lane_shift = 0;
    int64_t quad_capacity = 0;
    int64_t n_quads = 0;
    unsigned* rows = nullptr;
    size_t rows_capacity = 0;  // entries
    int stride = 0;
    unsigned long long* member_stats = nullptr;   // 3 words: k_list_members
    void* cub_temp = nullptr;
    size_t cub_temp_bytes = 0;
    float2* lj = nullptr;
    float4* ewald = nullptr;
    int* excl_off = nullptr;
    int* excl_partner = nullptr;
    int64_t excl_n_global = 0;
    double* partials = nullptr;
    int64_t partial_blocks = 0;
    double* scalars = nullptr;      // 6 force scalars + 1 kinetic
    unsigned* tickets = nullptr;    // finished blocks of the sums: forces, kinetic energy, bonded terms, constraints;
                                    // from 4 on: displacement checks in turn
    Mail* mail = nullptr;           // pinned: kMailDisplacement .. + 3 in turn, kMailKinetic, kMailScalars
    double gate2 = HUGE_VAL;        // limit that the launches of the MD loop carry (gate_closed)
    bool captured = false;          // a call was captured into a graph: results are copied, not reported
    bool word_shared = false;       // the caller has the displacement word's address and may write there
    unsigned long long seq = 0;     // launches that reported something so far
    unsigned long long disp_seq = 0, scalars_seq = 0;   // the last displacement check / energy sum whose report still stands (0: none)
    Status* status = nullptr;
    Status* h_status = nullptr;     // pinned
    double* h_scalars = nullptr;    // pinned
    unsigned long long* h_disp[2] = {};   // pinned, lagged displacement read-back
    long long disp_epoch[2] = {-1, -1};   // list build each read-back slot was measured under
    int disp_pending = -1;                // slot queued by the previous lagged query
    long long build_epoch = 0;            // bumped by every list build (new reference positions)
    long long settled_epoch = -1;         // list build, and stream, of the last force launch (list_settled)
    cudaStream_t settled_stream = nullptr;
    cudaEvent_t disp_event[2] = {};
    double* stage = nullptr;              // pinned: rows on their way to the device (kStageRows)
    cudaEvent_t stage_free = nullptr;
    unsigned char* flag = nullptr;
    unsigned long long* offsets64 = nullptr;
    bool list_valid = false;
    // distance constraints (dsmd_constraints.cuh)
    // bonded terms (dsmd_set_bonded)
    struct Bonded {
        int64_t n_global = 0, n_bonds = 0, n_angles = 0, n_torsions = 0, n_specials = 0, n_entries = 0, blocks = 0;
        int *bond_atoms = nullptr, *angle_atoms = nullptr, *torsion_atoms = nullptr, *torsion_n = nullptr, *special_atoms = nullptr;
        double *bond_par = nullptr, *angle_par = nullptr, *torsion_par = nullptr, *special_par = nullptr;
        int* slot_of_gid = nullptr;          // [n_global]
        long long* entries_of = nullptr;     // [n_global + 1]
        int* place = nullptr;                // [n_entries]
        double* contrib = nullptr;           // [3 * n_entries], by global id
        double* partials = nullptr;          // [5 * blocks]
        double* scalars = nullptr;           // device: PE, W, Wxx, Wyy, Wzz
        unsigned* missing = nullptr;         // device: terms with an owned atom and a partner that is not on this rank
        double* h_scalars = nullptr;         // pinned: 5 scalars + the missing count
        int64_t map_epoch = -1;              // list build the gid -> slot map belongs to
        int64_t terms() const { return n_bonds + n_angles + n_torsions + n_specials; }
    } bonded;
    int n_clusters = 0;
    int64_t cons_n_global = 0;
    int* cl_gid = nullptr;
    int* cl_slot = nullptr;           // [n_clusters * kClusterAtoms] as of the last sort
    unsigned char* cl_member = nullptr;   // [cons_n_global] 1: the atom belongs to a cluster
    int64_t cl_atoms = 0;             // that do
    int cl_shape = 0;                 // 0: any, 1: triangles, 2: bonds
    unsigned char* cl_a = nullptr;
    unsigned char* cl_b = nullptr;
    double* cl_d2 = nullptr;
    int* slot_of_gid = nullptr;
    bool slot_map_valid = false;
    double cons_tolerance = 1e-8;
    int cons_max_iterations = 500;
    bool owned_sorted_only = false;   // the owned atoms lie as their last sort left them: a list build sorts the ghosts alone
    int64_t expect_dropped = 0;    // atoms the last owned-only sort was told to remove (checked with the build status)
    int64_t stat_entries = 0, stat_interior = 0;   // worked out when asked for (list_members)
    int stat_rechecked = 0;
    long long stat_epoch = -1;     // list build they belong to
};

namespace {

#define DSMD_CUDA(ctx, call)                                                                       \
    do {                                                                                           \
        cudaError_t err_ = (call);                                                                 \
        if (err_ != cudaSuccess) {                                                                 \
            (ctx)->error = std::string(#call) + ": " + cudaGetErrorString(err_);                   \
            return DSMD_ERR_CUDA;                                                                  \
        }                                                                                          \
    } while (0)

#define DSMD_LAUNCHED(ctx)                                                                         \
    do {                                                                                           \
        ++(ctx)->launches;                                                                         \
        cudaError_t err_ = cudaGetLastError();                                                     \
        if (err_ != cudaSuccess) {                                                                 \
            (ctx)->error = std::string("kernel launch: ") + cudaGetErrorString(err_);              \
            return DSMD_ERR_CUDA;                                                                  \
        }                                                                                          \
    } while (0)

void free_bonded(dsmd_ctx* c) {
    dsmd_ctx::Bonded& b = c->bonded;
    cudaFree(b.bond_atoms); cudaFree(b.angle_atoms); cudaFree(b.torsion_atoms); cudaFree(b.torsion_n); cudaFree(b.special_atoms);
    cudaFree(b.bond_par); cudaFree(b.angle_par); cudaFree(b.torsion_par); cudaFree(b.special_par);
    cudaFree(b.slot_of_gid); cudaFree(b.entries_of); cudaFree(b.place); cudaFree(b.contrib); cudaFree(b.partials);
    cudaFree(b.scalars); cudaFree(b.missing);
    if (b.h_scalars) cudaFreeHost(b.h_scalars);
    b = dsmd_ctx::Bonded();
}

int fail(dsmd_ctx* ctx, int code, const std::string& what) {
    ctx->error = what;
    return code;
}

RealArrays arrays_of(dsmd_ctx* c, int set) {
    RealArrays a;
    for (int f = 0; f < kNumReal; ++f) a.p[f] = c->real[set][f];
    return a;
}

// Chooses the fixed-point mapping and the cell grid for the current box, cutoff and skin.
int make_grid(dsmd_ctx* c) {
    if (!c->box_set || !c->params_set) return fail(c, DSMD_ERR_STATE, "box and pair parameters must be set first");
    Grid& g = c->grid;
    const double R = c->cutoff + c->skin;
    double max_scale = 0.0;
    bool split[3];
    for (int a = 0; a < 3; ++a) {
        const bool has_sub = c->hi[a] > c->lo[a];
        split[a] = has_sub && (c->hi[a] - c->lo[a]) < c->box[a] - 1e-6;
        g.box[a] = c->box[a];
        if (c->periodic[a] && !split[a]) {
            g.wrap[a] = 1;
            g.org[a] = 0.0;
            g.inv_len[a] = 1.0 / c->box[a];
            g.scale[a] = static_cast<float>(c->box[a] / 4294967296.0);
            max_scale = std::max(max_scale, c->box[a] / 4294967296.0);
        } else {
            const double lo = (has_sub ? c->lo[a] : 0.0) - c->halo;
            const double hi = (has_sub ? c->hi[a] : c->box[a]) + c->halo;
            g.wrap[a] = 0;
            g.org[a] = lo;
            g.inv_len[a] = 1.0 / (hi - lo);
            g.scale[a] = static_cast<float>((hi - lo) / 2147483648.0);
            max_scale = std::max(max_scale, (hi - lo) / 2147483648.0);
        }
    }
    // Cells at least R / stencil wide (a hair more, so that fixed-point rounding cannot push a partner one cell too far).
    int stencil = 2;
    int x_refine = kXRefine;
    if (const char* e = std::getenv("DSMD_XREFINE")) x_refine = std::max(1, std::min(8, std::atoi(e)));
    for (int attempt = 0; attempt < 2; ++attempt) {
        bool ok = true;
        for (int a = 0; a < 3; ++a) {
            const double len = 1.0 / g.inv_len[a];
            const double width = R / stencil * (1.0 + 1e-6);
            int nc = static_cast<int>(std::floor(len / width));
            nc = std::max(1, std::min(nc, 1024));
            if (g.wrap[a] && nc < 2 * stencil + 1) ok = false;
            g.nc[a] = nc;
        }
        if (ok) { g.stencil = stencil; break; }
        if (stencil == 1) {
            return fail(c, DSMD_ERR_BOX_TOO_SMALL,
                        "a periodic axis is shorter than three cells of width cutoff + skin");
        }
        stencil = 1;
    }
    // A cell row costs the list most of a quad's number and storage whether atoms are in it or not (quad_base): no more rows
    // than half the atoms there is room for. Emptier boxes get wider y and z cells.
    const int64_t rows_most = std::max<int64_t>(kRowsAlways, c->capacity / 2);
    for (bool narrower = true; narrower && static_cast<int64_t>(g.nc[1]) * g.nc[2] > rows_most;) {
        const double share = std::sqrt(static_cast<double>(rows_most) / (static_cast<double>(g.nc[1]) * g.nc[2]));
        narrower = false;
        for (int a = 1; a < 3; ++a) {
            const int fewer = std::max(g.wrap[a] ? 2 * g.stencil + 1 : 1, static_cast<int>(g.nc[a] * share));
            if (fewer >= g.nc[a]) continue;
            g.nc[a] = fewer;
            narrower = true;
        }
    }
    // Rows of cells along x are contiguous runs of slots, searched through a window that is rounded outwards to whole
    // cells: finer x cells (kXRefine per unrefined cell) make the windows tighter at no cost per row.
    g.x_reach = static_cast<float>(g.stencil * (1.0 / (g.inv_len[0] * g.nc[0])) * 0.9999999);
    {
        int refine = x_refine;
        while (refine > 1 && (static_cast<int64_t>(g.nc[0]) * refine > 4096 ||
                              2 * static_cast<int64_t>(g.nc[0]) * refine * g.nc[1] * g.nc[2] + 1 > (1ll << 26)))
            refine >>= 1;
        g.nc[0] *= refine;
    }
    const int64_t ncells = static_cast<int64_t>(g.nc[0]) * g.nc[1] * g.nc[2];
    if (2 * ncells + 1 > (1ll << 30)) return fail(c, DSMD_ERR_INVALID, "cell grid too large");
    g.ncells = static_cast<int>(ncells);
    g.r2_list = static_cast<float>(R * R);
    g.r2_list_d = R * R;
    double max_len = 0.0;
    for (int a = 0; a < 3; ++a) {
        g.cellw[a] = static_cast<float>(1.0 / (g.inv_len[a] * g.nc[a]));
        max_len = std::max(max_len, 1.0 / g.inv_len[a]);
    }
    g.r_pad = static_cast<float>(R * (1.0 + 1e-4) + 8.0 * max_len * 1.2e-7);
    // Rounding band of the list search: coordinates are single-precision differences of up to three list radii (a candidate
    // and an atom of a quad, both relative to the quad's first atom), each good to three roundings of 2^-24; squares and
    // sums add a few more of R^2; the fixed-point grid one unit per coordinate. Everything inside the band is listed.
    g.band_rows = static_cast<float>(5.9604645e-8 * 48.0 * R * R + 8.0 * R * max_scale);
    for (int a = 0; a < 3; ++a) {
        g.cells_per_unit[a] = static_cast<float>(g.nc[a] / (g.wrap[a] ? 4294967296.0 : 2147483648.0));
        g.quad_spread[a] = g.wrap[a] ? std::min(g.r_pad, static_cast<float>(0.49 * g.box[a]) - g.r_pad) : g.r_pad;
    }
    g.cells_per_length = 1.0f / g.cellw[0];
    c->grid_valid = true;
    return DSMD_OK;
}

int ensure_cells(dsmd_ctx* c) {
    const int64_t need = 2ll * c->grid.ncells + 2;
    if (need > c->cell_capacity) {
        cudaFree(c->cell_start);
        cudaFree(c->cell_count);
        c->cell_start = c->cell_count = nullptr;
        DSMD_CUDA(c, cudaMalloc(&c->cell_start, sizeof(int) * need));
        DSMD_CUDA(c, cudaMalloc(&c->cell_count, sizeof(int) * need));
        c->counts_zero = false;
        c->cell_capacity = need;
    }
    return DSMD_OK;
}

int ensure_rows(dsmd_ctx* c, int stride) {
    if (c->n_quads > c->quad_capacity) {
        // with headroom here and below: the owned count of a brick changes by a few atoms at every migration, and a
        // reallocation synchronises the device
        const int64_t grown = c->n_quads + c->n_quads / 8 + 64;
        cudaFree(c->quad); cudaFree(c->row_end); cudaFree(c->row_int); cudaFree(c->row_special); cudaFree(c->boundary_pairs);
        c->quad = nullptr;
        c->row_end = c->row_int = c->boundary_pairs = nullptr;
        c->row_special = nullptr;
        c->quad_capacity = 0;
        DSMD_CUDA(c, cudaMalloc(&c->quad, sizeof(unsigned) * grown));
        DSMD_CUDA(c, cudaMalloc(&c->row_end, sizeof(int) * 2 * grown));
        DSMD_CUDA(c, cudaMalloc(&c->row_int, sizeof(int) * 2 * grown));
        DSMD_CUDA(c, cudaMalloc(&c->row_special, sizeof(unsigned) * 2 * grown));
        DSMD_CUDA(c, cudaMalloc(&c->boundary_pairs, sizeof(int) * 2 * grown));
        c->quad_capacity = grown;
    }
    const size_t slices = static_cast<size_t>((2 * c->n_quads + 31) / 32);
    const size_t need = slices * static_cast<size_t>(stride) * 32;
    if (need > c->rows_capacity) {
        const size_t grown = need + need / 8 + 4096;
        cudaFree(c->rows);
        c->rows = nullptr;
        c->rows_capacity = 0;
        DSMD_CUDA(c, cudaMalloc(&c->rows, sizeof(unsigned) * grown));
        c->rows_capacity = grown;
    }
    return DSMD_OK;
}

int pair_lane_shift(const dsmd_ctx* c);

// Long rows have their entries in another order (dsmd_row_layout.cuh), and with Ewald several copies of the table in the force
// kernel's shared memory.
bool long_rows(const dsmd_ctx* c) { return c->stride >= kLongRow; }
int ewald_copies(const dsmd_ctx* c) { return !c->coulomb ? 0 : (long_rows(c) ? kEwaldCopiesMost : 1); }

// Rows for `row_entries` entries each: lanes per row, stride, storage.
int lay_out_rows(dsmd_ctx* c, int row_entries) {
    const int64_t yz_rows = static_cast<int64_t>(c->grid.nc[1]) * c->grid.nc[2];
    c->n_quads = quad_base(static_cast<int>(c->n_owned), static_cast<int>(yz_rows));
    c->stride = whole_groups<0>(row_entries);
    if (long_rows(c)) c->stride = whole_groups<kLongOrder>(row_entries);
    c->lane_shift = pair_lane_shift(c);
    return ensure_rows(c, c->stride);
}

RowArrays rows_of(const dsmd_ctx* c) { return RowArrays{c->quad, c->rows, c->stride, c->row_end, c->row_int, c->row_special}; }

// Lanes that share a pair's row in the force kernel: one (four if rows are long) where that fills the device, more for small systems, whose time
// is the chain of dependent reads along a row. A function of the system alone, so that a pass over a part of the atoms
// gives the same bits as a pass over all of them.
int pair_lane_shift(const dsmd_ctx* c) {
    const int64_t pairs = std::min(2 * c->n_quads, c->n_owned);   // as many rows at most have atoms
    const auto wanted = [&](int shift) { return ewald_copies(c) == kEwaldCopiesMost ? kPairLanesWantedEwald : pair_lanes_wanted(shift); };
    int shift = long_rows(c) ? kLongOrder : 0;
    while (shift < 5 && (pairs << shift) < wanted(shift) && (8 << shift) <= c->stride) ++shift;
    return shift;
}

// Blocks of the force kernel for that many rows: with Coulomb or energy sums no more than the device holds at a time (they
// take further rows in turn).
int64_t pair_blocks(const dsmd_ctx* c, int64_t pairs, bool energy) {
    const int64_t lanes = pairs << c->lane_shift;
    switch (ewald_copies(c)) {
        case kEwaldCopiesMost: return std::min<int64_t>(blocks_for(lanes, kPairThreads<kEwaldCopiesMost, kOneType>), kDeviceSms);
        case 1: return std::min<int64_t>(blocks_for(lanes, kPairThreads<1, kOneType>), kDeviceSms * kPairBlocks<1, kOneType, false>);
        default: break;
    }
    const int threads = c->ntypes == 1 ? kPairThreads<0, kOneType> : kPairThreads<0, kFewTypes>;
    return energy ? std::min<int64_t>(blocks_for(lanes, threads), kDeviceSms * (512 / threads)) : blocks_for(lanes, threads);
}

int ensure_cub_temp(dsmd_ctx* c, size_t need) {
    if (need > c->cub_temp_bytes) {
        cudaFree(c->cub_temp);
        c->cub_temp = nullptr;
        c->cub_temp_bytes = 0;
        DSMD_CUDA(c, cudaMalloc(&c->cub_temp, need + need / 4));
        c->cub_temp_bytes = need + need / 4;
    }
    return DSMD_OK;
}

int ensure_partials(dsmd_ctx* c, int64_t blocks) {
    if (blocks > c->partial_blocks) {
        if (c->partials) cudaFree(c->partials);
        c->partials = nullptr;
        DSMD_CUDA(c, cudaMalloc(&c->partials, sizeof(double) * 6 * blocks));
        c->partial_blocks = blocks;
    }
    return DSMD_OK;
}

// What a sort does about the status words.
enum class StatusWords {
    kClear,       // all of them to zero, first
    kAreZero,     // those that the sort counts in are zero since the last list build, the others are nobody's concern until the build's end
    kKeep,        // a sort before this one has counted in them
};

// Sorts slots [first, n_total) by cell and gathers everything into the other buffer set. bounds (owned-only sorts): atoms
// outside the brick sort behind every cell and fall off the end. quads: to be worked out as well, or null.
int sort_range(dsmd_ctx* c, int64_t first, cudaStream_t s, StatusWords words, const Brick* bounds = nullptr, bool forces = true,
               const QuadArgs* quads = nullptr) {
    const int64_t n = c->n_total - first;
    const int from = c->cur, to = 1 - c->cur;
    if (words != StatusWords::kKeep) c->disp_seq = 0;   // reports of displacement checks are void
    const bool clear = words == StatusWords::kClear || (words == StatusWords::kAreZero && !c->sort_words_zero);
    c->sort_words_zero = false;
    const unsigned quad_blocks = quads ? blocks_for(static_cast<int64_t>(quads->rows) * 32, kThreads) : 0;
    if (n > 0) {
        Brick brick{};
        if (bounds) { brick = *bounds; brick.drop = 1; }
        const int in = static_cast<int>(c->n_total), i0 = static_cast<int>(first);
        // cells this sort is about: the owned ones, the ghosts', or both; and one behind them
        const int cell0 = first > 0 ? c->grid.ncells : 0, cells = (c->n_total > c->n_owned ? 2 : 1) * c->grid.ncells + 2 - cell0;
        if (!c->counts_zero || clear) {
            const int all = c->counts_zero ? 0 : static_cast<int>(c->cell_capacity);
            dsmd::launch_next(k_cell_begin, std::min<unsigned>(blocks_for(std::max(all, 1), kThreads), kDeviceSms * 8), kThreads, 0, s, all,
                              c->cell_count, clear ? c->status : nullptr);
            DSMD_LAUNCHED(c);
        }
        c->counts_zero = false;
        dsmd::launch_next(k_cell_keys, blocks_for(n, kThreads), kThreads, 0, s, c->grid, brick, i0, static_cast<int>(c->n_owned), in,
                          c->real[from][0], c->real[from][1], c->real[from][2], c->key, c->arrival, c->cell_count, c->status);
        DSMD_LAUNCHED(c);
        if (cells <= dsmd::kScanMost) {
            const int launched = dsmd::launch_cell_scan(cells, i0, c->cell_count + cell0, c->scan_sums, c->cell_start + cell0, s);
            if (launched == 2) ++c->launches;
            DSMD_LAUNCHED(c);
        } else {
            size_t need = 0;
            cub::DeviceScan::ExclusiveScan(nullptr, need, c->cell_count, c->cell_start, cuda::std::plus<int>(), i0, cells, s);
            { const int rc = ensure_cub_temp(c, need); if (rc) return rc; }
            DSMD_CUDA(c, cub::DeviceScan::ExclusiveScan(c->cub_temp, need, c->cell_count + cell0, c->cell_start + cell0,
                                                        cuda::std::plus<int>(), i0, cells, s));
        }
        const unsigned place_blocks = blocks_for(n, kThreads);
        dsmd::launch_next(k_place, place_blocks + quad_blocks, kThreads, 0, s, static_cast<int>(place_blocks), i0, in, c->key, c->arrival, c->cell_start,
                          c->list, cells, c->cell_count + cell0, quads ? *quads : QuadArgs{});
        DSMD_LAUNCHED(c);
        c->counts_zero = true;
        const auto reorder = forces ? k_reorder<true> : k_reorder<false>;
        dsmd::launch_next(reorder, blocks_for(n, kThreads), kThreads, 0, s, c->grid, i0, static_cast<int>(c->n_owned), in,
                          brick.drop ? static_cast<unsigned>(c->grid.ncells) : 0xFFFFFFFFu, c->key, c->list, c->cell_start, arrays_of(c, from),
                          arrays_of(c, to), c->type[from], c->gid[from], c->type[to], c->gid[to], c->pq, c->qf, c->ref[0], c->ref[1], c->ref[2],
                          c->ghost_slot);
        DSMD_LAUNCHED(c);
    } else {
        if (clear) DSMD_CUDA(c, cudaMemsetAsync(c->status, 0, sizeof(Status), s));
        if (quads) {
            dsmd::launch_next(k_place, quad_blocks, kThreads, 0, s, 0, 0, 0, c->key, c->arrival, c->cell_start, c->list, 0, c->cell_count, *quads);
            DSMD_LAUNCHED(c);
        }
    }
    if (first > 0) {
        // a ghost-only sort: the owned atoms are in place in the current set, the sorted ghosts come back to it (far
        // fewer bytes than carrying the owned atoms across, and one launch instead of thirteen copies)
        if (n > 0) {
            dsmd::launch_next(k_copy_back, blocks_for(n, kThreads), kThreads, 0, s, static_cast<int>(first), static_cast<int>(n),
                              arrays_of(c, to), arrays_of(c, from), c->type[to], c->gid[to], c->type[from], c->gid[from]);
            DSMD_LAUNCHED(c);
        }
    } else {
        c->cur = to;
    }
    c->slot_map_valid = false;
    return DSMD_OK;
}

int wait_mail(dsmd_ctx* c, int slot, int n, unsigned long long seq, cudaStream_t s) {
    const cudaError_t e = dsmd::wait_report(c->mail + slot, n, seq, s);
    return e == cudaSuccess ? static_cast<int>(DSMD_OK) : fail(c, DSMD_ERR_CUDA, std::string("waiting for a kernel's report: ") + cudaGetErrorString(e));
}

// Reports carry the number of their launch, which a replayed graph would repeat: a context that was ever captured copies.
bool reports_count(dsmd_ctx* c, cudaStream_t s) {
    cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(s, &status) != cudaSuccess || status != cudaStreamCaptureStatusNone) c->captured = true;
    return !c->captured;
}

// The report of a displacement check about to be launched: of all owned atoms, or none (a part says little, and parts may
// run side by side on several streams; nor where the caller has the word, which is then what counts). Slot and ticket follow from the launch's number: the MD loop has a check unread while
// the next one is under way, and their numbers differ by one (only a list build takes numbers in between, and it voids the check).
DisplacementReport displacement_report(dsmd_ctx* c, bool all_atoms, int64_t threads, cudaStream_t s) {
    c->disp_seq = 0;
    if (!all_atoms || !reports_count(c, s) || c->word_shared) return DisplacementReport{c->status, nullptr, nullptr, 0, c->gate2};
    c->disp_seq = ++c->seq;
    const int slot = static_cast<int>(c->seq & 3);
    return DisplacementReport{c->status, threads > kTicketThreadsMost ? nullptr : c->tickets + 4 + slot, c->mail + kMailDisplacement + slot, c->seq, c->gate2};
}

// Behind the launch that was given `report`.
int displacement_posted(dsmd_ctx* c, const DisplacementReport& report, cudaStream_t s) {
    if (!report.mail || report.ticket) return DSMD_OK;
    dsmd::launch_next(k_post_displacement, 1, 1, 0, s, report);
    DSMD_LAUNCHED(c);
    return DSMD_OK;
}

int read_status(dsmd_ctx* c, cudaStream_t s) {
    DSMD_CUDA(c, cudaMemcpyAsync(c->h_status, c->status, sizeof(Status), cudaMemcpyDeviceToHost, s));
    DSMD_CUDA(c, cudaStreamSynchronize(s));
    return DSMD_OK;
}

}  // namespace

// ---------------------------------------------------------------------------------------------------------------------
// C ABI
// ---------------------------------------------------------------------------------------------------------------------

extern "C" {

int dsmd_create(int device, int64_t capacity, dsmd_ctx** out) {
    if (!out || capacity <= 0 || capacity >= (1ll << 30)) return DSMD_ERR_INVALID;
    int count = 0;
    if (cudaGetDeviceCount(&count) != cudaSuccess || device < 0 || device >= count) return DSMD_ERR_CUDA;
    dsmd_ctx* c = new dsmd_ctx();
    c->device = device;
    c->capacity = capacity;
    *out = c;
    DSMD_CUDA(c, cudaSetDevice(device));
    for (int set = 0; set < 2; ++set) {
        for (int f = 0; f < kNumReal; ++f) {
            DSMD_CUDA(c, cudaMalloc(&c->real[set][f], sizeof(double) * capacity));
            DSMD_CUDA(c, cudaMemset(c->real[set][f], 0, sizeof(double) * capacity));
        }
        DSMD_CUDA(c, cudaMalloc(&c->type[set], sizeof(int) * capacity));
        DSMD_CUDA(c, cudaMalloc(&c->gid[set], sizeof(int) * capacity));
    }
    DSMD_CUDA(c, cudaMalloc(&c->pq, sizeof(int4) * capacity));
    DSMD_CUDA(c, cudaMalloc(&c->pq_next, sizeof(int4) * capacity));
    DSMD_CUDA(c, cudaMalloc(&c->key, sizeof(unsigned) * capacity));
    DSMD_CUDA(c, cudaMalloc(&c->arrival, sizeof(int) * capacity));
    DSMD_CUDA(c, cudaMalloc(&c->list, sizeof(int) * capacity));
    DSMD_CUDA(c, cudaMalloc(&c->scan_sums, sizeof(int) * dsmd::kScanBlocksMost));
    DSMD_CUDA(c, cudaMalloc(&c->qf, sizeof(float) * capacity));
    for (int a = 0; a < 3; ++a) DSMD_CUDA(c, cudaMalloc(&c->ref[a], sizeof(double) * capacity));
    DSMD_CUDA(c, cudaMalloc(&c->ghost_slot, sizeof(int) * capacity));
    DSMD_CUDA(c, cudaMalloc(&c->member_stats, sizeof(unsigned long long) * 3));
    DSMD_CUDA(c, cudaMalloc(&c->flag, capacity));
    DSMD_CUDA(c, cudaMalloc(&c->offsets64, sizeof(unsigned long long) * capacity));
    DSMD_CUDA(c, cudaMalloc(&c->scalars, sizeof(double) * 8));
    DSMD_CUDA(c, cudaMemset(c->scalars, 0, sizeof(double) * 8));
    DSMD_CUDA(c, cudaMalloc(&c->tickets, sizeof(unsigned) * 8));
    DSMD_CUDA(c, cudaMemset(c->tickets, 0, sizeof(unsigned) * 8));
    DSMD_CUDA(c, cudaMallocHost(&c->mail, sizeof(Mail) * kMailSlots));
    std::memset(c->mail, 0, sizeof(Mail) * kMailSlots);
    DSMD_CUDA(c, cudaMalloc(&c->status, sizeof(Status)));
    DSMD_CUDA(c, cudaMemset(c->status, 0, sizeof(Status)));
    DSMD_CUDA(c, cudaMallocHost(&c->h_status, sizeof(Status)));
    DSMD_CUDA(c, cudaMallocHost(&c->h_scalars, sizeof(double) * 8));
    for (int k = 0; k < 2; ++k) {
        DSMD_CUDA(c, cudaMallocHost(&c->h_disp[k], sizeof(unsigned long long)));
        *c->h_disp[k] = 0ull;
        DSMD_CUDA(c, cudaEventCreateWithFlags(&c->disp_event[k], cudaEventDisableTiming));
    }
    return DSMD_OK;
}

void dsmd_destroy(dsmd_ctx* c) {
    if (!c) return;
    cudaSetDevice(c->device);
    for (int set = 0; set < 2; ++set) {
        for (int f = 0; f < kNumReal; ++f) cudaFree(c->real[set][f]);
        cudaFree(c->type[set]); cudaFree(c->gid[set]); 
    }
    cudaFree(c->pq); cudaFree(c->pq_next); cudaFree(c->key); cudaFree(c->arrival); cudaFree(c->list); cudaFree(c->scan_sums); cudaFree(c->cell_count); cudaFree(c->qf); cudaFree(c->type_charge);
    for (int a = 0; a < 3; ++a) cudaFree(c->ref[a]);
    cudaFree(c->ghost_slot); cudaFree(c->cell_start); cudaFree(c->ghost_rows);
    cudaFree(c->rows); cudaFree(c->quad); cudaFree(c->row_end); cudaFree(c->row_int); cudaFree(c->row_special); cudaFree(c->boundary_pairs);
    cudaFree(c->member_stats);
    cudaFree(c->cub_temp); cudaFree(c->lj); cudaFree(c->ewald); cudaFree(c->excl_off); cudaFree(c->excl_partner);
    cudaFree(c->partials); cudaFree(c->scalars); cudaFree(c->tickets); cudaFree(c->status); cudaFree(c->flag); cudaFree(c->offsets64);
    cudaFree(c->cl_gid); cudaFree(c->cl_a); cudaFree(c->cl_b); cudaFree(c->cl_d2); cudaFree(c->slot_of_gid);
    cudaFree(c->cl_slot); cudaFree(c->cl_member);
    free_bonded(c);
    if (c->h_layer_start) cudaFreeHost(c->h_layer_start);
    if (c->copy_in) cudaStreamDestroy(c->copy_in);
    if (c->copy_out) cudaStreamDestroy(c->copy_out);
    for (int k = 0; k < 16; ++k) {
        if (c->piece_up[k]) cudaEventDestroy(c->piece_up[k]);
        if (c->piece_done[k]) cudaEventDestroy(c->piece_done[k]);
    }
    if (c->pipe_begin) cudaEventDestroy(c->pipe_begin);
    if (c->pipe_end) cudaEventDestroy(c->pipe_end);
    cudaFreeHost(c->h_status); cudaFreeHost(c->h_scalars); cudaFreeHost(c->mail);
    for (int k = 0; k < 2; ++k) {
        cudaFreeHost(c->h_disp[k]);
        if (c->disp_event[k]) cudaEventDestroy(c->disp_event[k]);
    }
    if (c->stage) cudaFreeHost(c->stage);
    if (c->stage_free) cudaEventDestroy(c->stage_free);
    delete c;
}

const char* dsmd_last_error(const dsmd_ctx* c) { return c ? c->error.c_str() : "null context"; }

int64_t dsmd_launch_count(const dsmd_ctx* c) { return c ? c->launches : 0; }

int dsmd_set_box(dsmd_ctx* c, const double box[3], const int periodic[3], const double lo[3], const double hi[3],
                 double halo) {
    if (!c || !box || !periodic) return DSMD_ERR_INVALID;
    for (int a = 0; a < 3; ++a) {
        if (!(box[a] > 0.0) || !std::isfinite(box[a])) return fail(c, DSMD_ERR_INVALID, "box lengths must be positive");
        c->box[a] = box[a];
        c->periodic[a] = periodic[a] != 0;
        c->lo[a] = lo ? lo[a] : 0.0;
        c->hi[a] = hi ? hi[a] : 0.0;
    }
    c->halo = halo > 0.0 ? halo : 0.0;
    c->box_set = true;
    c->grid_valid = false;
    c->list_valid = false;
    c->disp_seq = 0;
    return DSMD_OK;
}

int dsmd_set_pair_params(dsmd_ctx* c, int ntypes, const double* eps, const double* sig, double cutoff, double skin,
                         double switch_distance) {
    if (!c || ntypes <= 0 || ntypes > 64 || !eps || !sig) return DSMD_ERR_INVALID;
    if (!(cutoff > 0.0) || skin < 0.0) return fail(c, DSMD_ERR_INVALID, "cutoff must be positive, skin non-negative");
    if (switch_distance >= cutoff) return fail(c, DSMD_ERR_INVALID, "switch distance must be below the cutoff");
    DSMD_CUDA(c, cudaSetDevice(c->device));
    std::vector<float2> table(static_cast<size_t>(ntypes) * ntypes);
    for (int k = 0; k < ntypes * ntypes; ++k) {
        const double s2 = sig[k] * sig[k], s6 = s2 * s2 * s2;
        const double c6 = 4.0 * eps[k] * s6;
        table[k] = make_float2(static_cast<float>(12.0 * c6 * s6), static_cast<float>(-6.0 * c6));
    }
    if (c->lj) cudaFree(c->lj);
    c->lj = nullptr;
    DSMD_CUDA(c, cudaMalloc(&c->lj, sizeof(float2) * table.size()));
    DSMD_CUDA(c, cudaMemcpy(c->lj, table.data(), sizeof(float2) * table.size(), cudaMemcpyHostToDevice));
    c->ntypes = ntypes;
    c->cutoff = cutoff;
    c->skin = skin;
    c->switch_distance = switch_distance;
    c->params_set = true;
    c->grid_valid = false;
    c->list_valid = false;
    if (c->coulomb) return dsmd_set_coulomb(c, 1, c->alpha);
    return DSMD_OK;
}

int dsmd_set_coulomb(dsmd_ctx* c, int enabled, double alpha) {
    if (!c) return DSMD_ERR_INVALID;
    c->coulomb = enabled != 0;
    if (!c->coulomb) return DSMD_OK;
    if (!c->params_set) return fail(c, DSMD_ERR_STATE, "set the pair parameters (cutoff) before Coulomb");
    DSMD_CUDA(c, cudaSetDevice(c->device));
    c->alpha = alpha > 0.0 ? alpha : dsmd::ewald_alpha_for(c->cutoff);
    c->ewald_intervals = dsmd::ewald_intervals(c->cutoff * c->cutoff);
    const std::vector<float> coef = dsmd::ewald_build_table(c->alpha, c->ewald_intervals);
    if (c->ewald) cudaFree(c->ewald);
    c->ewald = nullptr;
    DSMD_CUDA(c, cudaMalloc(&c->ewald, sizeof(float) * coef.size()));
    DSMD_CUDA(c, cudaMemcpy(c->ewald, coef.data(), sizeof(float) * coef.size(), cudaMemcpyHostToDevice));
    return DSMD_OK;
}

int dsmd_get_ewald_alpha(const dsmd_ctx* c, double* alpha) {
    if (!c || !alpha) return DSMD_ERR_INVALID;
    *alpha = c->alpha;
    return DSMD_OK;
}

int dsmd_set_exclusions(dsmd_ctx* c, int64_t n_global, int64_t n_pairs, const int32_t* a, const int32_t* b) {
    if (!c || n_global < 0 || n_pairs < 0 || (n_pairs > 0 && (!a || !b))) return DSMD_ERR_INVALID;
    DSMD_CUDA(c, cudaSetDevice(c->device));
    if (c->excl_off) cudaFree(c->excl_off);
    if (c->excl_partner) cudaFree(c->excl_partner);
    c->excl_off = c->excl_partner = nullptr;
    c->excl_n_global = 0;
    c->list_valid = false;
    if (n_pairs == 0) return DSMD_OK;
    std::vector<std::pair<int, int>> directed;
    directed.reserve(2 * n_pairs);
    for (int64_t k = 0; k < n_pairs; ++k) {
        if (a[k] < 0 || b[k] < 0 || a[k] >= n_global || b[k] >= n_global || a[k] == b[k])
            return fail(c, DSMD_ERR_INVALID, "exclusion pair out of range");
        directed.emplace_back(a[k], b[k]);
        directed.emplace_back(b[k], a[k]);
    }
    std::sort(directed.begin(), directed.end());
    directed.erase(std::unique(directed.begin(), directed.end()), directed.end());
    std::vector<int> off(n_global + 1, 0), partner(directed.size());
    for (const auto& d : directed) ++off[d.first + 1];
    for (int64_t g = 0; g < n_global; ++g) off[g + 1] += off[g];
    for (size_t k = 0; k < directed.size(); ++k) partner[k] = directed[k].second;
    DSMD_CUDA(c, cudaMalloc(&c->excl_off, sizeof(int) * off.size()));
    DSMD_CUDA(c, cudaMalloc(&c->excl_partner, sizeof(int) * std::max<size_t>(partner.size(), 1)));
    DSMD_CUDA(c, cudaMemcpy(c->excl_off, off.data(), sizeof(int) * off.size(), cudaMemcpyHostToDevice));
    DSMD_CUDA(c, cudaMemcpy(c->excl_partner, partner.data(), sizeof(int) * partner.size(), cudaMemcpyHostToDevice));
    c->excl_n_global = n_global;
    return DSMD_OK;
}

// The fields an upload gives (or not) besides positions.
static int upload_rest(dsmd_ctx* c, int64_t n_owned, int64_t n_total, const double* const (&src)[kNumReal], bool rows_v, const int32_t* type,
                       const int32_t* gid, cudaStream_t s) {
    RealArrays missing{};
    for (int f = DSMD_VX; f < kNumReal; ++f) {
        if (src[f]) DSMD_CUDA(c, cudaMemcpyAsync(c->real[c->cur][f], src[f], sizeof(double) * n_total, cudaMemcpyHostToDevice, s));
        else if (!(rows_v && f <= DSMD_VZ)) missing.p[f] = c->real[c->cur][f];
    }
    if (type) DSMD_CUDA(c, cudaMemcpyAsync(c->type[c->cur], type, sizeof(int) * n_total, cudaMemcpyHostToDevice, s));
    if (gid) DSMD_CUDA(c, cudaMemcpyAsync(c->gid[c->cur], gid, sizeof(int) * n_total, cudaMemcpyHostToDevice, s));
    if (n_total > 0) {
        dsmd::launch_next(k_upload_defaults, blocks_for(n_total, kThreads), kThreads, 0, s, static_cast<int>(n_total), missing, type ? nullptr : c->type[c->cur],
                                                                            gid ? nullptr : c->gid[c->cur]);
        DSMD_LAUNCHED(c);
    }
    c->n_owned = n_owned;
    c->n_total = n_total;
    c->list_valid = false;
    c->slot_map_valid = false;
    c->owned_sorted_only = false;
    return DSMD_OK;
}

int dsmd_upload(dsmd_ctx* c, int64_t n_owned, int64_t n_total, const double* x, const double* y, const double* z,
                const double* vx, const double* vy, const double* vz, const double* mass, const double* charge,
                const int32_t* type, const int32_t* gid, void* stream) {
    if (!c || n_owned < 0 || n_total < n_owned || !x || !y || !z) return DSMD_ERR_INVALID;
    if (n_total > c->capacity) return fail(c, DSMD_ERR_CAPACITY, "more atoms than the context's capacity");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    DSMD_CUDA(c, cudaSetDevice(c->device));
    const double* const src[kNumReal] = {x, y, z, vx, vy, vz, nullptr, nullptr, nullptr, mass, charge};
    for (int f = 0; f < 3; ++f)
        DSMD_CUDA(c, cudaMemcpyAsync(c->real[c->cur][f], src[f], sizeof(double) * n_total, cudaMemcpyHostToDevice, s));
    return upload_rest(c, n_owned, n_total, src, false, type, gid, s);
}

static int split_rows(dsmd_ctx* c, const double* rows0, const double* rows1, const double* rows2, int64_t n, double* const* to, cudaStream_t s) {
    dsmd::launch_next(k_split_rows, std::min<unsigned>(blocks_for(3 * n, kThreads), kDeviceSms * 8), kThreads, 0, s, static_cast<int>(n), rows0, rows1,
                      rows2, to[0], to[1], to[2]);
    DSMD_LAUNCHED(c);
    return DSMD_OK;
}

// Rows of any memory into pinned memory of the context, kStageRows at a time, from where a kernel takes them in its turn. used: rows
// of it that kernels of this call have been given.
static int stage_rows(dsmd_ctx* c, const double* rows, int64_t n, double* const* to, int64_t& used, cudaStream_t s) {
    const int64_t most = std::min(kStageRows, 2 * c->capacity);
    if (!c->stage) {
        DSMD_CUDA(c, cudaEventCreateWithFlags(&c->stage_free, cudaEventDisableTiming));
        DSMD_CUDA(c, cudaMallocHost(&c->stage, sizeof(double) * 3 * most));
    }
    for (int64_t first = 0; first < n;) {
        if (used == 0 || used == most) {   // the rows of another call, or of this one's beginning, are still there
            DSMD_CUDA(c, cudaEventSynchronize(c->stage_free));
            used = 0;
        }
        const int64_t m = std::min(most - used, n - first);
        double* const at = c->stage + 3 * used;
        std::memcpy(at, rows + 3 * first, sizeof(double) * 3 * m);
        double* const columns[3] = {to[0] + first, to[1] + first, to[2] + first};
        const int rc = split_rows(c, at, at + m, at + 2 * m, m, columns, s);
        DSMD_CUDA(c, cudaEventRecord(c->stage_free, s));
        if (rc) return rc;
        used += m;
        first += m;
    }
    return DSMD_OK;
}

// [n][3] host rows (any memory) to three device arrays. Few rows are staged: the host waits for nothing but the upload before. More are
// copied by the runtime, through three arrays of the same size (from pageable memory 100,000 atoms 0.16 ms,
// 400,000 0.57; staged 0.20 and 0.69), but that waits for what is queued in the stream. The runtime takes a copy by where it starts: out
// of pageable memory it has read all of it when it returns; out of memory that it knows it only queues the copy (queued: the
// caller of the upload is to get the rows back when that is over), and refuses it if part of it is not known. Those rows are staged.
static int upload_columns(dsmd_ctx* c, const double* rows, int64_t n, double* const* to, double* const* scratch, bool few, int64_t& used, bool& queued,
                          cudaStream_t s) {
    if (few) return stage_rows(c, rows, n, to, used, s);
    for (int k = 0; k < 3; ++k) {
        cudaPointerAttributes memory{};
        if (cudaPointerGetAttributes(&memory, rows + k * n) != cudaSuccess) cudaGetLastError();   // not known to the runtime: pageable
        else if (memory.type != cudaMemoryTypeUnregistered) queued = true;
        const cudaError_t e = cudaMemcpyAsync(scratch[k], rows + k * n, sizeof(double) * n, cudaMemcpyHostToDevice, s);
        if (e == cudaErrorInvalidValue && queued) {
            cudaGetLastError();
            return stage_rows(c, rows, n, to, used, s);
        }
        DSMD_CUDA(c, e);
    }
    return split_rows(c, scratch[0], scratch[1], scratch[2], n, to, s);
}

int dsmd_upload_rows(dsmd_ctx* c, int64_t n_owned, int64_t n_total, const double* pos, const double* vel, const double* mass,
                     const double* charge, const int32_t* type, const int32_t* gid, void* stream) {
    if (!c || n_owned < 0 || n_total < n_owned || !pos) return DSMD_ERR_INVALID;
    if (n_total > c->capacity) return fail(c, DSMD_ERR_CAPACITY, "more atoms than the context's capacity");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    DSMD_CUDA(c, cudaSetDevice(c->device));
    const bool few = n_total * (vel ? 2 : 1) <= kStageRows;
    bool queued = false;
    int64_t used = 0;
    int rc = DSMD_OK;
    if (n_total > 0) rc = upload_columns(c, pos, n_total, c->real[c->cur], c->real[1 - c->cur], few, used, queued, s);
    if (n_total > 0 && !rc && vel)
        rc = upload_columns(c, vel, n_total, c->real[c->cur] + DSMD_VX, c->real[1 - c->cur] + DSMD_VX, few, used, queued, s);
    const double* const src[kNumReal] = {nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, mass, charge};
    if (!rc) rc = upload_rest(c, n_owned, n_total, src, vel != nullptr, type, gid, s);
    if (queued) {
        const cudaError_t e = cudaStreamSynchronize(s);
        if (!rc) DSMD_CUDA(c, e);
    }
    return rc;
}

int dsmd_upload_positions(dsmd_ctx* c, const double* x, const double* y, const double* z, void* stream) {
    if (!c || !x || !y || !z) return DSMD_ERR_INVALID;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const double* src[3] = {x, y, z};
    for (int a = 0; a < 3; ++a)
        DSMD_CUDA(c, cudaMemcpyAsync(c->real[c->cur][a], src[a], sizeof(double) * c->n_total, cudaMemcpyHostToDevice, s));
    c->owned_sorted_only = false;
    return DSMD_OK;
}

int dsmd_download(dsmd_ctx* c, int field, int64_t n, void* host_out, void* stream) {
    if (!c || field < 0 || field >= DSMD_FIELD_COUNT || n < 0 || n > c->capacity || !host_out) return DSMD_ERR_INVALID;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const void* src = field < kNumReal ? static_cast<const void*>(c->real[c->cur][field])
                                       : (field == DSMD_TYPE ? static_cast<const void*>(c->type[c->cur])
                                                             : static_cast<const void*>(c->gid[c->cur]));
    const size_t bytes = (field < kNumReal ? sizeof(double) : sizeof(int)) * static_cast<size_t>(n);
    DSMD_CUDA(c, cudaMemcpyAsync(host_out, src, bytes, cudaMemcpyDeviceToHost, s));
    DSMD_CUDA(c, cudaStreamSynchronize(s));
    return DSMD_OK;
}

int dsmd_device_pointer(dsmd_ctx* c, int field, void** out) {
    if (!c || field < 0 || field >= DSMD_FIELD_COUNT || !out) return DSMD_ERR_INVALID;
    *out = field < kNumReal ? static_cast<void*>(c->real[c->cur][field])
                            : (field == DSMD_TYPE ? static_cast<void*>(c->type[c->cur])
                                                  : static_cast<void*>(c->gid[c->cur]));
    return DSMD_OK;
}

int dsmd_counts(const dsmd_ctx* c, int64_t* n_owned, int64_t* n_total) {
    if (!c) return DSMD_ERR_INVALID;
    if (n_owned) *n_owned = c->n_owned;
    if (n_total) *n_total = c->n_total;
    return DSMD_OK;
}

int dsmd_set_counts(dsmd_ctx* c, int64_t n_owned, int64_t n_total) {
    if (!c || n_owned < 0 || n_total < n_owned) return DSMD_ERR_INVALID;
    if (n_total > c->capacity) return fail(c, DSMD_ERR_CAPACITY, "more atoms than the context's capacity");
    c->n_owned = n_owned;
    c->n_total = n_total;
    c->list_valid = false;
    return DSMD_OK;
}

static int sort_owned_impl(dsmd_ctx* c, const Brick* bounds, int64_t n_outside, bool check_now, cudaStream_t s) {
    DSMD_CUDA(c, cudaSetDevice(c->device));
    if (n_outside < 0 || n_outside >= c->n_owned) return fail(c, DSMD_ERR_INVALID, "sort: bad count of atoms to remove");
    if (!c->grid_valid) { const int rc = make_grid(c); if (rc) return rc; }
    { const int rc = ensure_cells(c); if (rc) return rc; }
    const int64_t keep_total = c->n_total;
    c->n_total = c->n_owned;   // sort the owned segment alone
    const int rc = sort_range(c, 0, s, StatusWords::kClear, n_outside > 0 ? bounds : nullptr);
    c->n_total = keep_total;
    if (rc) return rc;
    c->n_owned -= n_outside;
    c->n_total = c->n_owned;   // ghosts (if any were present) are dropped: the caller appends the new ones
    c->list_valid = false;
    c->owned_sorted_only = true;
    c->expect_dropped = n_outside;
    if (!check_now) return DSMD_OK;   // the status words stay and are read with the list build's
    { const int rc2 = read_status(c, s); if (rc2) return rc2; }
    if (c->h_status->sort_outside)
        return fail(c, DSMD_ERR_OUT_OF_DOMAIN, "an atom lies outside the subdomain + halo, or has a NaN position");
    if (c->h_status->dropped != static_cast<unsigned>(n_outside))
        return fail(c, DSMD_ERR_STATE, "sort: the number of atoms outside the brick differs from the caller's count");
    return DSMD_OK;
}

int dsmd_sort_owned(dsmd_ctx* c, void* stream) {
    if (!c) return DSMD_ERR_INVALID;
    return sort_owned_impl(c, nullptr, 0, true, static_cast<cudaStream_t>(stream));
}

int dsmd_sort_owned_in_brick(dsmd_ctx* c, const double lo[3], const double hi[3], const int split[3], int64_t n_outside,
                             void* stream) {
    if (!c || !lo || !hi || !split) return DSMD_ERR_INVALID;
    Brick bounds{};
    for (int a = 0; a < 3; ++a) {
        bounds.lo[a] = lo[a];
        bounds.hi[a] = hi[a];
        bounds.split[a] = split[a] != 0;
    }
    return sort_owned_impl(c, &bounds, n_outside, false, static_cast<cudaStream_t>(stream));
}

// forces: the force arrays move with the atoms. queue_next (or null): called once everything is launched and before the host waits for the
// build's report; what it launches must do nothing behind a closed gate. If the build has to be done again, or fails, the gate
// was closed, and what it swapped is put back; in the first case it is called again. After an error behind the first launch there
// is no list: the atoms may have been sorted, and rows rewritten.
static int build_list(dsmd_ctx* c, bool forces, cudaStream_t s, const std::function<int()>& queue_next = nullptr) {
    DSMD_CUDA(c, cudaSetDevice(c->device));
    if (c->n_owned <= 0) return fail(c, DSMD_ERR_STATE, "no atoms uploaded");
    if (!c->grid_valid) { const int rc = make_grid(c); if (rc) return rc; }
    { const int rc = ensure_cells(c); if (rc) return rc; }
    // what the list needs room for
    int row_entries = c->stride;
    if (c->stride == 0) {
        double volume = 1.0;
        for (int a = 0; a < 3; ++a) volume *= 1.0 / c->grid.inv_len[a];
        const double R = c->cutoff + c->skin;
        // partners of one atom, and how many more its pair-mate adds (the sphere that the pair's distance, about one atom
        // spacing in a dense system, moves out of the first one)
        const double expect = static_cast<double>(c->n_total) / volume * 4.18879020479 * R * R * R;
        const double apart = std::min(std::cbrt(volume / static_cast<double>(c->n_total)) / R, 1.0);
        row_entries = std::max(32, static_cast<int>(expect * (1.0 + std::min(0.9 * apart, 1.0)) * 1.2) + 32);
    }
    const int64_t rows = static_cast<int64_t>(c->grid.nc[1]) * c->grid.nc[2];
    if (4 * rows > c->ghost_rows_capacity) {
        if (c->ghost_rows) cudaFree(c->ghost_rows);
        c->ghost_rows = nullptr;
        DSMD_CUDA(c, cudaMalloc(&c->ghost_rows, sizeof(int) * 4 * rows));
        c->ghost_rows_capacity = 4 * rows;
    }
    {   // slab boundaries for the pipelined host-buffer call; written with the quads
        const int layers = c->grid.nc[2];
        if (layers + 1 > c->layer_capacity) {
            if (c->h_layer_start) cudaFreeHost(c->h_layer_start);
            c->h_layer_start = nullptr;
            DSMD_CUDA(c, cudaMallocHost(&c->h_layer_start, sizeof(unsigned long long) * (layers + 1)));
            std::memset(c->h_layer_start, 0, sizeof(unsigned long long) * (layers + 1));
            c->layer_capacity = layers + 1;
        }
    }
    c->list_valid = false;
    { const int rc = lay_out_rows(c, row_entries); if (rc) return rc; }
    // 1. bin + sort + reorder (everything, or only the ghosts when the owned segment was sorted just before: the
    //    status words of that sort are then still unread and are kept), and the quads
    const int64_t first = c->owned_sorted_only ? c->n_owned : 0;
    const int64_t expect_dropped = c->owned_sorted_only ? c->expect_dropped : 0;
    const StatusWords words = c->owned_sorted_only ? StatusWords::kKeep : StatusWords::kAreZero;
    c->owned_sorted_only = false;
    c->expect_dropped = 0;
    c->layer_tag = static_cast<unsigned>(++c->seq);
    const QuadArgs quads{c->grid.nc[0], c->grid.nc[1], static_cast<int>(rows), static_cast<int>(c->n_owned), c->quad, c->h_layer_start, c->layer_tag};
    { const int rc = sort_range(c, first, s, words, nullptr, forces, &quads); if (rc) return rc; }
    // 2. list rows
    if (c->n_total > c->n_owned) {
        dsmd::launch_next(k_ghost_row_extent, blocks_for(rows * 32, kThreads), kThreads, 0, s, c->grid, c->cell_start + c->grid.ncells, c->ghost_rows,
                          c->ghost_rows + rows);
        DSMD_LAUNCHED(c);
        dsmd::launch_next(k_ghost_rows_near, blocks_for(rows, kThreads), kThreads, 0, s, c->grid, c->ghost_rows, c->ghost_rows + rows,
                          c->ghost_rows + 2 * rows, c->ghost_rows + 3 * rows);
        DSMD_LAUNCHED(c);
    }
    int4* const places[2] = {c->pq, c->pq_next};
    const auto take_back = [&] {   // what was queued behind the build
        c->list_valid = false;
        c->disp_seq = 0;
        c->pq = places[0];
        c->pq_next = places[1];
    };
    const auto failed = [&](int rc) {
        take_back();
        return rc;
    };
    for (int attempt = 0; attempt < 4; ++attempt) {
        if (attempt > 0) { const int rc = lay_out_rows(c, row_entries); if (rc) return rc; }
        const ExclusionTable ex{c->excl_off, c->excl_partner, static_cast<int>(c->excl_n_global)};
        const unsigned blocks = blocks_for(c->n_quads * 32, kBuildThreads);
        const auto build = ex.offsets ? (long_rows(c) ? k_build_rows<true, kLongOrder> : k_build_rows<true, 0>)
                                      : (long_rows(c) ? k_build_rows<false, kLongOrder> : k_build_rows<false, 0>);
        dsmd::launch_next(build, blocks, kBuildThreads, 0, s, c->grid, static_cast<int>(c->n_owned), static_cast<int>(c->n_total),
                          static_cast<int>(c->n_quads), c->pq, c->gid[c->cur], ex, c->cell_start, c->ghost_rows + 2 * rows, c->ghost_rows + 3 * rows,
                          rows_of(c), c->boundary_pairs, c->status);
        DSMD_LAUNCHED(c);
        const unsigned long long seq = ++c->seq;
        dsmd::launch_next(k_build_done, 1, 1, 0, s, c->status, attempt == 0 ? static_cast<unsigned>(expect_dropped) : 0u, static_cast<unsigned>(c->stride),
                          c->mail + kMailBuild, seq);
        DSMD_LAUNCHED(c);
        c->disp_seq = 0;   // the displacement word starts again at zero
        ++c->build_epoch;
        c->list_valid = true;   // for what is queued behind it
        if (queue_next) { const int rc = queue_next(); if (rc) return failed(rc); }
        { const int rc = wait_mail(c, kMailBuild, 4, seq, s); if (rc) return failed(rc); }
        const Mail& report = c->mail[kMailBuild];
        const bool outside = report.value(0) != 0.0, miscounted = attempt == 0 && report.value(1) != static_cast<double>(expect_dropped);
        const bool overflowed = report.value(2) > c->stride;
        if (outside || miscounted || overflowed) take_back();
        if (outside) return fail(c, DSMD_ERR_OUT_OF_DOMAIN, "an atom lies outside the subdomain + halo, or has a NaN position");
        if (miscounted) return fail(c, DSMD_ERR_STATE, "sort: the number of atoms outside the brick differs from the caller's count");
        c->n_boundary = static_cast<int64_t>(report.value(3));
        c->sort_words_zero = true;
        if (!overflowed) break;
        // a row overflowed: grow and build again
        row_entries = static_cast<int>(report.value(2) * 1.1) + 8;
        if (attempt == 3) return fail(c, DSMD_ERR_CAPACITY, "neighbour rows kept overflowing");
    }
    return DSMD_OK;
}

int dsmd_build_neighbor_list(dsmd_ctx* c, void* stream) {
    return c ? build_list(c, true, static_cast<cudaStream_t>(stream)) : DSMD_ERR_INVALID;
}

int dsmd_ghost_slots(dsmd_ctx* c, const int32_t** out) {
    if (!c || !out) return DSMD_ERR_INVALID;
    *out = c->ghost_slot;
    return DSMD_OK;
}

// The list proper (k_list_members): where each atom's partners start (c->offsets64), sums into the context. Worked out once
// per list build, when somebody asks for it; forces need no membership finer than the rows'.
static unsigned member_blocks(const dsmd_ctx* c) {
    return std::min<unsigned>(blocks_for(2 * c->n_quads * 32, kMemberThreads), kDeviceSms * 8);
}

static int list_members(dsmd_ctx* c, cudaStream_t s) {
    if (c->stat_epoch == c->build_epoch) return DSMD_OK;
    const int n = static_cast<int>(c->n_owned);
    DSMD_CUDA(c, cudaSetDevice(c->device));
    DSMD_CUDA(c, cudaMemsetAsync(c->member_stats, 0, sizeof(unsigned long long) * 3, s));
    const auto count = long_rows(c) ? k_list_members<false, kLongOrder> : k_list_members<false, 0>;
    count<<<member_blocks(c), kMemberThreads, 0, s>>>(c->grid, static_cast<int>(2 * c->n_quads), rows_of(c), c->ref[0], c->ref[1],
                                                                   c->ref[2], c->offsets64, c->member_stats, nullptr, nullptr, nullptr);
    DSMD_LAUNCHED(c);
    size_t need = 0;
    cub::DeviceScan::ExclusiveSum(nullptr, need, c->offsets64, c->offsets64, n, s);
    { const int rc = ensure_cub_temp(c, need); if (rc) return rc; }
    DSMD_CUDA(c, cub::DeviceScan::ExclusiveSum(c->cub_temp, need, c->offsets64, c->offsets64, n, s));
    unsigned long long sums[3] = {0, 0, 0};
    DSMD_CUDA(c, cudaMemcpyAsync(sums, c->member_stats, sizeof(sums), cudaMemcpyDeviceToHost, s));
    DSMD_CUDA(c, cudaStreamSynchronize(s));
    c->stat_entries = static_cast<int64_t>(sums[0]);
    c->stat_interior = static_cast<int64_t>(sums[1]);
    c->stat_rechecked = static_cast<int>(sums[2]);
    c->stat_epoch = c->build_epoch;
    return DSMD_OK;
}

int dsmd_list_stats(dsmd_ctx* c, int64_t* directed_entries, int64_t* interior_entries, int32_t* row_stride,
                    int32_t* cells, int32_t* rechecked) {
    if (!c) return DSMD_ERR_INVALID;
    if (!c->list_valid) return fail(c, DSMD_ERR_STATE, "no neighbour list");
    if (directed_entries || interior_entries || rechecked) {
        const int rc = list_members(c, nullptr);
        if (rc) return rc;
    }
    if (directed_entries) *directed_entries = c->stat_entries;
    if (interior_entries) *interior_entries = c->stat_interior;
    if (row_stride) *row_stride = c->stride;
    if (cells) *cells = c->grid.ncells;
    if (rechecked) *rechecked = c->stat_rechecked;
    return DSMD_OK;
}

int dsmd_list_export(dsmd_ctx* c, int32_t* d_i, int32_t* d_j, uint8_t* d_flags, int64_t capacity, int64_t* n_pairs,
                     void* stream) {
    if (!c || !n_pairs) return DSMD_ERR_INVALID;
    if (!c->list_valid) return fail(c, DSMD_ERR_STATE, "no neighbour list");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    { const int rc = list_members(c, s); if (rc) return rc; }
    *n_pairs = c->stat_entries;
    if (!d_i || !d_j || capacity < c->stat_entries) return DSMD_OK;   // size query
    const auto write = long_rows(c) ? k_list_members<true, kLongOrder> : k_list_members<true, 0>;
    write<<<member_blocks(c), kMemberThreads, 0, s>>>(c->grid, static_cast<int>(2 * c->n_quads), rows_of(c), c->ref[0], c->ref[1],
                                                                  c->ref[2], c->offsets64, nullptr, d_i, d_j, d_flags);
    DSMD_LAUNCHED(c);
    DSMD_CUDA(c, cudaStreamSynchronize(s));
    return DSMD_OK;
}

// kick: 0.5 for the first velocity-Verlet half, 1.0 for the merged second-and-first half.
static int pack_impl(dsmd_ctx* c, int64_t first, int64_t count, bool integrate, double dt, double f2a, cudaStream_t s,
                     double kick = 0.5, const ClusterMembers& skip = {}, const BondedForces* bonded = nullptr) {
    if (count <= 0) return DSMD_OK;
    const DisplacementReport report = displacement_report(c, first == 0 && count >= c->n_owned, count, s);
    double** r = c->real[c->cur];
    const auto kernel = !integrate ? k_pack<false, false> : (bonded ? k_pack<true, true> : k_pack<true, false>);
    // (a part of the atoms follows a copy on another stream: nothing to overlap with)
    dsmd::launch_next_if(first == 0 && count >= c->n_owned, kernel, blocks_for(count, kThreads), kThreads, 0, s, c->grid, static_cast<int>(first), static_cast<int>(count), static_cast<int>(c->n_owned), r[0], r[1], r[2], r[3], r[4], r[5],
        r[6], r[7], r[8], r[9], c->type[c->cur], c->ref[0], c->ref[1], c->ref[2], c->pq, dt, kick * dt * f2a, skip,
        bonded ? *bonded : BondedForces{}, report);
    DSMD_LAUNCHED(c);
    return displacement_posted(c, report, s);
}

int dsmd_pack_positions(dsmd_ctx* c, int64_t first, int64_t count, void* stream) {
    if (!c || first < 0 || count < 0 || first + count > c->n_total) return DSMD_ERR_INVALID;
    if (!c->grid_valid) return fail(c, DSMD_ERR_STATE, "no neighbour list built yet");
    return pack_impl(c, first, count, false, 0.0, 0.0, static_cast<cudaStream_t>(stream));
}

int dsmd_max_displacement_sq(dsmd_ctx* c, double* out, void* stream) {
    if (!c || !out) return DSMD_ERR_INVALID;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    bool outside;
    if (c->disp_seq && !c->captured && !c->word_shared) {   // nothing has touched the status since the last displacement check: its report says it all
        DSMD_CUDA(c, cudaStreamSynchronize(s));
        const int slot = kMailDisplacement + static_cast<int>(c->disp_seq & 3);
        { const int rc = wait_mail(c, slot, 2, c->disp_seq, s); if (rc) return rc; }
        *out = c->mail[slot].value(0);
        outside = c->mail[slot].value(1) != 0.0;
    } else {
        { const int rc = read_status(c, s); if (rc) return rc; }
        std::memcpy(out, &c->h_status->max_disp2, sizeof(*out));
        outside = c->h_status->out_of_domain != 0;
    }
    if (outside) return fail(c, DSMD_ERR_OUT_OF_DOMAIN, "an atom left the subdomain + halo, or has a NaN position");
    return DSMD_OK;
}

int dsmd_max_displacement_sq_lagged(dsmd_ctx* c, double* out, void* stream) {
    if (!c || !out) return DSMD_ERR_INVALID;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    *out = -1.0;
    if (c->disp_pending >= 0) {
        const int slot = c->disp_pending;
        DSMD_CUDA(c, cudaEventSynchronize(c->disp_event[slot]));   // queued one call ago: long finished
        if (c->disp_epoch[slot] == c->build_epoch) {   // else it was measured against reference positions that are gone
            double v;
            const unsigned long long bits = *c->h_disp[slot];
            std::memcpy(&v, &bits, sizeof(v));
            *out = v;
        }
    }
    const int next = c->disp_pending == 0 ? 1 : 0;
    DSMD_CUDA(c, cudaMemcpyAsync(c->h_disp[next], &c->status->max_disp2, sizeof(unsigned long long), cudaMemcpyDeviceToHost, s));
    DSMD_CUDA(c, cudaEventRecord(c->disp_event[next], s));
    c->disp_epoch[next] = c->build_epoch;
    c->disp_pending = next;
    return DSMD_OK;
}

// Whether the force launch about to be made in `s` may read the list before the launch before it has ended: a force launch in the same
// stream came between the build and this one, and has itself waited for the build. (Never in a graph, whose edges are its own.)
static bool list_settled(const dsmd_ctx* c, cudaStream_t s) {
    return !c->captured && c->settled_epoch == c->build_epoch && c->settled_stream == s;
}

static void force_launched(dsmd_ctx* c, cudaStream_t s) {
    ++c->launches;
    if (c->captured) return;   // perhaps into a graph only
    c->settled_epoch = c->build_epoch;
    c->settled_stream = s;
}

static PairParams pair_params(const dsmd_ctx* c) {
    PairParams p{};
    for (int a = 0; a < 3; ++a) p.scale[a] = c->grid.scale[a];
    p.rc2 = static_cast<float>(c->cutoff * c->cutoff);
    if (c->switch_distance > 0.0) {
        const double rs2 = c->switch_distance * c->switch_distance, d = c->cutoff * c->cutoff - rs2;
        p.rs2 = static_cast<float>(rs2);
        p.inv_denom = static_cast<float>(1.0 / (d * d * d));
    } else {
        p.rs2 = -1.f;
    }
    p.kq = static_cast<float>(kCoulomb);
    p.alpha = static_cast<float>(c->alpha);
    p.two_alpha_sqrtpi = static_cast<float>(2.0 * c->alpha / std::sqrt(3.14159265358979323846));
    p.ewald_intervals = c->ewald_intervals;
    p.ewald_most = std::nextafter(std::ldexp(kEwaldFirst, c->ewald_intervals >> dsmd::kEwaldBits), 0.0f);
    p.ewald = c->ewald;
    p.ntypes = c->ntypes;
    p.lj = c->lj;
    p.type_charge = c->coulomb ? c->type_charge : nullptr;
    return p;
}

// The pair kernel over the pair rows first .. first + count of a FULL or INTERIOR pass without energy (count < 0: all of
// them, any phase), or over the pairs with a ghost partner (BOUNDARY).
static int compute_forces_impl(dsmd_ctx* c, int phase, int want_energy, int64_t first, int64_t count, void* stream) {
    if (!c || phase < DSMD_PHASE_FULL || phase > DSMD_PHASE_BOUNDARY) return DSMD_ERR_INVALID;
    if (!c->list_valid) return fail(c, DSMD_ERR_STATE, "build the neighbour list before computing forces");
    const bool ranged = count >= 0;
    if (ranged && (phase == DSMD_PHASE_BOUNDARY || want_energy || first < 0 || first + count > 2 * c->n_quads))
        return fail(c, DSMD_ERR_INVALID, "a range of pair rows is for FULL or INTERIOR passes without energy");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const bool sw = c->switch_distance > 0.0;
    const PairParams p = pair_params(c);
    // the boundary pass runs over the pairs the list build found a ghost partner for (none: nothing to launch)
    const int64_t pairs = phase == DSMD_PHASE_BOUNDARY ? c->n_boundary : (ranged ? count : 2 * c->n_quads);
    const bool e = want_energy != 0;
    if (e) { const int rc = ensure_partials(c, std::max<int64_t>(pair_blocks(c, pairs, true), 1)); if (rc) return rc; }
    const bool report = reports_count(c, s) && e;
    double** r = c->real[c->cur];
    const ForceArgs a{c->pq, c->qf, rows_of(c), phase, phase == DSMD_PHASE_BOUNDARY ? c->boundary_pairs : nullptr,
                      static_cast<int>(ranged ? first : 0), static_cast<int>(pairs), c->lane_shift, r[DSMD_FX], r[DSMD_FY], r[DSMD_FZ], c->partials,
                      c->tickets, c->scalars, report ? c->mail + kMailScalars : nullptr, report ? ++c->seq : 0, c->status, c->gate2, list_settled(c, s)};
    if (e && pairs > 0) c->scalars_seq = a.seq;
    if (pairs > 0) {   // else nothing to add to the forces; the energy sums of a boundary pass stay as the interior pass left them
        const unsigned blocks = static_cast<unsigned>(pair_blocks(c, pairs, e));
        const int copies = ewald_copies(c);
        const auto launch = copies == 0 ? (long_rows(c) ? (e ? dsmd::launch_pair<0, true, kLongOrder> : dsmd::launch_pair<0, false, kLongOrder>)
                                                       : (e ? dsmd::launch_pair<0, true, 0> : dsmd::launch_pair<0, false, 0>))
                            : copies == 1 ? (e ? dsmd::launch_pair<1, true, 0> : dsmd::launch_pair<1, false, 0>)
                                          : (e ? dsmd::launch_pair<kEwaldCopiesMost, true, kLongOrder> : dsmd::launch_pair<kEwaldCopiesMost, false, kLongOrder>);
        // (ranges and boundary passes follow work of other streams: nothing to overlap with)
        DSMD_CUDA(c, launch(p, a, sw, blocks, !ranged && phase != DSMD_PHASE_BOUNDARY, s));
        force_launched(c, s);
    }
    return DSMD_OK;
}

// Pair forces and, with them, the second half of this step and the first half of the next in one kernel (plain
// Lennard-Jones systems of one rank). The atoms' forces stay inside the kernel.
static int force_step(dsmd_ctx* c, double dt, double f2a, cudaStream_t s) {
    const PairParams p = pair_params(c);
    const int64_t pairs = 2 * c->n_quads;
    double** r = c->real[c->cur];
    const ForceArgs a{c->pq, c->qf, rows_of(c), DSMD_PHASE_FULL, nullptr, 0, static_cast<int>(pairs), c->lane_shift,
                      nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, 0, c->status, c->gate2, list_settled(c, s)};
    const StepArgs at{r[0], r[1], r[2], r[3], r[4], r[5], r[9], c->ref[0], c->ref[1], c->ref[2], c->pq_next, dt, dt * f2a};
    const unsigned blocks = static_cast<unsigned>(pair_blocks(c, pairs, false));
    const DisplacementReport report = displacement_report(c, true, pairs << c->lane_shift, s);
    const auto launch = long_rows(c) ? dsmd::launch_step<kLongOrder> : dsmd::launch_step<0>;
    DSMD_CUDA(c, launch(p, a, c->grid, at, report, c->switch_distance > 0.0, blocks, s));
    force_launched(c, s);
    std::swap(c->pq, c->pq_next);
    return displacement_posted(c, report, s);
}

int dsmd_compute_forces(dsmd_ctx* c, int phase, int want_energy, void* stream) {
    return compute_forces_impl(c, phase, want_energy, 0, -1, stream);
}

int dsmd_read_scalars(dsmd_ctx* c, double out[6], void* stream) {
    if (!c || !out) return DSMD_ERR_INVALID;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (c->scalars_seq && !c->captured) {
        DSMD_CUDA(c, cudaStreamSynchronize(s));
        { const int rc = wait_mail(c, kMailScalars, 6, c->scalars_seq, s); if (rc) return rc; }
        for (int k = 0; k < 6; ++k) out[k] = c->mail[kMailScalars].value(k);
        return DSMD_OK;
    }
    DSMD_CUDA(c, cudaMemcpyAsync(c->h_scalars, c->scalars, sizeof(double) * 6, cudaMemcpyDeviceToHost, s));
    DSMD_CUDA(c, cudaStreamSynchronize(s));
    for (int k = 0; k < 6; ++k) out[k] = c->h_scalars[k];
    return DSMD_OK;
}

namespace {

ClusterTable cluster_table(const dsmd_ctx* c) {
    ClusterTable t{};
    t.n_clusters = c->n_clusters;
    t.atom_slot = c->cl_slot;
    t.con_a = c->cl_a;
    t.con_b = c->cl_b;
    t.con_d2 = c->cl_d2;
    for (int a = 0; a < 3; ++a) {
        t.box[a] = c->box[a];
        t.periodic[a] = c->periodic[a];
    }
    return t;
}

// Where the clusters' atoms are since the last sort.
int ensure_slot_map(dsmd_ctx* c, cudaStream_t s) {
    if (c->slot_map_valid) return DSMD_OK;
    dsmd::launch_next(k_slot_of_gid, blocks_for(c->n_owned, kThreads), kThreads, 0, s, static_cast<int>(c->n_owned), c->gid[c->cur],
                                                                         static_cast<int>(c->cons_n_global), c->slot_of_gid);
    DSMD_LAUNCHED(c);
    const int n = c->n_clusters * kClusterAtoms;
    dsmd::launch_next(k_cluster_slots, blocks_for(n, kThreads), kThreads, 0, s, n, c->cl_gid, c->slot_of_gid, c->cl_slot);
    DSMD_LAUNCHED(c);
    c->slot_map_valid = true;
    return DSMD_OK;
}

int launch_constrained(dsmd_ctx* c, bool finish, bool start, double half_kick, double dt, double prefactor, double* d_virial3, bool behind_forces,
                       cudaStream_t s) {
    double** r = c->real[c->cur];
    const AtomArrays at{r[0], r[1], r[2], r[3], r[4], r[5], r[6], r[7], r[8], r[9], c->type[c->cur], c->ref[0], c->ref[1], c->ref[2], c->pq};
    const unsigned blocks = blocks_for(c->n_clusters, 128);
    const DisplacementReport report = start ? displacement_report(c, c->cl_atoms == c->n_owned, c->n_clusters, s) : DisplacementReport{c->status, nullptr, nullptr, 0, HUGE_VAL};
    const auto launch = [&](auto shape) {
        const auto kernel = finish && start ? k_constrained<decltype(shape), true, true>
                                            : (finish ? k_constrained<decltype(shape), true, false> : k_constrained<decltype(shape), false, true>);
        dsmd::launch_next(kernel, blocks, 128, 0, s, cluster_table(c), c->grid, at, half_kick, dt, c->cons_tolerance, c->cons_max_iterations, prefactor,
                                      c->partials, c->tickets + 3, d_virial3, report, behind_forces);
    };
    if (c->cl_shape == 1) launch(TriangleCluster());
    else if (c->cl_shape == 2) launch(BondCluster());
    else launch(AnyCluster());
    DSMD_LAUNCHED(c);
    return displacement_posted(c, report, s);
}

// The velocity-Verlet halves of a system with constraints: the second half of a step with RATTLE (finish), the first half
// with SHAKE (start), or both in one pass (a second half and the first half of the next step, the same forces).
// behind_forces: the launch before was the force kernel, in the same stream.
int constrained_halves(dsmd_ctx* c, bool finish, bool start, double dt, double f2a, bool behind_forces, cudaStream_t s) {
    behind_forces = behind_forces && c->slot_map_valid;
    { const int rc = ensure_slot_map(c, s); if (rc) return rc; }
    const double half_kick = 0.5 * dt * f2a;
    const int rc = launch_constrained(c, finish, start, half_kick, dt, 0.0, nullptr, behind_forces, s);
    if (rc || c->cl_atoms == c->n_owned) return rc;
    // the free atoms
    const ClusterMembers members{c->cl_member, static_cast<int>(c->cons_n_global), c->gid[c->cur]};
    if (start) return pack_impl(c, 0, c->n_owned, true, dt, f2a, s, finish ? 1.0 : 0.5, members);
    double** r = c->real[c->cur];
    dsmd::launch_next(k_vv2, blocks_for(c->n_owned, kThreads), kThreads, 0, s, static_cast<int>(c->n_owned), half_kick, r[3], r[4], r[5], r[6], r[7], r[8],
                                                               r[9], members);
    DSMD_LAUNCHED(c);
    return DSMD_OK;
}

int rattle_impl(dsmd_ctx* c, double dt, double f2a, double* d_virial3, cudaStream_t s) {
    { const int rc = ensure_slot_map(c, s); if (rc) return rc; }
    if (d_virial3) { const int rc = ensure_partials(c, blocks_for(c->n_clusters, 128)); if (rc) return rc; }
    return launch_constrained(c, true, false, 0.0, dt, -2.0 / (f2a * dt), d_virial3, false, s);
}

}  // namespace

int dsmd_set_constraints(dsmd_ctx* c, int64_t n_global, int64_t n_constraints, const int32_t* a, const int32_t* b,
                         const double* distance, double tolerance, int max_iterations) {
    if (!c || n_global < 0 || n_constraints < 0 || (n_constraints > 0 && (!a || !b || !distance))) return DSMD_ERR_INVALID;
    DSMD_CUDA(c, cudaSetDevice(c->device));
    cudaFree(c->cl_gid); cudaFree(c->cl_a); cudaFree(c->cl_b); cudaFree(c->cl_d2); cudaFree(c->slot_of_gid);
    cudaFree(c->cl_slot); cudaFree(c->cl_member);
    c->cl_gid = c->slot_of_gid = c->cl_slot = nullptr;
    c->cl_a = c->cl_b = c->cl_member = nullptr;
    c->cl_d2 = nullptr;
    c->n_clusters = 0;
    c->slot_map_valid = false;
    if (tolerance > 0.0) c->cons_tolerance = tolerance;
    if (max_iterations > 0) c->cons_max_iterations = max_iterations;
    if (n_constraints == 0) return DSMD_OK;
    // clusters = connected groups of constraints (union-find over the atoms), in the order of their first constraint;
    // inside a cluster the constraints keep their given order
    std::vector<int> parent(static_cast<size_t>(n_global));
    for (int64_t g = 0; g < n_global; ++g) parent[g] = static_cast<int>(g);
    auto find = [&](int v) {
        while (parent[v] != v) v = parent[v] = parent[parent[v]];
        return v;
    };
    for (int64_t k = 0; k < n_constraints; ++k) {
        if (a[k] < 0 || b[k] < 0 || a[k] >= n_global || b[k] >= n_global || a[k] == b[k] || !(distance[k] > 0.0))
            return fail(c, DSMD_ERR_INVALID, "constraint names an atom outside the system, or its distance is not positive");
        parent[find(a[k])] = find(b[k]);
    }
    std::vector<int> cluster_of(static_cast<size_t>(n_global), -1);
    std::vector<int> gids;
    std::vector<unsigned char> ca, cb;
    std::vector<double> d2;
    std::vector<int> n_atoms, n_cons;
    for (int64_t k = 0; k < n_constraints; ++k) {
        const int root = find(a[k]);
        int cl = cluster_of[root];
        if (cl < 0) {
            cl = cluster_of[root] = static_cast<int>(n_atoms.size());
            n_atoms.push_back(0);
            n_cons.push_back(0);
            gids.resize(gids.size() + kClusterAtoms, -1);
            ca.resize(ca.size() + kClusterCons, 255);
            cb.resize(cb.size() + kClusterCons, 255);
            d2.resize(d2.size() + kClusterCons, 1.0);
        }
        int local[2];
        const int ends[2] = {a[k], b[k]};
        for (int e = 0; e < 2; ++e) {
            local[e] = -1;
            for (int q = 0; q < n_atoms[cl]; ++q)
                if (gids[static_cast<size_t>(cl) * kClusterAtoms + q] == ends[e]) local[e] = q;
            if (local[e] < 0) {
                if (n_atoms[cl] == kClusterAtoms)
                    return fail(c, DSMD_ERR_CAPACITY, "a group of connected constraints has more than 4 atoms");
                local[e] = n_atoms[cl]++;
                gids[static_cast<size_t>(cl) * kClusterAtoms + local[e]] = ends[e];
            }
        }
        if (n_cons[cl] == kClusterCons) return fail(c, DSMD_ERR_CAPACITY, "a group of connected constraints has more than 6 constraints");
        const size_t at = static_cast<size_t>(cl) * kClusterCons + n_cons[cl]++;
        ca[at] = static_cast<unsigned char>(local[0]);
        cb[at] = static_cast<unsigned char>(local[1]);
        d2[at] = distance[k] * distance[k];
    }
    const size_t ncl = n_atoms.size();
    DSMD_CUDA(c, cudaMalloc(&c->cl_gid, sizeof(int) * gids.size()));
    DSMD_CUDA(c, cudaMalloc(&c->cl_a, ca.size()));
    DSMD_CUDA(c, cudaMalloc(&c->cl_b, cb.size()));
    DSMD_CUDA(c, cudaMalloc(&c->cl_d2, sizeof(double) * d2.size()));
    DSMD_CUDA(c, cudaMalloc(&c->slot_of_gid, sizeof(int) * static_cast<size_t>(n_global)));
    DSMD_CUDA(c, cudaMemcpy(c->cl_gid, gids.data(), sizeof(int) * gids.size(), cudaMemcpyHostToDevice));
    DSMD_CUDA(c, cudaMemcpy(c->cl_a, ca.data(), ca.size(), cudaMemcpyHostToDevice));
    DSMD_CUDA(c, cudaMemcpy(c->cl_b, cb.data(), cb.size(), cudaMemcpyHostToDevice));
    DSMD_CUDA(c, cudaMemcpy(c->cl_d2, d2.data(), sizeof(double) * d2.size(), cudaMemcpyHostToDevice));
    DSMD_CUDA(c, cudaMalloc(&c->cl_slot, sizeof(int) * gids.size()));
    std::vector<unsigned char> member(static_cast<size_t>(n_global), 0);
    for (int g : gids)
        if (g >= 0) member[static_cast<size_t>(g)] = 1;
    c->cl_atoms = std::count(member.begin(), member.end(), 1);
    DSMD_CUDA(c, cudaMalloc(&c->cl_member, member.size()));
    DSMD_CUDA(c, cudaMemcpy(c->cl_member, member.data(), member.size(), cudaMemcpyHostToDevice));
    // one shape for all: compiled with the constraint order known
    const auto all_are = [&](auto shape) {
        for (size_t k = 0; k < ncl; ++k) {
            if (n_atoms[k] != shape.atoms || n_cons[k] != shape.constraints) return false;
            for (int j = 0; j < shape.constraints; ++j)
                if (ca[k * kClusterCons + j] != shape.a(j) || cb[k * kClusterCons + j] != shape.b(j)) return false;
        }
        return true;
    };
    c->cl_shape = all_are(TriangleCluster()) ? 1 : (all_are(BondCluster()) ? 2 : 0);
    c->n_clusters = static_cast<int>(ncl);
    c->cons_n_global = n_global;
    return DSMD_OK;
}

int dsmd_constraint_failures(dsmd_ctx* c, int64_t* failed, void* stream) {
    if (!c || !failed) return DSMD_ERR_INVALID;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    { const int rc = read_status(c, s); if (rc) return rc; }
    *failed = c->h_status->constraint_failed;
    return DSMD_OK;
}

int dsmd_rattle(dsmd_ctx* c, double dt, double f2a, double* d_virial_diag, void* stream) {
    if (!c || !(dt > 0.0)) return DSMD_ERR_INVALID;
    if (c->n_clusters == 0) return DSMD_OK;
    if (c->n_total != c->n_owned) return fail(c, DSMD_ERR_STATE, "constraints are solved on single-rank systems only");
    return rattle_impl(c, dt, f2a, d_virial_diag, static_cast<cudaStream_t>(stream));
}

int dsmd_integrate(dsmd_ctx* c, int half, double dt, double f2a, void* stream) {
    if (!c || half < 1 || half > 3) return DSMD_ERR_INVALID;
    if (!c->grid_valid) return fail(c, DSMD_ERR_STATE, "no neighbour list built yet");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const bool constrained = c->n_clusters > 0;
    if (constrained && c->n_total != c->n_owned)
        return fail(c, DSMD_ERR_STATE, "constraints are solved on single-rank systems only");
    if (half == 3) {
        if (constrained) return fail(c, DSMD_ERR_STATE, "the merged half steps are not available with constraints");
        return pack_impl(c, 0, c->n_owned, true, dt, f2a, s, 1.0);
    }
    if (constrained) return constrained_halves(c, half == 2, half == 1, dt, f2a, false, s);
    if (half == 1) return pack_impl(c, 0, c->n_owned, true, dt, f2a, s);
    double** r = c->real[c->cur];
    dsmd::launch_next(k_vv2, blocks_for(c->n_owned, kThreads), kThreads, 0, s, static_cast<int>(c->n_owned), 0.5 * dt * f2a, r[3], r[4],
                                                               r[5], r[6], r[7], r[8], r[9], ClusterMembers{});
    DSMD_LAUNCHED(c);
    return DSMD_OK;
}

// ---- bonded terms ------------------------------------------------------------------------------------------------------


static int to_device_bytes(dsmd_ctx* c, void** dst, const void* src, size_t bytes) {
    *dst = nullptr;
    if (bytes == 0) return DSMD_OK;
    DSMD_CUDA(c, cudaMalloc(dst, bytes));
    DSMD_CUDA(c, cudaMemcpy(*dst, src, bytes, cudaMemcpyHostToDevice));
    return DSMD_OK;
}
#define DSMD_TO_DEVICE(c, dst, vec)                                                                                    \
    do {                                                                                                               \
        const int rc_ = to_device_bytes(c, reinterpret_cast<void**>(&(dst)), (vec).data(), sizeof((vec)[0]) * (vec).size()); \
        if (rc_) return rc_;                                                                                           \
    } while (0)

int dsmd_set_type_charges(dsmd_ctx* c, int ntypes, const double* charge_of_type) {
    if (!c) return DSMD_ERR_INVALID;
    DSMD_CUDA(c, cudaSetDevice(c->device));
    cudaFree(c->type_charge);
    c->type_charge = nullptr;
    if (!charge_of_type || ntypes <= 0) return DSMD_OK;
    if (!c->params_set || ntypes != c->ntypes)
        return fail(c, DSMD_ERR_INVALID, "dsmd_set_type_charges: the number of types differs from dsmd_set_pair_params'");
    // the atoms already on the device must agree with the table (those that arrive later are the caller's word)
    if (c->n_total > 0) {
        std::vector<double> q(static_cast<size_t>(c->n_total));
        std::vector<int> t(static_cast<size_t>(c->n_total));
        DSMD_CUDA(c, cudaMemcpy(q.data(), c->real[c->cur][10], sizeof(double) * q.size(), cudaMemcpyDeviceToHost));
        DSMD_CUDA(c, cudaMemcpy(t.data(), c->type[c->cur], sizeof(int) * t.size(), cudaMemcpyDeviceToHost));
        for (size_t k = 0; k < q.size(); ++k)
            if (t[k] < 0 || t[k] >= ntypes || q[k] != charge_of_type[t[k]])
                return fail(c, DSMD_ERR_INVALID, "dsmd_set_type_charges: an atom's charge is not the charge given for its type");
    }
    std::vector<float> table(static_cast<size_t>(ntypes));
    for (int k = 0; k < ntypes; ++k) table[static_cast<size_t>(k)] = static_cast<float>(charge_of_type[k]);
    DSMD_CUDA(c, cudaMalloc(&c->type_charge, sizeof(float) * table.size()));
    DSMD_CUDA(c, cudaMemcpy(c->type_charge, table.data(), sizeof(float) * table.size(), cudaMemcpyHostToDevice));
    return DSMD_OK;
}

int dsmd_set_bonded(dsmd_ctx* c, int64_t n_global, int64_t n_bonds, const int32_t* bond_atoms, const double* bond_k,
                    const double* bond_r0, int64_t n_angles, const int32_t* angle_atoms, const double* angle_k,
                    const double* angle_theta0, int64_t n_torsions, const int32_t* torsion_atoms, const double* torsion_k,
                    const double* torsion_phi0, const int32_t* torsion_n, int64_t n_specials, const int32_t* special_atoms,
                    const double* special_sigma, const double* special_epsilon, const double* special_lj_scale,
                    const double* special_coulomb_scale) {
    if (!c || n_global < 0 || n_bonds < 0 || n_angles < 0 || n_torsions < 0 || n_specials < 0) return DSMD_ERR_INVALID;
    if ((n_bonds > 0 && (!bond_atoms || !bond_k || !bond_r0)) || (n_angles > 0 && (!angle_atoms || !angle_k || !angle_theta0)) ||
        (n_torsions > 0 && (!torsion_atoms || !torsion_k || !torsion_phi0 || !torsion_n)) ||
        (n_specials > 0 && (!special_atoms || !special_sigma || !special_epsilon || !special_lj_scale || !special_coulomb_scale)))
        return DSMD_ERR_INVALID;
    DSMD_CUDA(c, cudaSetDevice(c->device));
    free_bonded(c);
    const int64_t terms = n_bonds + n_angles + n_torsions + n_specials;
    if (terms == 0) return DSMD_OK;
    if (n_global >= (1ll << 31) || terms >= (1ll << 29)) return fail(c, DSMD_ERR_INVALID, "too many atoms or bonded terms");
    // term tables, and for every global id the places (3-double groups of the scratch array) its forces are written to,
    // in the order bonds, angles, torsions, specials and, inside a kind, term by term: the order the forces are added in
    std::vector<int> ba(bond_atoms, bond_atoms + 2 * n_bonds), aa(angle_atoms, angle_atoms + 3 * n_angles),
        ta(torsion_atoms, torsion_atoms + 4 * n_torsions), tn(torsion_n, torsion_n + n_torsions),
        sa(special_atoms, special_atoms + 2 * n_specials);
    std::vector<double> bp(2 * n_bonds), ap(2 * n_angles), tp(2 * n_torsions), sp(4 * n_specials);
    for (int64_t k = 0; k < n_bonds; ++k) { bp[2 * k] = bond_k[k]; bp[2 * k + 1] = bond_r0[k]; }
    for (int64_t k = 0; k < n_angles; ++k) { ap[2 * k] = angle_k[k]; ap[2 * k + 1] = angle_theta0[k]; }
    for (int64_t k = 0; k < n_torsions; ++k) { tp[2 * k] = torsion_k[k]; tp[2 * k + 1] = torsion_phi0[k]; }
    for (int64_t k = 0; k < n_specials; ++k) {
        sp[4 * k] = special_sigma[k]; sp[4 * k + 1] = special_epsilon[k];
        sp[4 * k + 2] = special_lj_scale[k]; sp[4 * k + 3] = special_coulomb_scale[k];
    }
    const int64_t n_entries = 2 * n_bonds + 3 * n_angles + 4 * n_torsions + 2 * n_specials;
    std::vector<long long> entries_of(static_cast<size_t>(n_global) + 1, 0);
    const std::vector<int>* tables[4] = {&ba, &aa, &ta, &sa};
    for (const std::vector<int>* t : tables)
        for (int g : *t) {
            if (g < 0 || g >= n_global) return fail(c, DSMD_ERR_INVALID, "a bonded term names an atom id outside [0, n_global)");
            ++entries_of[static_cast<size_t>(g) + 1];
        }
    for (int64_t g = 0; g < n_global; ++g) entries_of[g + 1] += entries_of[g];
    std::vector<int> place(static_cast<size_t>(n_entries));
    {
        std::vector<long long> next(entries_of.begin(), entries_of.end() - 1);
        size_t k = 0;
        for (const std::vector<int>* t : tables)
            for (int g : *t) place[k++] = static_cast<int>(next[g]++);
    }
    dsmd_ctx::Bonded& b = c->bonded;
    DSMD_TO_DEVICE(c, b.bond_atoms, ba);
    DSMD_TO_DEVICE(c, b.angle_atoms, aa);
    DSMD_TO_DEVICE(c, b.torsion_atoms, ta);
    DSMD_TO_DEVICE(c, b.torsion_n, tn);
    DSMD_TO_DEVICE(c, b.special_atoms, sa);
    DSMD_TO_DEVICE(c, b.bond_par, bp);
    DSMD_TO_DEVICE(c, b.angle_par, ap);
    DSMD_TO_DEVICE(c, b.torsion_par, tp);
    DSMD_TO_DEVICE(c, b.special_par, sp);
    DSMD_TO_DEVICE(c, b.entries_of, entries_of);
    DSMD_TO_DEVICE(c, b.place, place);
    b.blocks = blocks_for(terms, kBondedThreads);
    DSMD_CUDA(c, cudaMalloc(&b.slot_of_gid, sizeof(int) * std::max<int64_t>(n_global, 1)));
    DSMD_CUDA(c, cudaMalloc(&b.contrib, sizeof(double) * 3 * n_entries));
    DSMD_CUDA(c, cudaMalloc(&b.partials, sizeof(double) * 5 * b.blocks));
    DSMD_CUDA(c, cudaMalloc(&b.scalars, sizeof(double) * 5));
    DSMD_CUDA(c, cudaMemset(b.scalars, 0, sizeof(double) * 5));
    DSMD_CUDA(c, cudaMalloc(&b.missing, sizeof(unsigned)));
    DSMD_CUDA(c, cudaMemset(b.missing, 0, sizeof(unsigned)));
    DSMD_CUDA(c, cudaMallocHost(&b.h_scalars, sizeof(double) * 6));
    b.n_global = n_global;
    b.n_bonds = n_bonds; b.n_angles = n_angles; b.n_torsions = n_torsions; b.n_specials = n_specials;
    b.n_entries = n_entries;
    b.map_epoch = -1;
    return DSMD_OK;
}

// The terms' contributions into their scratch array. behind_forces: the launch before is the force kernel at the same positions.
static int bonded_terms(dsmd_ctx* c, bool sums, bool behind_forces, cudaStream_t s) {
    dsmd_ctx::Bonded& b = c->bonded;
    if (b.terms() == 0) return DSMD_OK;
    if (!c->list_valid) return fail(c, DSMD_ERR_STATE, "no neighbour list built yet (bonded terms find their atoms through the sorted arrays)");
    if (b.map_epoch != c->build_epoch) {   // the sort of a list build moved the atoms
        DSMD_CUDA(c, cudaMemsetAsync(b.slot_of_gid, 0x7F, sizeof(int) * b.n_global, s));   // 0x7F7F7F7F: beyond any slot
        dsmd::launch_next(k_bonded_slot_map, blocks_for(c->n_total, kThreads), kThreads, 0, s, static_cast<int>(c->n_total), c->gid[c->cur],
                                                                               static_cast<int>(b.n_global), b.slot_of_gid);
        DSMD_LAUNCHED(c);
        b.map_epoch = c->build_epoch;
        behind_forces = false;
    }
    BondedTable t{};
    t.place = b.place;
    t.n_bonds = static_cast<int>(b.n_bonds); t.n_angles = static_cast<int>(b.n_angles);
    t.n_torsions = static_cast<int>(b.n_torsions); t.n_specials = static_cast<int>(b.n_specials);
    t.bond_atoms = b.bond_atoms; t.bond_par = b.bond_par; t.angle_atoms = b.angle_atoms; t.angle_par = b.angle_par;
    t.torsion_atoms = b.torsion_atoms; t.torsion_par = b.torsion_par; t.torsion_n = b.torsion_n;
    t.special_atoms = b.special_atoms; t.special_par = b.special_par;
    t.slot_of_gid = b.slot_of_gid;
    t.n_global = static_cast<int>(b.n_global);
    t.n_owned = static_cast<int>(c->n_owned);
    for (int a = 0; a < 3; ++a) { t.box[a] = c->box[a]; t.periodic[a] = c->periodic[a]; }
    double** r = c->real[c->cur];
    const auto kernel = sums ? k_bonded_terms<true> : k_bonded_terms<false>;
    dsmd::launch_next(kernel, static_cast<unsigned>(b.blocks), kBondedThreads, 0, s, t, r[0], r[1], r[2], r[10], b.contrib, b.partials, c->tickets + 2,
                                                                      b.scalars, b.missing, behind_forces);
    DSMD_LAUNCHED(c);
    return DSMD_OK;
}

static BondedForces bonded_forces(const dsmd_ctx* c) {
    return BondedForces{c->gid[c->cur], static_cast<int>(c->bonded.n_global), c->bonded.entries_of, c->bonded.contrib};
}

int dsmd_compute_bonded(dsmd_ctx* c, void* stream) {
    if (!c) return DSMD_ERR_INVALID;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (c->bonded.terms() == 0) return DSMD_OK;
    { const int rc = bonded_terms(c, true, false, s); if (rc) return rc; }
    double** r = c->real[c->cur];
    dsmd::launch_next(k_bonded_gather, blocks_for(c->n_owned, kThreads), kThreads, 0, s, static_cast<int>(c->n_owned), bonded_forces(c), r[6], r[7], r[8]);
    DSMD_LAUNCHED(c);
    return DSMD_OK;
}

int dsmd_read_bonded_scalars(dsmd_ctx* c, double out[5], void* stream) {
    if (!c || !out) return DSMD_ERR_INVALID;
    dsmd_ctx::Bonded& b = c->bonded;
    for (int k = 0; k < 5; ++k) out[k] = 0.0;
    if (b.terms() == 0) return DSMD_OK;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    unsigned* h_missing = reinterpret_cast<unsigned*>(b.h_scalars + 5);
    DSMD_CUDA(c, cudaMemcpyAsync(b.h_scalars, b.scalars, sizeof(double) * 5, cudaMemcpyDeviceToHost, s));
    DSMD_CUDA(c, cudaMemcpyAsync(h_missing, b.missing, sizeof(unsigned), cudaMemcpyDeviceToHost, s));
    DSMD_CUDA(c, cudaMemsetAsync(b.missing, 0, sizeof(unsigned), s));
    DSMD_CUDA(c, cudaStreamSynchronize(s));
    for (int k = 0; k < 5; ++k) out[k] = b.h_scalars[k];
    if (*h_missing)
        return fail(c, DSMD_ERR_STATE, std::to_string(*h_missing) + " bonded term(s) have an owned atom whose partner is not on "
                                       "this rank: the halo is narrower than the term is long");
    return DSMD_OK;
}

int dsmd_kinetic_energy(dsmd_ctx* c, double* out, void* stream) {
    if (!c || !out) return DSMD_ERR_INVALID;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const int64_t blocks = std::min<int64_t>(blocks_for(c->n_owned, kThreads), kDeviceSms * 8);
    { const int rc = ensure_partials(c, blocks); if (rc) return rc; }
    double** r = c->real[c->cur];
    dsmd::launch_next(k_kinetic, static_cast<unsigned>(blocks), kThreads, 0, s, static_cast<int>(c->n_owned), r[3], r[4], r[5], r[9],
                                                                 c->partials, c->tickets + 1, c->scalars + 6, c->mail + kMailKinetic, ++c->seq);
    DSMD_LAUNCHED(c);
    DSMD_CUDA(c, cudaStreamSynchronize(s));
    { const int rc = wait_mail(c, kMailKinetic, 1, c->seq, s); if (rc) return rc; }
    *out = c->mail[kMailKinetic].value(0);
    return DSMD_OK;
}

int dsmd_scale_velocities(dsmd_ctx* c, double factor, void* stream) {
    if (!c || !std::isfinite(factor)) return DSMD_ERR_INVALID;
    if (c->n_owned == 0) return DSMD_OK;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    double** r = c->real[c->cur];
    dsmd::launch_next(k_scale_velocities, blocks_for(c->n_owned, kThreads), kThreads, 0, s, static_cast<int>(c->n_owned), factor, r[3], r[4],
                                                                             r[5]);
    DSMD_LAUNCHED(c);
    return DSMD_OK;
}

int dsmd_run_nve(dsmd_ctx* c, int64_t n_steps, double dt, double f2a, double hi_frac, int every, int lagged,
                 int64_t* n_rebuilds, double* worst_disp_sq, void* stream) {
    if (!c || n_steps < 0) return DSMD_ERR_INVALID;
    if (c->n_total != c->n_owned) return fail(c, DSMD_ERR_STATE, "dsmd_run_nve handles single-rank systems only");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (!c->list_valid) {
        const int rc = dsmd_build_neighbor_list(c, s);
        if (rc) return rc;
        const int rc2 = dsmd_compute_forces(c, DSMD_PHASE_FULL, 0, s);
        if (rc2) return rc2;
        const int rc3 = dsmd_compute_bonded(c, s);
        if (rc3) return rc3;
    }
    const double limit2 = (hi_frac * c->skin) * (hi_frac * c->skin);
    int64_t rebuilds = 0;
    double worst = 0.0;
    int since_build = 0;
    double d_prev = 0.0, d_prev2 = 0.0;    // displacement (not squared) seen one and two steps ago (lagged mode)
    unsigned long long pending = 0;        // the last displacement check whose report has not been looked at
    // the loop reads the reports of its own launches only, whatever was captured before and whoever has the displacement word
    struct Reporting {
        dsmd_ctx* c;
        bool captured, word_shared;
        ~Reporting() {
            c->captured |= captured;
            c->word_shared = word_shared;
        }
    } reporting{c, c->captured, c->word_shared};
    c->captured = c->word_shared = false;
    const auto reported = [&](unsigned long long seq, double& d2) {
        d2 = 0.0;
        if (!seq) return static_cast<int>(DSMD_OK);   // no atoms, no check
        const int slot = kMailDisplacement + static_cast<int>(seq & 3);
        const int rc = wait_mail(c, slot, 2, seq, s);
        d2 = c->mail[slot].value(0);
        if (!rc && !lagged && c->mail[slot].value(1) != 0.0)
            return fail(c, DSMD_ERR_OUT_OF_DOMAIN, "an atom left the subdomain + halo, or has a NaN position");
        return rc;
    };
    // Between two steps of this loop nobody reads the velocities, so the second half of one step and the first half of the
    // next (the same forces) are one pass over the atoms, with RATTLE between them where there are constraints; and where
    // the pair forces are all the forces there are, that pass is the end of the force kernel (k_step).
    const bool constrained = c->n_clusters > 0, bonded = !constrained && c->bonded.terms() > 0;
    // (Not for a context that was ever captured: the loop of such steps swaps the two buffers of positions that kernels read,
    // and a graph holds the address of one of them.)
    const bool fused = !constrained && !bonded && !c->coulomb && c->n_owned > 0 && !reporting.captured;
    // Forces at the current positions and on to the next ones, up to their displacement check; nothing happens on the device
    // when the check of the current ones went beyond `gate2`.
    const auto advance = [&](double gate2) {
        c->gate2 = gate2;
        int rc = DSMD_OK;
        if (fused) {
            rc = force_step(c, dt, f2a, s);
        } else {
            rc = dsmd_compute_forces(c, DSMD_PHASE_FULL, 0, s);
            if (bonded) {   // the bonded contributions go straight into the pass over the atoms
                if (!rc) rc = bonded_terms(c, false, true, s);
                const BondedForces terms = bonded_forces(c);
                if (!rc) rc = pack_impl(c, 0, c->n_owned, true, dt, f2a, s, 1.0, {}, &terms);
            } else {
                if (!rc) rc = dsmd_compute_bonded(c, s);
                if (!rc) rc = constrained ? constrained_halves(c, true, true, dt, f2a, c->bonded.terms() == 0, s) : dsmd_integrate(c, 3, dt, f2a, s);
            }
        }
        c->gate2 = HUGE_VAL;
        return rc;
    };
    // With constraints and bonded terms at once the forces are added to in place: not a thing to do twice.
    const bool ahead_of_check = !lagged && !(constrained && c->bonded.terms() > 0);
    if (n_steps > 0) { const int rc = dsmd_integrate(c, 1, dt, f2a, s); if (rc) return rc; }
    for (int64_t step = 0; step < n_steps; ++step) {
        const unsigned long long check = c->disp_seq;   // the displacement check of the positions that are current now
        const bool last = step + 1 == n_steps;
        ++since_build;
        bool rebuild = every > 0 && since_build >= every, advanced = false, built_ahead = false;
        if (!lagged) {
            // unless a rebuild is due or this is the end, the next kernels are queued before the host looks at the check
            if (ahead_of_check && !rebuild && !last) {
                const int rc = advance(limit2);
                if (rc) return rc;
                advanced = true;
            }
            double d2 = 0.0;
            const int rc = reported(check, d2);
            if (rc) {
                // an atom outside closed the gate: the kernel queued above left its buffer of positions unwritten, and reports nothing
                if (advanced && limit2 < dsmd::kGateOpen) {
                    if (fused) std::swap(c->pq, c->pq_next);
                    c->disp_seq = 0;
                }
                return rc;
            }
            if (d2 > limit2) rebuild = true;
            if (!rebuild) worst = std::max(worst, d2);
        } else {
            // Look at what the previous step saw (its report came long ago) and decide on the linear extrapolation of the
            // last two values, as the reference does on several ranks (src/md_simulation.cpp:1232-1245). The previous
            // step's forces were evaluated under d_prev.
            if (pending) {
                double d2 = 0.0;
                const int rc = reported(pending, d2);
                if (rc) return rc;
                d_prev2 = d_prev;
                d_prev = std::sqrt(d2);
                worst = std::max(worst, d_prev * d_prev);
            }
            pending = check;
            const double predicted = d_prev + 1.5 * std::max(d_prev - d_prev2, 0.0);
            if (predicted * predicted > limit2) rebuild = true;
        }
        if (rebuild) {
            // Forces are evaluated next, as a rule queued behind the build before the host hears of it.
            const bool queue = ahead_of_check && !last && limit2 < dsmd::kGateOpen;
            const int rc = queue ? build_list(c, false, s, [&] { return advance(limit2); })
                                 : build_list(c, false, s);
            if (rc) return rc;
            built_ahead = queue;
            ++rebuilds;
            since_build = 0;
            d_prev = d_prev2 = 0.0;
            pending = 0;   // that check was made against reference positions that are gone
        }
        if (last) {
            { const int rc = dsmd_compute_forces(c, DSMD_PHASE_FULL, 0, s); if (rc) return rc; }
            { const int rc = dsmd_compute_bonded(c, s); if (rc) return rc; }
            { const int rc = dsmd_integrate(c, 2, dt, f2a, s); if (rc) return rc; }
        } else if (!built_ahead && (!advanced || rebuild)) {
            const int rc = advance(HUGE_VAL);
            if (rc) return rc;
        }
    }
    if (lagged && pending) {
        double d2 = 0.0;
        const int rc = reported(pending, d2);
        if (rc) return rc;
        const double d = std::sqrt(d2);
        worst = std::max(worst, d * d);
    }
    DSMD_CUDA(c, cudaStreamSynchronize(s));
    if (n_rebuilds) *n_rebuilds = rebuilds;
    if (worst_disp_sq) *worst_disp_sq = worst;
    return DSMD_OK;
}

// Device address of `n` doubles of pinned (or registered) host memory, or null.
static double* pinned(const double* p, int64_t n) {
    cudaPointerAttributes lo{}, hi{};
    if (cudaPointerGetAttributes(&lo, p) != cudaSuccess || cudaPointerGetAttributes(&hi, p + n - 1) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    if (lo.type != cudaMemoryTypeHost || hi.type != cudaMemoryTypeHost || !lo.devicePointer || !hi.devicePointer) return nullptr;
    return static_cast<double*>(lo.devicePointer) + (n - 1) == static_cast<double*>(hi.devicePointer) ? static_cast<double*>(lo.devicePointer) : nullptr;
}

// Three host arrays that kernels can read (or write) directly.
struct PinnedArrays {
    double* p[3];
    bool all;
    PinnedArrays(const double* x, const double* y, const double* z, int64_t n) : p{pinned(x, n), pinned(y, n), pinned(z, n)} {
        all = p[0] && p[1] && p[2];
    }
};

static int pull_positions(dsmd_ctx* c, const PinnedArrays& from, int64_t first, int64_t count, cudaStream_t s) {
    double** r = c->real[c->cur];
    k_pull<<<std::min<unsigned>(blocks_for(count, kThreads), kLinkBlocks), kThreads, 0, s>>>(
        static_cast<int>(first), static_cast<int>(count), from.p[0], from.p[1], from.p[2], r[0], r[1], r[2]);
    DSMD_LAUNCHED(c);
    return DSMD_OK;
}

static int push_forces(dsmd_ctx* c, const PinnedArrays& to, int64_t first, int64_t count, cudaStream_t s) {
    double** r = c->real[c->cur];
    k_push<<<std::min<unsigned>(blocks_for(count, kThreads), kLinkBlocks), kThreads, 0, s>>>(
        static_cast<int>(first), static_cast<int>(count), r[DSMD_FX], r[DSMD_FY], r[DSMD_FZ], to.p[0], to.p[1], to.p[2]);
    DSMD_LAUNCHED(c);
    return DSMD_OK;
}

// The pipelined form of the host-buffer call, for a step without rebuild and without energy on a single-rank system:
// the sorted atoms are cut into slabs of z layers of cells; positions go up slab by slab on one copy stream, and behind slab k
// the pair kernel takes the layers whose partners are on the device by then: those of slab k but for its last `stencil` layers,
// and the last of slab k - 1 before them (the box's first and last layers, neighbours through the periodic boundary, come at the
// end). Their forces go down on a second copy stream: the two directions of the host link and the kernels run side by side,
// one slab apart.
// What bounds it: the link, 0.55 ms for 24 MB each way at once (0.46 ms one way), and about 7 us per copy when both directions
// are busy, six copies per slab: few and large slabs (kSlabAtoms).
// Returns DSMD_ERR_STATE when the system does not cut into at least four slabs (the caller falls back).
static int forces_host_pipelined(dsmd_ctx* c, const double* x, const double* y, const double* z, double* fx, double* fy,
                                 double* fz, const PinnedArrays& to, cudaStream_t s) {
    const int layers = c->grid.nc[2], S = c->grid.stencil;
    const int pieces = std::min(std::max(4, std::min(kSlabs, static_cast<int>(c->n_owned / kSlabAtoms))), layers / (2 * S));
    if (pieces < 4 || !c->h_layer_start || c->n_total != c->n_owned) return DSMD_ERR_STATE;
    // the build's own report says nothing about words that an earlier kernel wrote to the host: each one says it for itself
    const volatile unsigned long long* layer_start = c->h_layer_start;
    for (int l = 0; l <= layers; ++l)
        if (static_cast<unsigned>(layer_start[l] >> 32) != c->layer_tag) {
            DSMD_CUDA(c, cudaDeviceSynchronize());
            break;
        }
    if (!c->copy_in) {
        DSMD_CUDA(c, cudaStreamCreateWithFlags(&c->copy_in, cudaStreamNonBlocking));
        DSMD_CUDA(c, cudaStreamCreateWithFlags(&c->copy_out, cudaStreamNonBlocking));
        for (int k = 0; k < 16; ++k) {
            DSMD_CUDA(c, cudaEventCreateWithFlags(&c->piece_up[k], cudaEventDisableTiming));
            DSMD_CUDA(c, cudaEventCreateWithFlags(&c->piece_done[k], cudaEventDisableTiming));
        }
        DSMD_CUDA(c, cudaEventCreateWithFlags(&c->pipe_begin, cudaEventDisableTiming));
        DSMD_CUDA(c, cudaEventCreateWithFlags(&c->pipe_end, cudaEventDisableTiming));
    }
    const auto layer_of = [&](int k) { return static_cast<int>(static_cast<int64_t>(layers) * k / pieces); };
    const auto slot_of = [&](int layer) { return layer == 0 ? 0 : (layer == layers ? c->n_owned : static_cast<int64_t>(layer_start[layer] & 0xFFFFFFFFull)); };
    // everything queued on the caller's stream so far comes first
    DSMD_CUDA(c, cudaEventRecord(c->pipe_begin, s));
    DSMD_CUDA(c, cudaStreamWaitEvent(c->copy_in, c->pipe_begin, 0));
    DSMD_CUDA(c, cudaStreamWaitEvent(c->copy_out, c->pipe_begin, 0));
    const double* src[3] = {x, y, z};
    double* dst[3] = {fx, fy, fz};
    for (int k = 0; k < pieces; ++k) {
        const int64_t first = slot_of(layer_of(k)), count = slot_of(layer_of(k + 1)) - first;
        for (int a = 0; a < 3 && count > 0; ++a)
            DSMD_CUDA(c, cudaMemcpyAsync(c->real[c->cur][a] + first, src[a] + first, sizeof(double) * count,
                                         cudaMemcpyHostToDevice, c->copy_in));
        DSMD_CUDA(c, cudaEventRecord(c->piece_up[k], c->copy_in));
    }
    for (int k = 0; k <= pieces; ++k) {
        if (k < pieces) {
            const int64_t first = slot_of(layer_of(k)), count = slot_of(layer_of(k + 1)) - first;
            DSMD_CUDA(c, cudaStreamWaitEvent(s, c->piece_up[k], 0));
            const int rc = pack_impl(c, first, count, false, 0.0, 0.0, s);
            if (rc) return rc;
        }
        // layers [lo, hi) of this turn; at the end both ends of the box
        const int ranges[2][2] = {{k == 0 ? S : layer_of(k) - S, k < pieces ? layer_of(k + 1) - S : layers}, {0, k < pieces ? 0 : S}};
        for (const int (&range)[2] : ranges) {
            // their pair rows: a cell row's number fixes the first of them
            const int64_t pair_lo = 2ll * quad_base(static_cast<int>(slot_of(range[0])), range[0] * c->grid.nc[1]) * (range[0] > 0 ? 1 : 0);
            const int64_t pair_hi = 2ll * quad_base(static_cast<int>(slot_of(range[1])), range[1] * c->grid.nc[1]);
            if (slot_of(range[1]) == slot_of(range[0])) continue;
            const int rc = compute_forces_impl(c, DSMD_PHASE_FULL, 0, pair_lo, pair_hi - pair_lo, s);
            if (rc) return rc;
        }
        DSMD_CUDA(c, cudaEventRecord(c->piece_done[k], s));
        DSMD_CUDA(c, cudaStreamWaitEvent(c->copy_out, c->piece_done[k], 0));
        for (const int (&range)[2] : ranges) {
            const int64_t first = slot_of(range[0]), count = slot_of(range[1]) - first;
            if (count == 0) continue;
            if (k == pieces && to.all) {   // two small pieces
                const int rc = push_forces(c, to, first, count, c->copy_out);
                if (rc) return rc;
                continue;
            }
            for (int a = 0; a < 3; ++a)
                DSMD_CUDA(c, cudaMemcpyAsync(dst[a] + first, c->real[c->cur][DSMD_FX + a] + first, sizeof(double) * count,
                                             cudaMemcpyDeviceToHost, c->copy_out));
        }
    }
    DSMD_CUDA(c, cudaEventRecord(c->pipe_end, c->copy_out));
    DSMD_CUDA(c, cudaStreamWaitEvent(s, c->pipe_end, 0));
    DSMD_CUDA(c, cudaStreamSynchronize(s));
    return DSMD_OK;
}

int dsmd_forces_host(dsmd_ctx* c, const double* x, const double* y, const double* z, int rebuild, double* fx,
                     double* fy, double* fz, double* out6, void* stream) {
    if (!c || !x || !y || !z || !fx || !fy || !fz) return DSMD_ERR_INVALID;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const PinnedArrays from(x, y, z, std::max<int64_t>(c->n_total, 1)), to(fx, fy, fz, std::max<int64_t>(c->n_owned, 1));
    if (!rebuild && c->list_valid && !out6 && (c->n_owned >= kPipelineLeast || !from.all || !to.all)) {
        const int rc = forces_host_pipelined(c, x, y, z, fx, fy, fz, to, s);
        if (rc != DSMD_ERR_STATE) return rc;   // DSMD_ERR_STATE: too small to cut into slabs, the plain way below
    }
    {
        const int rc = from.all && c->n_total > 0 ? pull_positions(c, from, 0, c->n_total, s) : dsmd_upload_positions(c, x, y, z, s);
        if (rc) return rc;
        c->owned_sorted_only = false;
    }
    if (rebuild || !c->list_valid) {
        const int rc = dsmd_build_neighbor_list(c, s);
        if (rc) return rc;
    } else {
        const int rc = pack_impl(c, 0, c->n_total, false, 0.0, 0.0, s);
        if (rc) return rc;
    }
    { const int rc = dsmd_compute_forces(c, DSMD_PHASE_FULL, out6 ? 1 : 0, s); if (rc) return rc; }
    if (to.all && c->n_owned > 0) { const int rc = push_forces(c, to, 0, c->n_owned, s); if (rc) return rc; }
    double* dst[3] = {fx, fy, fz};
    for (int a = 0; a < 3 && !to.all; ++a)
        DSMD_CUDA(c, cudaMemcpyAsync(dst[a], c->real[c->cur][DSMD_FX + a], sizeof(double) * c->n_owned,
                                     cudaMemcpyDeviceToHost, s));
    if (out6) { const int rc = dsmd_read_scalars(c, out6, s); if (rc) return rc; }
    DSMD_CUDA(c, cudaStreamSynchronize(s));
    return DSMD_OK;
}

int dsmd_fma_probe(dsmd_ctx* c, int iters, double* flops, void* stream) {
    if (!c || iters <= 0 || !flops) return DSMD_ERR_INVALID;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    int sms = 0;
    DSMD_CUDA(c, cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c->device));
    const int blocks = sms * 8;
    k_fma_probe<<<blocks, 256, 0, s>>>(iters, 1.0f, reinterpret_cast<float*>(c->flag));
    DSMD_LAUNCHED(c);
    *flops = static_cast<double>(blocks) * 256.0 * static_cast<double>(iters) * 8.0 * 2.0;
    return DSMD_OK;
}

// ---- ghosts ---------------------------------------------------------------------------------------------------------

int dsmd_halo_pack(dsmd_ctx* c, const int32_t* d_index, const int8_t* d_image, int64_t count, double* d_out,
                   void* stream) {
    if (!c || count < 0 || (count > 0 && (!d_index || !d_out))) return DSMD_ERR_INVALID;
    if (count == 0) return DSMD_OK;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    double** r = c->real[c->cur];
    k_halo_pack<<<blocks_for(count, kThreads), kThreads, 0, s>>>(static_cast<int>(count), d_index,
                                                                reinterpret_cast<const signed char*>(d_image), r[0], r[1],
                                                                r[2], c->box[0], c->box[1], c->box[2], d_out);
    DSMD_LAUNCHED(c);
    return DSMD_OK;
}

int dsmd_displacement_word(dsmd_ctx* c, void** device_word) {
    if (!c || !device_word) return DSMD_ERR_INVALID;
    *device_word = &c->status->max_disp2;
    c->word_shared = true;
    return DSMD_OK;
}

int dsmd_halo_unpack(dsmd_ctx* c, const double* d_in, int64_t first_ghost, int64_t count, void* stream) {
    if (!c || count < 0 || first_ghost < 0 || first_ghost + count > c->n_total - c->n_owned) return DSMD_ERR_INVALID;
    if (count == 0) return DSMD_OK;
    if (!c->list_valid) return fail(c, DSMD_ERR_STATE, "halo unpack needs the ghost slots of a built list");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    double** r = c->real[c->cur];
    c->disp_seq = 0;
    k_halo_unpack<<<blocks_for(count, kThreads), kThreads, 0, s>>>(c->grid, static_cast<int>(first_ghost),
                                                                  static_cast<int>(count), d_in, c->ghost_slot, r[0],
                                                                  r[1], r[2], c->type[c->cur], c->pq, c->status);
    DSMD_LAUNCHED(c);
    return DSMD_OK;
}

int dsmd_halo_select(dsmd_ctx* c, const double lo[3], const double hi[3], int32_t* d_index, int64_t capacity,
                     int64_t* count, void* stream) {
    if (!c || !lo || !hi || !count) return DSMD_ERR_INVALID;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const int n = static_cast<int>(c->n_owned);
    *count = 0;
    if (n == 0) return DSMD_OK;
    double** r = c->real[c->cur];
    k_halo_flag<<<blocks_for(n, kThreads), kThreads, 0, s>>>(n, r[0], r[1], r[2], lo[0], lo[1], lo[2], hi[0], hi[1],
                                                            hi[2], c->flag);
    DSMD_LAUNCHED(c);
    size_t need = 0;
    thrust::counting_iterator<int> iota(0);
    int* d_selected = c->list;   // scratch of capacity entries
    cub::DeviceSelect::Flagged(nullptr, need, iota, c->flag, d_selected, &c->status->select_count, n, s);
    if (need > c->cub_temp_bytes) {
        if (c->cub_temp) cudaFree(c->cub_temp);
        c->cub_temp = nullptr;
        DSMD_CUDA(c, cudaMalloc(&c->cub_temp, need));
        c->cub_temp_bytes = need;
    }
    DSMD_CUDA(c, cub::DeviceSelect::Flagged(c->cub_temp, need, iota, c->flag, d_selected, &c->status->select_count, n, s));
    unsigned long long selected = 0;
    DSMD_CUDA(c, cudaMemcpyAsync(&selected, &c->status->select_count, sizeof(selected), cudaMemcpyDeviceToHost, s));
    DSMD_CUDA(c, cudaStreamSynchronize(s));
    *count = static_cast<int64_t>(selected);
    if (d_index && static_cast<int64_t>(selected) <= capacity && selected > 0)
        DSMD_CUDA(c, cudaMemcpyAsync(d_index, d_selected, sizeof(int) * selected, cudaMemcpyDeviceToDevice, s));
    DSMD_CUDA(c, cudaStreamSynchronize(s));
    return DSMD_OK;
}

int dsmd_halo_pack_records(dsmd_ctx* c, const int32_t* d_index, int64_t count, const double shift[3],
                           double* d_real_out, int32_t* d_int_out, void* stream) {
    if (!c || count < 0 || (count > 0 && (!d_index || !d_real_out || !d_int_out))) return DSMD_ERR_INVALID;
    if (count == 0) return DSMD_OK;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    k_halo_pack_records<<<blocks_for(count, kThreads), kThreads, 0, s>>>(
        static_cast<int>(count), d_index, arrays_of(c, c->cur), c->type[c->cur], c->gid[c->cur], shift ? shift[0] : 0.0,
        shift ? shift[1] : 0.0, shift ? shift[2] : 0.0, d_real_out, d_int_out);
    DSMD_LAUNCHED(c);
    return DSMD_OK;
}

int dsmd_halo_append_records(dsmd_ctx* c, const double* d_real_in, const int32_t* d_int_in, int64_t count,
                             void* stream) {
    if (!c || count < 0 || (count > 0 && (!d_real_in || !d_int_in))) return DSMD_ERR_INVALID;
    if (c->n_total + count > c->capacity) return fail(c, DSMD_ERR_CAPACITY, "ghosts exceed the context's capacity");
    if (count == 0) return DSMD_OK;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    k_halo_append_records<<<blocks_for(count, kThreads), kThreads, 0, s>>>(
        static_cast<int>(count), static_cast<int>(c->n_total), d_real_in, d_int_in, arrays_of(c, c->cur),
        c->type[c->cur], c->gid[c->cur]);
    DSMD_LAUNCHED(c);
    c->n_total += count;
    c->list_valid = false;
    return DSMD_OK;
}

int dsmd_halo_append_packed(dsmd_ctx* c, const double* d_records, int64_t count, void* stream) {
    if (!c || count < 0 || (count > 0 && !d_records)) return DSMD_ERR_INVALID;
    if (c->n_total + count > c->capacity) return fail(c, DSMD_ERR_CAPACITY, "atoms exceed the context's capacity");
    if (count == 0) return DSMD_OK;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    k_halo_append_packed<<<blocks_for(count, kThreads), kThreads, 0, s>>>(
        static_cast<int>(count), static_cast<int>(c->n_total), d_records, arrays_of(c, c->cur), c->type[c->cur],
        c->gid[c->cur]);
    DSMD_LAUNCHED(c);
    c->n_total += count;
    c->list_valid = false;
    return DSMD_OK;
}

int dsmd_capacity(const dsmd_ctx* c, int64_t* capacity) {
    if (!c || !capacity) return DSMD_ERR_INVALID;
    *capacity = c->capacity;
    return DSMD_OK;
}

}  // extern "C"
