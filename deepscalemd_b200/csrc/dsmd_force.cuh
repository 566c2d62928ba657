// What the force kernels (dsmd_pair.cuh) are given and how they are launched. The kernels are compiled in several translation
// units, forces and energy sums, with and without Ewald apart (dsmd_pair_*.cu): the device loads a unit's code when a kernel of it
// is first launched, and all forms together took 17 ms of a program's first call, most of it for forms that the program never
// uses (apart: 2.7 ms for the rest of the library and 0.6 for Lennard-Jones forces).
#pragma once

#include <cuda_runtime.h>

#include "dsmd_common.cuh"
#include "dsmd_report.cuh"

namespace dsmd {

struct RowArrays {
    const unsigned* quad;
    unsigned* rows;
    int stride;             // entries a row has room for, whole groups
    int* row_end;
    int* row_int;
    unsigned* row_special;
};

// Who writes where when a displacement check ends.
struct DisplacementReport {
    Status* st;
    unsigned* ticket;      // blocks that have finished, or null: see report_displacement
    Mail* mail;            // or null: no report
    unsigned long long seq;
    double gate2;          // see gate_closed
};

struct PairParams {
    float scale[3];
    float rc2;
    float rs2, inv_denom;        // CHARMM switch on r^2 (rs2 < 0: off)
    float kq;                    // Coulomb constant
    float alpha, two_alpha_sqrtpi;
    int ntypes;
    int ewald_intervals;
    float ewald_most;            // largest r^2 looked up: the last float inside the last interval
    const float2* lj;            // [ntypes * ntypes] {12 c12, -6 c6}
    const float4* ewald;         // [2 * intervals]: force cubic, energy cubic
    const float* type_charge;    // [ntypes] when every atom's charge is that of its type (dsmd_set_type_charges), else null
};

// Pair parameters by type. kOneType: constants. kTwoTypes (without Ewald): both in registers, the partner's type picks. kFewTypes: a table over (type of the first atom, type of the second, type
// of the partner) that holds what both atoms need side by side - up to 8 types, 8 KB (12 KB with charges by type). kManyTypes: a table over two types,
// read once per atom.
enum { kOneType = 0, kFewTypes = 1, kManyTypes = 2, kTwoTypes = 3 };
constexpr int kFewTypesMost = 8;

constexpr int kEwaldCopiesMost = 8;   // see EwaldTable
constexpr float kEwaldFirst = 0.5f;   // r^2 at which the table starts

struct ForceArgs {
    const int4* pq;
    const float* qf;
    RowArrays rows;
    int phase;
    const int* pair_list;    // the pairs to work on (boundary pass), or null: first_pair ...
    int first_pair, n_pairs; // ... first_pair + n_pairs
    int lane_shift;          // log2 of the lanes that share one row
    double *fx, *fy, *fz;
    double* partials;        // energy sums: per block, a count of finished blocks, and the total
    unsigned* ticket;
    double* scalars;
    Mail* mail;              // where the total is reported to the host
    unsigned long long seq;
    const Status* st;
    double gate2;            // see gate_closed
    bool list_settled;       // the list was complete before the launch before this one began: it may be read without waiting
};

struct StepArgs {
    double *x, *y, *z, *vx, *vy, *vz;
    const double *mass, *xref, *yref, *zref;
    int4* pq_next;
    double dt, kick;    // kick = dt times the force-to-acceleration factor: half of it ends this step, half begins the next
};

// Threads per block and blocks per SM, which fix the registers and with them how the compiler interleaves the partners of a
// chunk; measured on a B200, the best of five to nine settings each. Long rows with Ewald: one block of 512 per SM, 128 registers
// (0.97 ms per pass over 648,000 water atoms; 0.97 to 1.16 ms with one of 384 to 768 or two to four smaller ones; 1.12 ms with a row per
// lane). One type: 64 registers, 0.356 ms at 4,000,000 Lennard-Jones atoms (0.37 to 0.41 ms at 14 to 20 blocks; 0.418 ms while what the
// end of a row needs was kept in registers through its loop). Two types: 80 registers, 0.164 ms for the 1,048,576-atom mixture
// (0.17 to 0.19 ms at other settings, 0.174 with the pair table in shared memory, 0.185 before).
template <int COPIES, int TYPES>
constexpr int kPairThreads = COPIES == kEwaldCopiesMost ? 512 : (COPIES == 0 && TYPES == kOneType ? 64 : 128);
template <int COPIES, int TYPES, bool ENERGY>
constexpr int kPairBlocks = ENERGY || COPIES == kEwaldCopiesMost ? 1 : (COPIES > 0 ? 5 : (TYPES == kOneType ? 16 : 6));

// Both return what the launch returned. sw: with the switching function. overlap: dsmd_launch.cuh. ENERGY: with energy sums. ORDER: of the rows' entries
// (dsmd_row_layout.cuh).
template <int COPIES, bool ENERGY, int ORDER>
cudaError_t launch_pair(const PairParams& p, const ForceArgs& a, bool sw, unsigned blocks, bool overlap, cudaStream_t s);
template <int ORDER>
cudaError_t launch_step(const PairParams& p, const ForceArgs& a, const Grid& g, const StepArgs& at, const DisplacementReport& report,
                        bool sw, unsigned blocks, cudaStream_t s);

}  // namespace dsmd
