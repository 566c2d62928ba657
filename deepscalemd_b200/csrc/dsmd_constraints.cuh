// Holonomic distance constraints of small rigid groups (rigid water and the like): SHAKE after the drift, RATTLE after
// the second velocity half, together with the velocity-Verlet halves around them. Included by dsmd_core.cu.
//
// What the reference does in shake_cluster_kernel / rattle_cluster_kernel (src/force_calculator_cuda.cu:6168-6333) and,
// on the host, ConstraintSolver (src/constraint_solver.cpp:15-146): every connected group of constraints (a "cluster":
// the three O-H, O-H, H-H constraints of a water molecule) is solved by ONE thread, sweeping its constraints in their
// given order until each |r_ij|^2 is within `tolerance` (relative) of its target (SHAKE: corrections along the bond
// vectors the pairs had before the drift; velocities take the displacement over dt), or until the relative velocity
// along every bond is below `tolerance` (RATTLE). A cluster converged is a cluster left alone, so the result is the one
// of sweeping all constraints of the system in order, as the host solver does.
//
// A cluster's atoms meet nobody else between two force evaluations, so one thread takes them through the whole of it:
// second half-kick and RATTLE, first half-kick, drift, SHAKE, conversion to fixed point and displacement check.
// What bounds it: fp64 arithmetic of the sweeps (about 10 of them). The shapes that occur in numbers (three atoms with three
// constraints, two atoms with one) are compiled with their constraint order known, which keeps the cluster in registers:
// 648,000 water atoms, one step: 0.08 ms, against 0.78 ms for separate passes over clusters in local memory.
//
// Atoms are re-sorted by cell at every list build, so clusters name their atoms by global id; the slots are looked up
// once per build. Clusters hold at most kClusterAtoms atoms and kClusterCons constraints.
#pragma once

namespace {

constexpr int kClusterAtoms = 4;
constexpr int kClusterCons = 6;

struct ClusterTable {
    int n_clusters;
    const int* atom_slot;           // [n_clusters * kClusterAtoms], -1: unused
    const unsigned char* con_a;     // [n_clusters * kClusterCons] atom of the cluster (0 .. kClusterAtoms - 1), 255: unused
    const unsigned char* con_b;
    const double* con_d2;           // squared target distance
    double box[3];
    int periodic[3];
};

__device__ __forceinline__ void half_box_image(double d[3], const ClusterTable& t) {
#pragma unroll
    for (int a = 0; a < 3; ++a)
        if (t.periodic[a]) {
            if (d[a] > 0.5 * t.box[a]) d[a] -= t.box[a];
            else if (d[a] < -0.5 * t.box[a]) d[a] += t.box[a];
        }
}

__global__ void k_slot_of_gid(int n, const int* __restrict__ gid, int n_global, int* __restrict__ slot_of) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n) return;
    const int g = gid[s];
    if (g >= 0 && g < n_global) slot_of[g] = s;
}

__global__ void k_cluster_slots(int n, const int* __restrict__ atom_gid, const int* __restrict__ slot_of_gid, int* __restrict__ slot) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < n) slot[k] = atom_gid[k] < 0 ? -1 : slot_of_gid[atom_gid[k]];
}

// Shapes of clusters: how many atoms and constraints, and which atoms constraint j joins.
struct AnyCluster {
    static constexpr int atoms = kClusterAtoms, constraints = kClusterCons;
    static constexpr bool known = false;
    static constexpr __host__ __device__ int a(int) { return 0; }
    static constexpr __host__ __device__ int b(int) { return 0; }
};
struct TriangleCluster {   // rigid water: 0-1, 0-2, 1-2
    static constexpr int atoms = 3, constraints = 3;
    static constexpr bool known = true;
    static constexpr __host__ __device__ int a(int j) { return j < 2 ? 0 : 1; }
    static constexpr __host__ __device__ int b(int j) { return j == 0 ? 1 : 2; }
};
struct BondCluster {       // one bond
    static constexpr int atoms = 2, constraints = 1;
    static constexpr bool known = true;
    static constexpr __host__ __device__ int a(int) { return 0; }
    static constexpr __host__ __device__ int b(int) { return 1; }
};

template <class Shape>
struct Cluster {
    double p[Shape::atoms][3], v[Shape::atoms][3], w[Shape::atoms];   // position, velocity, 1 / mass
    int slot[Shape::atoms];
    int n;

    // One constraint, given the places of its atoms: SHAKE (true: nothing left to correct).
    __device__ __forceinline__ bool shake_one(const ClusterTable& t, const double (&q)[Shape::atoms][3], int a, int b, double target2,
                                              double inv_dt, double tolerance) {
        double d[3] = {p[a][0] - p[b][0], p[a][1] - p[b][1], p[a][2] - p[b][2]};
        half_box_image(d, t);
        const double excess = (d[0] * d[0] + d[1] * d[1] + d[2] * d[2]) - target2;
        if (fabs(excess) < tolerance * target2) return true;
        double o[3] = {q[a][0] - q[b][0], q[a][1] - q[b][1], q[a][2] - q[b][2]};
        half_box_image(o, t);
        const double along = o[0] * d[0] + o[1] * d[1] + o[2] * d[2];
        if (fabs(along) >= 1e-12) {   // else degenerate geometry: the next sweep tries again
            const double gm = excess / (2.0 * (w[a] + w[b]) * along);
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const double corr = gm * o[c];
                p[a][c] -= corr * w[a];
                p[b][c] += corr * w[b];
                v[a][c] -= corr * w[a] * inv_dt;
                v[b][c] += corr * w[b] * inv_dt;
            }
        }
        return false;
    }

    // RATTLE, one constraint; wsum: diagonal of the constraint virial, prefactor * k r_a^2.
    __device__ __forceinline__ bool rattle_one(const ClusterTable& t, int a, int b, double tolerance, double prefactor, double (&wsum)[3]) {
        double d[3] = {p[a][0] - p[b][0], p[a][1] - p[b][1], p[a][2] - p[b][2]};
        half_box_image(d, t);
        const double r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2];
        if (r2 < 1e-20) return true;
        const double along = d[0] * (v[a][0] - v[b][0]) + d[1] * (v[a][1] - v[b][1]) + d[2] * (v[a][2] - v[b][2]);
        if (fabs(along) < tolerance) return true;
        const double km = along / ((w[a] + w[b]) * r2);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            v[a][c] -= km * w[a] * d[c];
            v[b][c] += km * w[b] * d[c];
            wsum[c] += prefactor * km * d[c] * d[c];
        }
        return false;
    }

    template <bool SHAKE>
    __device__ __forceinline__ bool solve(const ClusterTable& t, int k, const double (&q)[Shape::atoms][3], double inv_dt, double tolerance,
                                          int max_iterations, double prefactor, double (&wsum)[3]) {
        if (Shape::known) {
            double target2[Shape::constraints];
#pragma unroll
            for (int j = 0; j < Shape::constraints; ++j) target2[j] = t.con_d2[k * kClusterCons + j];
            for (int sweep = 0; sweep < max_iterations; ++sweep) {
                bool done = true;
#pragma unroll
                for (int j = 0; j < Shape::constraints; ++j)
                    done &= SHAKE ? shake_one(t, q, Shape::a(j), Shape::b(j), target2[j], inv_dt, tolerance)
                                  : rattle_one(t, Shape::a(j), Shape::b(j), tolerance, prefactor, wsum);
                if (done) return true;
            }
        } else {
            for (int sweep = 0; sweep < max_iterations; ++sweep) {
                bool done = true;
                for (int j = 0; j < Shape::constraints; ++j) {
                    const int a = t.con_a[k * kClusterCons + j], b = t.con_b[k * kClusterCons + j];
                    if (a == 255) break;
                    done &= SHAKE ? shake_one(t, q, a, b, t.con_d2[k * kClusterCons + j], inv_dt, tolerance)
                                  : rattle_one(t, a, b, tolerance, prefactor, wsum);
                }
                if (done) return true;
            }
        }
        return false;
    }
};

struct AtomArrays {
    double *x, *y, *z, *vx, *vy, *vz;
    const double *fx, *fy, *fz, *mass;
    const int* type;
    const double *xref, *yref, *zref;
    int4* pq;
};

// FINISH: v += half_kick f / m, RATTLE; START: v += half_kick f / m, x += dt v, SHAKE, fixed point, displacement check (of
// the drifted position and of the corrected one). virial (may be null): the diagonal of the constraint virial of RATTLE,
// -2 / (force_to_accel dt) * sum over corrections of k r_a^2 (`prefactor`).
template <class Shape, bool FINISH, bool START>
__global__ void __launch_bounds__(128) k_constrained(ClusterTable t, Grid g, AtomArrays at, double half_kick, double dt, double tolerance,
                                                     int max_iterations, double prefactor, double* __restrict__ partials, unsigned* __restrict__ ticket,
                                                     double* __restrict__ virial, DisplacementReport report) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    double wsum[3] = {0.0, 0.0, 0.0}, worst2 = 0.0;
    if (k < t.n_clusters) {
        Cluster<Shape> c;
        c.n = 0;
        double a[Shape::atoms][3];   // half_kick f / m
#pragma unroll
        for (int m = 0; m < Shape::atoms; ++m) {
            const int s = t.atom_slot[k * kClusterAtoms + m];
            c.slot[m] = s;
            if (!Shape::known && s < 0) continue;
            c.n = m + 1;
            c.p[m][0] = at.x[s]; c.p[m][1] = at.y[s]; c.p[m][2] = at.z[s];
            c.v[m][0] = at.vx[s]; c.v[m][1] = at.vy[s]; c.v[m][2] = at.vz[s];
            c.w[m] = 1.0 / at.mass[s];
            if (half_kick != 0.0) {
                const double h = half_kick / at.mass[s];
                a[m][0] = h * at.fx[s]; a[m][1] = h * at.fy[s]; a[m][2] = h * at.fz[s];
            } else {
                a[m][0] = a[m][1] = a[m][2] = 0.0;
            }
        }
        bool good = true;
        if (FINISH) {
#pragma unroll
            for (int m = 0; m < Shape::atoms; ++m)
                if (Shape::known || m < c.n)
                    for (int x = 0; x < 3; ++x) c.v[m][x] += a[m][x];
            good &= c.template solve<false>(t, k, c.p, 0.0, tolerance, max_iterations, prefactor, wsum);
        }
        if (START) {
            double q[Shape::atoms][3];
#pragma unroll
            for (int m = 0; m < Shape::atoms; ++m)
                if (Shape::known || m < c.n) {
                    const double ref[3] = {at.xref[c.slot[m]], at.yref[c.slot[m]], at.zref[c.slot[m]]};
                    double d2 = 0.0;
#pragma unroll
                    for (int x = 0; x < 3; ++x) {
                        q[m][x] = c.p[m][x];
                        c.v[m][x] += a[m][x];
                        c.p[m][x] += dt * c.v[m][x];
                        d2 += (c.p[m][x] - ref[x]) * (c.p[m][x] - ref[x]);
                    }
                    worst2 = fmax(worst2, d2 == d2 ? d2 : __longlong_as_double(0x7FF0000000000000ll));   // see k_pack
                }
            good &= c.template solve<true>(t, k, q, 1.0 / dt, tolerance, max_iterations, 0.0, wsum);
        }
        unsigned bad = 0;
#pragma unroll
        for (int m = 0; m < Shape::atoms; ++m)
            if (Shape::known || m < c.n) {
                const int s = c.slot[m];
                at.vx[s] = c.v[m][0]; at.vy[s] = c.v[m][1]; at.vz[s] = c.v[m][2];
                if (START) {
                    at.x[s] = c.p[m][0]; at.y[s] = c.p[m][1]; at.z[s] = c.p[m][2];
                    int4 f;
                    f.x = static_cast<int>(dsmd::to_fixed(c.p[m][0], 0, g, bad));
                    f.y = static_cast<int>(dsmd::to_fixed(c.p[m][1], 1, g, bad));
                    f.z = static_cast<int>(dsmd::to_fixed(c.p[m][2], 2, g, bad));
                    f.w = at.type[s];
                    at.pq[s] = f;
                    const double dx = c.p[m][0] - at.xref[s], dy = c.p[m][1] - at.yref[s], dz = c.p[m][2] - at.zref[s];
                    const double d2 = dx * dx + dy * dy + dz * dz;
                    worst2 = fmax(worst2, d2 == d2 ? d2 : __longlong_as_double(0x7FF0000000000000ll));
                }
            }
        if (bad) atomicAdd(&report.st->out_of_domain, 1u);
        if (!good) atomicAdd(&report.st->constraint_failed, 1u);
    }
    if (START) report_displacement(worst2, report);
    if (virial) sum_over_grid<3>(wsum, partials, ticket, virial, false);
}

}  // namespace
