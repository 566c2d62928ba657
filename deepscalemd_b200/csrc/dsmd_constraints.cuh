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
// What bounds it: the chain of fp64 operations of the sweeps (some 20 of each kind). The shapes that occur in numbers (three
// atoms with three constraints, two atoms with one) are compiled with their constraint order known, which keeps the cluster
// in registers, and sweep over what the sweeps are about instead of over atoms (rattle_known, shake_known). Rigid water,
// second half of a step and first half of the next: 0.098 ms at 648,000 atoms, 22 us at 3,993 (sweeps over the atoms'
// positions and velocities: 0.277 ms and 60 us).
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

__global__ void k_slot_of_gid(int n, const int* gid, int n_global, int* __restrict__ slot_of) {
    if (!dsmd::after_previous()) return;
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n) return;
    const int g = gid[s];
    if (g >= 0 && g < n_global) slot_of[g] = s;
}

__global__ void k_cluster_slots(int n, const int* atom_gid, const int* slot_of_gid, int* __restrict__ slot) {
    if (!dsmd::after_previous()) return;
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

    // How the bond vector (or relative velocity) of constraint i changes per unit of a correction along constraint j, in
    // which atom a(j) goes by -w and atom b(j) by +w.
    __device__ __forceinline__ double coupling(int i, int j) const {
        const int ai = Shape::a(i), bi = Shape::b(i), aj = Shape::a(j), bj = Shape::b(j);
        double m = 0.0;
        if (ai == aj) m -= w[aj];
        if (ai == bj) m += w[bj];
        if (bi == aj) m += w[aj];
        if (bi == bj) m -= w[bj];
        return m;
    }

    // The bond vectors of a known shape.
    __device__ __forceinline__ void bonds(const ClusterTable& t, double (&d)[Shape::constraints][3]) const {
#pragma unroll
        for (int j = 0; j < Shape::constraints; ++j) {
#pragma unroll
            for (int x = 0; x < 3; ++x) d[j][x] = p[Shape::a(j)][x] - p[Shape::b(j)][x];
            half_box_image(d[j], t);
        }
    }

    // RATTLE of a known shape. A correction along one bond changes the relative velocity along the others by amounts that
    // do not depend on the velocities, so the sweeps work on one number per constraint, d . (v_a - v_b): one dependent
    // multiply-add per constraint instead of a pass through the atoms' velocities with a division. Atoms take the sum.
    __device__ __forceinline__ bool rattle_known(const double (&d)[Shape::constraints][3], double tolerance, int max_iterations,
                                                 double prefactor, double (&wsum)[3]) {
        constexpr int N = Shape::constraints;
        double along[N], inv[N], g[N][N], sum[N];
#pragma unroll
        for (int j = 0; j < N; ++j) {
            const int a = Shape::a(j), b = Shape::b(j);
            const double r2 = d[j][0] * d[j][0] + d[j][1] * d[j][1] + d[j][2] * d[j][2];
            along[j] = d[j][0] * (v[a][0] - v[b][0]) + d[j][1] * (v[a][1] - v[b][1]) + d[j][2] * (v[a][2] - v[b][2]);
            inv[j] = r2 < 1e-20 ? 0.0 : 1.0 / ((w[a] + w[b]) * r2);   // no bond vector: nothing to correct
            sum[j] = 0.0;
        }
#pragma unroll
        for (int j = 0; j < N; ++j)
#pragma unroll
            for (int i = 0; i < N; ++i) g[i][j] = inv[j] * coupling(i, j) * (d[i][0] * d[j][0] + d[i][1] * d[j][1] + d[i][2] * d[j][2]);
        bool done = false;
        for (int sweep = 0; sweep < max_iterations && !done; ++sweep) {
            done = true;
#pragma unroll
            for (int j = 0; j < N; ++j) {   // a constraint that holds is left alone (selected, not branched over)
                const double now = along[j];
                const bool holds = fabs(now) < tolerance || inv[j] == 0.0;
                done &= holds;
                sum[j] = holds ? sum[j] : fma(now, inv[j], sum[j]);
#pragma unroll
                for (int i = 0; i < N; ++i) along[i] = holds ? along[i] : fma(now, g[i][j], along[i]);
            }
        }
#pragma unroll
        for (int j = 0; j < N; ++j)
#pragma unroll
            for (int x = 0; x < 3; ++x) {
                v[Shape::a(j)][x] -= sum[j] * w[Shape::a(j)] * d[j][x];
                v[Shape::b(j)][x] += sum[j] * w[Shape::b(j)] * d[j][x];
                wsum[x] += prefactor * sum[j] * d[j][x] * d[j][x];
            }
        return done;
    }

    // SHAKE of a known shape, o: the bond vectors before the drift. The sweeps work on the bond vectors and on their
    // components along o (which change by amounts known in advance); atoms take the sum. Each component's reciprocal follows
    // it from sweep to sweep by Newton's iteration, of third order, where it moved by less than 1 % (relative error below
    // 1e-6 of a correction, gone with the next sweep; nothing is left of it when the sweeps end at 1e-8): half as long a
    // chain of dependent operations as a division, and no branch.
    __device__ __forceinline__ bool shake_known(const ClusterTable& t, int k, const double (&o)[Shape::constraints][3], double inv_dt,
                                                double tolerance, int max_iterations) {
        constexpr int N = Shape::constraints;
        double d[N][3], target2[N], half_inv[N], sum[N], along[N], inv[N], move[N][N], change[N][N];
        bonds(t, d);
#pragma unroll
        for (int j = 0; j < N; ++j) {
            target2[j] = t.con_d2[k * kClusterCons + j];
            half_inv[j] = 0.5 / (w[Shape::a(j)] + w[Shape::b(j)]);
            sum[j] = 0.0;
            along[j] = o[j][0] * d[j][0] + o[j][1] * d[j][1] + o[j][2] * d[j][2];
            inv[j] = fabs(along[j]) >= 1e-12 ? 1.0 / along[j] : 0.0;
#pragma unroll
            for (int i = 0; i < N; ++i) {
                move[i][j] = coupling(i, j);
                change[i][j] = move[i][j] * (o[i][0] * o[j][0] + o[i][1] * o[j][1] + o[i][2] * o[j][2]);
            }
        }
        bool done = false;
        for (int sweep = 0; sweep < max_iterations && !done; ++sweep) {
            done = true;
#pragma unroll
            for (int j = 0; j < N; ++j) {
                const double off = fma(-along[j], inv[j], 1.0);
                double y = fma(inv[j], fma(off, off, off), inv[j]);
                if (fabs(off) > 0.01) y = fabs(along[j]) >= 1e-12 ? 1.0 / along[j] : 0.0;   // 0, degenerate geometry: the next sweep tries again
                inv[j] = y;
                const double excess = fma(d[j][0], d[j][0], fma(d[j][1], d[j][1], fma(d[j][2], d[j][2], -target2[j])));
                const bool holds = fabs(excess) < tolerance * target2[j];
                done &= holds;
                const double gm = holds ? 0.0 : excess * (half_inv[j] * y);
                sum[j] += gm;
#pragma unroll
                for (int i = 0; i < N; ++i) {
                    along[i] = fma(gm, change[i][j], along[i]);
                    const double c = gm * move[i][j];
#pragma unroll
                    for (int x = 0; x < 3; ++x) d[i][x] = fma(c, o[j][x], d[i][x]);
                }
            }
        }
#pragma unroll
        for (int j = 0; j < N; ++j)
#pragma unroll
            for (int x = 0; x < 3; ++x) {
                const int a = Shape::a(j), b = Shape::b(j);
                const double corr = sum[j] * o[j][x];
                p[a][x] -= corr * w[a];
                p[b][x] += corr * w[b];
                v[a][x] -= corr * w[a] * inv_dt;
                v[b][x] += corr * w[b] * inv_dt;
            }
        return done;
    }

    // Any other shape: sweeps over the atoms.
    template <bool SHAKE>
    __device__ __forceinline__ bool solve(const ClusterTable& t, int k, const double (&q)[Shape::atoms][3], double inv_dt, double tolerance,
                                          int max_iterations, double prefactor, double (&wsum)[3]) {
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
// behind_forces: the launch before is the force kernel, which has waited for all before itself and writes nothing but forces: the atoms'
// state is read while it ends.
template <class Shape, bool FINISH, bool START>
__global__ void __launch_bounds__(128) k_constrained(ClusterTable t, Grid g, AtomArrays at, double half_kick, double dt, double tolerance,
                                                     int max_iterations, double prefactor, double* __restrict__ partials, unsigned* __restrict__ ticket,
                                                     double* __restrict__ virial, DisplacementReport report, bool behind_forces) {
    if (!behind_forces && !dsmd::after_previous()) return;
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    double wsum[3] = {0.0, 0.0, 0.0}, worst2 = 0.0;
    Cluster<Shape> c;
    c.n = 0;
    double a[Shape::atoms][3];   // half_kick f / m
    if (k < t.n_clusters) {
#pragma unroll
        for (int m = 0; m < Shape::atoms; ++m) {
            const int s = t.atom_slot[k * kClusterAtoms + m];
            c.slot[m] = s;
            if (!Shape::known && s < 0) continue;
            c.n = m + 1;
            c.p[m][0] = at.x[s]; c.p[m][1] = at.y[s]; c.p[m][2] = at.z[s];
            c.v[m][0] = at.vx[s]; c.v[m][1] = at.vy[s]; c.v[m][2] = at.vz[s];
            const double mass = at.mass[s];
            c.w[m] = 1.0 / mass;
            a[m][0] = half_kick / mass;
        }
    }
    if (behind_forces && !dsmd::after_previous()) return;
    if (START && dsmd::gate_closed(report.st, report.gate2)) return;
    if (k < t.n_clusters) {
#pragma unroll
        for (int m = 0; m < Shape::atoms; ++m) {
            const int s = c.slot[m];
            if (!Shape::known && s < 0) continue;
            if (half_kick != 0.0) {
                const double h = a[m][0];
                a[m][0] = h * at.fx[s]; a[m][1] = h * at.fy[s]; a[m][2] = h * at.fz[s];
            } else {
                a[m][0] = a[m][1] = a[m][2] = 0.0;
            }
        }
        double o[Shape::constraints][3];   // bond vectors before the drift
        if constexpr (Shape::known) c.bonds(t, o);
        bool good = true;
        if (FINISH) {
#pragma unroll
            for (int m = 0; m < Shape::atoms; ++m)
                if (Shape::known || m < c.n)
                    for (int x = 0; x < 3; ++x) c.v[m][x] += a[m][x];
            if constexpr (Shape::known) good &= c.rattle_known(o, tolerance, max_iterations, prefactor, wsum);
            else good &= c.template solve<false>(t, k, c.p, 0.0, tolerance, max_iterations, prefactor, wsum);
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
            if constexpr (Shape::known) good &= c.shake_known(t, k, o, 1.0 / dt, tolerance, max_iterations);
            else good &= c.template solve<true>(t, k, q, 1.0 / dt, tolerance, max_iterations, 0.0, wsum);
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
