// LJ + real-space Ewald over the pair rows of dsmd_row_layout.cuh. Included by dsmd_pair_*.cu, each of which compiles some of the forms.
#pragma once

#include <type_traits>

#include "../../include/dsmd_b200.h"
#include "dsmd_f32x2.cuh"
#include "dsmd_launch.cuh"
#include "dsmd_force.cuh"
#include "dsmd_row_layout.cuh"
#include "dsmd_sums.cuh"
#include "ewald_table.hpp"

namespace {

using namespace dsmd;

// 1 / v: the hardware approximation (1 ulp) for the force-only kernels, one Newton step more (full single precision)
// where energy and virial sums are taken.
template <bool REFINE>
__device__ __forceinline__ float reciprocal(float v) {
    const float r = rcp_approx(v);
    return REFINE ? fmaf(r, fmaf(-v, r, 1.0f), r) : r;
}

// The real-space Ewald functions of r^2 as cubics on intervals of constant relative width (ewald_table.hpp). For rows of
// hundreds of entries the table lies in shared memory eight times over, copy c in the 16-byte bank group c, and a lane reads
// the copy of its place in its group of eight: a look-up by 32 lanes is 4 wavefronts whatever the intervals (8 to 11 with one
// copy). For short rows, where laying the table out (36 KB at a cutoff of 10 A) would be most of the work, one copy.

template <int COPIES>
struct EwaldTable {
    const float4* mine;   // this lane's copy of interval 0
    int intervals;
};

__device__ __forceinline__ float ewald_cubic(const float4* at, float t) {
    const float4 c = *at;   // coefficients of 32 t: powers of two, the same roundings
    return ((c.w * t + c.z) * t + c.y) * t + c.x;
}

template <bool ENERGY, int COPIES>
__device__ __forceinline__ void ewald_functions(const EwaldTable<COPIES>& table, float r2, float most, float& ff, float& ef) {
    // the interval and the place in it (1 / 32 octave: the low 18 bits of the mantissa); beyond the cutoff the last one,
    // below the table (the caller deals with that) the first one
    const unsigned bits = __float_as_uint(fmaxf(fminf(r2, most), kEwaldFirst));
    const unsigned idx = (bits - dsmd::kEwaldBaseBits) >> dsmd::kEwaldIndexShift;
    const float t = __uint_as_float(0x3F800000u | (bits & ((1u << dsmd::kEwaldIndexShift) - 1u))) - 1.0f;
    ff = ewald_cubic(table.mine + idx * COPIES, t);
    if (ENERGY) ef = ewald_cubic(table.mine + (table.intervals + idx) * COPIES, t);
}

// The same in closed form, for r^2 below the table.
__device__ __forceinline__ void ewald_functions_analytic(const PairParams& p, float r2, float& ff, float& ef) {
    const float r = sqrtf(r2), ar = p.alpha * r, ec = erfcf(ar) / r;
    ff = (ec + p.two_alpha_sqrtpi * __expf(-ar * ar)) / r2;
    ef = ec;
}

// What one evaluation needs to know of the two pairs.
struct PairTerms {
    F2 rep, att;   // 12 c12, -6 c6
    F2 qq;         // Coulomb constant times the charges
};

// Sums of the two atoms of a pair row.
//
// What bounds the force kernel: the multiply-add and the integer / select pipes, each busy half of the time and often at once (a packed
// instruction, two lanes: the two atoms, counts twice; about 55 scalar operations per entry (two pairs) for Lennard-Jones, 75 with Ewald),
// and beside them the L1 unit (13 wavefronts per gather of 32 random partners, half of that where four lanes gather neighbours).
// So what counts is the number of operations and that the compiler has registers to interleave four partners with. The plain form
// therefore leaves out what no pair of a sane system needs: with Ewald or energies it keeps the smallest r^2 for a look
// afterwards, without them a pair that coincides leaves sums that are not finite.
template <int COPIES, bool ENERGY, bool SWITCH>
struct PairAccumulator {
    static constexpr bool COULOMB = COPIES > 0;
    F2 ax{0}, ay{0}, az{0};
    F2 e_sum{0}, w_sum{0}, wx{0}, wy{0}, wz{0};
    float least = 3.0e38f;   // smallest r^2 seen (Ewald or energies)
    int n_in = 0;

    // Forces of the two atoms out, and the sums back to zero.
    __device__ __forceinline__ void take_forces(float (&a)[3], float (&b)[3]) {
        parts(ax, a[0], b[0]);
        parts(ay, a[1], b[1]);
        parts(az, a[2], b[2]);
        ax = ay = az = F2{0};
    }

    // Half of the energy sums (every pair is listed from both sides) added to v, and back to zero.
    __device__ __forceinline__ void take_energies(bool both_lanes, double (&v)[6]) {
        const F2 sums[5] = {e_sum, w_sum, wx, wy, wz};
#pragma unroll
        for (int k = 0; k < 5; ++k) {
            float a, b;
            parts(sums[k], a, b);
            v[k] += 0.5 * (static_cast<double>(a) + (both_lanes ? static_cast<double>(b) : 0.0));
        }
        v[5] += (both_lanes ? 0.5 : 0.25) * static_cast<double>(n_in);
        e_sum = w_sum = wx = wy = wz = F2{0};
        n_in = 0;
    }

    // Pair terms at the distances r2 of the two pairs: force over distance and energy. CAREFUL: Ewald functions below their
    // table, excluded pairs (Lennard-Jones off; the pair's 1/r is not part of the Ewald sum: erfc -> -erf).
    template <bool CAREFUL>
    __device__ __forceinline__ void evaluate(const PairParams& p, const EwaldTable<COPIES>& table, const PairTerms& k, F2 r2, float ra, float rb,
                                             bool ex_a, bool ex_b, F2& f, F2& u) {
        const F2 r2inv = f2(reciprocal<ENERGY>(ra), reciprocal<ENERGY>(rb));
        const F2 r6 = mul(mul(r2inv, r2inv), r2inv);
        f = mul(mul(r2inv, r6), fma(k.rep, r6, k.att));
        u = F2{0};
        if (ENERGY || SWITCH) u = mul(r6, fma(mul(k.rep, both(1.0f / 12.0f)), r6, mul(k.att, both(1.0f / 6.0f))));
        if (SWITCH) {
            // smooth for r^2 > rs2: f -> sw f + 12 u a (r^2 - rs2) / denom, u -> sw u (a = rc2 - r^2)
            const F2 a = fma(r2, both(-1.0f), both(p.rc2));
            const F2 above = add(r2, both(-p.rs2));
            const F2 aw = mul(a, both(p.inv_denom));
            const F2 b = fma(r2, both(2.0f), both(p.rc2 - 3.0f * p.rs2));
            float swa, swb, da, db;
            parts(mul(mul(a, b), aw), swa, swb);
            parts(mul(mul(mul(u, both(12.0f)), aw), above), da, db);
            const bool s_a = ra > p.rs2, s_b = rb > p.rs2;
            const F2 factor = f2(s_a ? swa : 1.0f, s_b ? swb : 1.0f);
            f = fma(factor, f, f2(s_a ? da : 0.0f, s_b ? db : 0.0f));
            u = mul(u, factor);
        }
        if (CAREFUL) {
            float va, vb;
            parts(f, va, vb);
            f = f2(ex_a ? 0.0f : va, ex_b ? 0.0f : vb);
            parts(u, va, vb);
            u = f2(ex_a ? 0.0f : va, ex_b ? 0.0f : vb);
        }
        if (COULOMB) {
            float ffa, ffb, efa = 0.0f, efb = 0.0f;
            ewald_functions<ENERGY>(table, ra, p.ewald_most, ffa, efa);
            ewald_functions<ENERGY>(table, rb, p.ewald_most, ffb, efb);
            if (CAREFUL) {
                if (ra < kEwaldFirst) ewald_functions_analytic(p, ra, ffa, efa);
                if (rb < kEwaldFirst) ewald_functions_analytic(p, rb, ffb, efb);
                const float ia = rsqrtf(ra), ib = rsqrtf(rb);
                if (ex_a) { ffa -= ia * ia * ia; efa -= ia; }
                if (ex_b) { ffb -= ib * ib * ib; efb -= ib; }
            }
            f = fma(k.qq, f2(ffa, ffb), f);
            if (ENERGY) u = fma(k.qq, f2(efa, efb), u);
        }
    }

    __device__ __forceinline__ void sum(F2 dx, F2 dy, F2 dz, F2 r2, F2 f, F2 u, bool in_a, bool in_b) {
        float va, vb;
        parts(f, va, vb);
        f = f2(in_a ? va : 0.0f, in_b ? vb : 0.0f);
        ax = fma(f, dx, ax);
        ay = fma(f, dy, ay);
        az = fma(f, dz, az);
        if (ENERGY) {
            parts(u, va, vb);
            e_sum = add(e_sum, f2(in_a ? va : 0.0f, in_b ? vb : 0.0f));
            w_sum = fma(f, r2, w_sum);
            wx = fma(mul(f, dx), dx, wx);
            wy = fma(mul(f, dy), dy, wy);
            wz = fma(mul(f, dz), dz, wz);
            n_in += (in_a ? 1 : 0) + (in_b ? 1 : 0);
        }
    }

    // What the plain form, which takes the table's first value for any distance below the table, left out of the Ewald terms of
    // two pairs at those distances. qq: Coulomb constant times the charges of the two pairs.
    __device__ __forceinline__ void add_close_rest(const PairParams& p, const EwaldTable<COPIES>& table, F2 dx, F2 dy, F2 dz, F2 r2, F2 qq) {
        float ra, rb;
        parts(r2, ra, rb);
        if (fminf(ra, rb) >= kEwaldFirst) return;
        float ffa, ffb, efa = 0.0f, efb = 0.0f, tfa, tfb, tea = 0.0f, teb = 0.0f;
        ewald_functions_analytic(p, ra, ffa, efa);
        ewald_functions_analytic(p, rb, ffb, efb);
        ewald_functions<ENERGY>(table, ra, p.ewald_most, tfa, tea);
        ewald_functions<ENERGY>(table, rb, p.ewald_most, tfb, teb);
        sum(dx, dy, dz, r2, mul(qq, f2(ffa - tfa, ffb - tfb)), mul(qq, f2(efa - tea, efb - teb)), ra < kEwaldFirst && ra < p.rc2,
            rb < kEwaldFirst && rb < p.rc2);
        n_in = 0;   // counted already
    }

    // Sums of all lanes of a warp, in every lane.
    __device__ __forceinline__ void over_warp() {
        F2* const sums[8] = {&ax, &ay, &az, &e_sum, &w_sum, &wx, &wy, &wz};
#pragma unroll
        for (int k = 0; k < (ENERGY ? 8 : 3); ++k)
            for (int o = 16; o > 0; o >>= 1) *sums[k] = add(*sums[k], F2{__shfl_xor_sync(0xFFFFFFFFu, sums[k]->v, o)});
    }
    __device__ __forceinline__ void add_sums(const PairAccumulator& other) {
        ax = add(ax, other.ax);
        ay = add(ay, other.ay);
        az = add(az, other.az);
        if (ENERGY) {
            e_sum = add(e_sum, other.e_sum);
            w_sum = add(w_sum, other.w_sum);
            wx = add(wx, other.wx);
            wy = add(wy, other.wy);
            wz = add(wz, other.wz);
        }
    }

    // (unsigned: the difference of two places half a box apart and more wraps, which signed arithmetic must not)
    static __device__ __forceinline__ float offset(int a, int b) {
        return static_cast<float>(static_cast<int>(static_cast<unsigned>(a) - static_cast<unsigned>(b)));
    }
    static __device__ __forceinline__ F2 distance(const PairParams& p, const int4& pa, const int4& pb, const int4& pj, F2& dx, F2& dy, F2& dz) {
        dx = mul(f2(offset(pa.x, pj.x), offset(pb.x, pj.x)), both(p.scale[0]));
        dy = mul(f2(offset(pa.y, pj.y), offset(pb.y, pj.y)), both(p.scale[1]));
        dz = mul(f2(offset(pa.z, pj.z), offset(pb.z, pj.z)), both(p.scale[2]));
        return fma(dz, dz, fma(dx, dx, mul(dy, dy)));   // (in this order: it decides which pairs lie inside a plain cutoff)
    }

    // The distance of the row's own two atoms, from each of them.
    static __device__ __forceinline__ F2 own_distance(const PairParams& p, const int4& pa, const int4& pb, F2& dx, F2& dy, F2& dz) {
        dx = mul(f2(offset(pa.x, pb.x), offset(pb.x, pa.x)), both(p.scale[0]));
        dy = mul(f2(offset(pa.y, pb.y), offset(pb.y, pa.y)), both(p.scale[1]));
        dz = mul(f2(offset(pa.z, pb.z), offset(pb.z, pa.z)), both(p.scale[2]));
        return fma(dz, dz, fma(dx, dx, mul(dy, dy)));
    }

    // The row's own two atoms, each the other's partner, in the plain form. k_a: terms of the second as the first sees it, k_b: of
    // the first as the second does. there: the pair counts.
    __device__ __forceinline__ void add_own(const PairParams& p, const EwaldTable<COPIES>& table, const int4& pa, const int4& pb,
                                            const PairTerms& k_a, const PairTerms& k_b, bool there) {
        F2 dx, dy, dz;
        const F2 r2 = own_distance(p, pa, pb, dx, dy, dz);
        float ra, rb;
        parts(r2, ra, rb);
        const PairTerms k{first_second(k_a.rep, k_b.rep), first_second(k_a.att, k_b.att), first_second(k_a.qq, k_b.qq)};
        F2 f, u;
        evaluate<false>(p, table, k, r2, ra, rb, false, false, f, u);
        if (there) least = fminf(least, fminf(ra, rb));
        sum(dx, dy, dz, r2, f, u, there && ra < p.rc2, there && rb < p.rc2);
    }

    // One entry, seen from the two atoms at pa and pb (fixed-point positions: the 32-bit difference is the nearest image).
    // The plain form takes every pair inside the cutoff; CAREFUL also tells pairs that coincide (r^2 < 1e-10: no force) and
    // those named above.
    template <bool CAREFUL>
    __device__ __forceinline__ void add_partner(const PairParams& p, const EwaldTable<COPIES>& table, const int4& pa, const int4& pb,
                                                const int4& pj, const PairTerms& k, unsigned entry) {
        F2 dx, dy, dz;
        const F2 r2 = distance(p, pa, pb, pj, dx, dy, dz);
        float ra, rb;
        parts(r2, ra, rb);
        F2 f, u;
        evaluate<CAREFUL>(p, table, k, r2, ra, rb, CAREFUL && (entry & kExclFirst) != 0u, CAREFUL && (entry & kExclSecond) != 0u, f, u);
        if (CAREFUL) {
            sum(dx, dy, dz, r2, f, u, ra < p.rc2 && ra >= 1e-10f, rb < p.rc2 && rb >= 1e-10f);
        } else {
            if (COULOMB || ENERGY) asm("min.f32 %0, %0, %1, %2;" : "+f"(least) : "f"(ra), "f"(rb));
            sum(dx, dy, dz, r2, f, u, ra < p.rc2, rb < p.rc2);
        }
    }
};

// Tables in shared memory: Ewald cubics and pair parameters by type. Every thread of the block calls it once.
template <int COPIES, bool ENERGY, int TYPES, bool QTYPE>
struct PairTables {
    static constexpr bool COULOMB = COPIES > 0;
    static constexpr bool few = TYPES == kFewTypes, many = TYPES == kManyTypes, by_type = COULOMB && QTYPE;
    static constexpr int functions = ENERGY ? 2 : 1;
    EwaldTable<COPIES> ewald;
    const ulonglong2* lj3;             // few: {rep, att} of both atoms by (type, type, partner's type)
    const unsigned long long* qq3;     // few, by_type: charges likewise
    const float2* lj2;                 // many
    const float* charge;               // by_type && !few

    __host__ __device__ static size_t bytes(int nt, int intervals) {
        size_t n = COULOMB ? sizeof(float4) * COPIES * functions * intervals : 0;
        if (few) n += static_cast<size_t>(nt) * nt * nt * (by_type ? 24 : 16);
        if (many) n += static_cast<size_t>(nt) * nt * sizeof(float2);
        if (by_type && !few) n += nt * sizeof(float);
        return n;
    }

    __device__ __forceinline__ PairTables(const PairParams& p, float4* smem) {
        const int nt = p.ntypes;
        float4* s_ewald = smem;
        ulonglong2* s_lj3 = reinterpret_cast<ulonglong2*>(s_ewald + (COULOMB ? functions * p.ewald_intervals * COPIES : 0));
        unsigned long long* s_qq3 = reinterpret_cast<unsigned long long*>(s_lj3 + (few ? nt * nt * nt : 0));
        float2* s_lj2 = reinterpret_cast<float2*>(s_qq3 + (few && by_type ? nt * nt * nt : 0));
        float* s_charge = reinterpret_cast<float*>(s_lj2 + (many ? nt * nt : 0));
        if (COULOMB)
            for (int k = threadIdx.x; k < functions * p.ewald_intervals * COPIES; k += blockDim.x) {
                const int entry = k / (COULOMB ? COPIES : 1);
                const float4 v = p.ewald[entry < p.ewald_intervals ? 2 * entry : 2 * (entry - p.ewald_intervals) + 1];
                s_ewald[k] = make_float4(v.x, v.y * 32.0f, v.z * 1024.0f, v.w * 32768.0f);
            }
        if (few)
            for (int k = threadIdx.x; k < nt * nt * nt; k += blockDim.x) {
                const int tj = k % nt, tb = (k / nt) % nt, ta = k / (nt * nt);
                const float2 la = p.lj[ta * nt + tj], lb = p.lj[tb * nt + tj];
                s_lj3[k] = make_ulonglong2(f2(la.x, lb.x).v, f2(la.y, lb.y).v);
                if (by_type) {
                    const float qj = p.type_charge[tj];
                    s_qq3[k] = f2(p.kq * p.type_charge[ta] * qj, p.kq * p.type_charge[tb] * qj).v;
                }
            }
        if (many)
            for (int k = threadIdx.x; k < nt * nt; k += blockDim.x) s_lj2[k] = p.lj[k];
        if (by_type && !few)
            for (int k = threadIdx.x; k < nt; k += blockDim.x) s_charge[k] = p.type_charge[k];
        if (COULOMB || few || many) __syncthreads();
        ewald = EwaldTable<COPIES>{s_ewald + (threadIdx.x & (COPIES > 0 ? COPIES - 1u : 0u)), p.ewald_intervals};
        lj3 = s_lj3;
        qq3 = s_qq3;
        lj2 = s_lj2;
        charge = s_charge;
    }
};

// What the plain form left out of a row's entries (add_close_rest), by all lanes of a warp.
template <int COPIES, bool ENERGY, bool SWITCH, bool BY_TYPE, int ORDER>
__device__ __forceinline__ PairAccumulator<COPIES, ENERGY, SWITCH> close_rest(const PairParams& p, const ForceArgs& a,
                                                                              const EwaldTable<COPIES>& table, int pair) {
    using Sums = PairAccumulator<COPIES, ENERGY, SWITCH>;
    Sums rest;
    int first;
    const int atoms = pair_atoms(a.rows.quad, pair, first), last = first + atoms - 1;
    const int4 pa = a.pq[first], pb = a.pq[last];
    const F2 q = mul(both(p.kq), BY_TYPE ? f2(p.type_charge[pa.w], p.type_charge[pb.w]) : f2(a.qf[first], a.qf[last]));
    const int mid = a.rows.row_int[pair], end = a.rows.row_end[pair], ghosts = whole_groups<ORDER>(mid);
    const int k0 = a.phase == DSMD_PHASE_BOUNDARY ? ghosts : 0, k1 = a.phase == DSMD_PHASE_INTERIOR ? mid : end;
    const unsigned* words = a.rows.rows + row_base<ORDER>(static_cast<unsigned>(pair), a.rows.stride);
#pragma unroll 1
    for (int k = k0 + (threadIdx.x & 31); k < k1; k += 32) {
        if (k >= mid && k < ghosts) continue;
        const unsigned e = words[row_offset<ORDER>(k)];
        const int4 pj = a.pq[e];
        F2 dx, dy, dz;
        const F2 r2 = Sums::distance(p, pa, pb, pj, dx, dy, dz);
        rest.add_close_rest(p, table, dx, dy, dz, r2, mul(q, both(BY_TYPE ? p.type_charge[pj.w] : a.qf[e])));
    }
    if ((threadIdx.x & 31) == 0 && atoms > 1 && a.phase != DSMD_PHASE_BOUNDARY && !(a.rows.row_special[pair] & kRowOwnExcluded)) {
        F2 dx, dy, dz;
        const F2 r2 = Sums::own_distance(p, pa, pb, dx, dy, dz);
        rest.add_close_rest(p, table, dx, dy, dz, r2, mul(q, BY_TYPE ? f2(p.type_charge[pb.w], p.type_charge[pa.w]) : f2(a.qf[last], a.qf[first])));
    }
    rest.over_warp();
    return rest;
}

// The row that thread t of a force kernel works on (-1: none) and its place among the lanes of the row.
__device__ __forceinline__ int row_of_thread(const ForceArgs& a, int t) {
    const int slot = t >> a.lane_shift;
    return slot < a.n_pairs ? (a.pair_list ? a.pair_list[slot] : a.first_pair + slot) : -1;
}

// t again, as a number that the compiler takes for another one: what follows from it is worked out (and read) anew instead of
// being kept in registers across the loop over a row's entries.
__device__ __forceinline__ int afresh(int t) {
    asm volatile("" : "+r"(t));
    return t;
}

// What a lane knows of its row from the list alone.
struct RowHead {
    int pair, first, atoms;   // no atoms: no row
    int c, c_end;             // this lane's first chunk of entries, one past the row's last
    unsigned special;
    uint4 e;                  // the first chunk
};

template <int ORDER>
__device__ __forceinline__ const uint4* row_chunks(const ForceArgs& a, int pair, int sub) {
    return reinterpret_cast<const uint4*>(a.rows.rows + row_base<ORDER>(static_cast<unsigned>(pair), a.rows.stride)) + (sub & ((1 << ORDER) - 1));
}

template <int ORDER>
__device__ __forceinline__ RowHead open_row(const ForceArgs& a, int t) {
    const int sub = t & ((1 << a.lane_shift) - 1);
    RowHead h{};
    h.pair = row_of_thread(a, t);
    if (h.pair < 0) return h;
    h.atoms = pair_atoms(a.rows.quad, h.pair, h.first);
    const int mid = a.rows.row_int[h.pair], end = a.rows.row_end[h.pair];
    h.special = a.rows.row_special[h.pair];
    // Chunks of entries, in groups of as many as lie side by side: those of owned partners, of ghosts, or all (what lies between
    // the two kinds are atoms out of reach).
    h.c = sub;
    if (a.phase == DSMD_PHASE_BOUNDARY) h.c += whole_groups<ORDER>(mid) >> 2;
    h.c_end = whole_groups<ORDER>(a.phase == DSMD_PHASE_INTERIOR ? mid : max(mid, end)) >> 2;
    if (h.special & kRowCareful) h.c_end = 0;
    if (h.c < h.c_end) h.e = __ldcs(row_chunks<ORDER>(a, h.pair, sub) + (h.c >> ORDER) * size_t(32));
    return h;
}

// Forces on the atoms of one pair row, worked on by 2^lane_shift lanes of a warp, which take the row's chunks of four entries in
// turn; the row's sums, in all its lanes. The next chunk of entries and the partners of the current one are in flight before
// any arithmetic starts; the list is streamed with an evict-first hint so that the positions stay in L2.
// Every listed pair is evaluated from the side of each of its owned atoms (a full list), so forces need no scatter and no
// atomics and the order of the sums is fixed (bitwise reproducible). Energy and virial take half of every directed entry;
// an owned-ghost pair is then counted half on each rank, as the reference's list kernel does
// (src/force_calculator_cuda.cu:1784-1789).
template <int COPIES, bool ENERGY, int TYPES, bool SWITCH, bool QTYPE, int ORDER>
__device__ __forceinline__ void row_forces(const PairParams& p, const ForceArgs& a, const PairTables<COPIES, ENERGY, TYPES, QTYPE>& tables,
                                           int t, const RowHead& head, float (&sum_a)[3], float (&sum_b)[3], double (&v)[6]) {
    constexpr bool COULOMB = COPIES > 0, few = TYPES == kFewTypes, many = TYPES == kManyTypes, by_type = COULOMB && QTYPE;
    constexpr bool two_types = TYPES == kTwoTypes;
    const int nt = p.ntypes, lanes = 1 << a.lane_shift, sub = t & (lanes - 1);
    const EwaldTable<COPIES>& table = tables.ewald;
    PairAccumulator<COPIES, ENERGY, SWITCH> acc;
    bool close = false;   // the row has a pair below the Ewald table
    bool two = false;     // the row has two atoms
    const int first = head.first, atoms = head.atoms;
    if (atoms > 0) {
        const int4 pa = a.pq[first], pb = a.pq[first + atoms - 1];
        const unsigned special = head.special;
        const uint4* row = row_chunks<ORDER>(a, head.pair, sub);
        F2 q{0};
        PairTerms one{};
        const int row3 = (pa.w * nt + pb.w) * nt;
        if (COULOMB && !(few && by_type))
            q = mul(both(p.kq), by_type ? f2(tables.charge[pa.w], tables.charge[pb.w]) : f2(a.qf[first], a.qf[first + atoms - 1]));
        if (TYPES == kOneType) {
            const float2 lj = p.lj[0];
            one.rep = both(lj.x);
            one.att = both(lj.y);
            if (by_type) one.qq = mul(q, both(tables.charge[0]));
        }
        // two types: what either asks for, in registers
        PairTerms of_type[2];
        if (two_types)
            for (int k = 0; k < 2; ++k) {
                const float2 la = p.lj[pa.w * 2 + k], lb = p.lj[pb.w * 2 + k];
                of_type[k].rep = f2(la.x, lb.x);
                of_type[k].att = f2(la.y, lb.y);
            }
        const auto take = [&](unsigned e, int4& pos, float& charge) {
            pos = a.pq[e];
            if (COULOMB && !by_type) charge = a.qf[e];
        };
        const auto terms = [&](int type, float charge) {
            PairTerms k = one;
            if (two_types) k = type ? of_type[1] : of_type[0];
            if (few) {
                const ulonglong2 lj = tables.lj3[row3 + type];
                k.rep.v = lj.x;
                k.att.v = lj.y;
                if (by_type) k.qq.v = tables.qq3[row3 + type];
            }
            if (many) {
                const float2 la = tables.lj2[pa.w * nt + type], lb = tables.lj2[pb.w * nt + type];
                k.rep = f2(la.x, lb.x);
                k.att = f2(la.y, lb.y);
            }
            if (COULOMB && by_type && many) k.qq = mul(q, both(tables.charge[type]));
            if (COULOMB && !by_type) k.qq = mul(q, both(charge));
            return k;
        };
        const auto add = [&](const int4& pos, float charge) {
            acc.template add_partner<false>(p, table, pa, pb, pos, terms(pos.w, charge), 0u);
        };
        int c = head.c;
        const int c_end = head.c_end;
        uint4 e = head.e;
        {   // the two atoms themselves: each is the other's partner
            two = atoms > 1;
            const bool own = two && a.phase != DSMD_PHASE_BOUNDARY && !(special & (kRowOwnExcluded | kRowCareful));
            float q_a = 0.0f, q_b = 0.0f;
            if (COULOMB && !by_type) { q_a = a.qf[first]; q_b = a.qf[first + atoms - 1]; }
            acc.add_own(p, table, pa, pb, terms(pb.w, q_b), terms(pa.w, q_a), own && sub == 0);
        }
        for (; c < c_end; c += lanes) {
            int4 p_x, p_y, p_z, p_w;
            float q_x, q_y, q_z, q_w;
            take(e.x, p_x, q_x);
            take(e.y, p_y, q_y);
            take(e.z, p_z, q_z);
            take(e.w, p_w, q_w);
            if (c + lanes < c_end) e = __ldcs(row + ((c + lanes) >> ORDER) * size_t(32));
            add(p_x, q_x);
            add(p_y, q_y);
            add(p_z, q_z);
            add(p_w, q_w);
        }
        // What needs care, an entry per lane: excluded partners, and all entries of a row with a pair that coincides (there is
        // none in a sane system), the two atoms' own with them.
        const unsigned row_lanes = (lanes == 32 ? 0xFFFFFFFFu : (1u << lanes) - 1u) << (threadIdx.x & 31 & -lanes);
        // (one vote per row as a rule)
        bool suspect;
        if (!COULOMB && !ENERGY) {   // r^2 < 1e-10: r^-8 is infinite, and so, or no number, is what any parameters make of it
            float s[6];
            parts(acc.ax, s[0], s[1]);
            parts(acc.ay, s[2], s[3]);
            parts(acc.az, s[4], s[5]);
            suspect = !(fabsf(s[0] + s[1]) + fabsf(s[2] + s[3]) + fabsf(s[4] + s[5]) < 3.0e38f);
        } else {
            suspect = acc.least < (COULOMB ? kEwaldFirst : 1e-10f);
        }
        bool again = __any_sync(row_lanes, suspect || (special & kRowCareful));
        if (COULOMB && again) {
            again = __any_sync(row_lanes, acc.least < 1e-10f || (special & kRowCareful));
            close = !again;
        }
        if (again || (special & ((kRowCountMask << kRowCountBits) | kRowCountMask))) {
            const int t2 = afresh(t), pair = row_of_thread(a, t2);
            int first;
            const int atoms = pair_atoms(a.rows.quad, pair, first);
            const int mid = a.rows.row_int[pair], end = max(mid, a.rows.row_end[pair]), ghosts = whole_groups<ORDER>(mid);
            const unsigned* words = a.rows.rows + row_base<ORDER>(static_cast<unsigned>(pair), a.rows.stride);
            if (again) acc = PairAccumulator<COPIES, ENERGY, SWITCH>();
            const bool interior = a.phase != DSMD_PHASE_BOUNDARY, boundary = a.phase != DSMD_PHASE_INTERIOR;
            const int ex_own = special & kRowCountMask, ex_all = ex_own + static_cast<int>((special >> kRowCountBits) & kRowCountMask);
            const int x0 = interior ? 0 : ex_own, x1 = boundary ? ex_all : ex_own;
            const int n_own = again && atoms > 1 && interior && !(special & kRowOwnExcluded) ? 2 : 0;
            const int n_first = interior ? mid : 0, n_second = boundary ? max(end - ghosts, 0) : 0;
            const int n_care = n_own + (x1 - x0) + (again ? n_first + n_second : 0);
#pragma unroll 1
            for (int i = t2 & (lanes - 1); i < n_care; i += lanes) {
                const int x = i - n_own, k = x - (x1 - x0);
                unsigned e = static_cast<unsigned>(first + i);
                if (x >= 0) e = words[row_offset<ORDER>(k < 0 ? a.rows.stride - 1 - (x0 + x) : (k < n_first ? k : ghosts + k - n_first))];
                int4 pj;
                float qj = 0.0f;
                take(e & kIndexMask, pj, qj);
                acc.template add_partner<true>(p, table, pa, pb, pj, terms(pj.w, qj), e);
            }
        }
    }
    // Rows with a pair below the Ewald table, one after the other by the whole warp, an entry per lane. A warp has such a row now
    // and then (a box of 648,000 water atoms, started from jittered places, has 15 such pairs), and one lane on its own would keep
    // the others, and in a grid of one round the device, waiting for hundreds of entries: 1.56 ms for that box with the row done
    // again by its lane, 1.14 this way, when a box without such pairs took 1.12 (1.53 with a row per atom and a branch per pair).
    if (COULOMB)
        for (unsigned todo = __ballot_sync(0xFFFFFFFFu, close && sub == 0); todo; todo &= todo - 1) {
            const int leader = __ffs(todo) - 1;
            const int its_row = row_of_thread(a, afresh(t));
            const auto rest = close_rest<COPIES, ENERGY, SWITCH, by_type, ORDER>(p, a, table, __shfl_sync(0xFFFFFFFFu, its_row, leader));
            if ((threadIdx.x & 31) == leader) acc.add_sums(rest);
        }
    if (ENERGY) acc.take_energies(two, v);   // a lone atom's sums are in both lanes; no atom: zeros
    acc.take_forces(sum_a, sum_b);
    // (From near to far or the other way, at the same cost; the last bits, and with them the path that a long run takes, are others. Its
    // energy drift is not: over 400 starts of 32,000 atoms 0.9e-5 +- 0.3e-5 and 1.1e-5 +- 0.3e-5 per atom and 10,000 steps.)
    for (int o = 1; o < lanes; o <<= 1) {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            sum_a[k] += __shfl_xor_sync(0xFFFFFFFFu, sum_a[k], o);
            sum_b[k] += __shfl_xor_sync(0xFFFFFFFFu, sum_b[k], o);
        }
    }
}

// QTYPE: charges by type (dsmd_set_type_charges): the partner's charge comes out of a table in shared memory, indexed by
// the type that arrives with its position, instead of a second gather from global memory.
// With Coulomb the blocks stay and take further rows in turn, so that the Ewald tables are laid out once per block; with
// energy sums, so that the last block has few partial sums to add up.
template <int COPIES, bool ENERGY, int TYPES, bool SWITCH, bool QTYPE, int ORDER>
__global__ void __launch_bounds__((kPairThreads<COPIES, TYPES>), (kPairBlocks<COPIES, TYPES, ENERGY>)) k_pair(PairParams p, ForceArgs a) {
    extern __shared__ float4 smem[];
    const PairTables<COPIES, ENERGY, TYPES, QTYPE> tables(p, smem);   // parameters: no kernel writes them
    const int t0 = blockIdx.x * blockDim.x + threadIdx.x;
    RowHead head{};
    if (a.list_settled) head = open_row<ORDER>(a, t0);   // while the launch before this one ends
    if (!dsmd::after_previous() || (!ENERGY && dsmd::gate_closed(a.st, a.gate2))) return;
    double v[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};   // energy, virial and its diagonal, pairs
    for (int t = t0; (t & ~31) >> a.lane_shift < a.n_pairs; t += gridDim.x * blockDim.x) {
        if (t != t0 || !a.list_settled) head = open_row<ORDER>(a, t);
        float sum_a[3], sum_b[3];
        row_forces<COPIES, ENERGY, TYPES, SWITCH, QTYPE, ORDER>(p, a, tables, t, head, sum_a, sum_b, v);
        const int t2 = afresh(t), pair = row_of_thread(a, t2), sub = t2 & ((1 << a.lane_shift) - 1);
        int first = 0;
        const int atoms = pair >= 0 ? pair_atoms(a.rows.quad, pair, first) : 0;
        if (sub == 0 && atoms > 0) {
            double* const out[3] = {a.fx, a.fy, a.fz};
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                double* f = out[k] + first;
                if (a.phase == DSMD_PHASE_BOUNDARY) {
                    f[0] += static_cast<double>(sum_a[k]);
                    if (atoms > 1) f[1] += static_cast<double>(sum_b[k]);
                } else {
                    f[0] = static_cast<double>(sum_a[k]);
                    if (atoms > 1) f[1] = static_cast<double>(sum_b[k]);
                }
            }
        }
        if (COPIES == 0 && !ENERGY) break;   // one row per lane group: the grid covers all
    }
    if (ENERGY) sum_over_grid<6>(v, a.partials, a.ticket, a.scalars, a.phase == DSMD_PHASE_BOUNDARY, a.mail, a.seq);
}

// The force pass of a step and what follows it up to the next force pass, for loops in which nobody reads forces or
// velocities in between: v += kick f / m, x += dt v, fixed-point positions of the next step (into the other buffer: rows
// still read this one's), displacement check. A separate pass would read and write the forces and read everything else again
// (172 bytes per atom, 0.11 ms at 4,000,000 atoms beside 0.356 for the forces; this kernel 0.441, the blocks' ends being little
// hidden by other blocks' force arithmetic), and a small system's step is one launch.
template <int TYPES, bool SWITCH, int ORDER>
__global__ void __launch_bounds__((kPairThreads<0, TYPES>), (kPairBlocks<0, TYPES, false>))
k_step(PairParams p, ForceArgs a, Grid g, StepArgs at, DisplacementReport report) {
    extern __shared__ float4 smem[];
    const PairTables<0, false, TYPES, false> tables(p, smem);   // parameters: no kernel writes them
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    RowHead head{};
    if (a.list_settled) head = open_row<ORDER>(a, t);   // while the launch before this one ends
    if (!dsmd::after_previous() || dsmd::gate_closed(report.st, report.gate2)) return;
    if (!a.list_settled) head = open_row<ORDER>(a, t);
    float sum_a[3], sum_b[3];
    double unused[6];
    row_forces<0, false, TYPES, SWITCH, false, ORDER>(p, a, tables, t, head, sum_a, sum_b, unused);
    const int t2 = afresh(t), pair = row_of_thread(a, t2), sub = t2 & ((1 << a.lane_shift) - 1);
    int first = 0;
    const int atoms = pair >= 0 ? pair_atoms(a.rows.quad, pair, first) : 0;
    // The atoms' turn: an atom per thread, neighbours side by side. (Two atoms by the lanes that hold their sums is four times
    // the instructions where rows have many lanes: 24.5 us per step of 32,000 atoms, 20.7 us this way.)
    __shared__ float s_force[2 * kPairThreads<0, TYPES>][3];
    __shared__ int s_slot[2 * kPairThreads<0, TYPES>];
    const int rows_here = blockDim.x >> a.lane_shift;
    if (sub == 0) {
        const int at2 = 2 * (threadIdx.x >> a.lane_shift);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            s_force[at2][k] = sum_a[k];
            s_force[at2 + 1][k] = sum_b[k];
        }
        s_slot[at2] = atoms > 0 ? first : -1;
        s_slot[at2 + 1] = atoms > 1 ? first + 1 : -1;
    }
    __syncthreads();
    double worst2 = 0.0;
    for (int t = threadIdx.x; t < 2 * rows_here; t += blockDim.x) {
        const int s = s_slot[t];
        if (s < 0) continue;
        const double h = at.kick / at.mass[s];
        const double ux = at.vx[s] + h * static_cast<double>(s_force[t][0]);
        const double uy = at.vy[s] + h * static_cast<double>(s_force[t][1]);
        const double uz = at.vz[s] + h * static_cast<double>(s_force[t][2]);
        const double px = at.x[s] + at.dt * ux, py = at.y[s] + at.dt * uy, pz = at.z[s] + at.dt * uz;
        at.vx[s] = ux; at.vy[s] = uy; at.vz[s] = uz;
        at.x[s] = px; at.y[s] = py; at.z[s] = pz;
        unsigned bad = 0;
        int4 f;
        f.x = static_cast<int>(dsmd::to_fixed(px, 0, g, bad));
        f.y = static_cast<int>(dsmd::to_fixed(py, 1, g, bad));
        f.z = static_cast<int>(dsmd::to_fixed(pz, 2, g, bad));
        f.w = a.pq[s].w;
        at.pq_next[s] = f;
        if (bad) atomicAdd(&report.st->out_of_domain, 1u);
        const double dx = px - at.xref[s], dy = py - at.yref[s], dz = pz - at.zref[s];
        const double d2 = dx * dx + dy * dy + dz * dz;
        worst2 = fmax(worst2, d2 == d2 ? d2 : __longlong_as_double(0x7FF0000000000000ll));   // see k_pack
    }
    report_displacement(worst2, report);
}

}  // namespace

namespace dsmd {

template <int COPIES, bool ENERGY, int ORDER>
cudaError_t launch_pair(const PairParams& p, const ForceArgs& a, bool sw, unsigned blocks, bool overlap, cudaStream_t s) {
    const auto launch = [&](auto types, auto switched, auto qtype) {
        constexpr int TYPES = decltype(types)::value;
        constexpr bool SWITCH = decltype(switched)::value, QTYPE = decltype(qtype)::value;
        const size_t smem = PairTables<COPIES, ENERGY, TYPES, QTYPE>::bytes(p.ntypes, p.ewald_intervals);
        const auto kernel = k_pair<COPIES, ENERGY, TYPES, SWITCH, QTYPE, ORDER>;
        if (smem > 48 * 1024) {
            const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
            if (e != cudaSuccess) return e;
        }
        return launch_next_if(overlap, kernel, blocks, kPairThreads<COPIES, TYPES>, smem, s, p, a);
    };
    const auto by_charge = [&](auto types, auto switched) {   // charges by type: only the kernels with Coulomb have this form
        if (COPIES > 0 && p.type_charge) return launch(types, switched, std::integral_constant<bool, (COPIES > 0)>());
        return launch(types, switched, std::false_type());
    };
    const auto by_switch = [&](auto types) { return sw ? by_charge(types, std::true_type()) : by_charge(types, std::false_type()); };
    if (p.ntypes == 1) return by_switch(std::integral_constant<int, kOneType>());
    if (COPIES == 0 && p.ntypes == 2) return by_switch(std::integral_constant<int, COPIES == 0 ? kTwoTypes : kFewTypes>());
    if (p.ntypes <= kFewTypesMost) return by_switch(std::integral_constant<int, kFewTypes>());
    return by_switch(std::integral_constant<int, kManyTypes>());
}

template <int ORDER>
cudaError_t launch_step(const PairParams& p, const ForceArgs& a, const Grid& g, const StepArgs& at, const DisplacementReport& report, bool sw,
                        unsigned blocks, cudaStream_t s) {
    const auto launch = [&](auto types) {
        constexpr int TYPES = decltype(types)::value;
        const size_t smem = PairTables<0, false, TYPES, false>::bytes(p.ntypes, 0);
        const auto kernel = sw ? k_step<TYPES, true, ORDER> : k_step<TYPES, false, ORDER>;
        return launch_next(kernel, blocks, kPairThreads<0, TYPES>, smem, s, p, a, g, at, report);
    };
    if (p.ntypes == 1) return launch(std::integral_constant<int, kOneType>());
    if (p.ntypes == 2) return launch(std::integral_constant<int, kTwoTypes>());
    if (p.ntypes <= kFewTypesMost) return launch(std::integral_constant<int, kFewTypes>());
    return launch(std::integral_constant<int, kManyTypes>());
}

}  // namespace dsmd
