// move_impl.cuh -- field interpolation and particle pushers of both movers.
//
// The selected ParticlePusher and FieldWeigthing of PICParcel::move
// (PICMCCFVM/parcels/Templates/PICParcel/PICParcel.C:38-144).  Instantiated
// twice: Real = double in move_fp64.cu (built with --fmad=false, evaluation
// order identical to the CPU oracle, so the FP64 form is bit-exact) and
// Real = float in move_fp32.cu (the mixed form).
#pragma once

#include "common.cuh"

namespace pgd {

// Per-precision access to the species and field constants.  The FP64 form
// evaluates q dt/2 / m exactly as the oracle does; the FP32 form uses the
// host-rounded float copies.
template <class Real> struct PC;
template <> struct PC<double> {
    static __device__ __forceinline__ double B(const MoveParams& P, int a) { return P.B[a]; }
    // the parcel's charge is the species charge times its charge modifier zf
    // (PICCloud.C:368); zf = 1 leaves q dt/2 / m as it is.  The two values of a
    // whole step come from the host (an FP64 division is some ten issues of
    // 64 cycles); the compares are of bits, off the FP64 pipe.
    static __device__ __forceinline__ double qdm(const MoveParams& P, double half_dt, double zf) {
        if (__double_as_longlong(zf) == __double_as_longlong(1.0)) {
            if (__double_as_longlong(half_dt) == __double_as_longlong(P.half_dt)) return P.qdm_half;
            if (__double_as_longlong(half_dt) == __double_as_longlong(P.dt)) return P.qdm_full;
        }
        return P.q * zf * half_dt / P.mass;
    }
};
template <> struct PC<float> {
    static __device__ __forceinline__ float B(const MoveParams& P, int a) { return P.B_f[a]; }
    static __device__ __forceinline__ float qdm(const MoveParams& P, float half_dt, float zf) {
        return P.qm_f * zf * half_dt;
    }
};

template <class Real>
__device__ __forceinline__ Real dot3(const Real* a, const Real* b) {
    return a[0] * b[0] + a[1] * b[1] + a[2] * b[2];
}
template <class Real>
__device__ __forceinline__ void cross3(const Real* a, const Real* b, Real* o) {
    o[0] = a[1] * b[2] - a[2] * b[1];
    o[1] = a[2] * b[0] - a[0] * b[2];
    o[2] = a[0] * b[1] - a[1] * b[0];
}

// sqrt(x) / c for x >= 0, the divisor known in advance (Markstein 1990; Cornea,
// Harrison, Tang 2002): 1 / c rounded to nearest is within 0.19 2^-53 of 1 / c,
// so v (1 / c) is less than one ulp off, its remainder is exact (a root is 0 or
// above 2^-538) and one correction rounds the quotient correctly: the bits of
// v / c from three FP64 instructions instead of some nine.
__device__ __forceinline__ double root_over_c(double x) {
    constexpr double r = 1.0 / kC;
    const double v = sqrt(x);
    if ((__double2hiint(v) & 0x7ff00000) == 0x7ff00000) return v / kC;
    const double q = v * r;
    return __fma_rn(__fma_rn(-q, kC, v), r, q);
}
__device__ __forceinline__ float root_over_c(float x) { return sqrt(x) / float(kC); }

template <class Real>
struct PState {
    int cell, tet;
    Real y[4];
    Real U[3];
    Real zf;      // charge modifier (1 without per-parcel attributes)
    double nw;    // nParticle (the species weight without per-parcel attributes)
};

// The parcel's charge modifier and weight: per parcel when the store has
// the arrays, else 1 and the species weight.
template <class Real>
__device__ __forceinline__ void load_attributes(const MoveParams& P, int i, PState<Real>& s) {
    if (P.p.nw) {
        s.zf = Real(P.p.zq[i]);
        s.nw = P.p.nw[i];
    } else {
        s.zf = Real(1);
        s.nw = P.weight;
    }
}

template <class Real> __device__ __forceinline__ const Real* e_cell(const MoveParams& P);
template <> __device__ __forceinline__ const double* e_cell<double>(const MoveParams& P) { return P.E; }
template <> __device__ __forceinline__ const float* e_cell<float>(const MoveParams& P) { return P.E32; }
template <class Real> __device__ __forceinline__ const Real* e_point(const MoveParams& P);
template <> __device__ __forceinline__ const double* e_point<double>(const MoveParams& P) { return P.Ept; }
template <> __device__ __forceinline__ const float* e_point<float>(const MoveParams& P) { return P.Ept32; }

// FieldWeigthing::getFieldVector: VolumeWeighting (VolumeWeightingFW.C:60-67)
// interpolates cell centre + three triangle points; CellAverage
// (CellAverageFW.C:58-65) returns the cell value.
template <class Real>
__device__ __forceinline__ void field_at(const MoveParams& P, const TetConst& T,
                                         const PState<Real>& s, Real* E) {
    const Real* Ec = e_cell<Real>(P) + 3 * size_t(s.cell);
    if (P.field_weighting == PICGPU_WEIGHTING_CELL_AVERAGE) {
        E[0] = Ec[0]; E[1] = Ec[1]; E[2] = Ec[2];
        return;
    }
    const int* cp = P.m.cell_pt + 8 * size_t(s.cell);
    const Real* Ep = e_point<Real>(P);
    const Real* e1 = Ep + 3 * size_t(cp[T.tri[s.tet][0]]);
    const Real* e2 = Ep + 3 * size_t(cp[T.tri[s.tet][1]]);
    const Real* e3 = Ep + 3 * size_t(cp[T.tri[s.tet][2]]);
#pragma unroll
    for (int a = 0; a < 3; ++a)
        E[a] = Ec[a] * s.y[0] + e1[a] * s.y[1] + e2[a] * s.y[2] + e3[a] * s.y[3];
}

// BorisPusher::updateVelocity (submodels/ParticlePusher/BorisPusher/BorisPusher.C:69-112)
template <class Real>
__device__ __forceinline__ void push_boris(const MoveParams& P, const Real* E, const Real* Bv, Real* U, Real tt,
                                      Real zf) {
    const Real dt2 = Real(0.5) * tt;
    const Real mU = root_over_c(dot3(U, U));
    const Real g0 = sqrt(Real(1) - mU * mU);
    Real rU[3] = {U[0] / g0, U[1] / g0, U[2] / g0};
    const Real oldrU[3] = {rU[0], rU[1], rU[2]};
    const Real qdm = PC<Real>::qdm(P, dt2, zf);
    const Real rUsm[3] = {qdm * E[0], qdm * E[1], qdm * E[2]};
    rU[0] = rU[0] + rUsm[0]; rU[1] = rU[1] + rUsm[1]; rU[2] = rU[2] + rUsm[2];
    if (P.rotation) {
        const Real a0 = root_over_c(dot3(oldrU, oldrU)), a1 = root_over_c(dot3(rU, rU));
        const Real lF = (sqrt(Real(1) + a0 * a0) + sqrt(Real(1) + a1 * a1)) / Real(2);
        const Real t[3] = {qdm * Bv[0] / lF, qdm * Bv[1] / lF, qdm * Bv[2] / lF};
        Real cr[3];
        cross3(rU, t, cr);
        const Real Ud[3] = {rU[0] + cr[0], rU[1] + cr[1], rU[2] + cr[2]};
        const Real den = Real(1) + dot3(t, t);
        const Real sv[3] = {Real(2) * t[0] / den, Real(2) * t[1] / den, Real(2) * t[2] / den};
        cross3(Ud, sv, cr);
        rU[0] = rU[0] + cr[0]; rU[1] = rU[1] + cr[1]; rU[2] = rU[2] + cr[2];
    }
    rU[0] = rU[0] + rUsm[0]; rU[1] = rU[1] + rUsm[1]; rU[2] = rU[2] + rUsm[2];
    const Real mr = root_over_c(dot3(rU, rU));
    const Real g1 = sqrt(Real(1) + mr * mr);
    U[0] = rU[0] / g1; U[1] = rU[1] / g1; U[2] = rU[2] / g1;
}

// BorisNRPusher::updateVelocity (BorisNRPusher.C:69-99)
template <class Real>
__device__ __forceinline__ void push_boris_nr(const MoveParams& P, const Real* E, const Real* Bv, Real* U, Real tt,
                                      Real zf) {
    const Real dt2 = Real(0.5) * tt;
    const Real alpha = PC<Real>::qdm(P, dt2, zf);
    Real W[3] = {U[0] + alpha * E[0], U[1] + alpha * E[1], U[2] + alpha * E[2]};
    if (P.rotation) {
        const Real t[3] = {alpha * Bv[0], alpha * Bv[1], alpha * Bv[2]};
        Real cr[3];
        cross3(W, t, cr);
        const Real Ud[3] = {W[0] + cr[0], W[1] + cr[1], W[2] + cr[2]};
        const Real den = Real(1) + dot3(t, t);
        const Real sv[3] = {Real(2) * t[0] / den, Real(2) * t[1] / den, Real(2) * t[2] / den};
        cross3(Ud, sv, cr);
        W[0] = W[0] + cr[0]; W[1] = W[1] + cr[1]; W[2] = W[2] + cr[2];
    }
    U[0] = W[0] + alpha * E[0]; U[1] = W[1] + alpha * E[1]; U[2] = W[2] + alpha * E[2];
}

// VayPusher::updateVelocity (VayPusher.C:54-100); U x T uses v (VayPusher.C:81).
template <class Real>
__device__ __forceinline__ void push_vay(const MoveParams& P, const Real* E, const Real* Bv, Real* U, Real tt,
                                      Real zf) {
    const Real c = Real(kC);
    const Real dt2 = Real(0.5) * tt;
    const Real mU = root_over_c(dot3(U, U));
    const Real lF = Real(1) / sqrt(Real(1) - mU * mU);
    const Real rU0[3] = {lF * U[0], lF * U[1], lF * U[2]};
    const Real qe = PC<Real>::qdm(P, tt, zf);
    Real Ud[3] = {rU0[0] + qe * E[0], rU0[1] + qe * E[1], rU0[2] + qe * E[2]};
    const Real qb = PC<Real>::qdm(P, dt2, zf);
    Real T[3] = {qb * Bv[0], qb * Bv[1], qb * Bv[2]};
    Real cr[3];
    cross3(U, T, cr);
    Ud[0] = Ud[0] + cr[0]; Ud[1] = Ud[1] + cr[1]; Ud[2] = Ud[2] + cr[2];
    const Real mUd = root_over_c(dot3(Ud, Ud));
    Real alpha = Real(1) + mUd * mUd;
    const Real T2 = dot3(T, T);
    Real s = alpha - T2;
    const Real udt = dot3(Ud, T) / c;
    const Real us2 = udt * udt;
    alpha = Real(1) / sqrt(Real(0.5) * (s + sqrt(s * s + Real(4) * (T2 + us2))));
    T[0] = alpha * T[0]; T[1] = alpha * T[1]; T[2] = alpha * T[2];
    s = Real(1) / (Real(1) + dot3(T, T));
    alpha = dot3(Ud, T);
    cross3(Ud, T, cr);
    Real rU[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) rU[a] = s * ((Ud[a] + alpha * T[a]) + cr[a]);
    const Real mr = root_over_c(dot3(rU, rU));
    const Real g1 = sqrt(Real(1) + mr * mr);
    U[0] = rU[0] / g1; U[1] = rU[1] / g1; U[2] = rU[2] / g1;
}

// HigueraCaryPusher::updateVelocity (HigueraCary.C:69-115)
template <class Real>
__device__ __forceinline__ void push_hc(const MoveParams& P, const Real* E, const Real* Bv, Real* U, Real tt,
                                      Real zf) {
    const Real dt2 = Real(0.5) * tt;
    const Real mU = root_over_c(dot3(U, U));
    const Real g0 = sqrt(Real(1) - mU * mU);
    Real rU[3] = {U[0] / g0, U[1] / g0, U[2] / g0};
    const Real qdm = PC<Real>::qdm(P, dt2, zf);
    const Real rUsm[3] = {qdm * E[0], qdm * E[1], qdm * E[2]};
    rU[0] = rU[0] + rUsm[0]; rU[1] = rU[1] + rUsm[1]; rU[2] = rU[2] + rUsm[2];
    if (P.rotation) {
        const Real mr0 = root_over_c(dot3(rU, rU));
        const Real gfm2 = Real(1) + mr0 * mr0;
        Real t[3] = {qdm * Bv[0], qdm * Bv[1], qdm * Bv[2]};
        const Real beta2 = dot3(t, t);
        const Real gb = gfm2 - beta2;
        const Real tr = dot3(t, rU);
        const Real iG = Real(1) / sqrt(Real(0.5) * (gb + sqrt(gb * gb + Real(4) * (beta2 + tr * tr))));
        t[0] = iG * t[0]; t[1] = iG * t[1]; t[2] = iG * t[2];
        Real cr[3];
        cross3(rU, t, cr);
        const Real Ud[3] = {rU[0] + cr[0], rU[1] + cr[1], rU[2] + cr[2]};
        const Real den = Real(1) + dot3(t, t);
        const Real sv[3] = {Real(2) * t[0] / den, Real(2) * t[1] / den, Real(2) * t[2] / den};
        cross3(Ud, sv, cr);
        rU[0] = rU[0] + cr[0]; rU[1] = rU[1] + cr[1]; rU[2] = rU[2] + cr[2];
    }
    rU[0] = rU[0] + rUsm[0]; rU[1] = rU[1] + rUsm[1]; rU[2] = rU[2] + rUsm[2];
    const Real mr = root_over_c(dot3(rU, rU));
    const Real g1 = sqrt(Real(1) + mr * mr);
    U[0] = rU[0] / g1; U[1] = rU[1] / g1; U[2] = rU[2] / g1;
}

// The magnetic field the pushers use: the cell value (B[celli], as every
// picFoam pusher reads it, e.g. BorisPusher.C:100) when a per-cell field is
// set, else the uniform one.
template <class Real>
__device__ __forceinline__ void cell_B(const MoveParams& P, int cell, Real* Bv) {
    if (P.Bc) {
#pragma unroll
        for (int a = 0; a < 3; ++a) Bv[a] = Real(P.Bc[3 * size_t(cell) + a]);
    } else {
#pragma unroll
        for (int a = 0; a < 3; ++a) Bv[a] = PC<Real>::B(P, a);
    }
}

template <class Real>
__device__ __forceinline__ void push(const MoveParams& P, const TetConst& T, PState<Real>& s, Real tt) {
    if (P.pusher == PICGPU_PUSHER_NONE) return;
    Real E[3], Bv[3];
    field_at(P, T, s, E);
    cell_B(P, s.cell, Bv);
    switch (P.pusher) {
        case PICGPU_PUSHER_BORIS: push_boris(P, E, Bv, s.U, tt, s.zf); break;
        case PICGPU_PUSHER_BORIS_NR: push_boris_nr(P, E, Bv, s.U, tt, s.zf); break;
        case PICGPU_PUSHER_VAY: push_vay(P, E, Bv, s.U, tt, s.zf); break;
        default: push_hc(P, E, Bv, s.U, tt, s.zf); break;
    }
}

template <class Real> __device__ __forceinline__ Real* ybuf(const DSpecies& p, int a);
template <> __device__ __forceinline__ double* ybuf<double>(const DSpecies& p, int a) { return p.y64[a]; }
template <> __device__ __forceinline__ float* ybuf<float>(const DSpecies& p, int a) { return p.y32[a]; }
template <class Real> __device__ __forceinline__ Real* ubuf(const DSpecies& p, int a);
template <> __device__ __forceinline__ double* ubuf<double>(const DSpecies& p, int a) { return p.u64[a]; }
template <> __device__ __forceinline__ float* ubuf<float>(const DSpecies& p, int a) { return p.u32[a]; }

template <class Real>
__device__ __forceinline__ void warp_add_counter(unsigned long long* dst, unsigned v) {
    unsigned long long x = v;
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1) x += __shfl_xor_sync(0xffffffffu, x, off);
    if ((threadIdx.x & 31) == 0 && x) atomicAdd(dst, x);
}

}  // namespace pgd
