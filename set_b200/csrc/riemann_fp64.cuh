// riemann_fp64.cuh -- the plain form's FP64 HLLD / HLLC flux and MUSCL face states, written for the
// instruction budget of the stage kernel, which is bound by instruction issue and the latency of
// dependent FP64 operations (FP64 pipe 44-46 % busy, issue 53-54 %, HBM 21-29 % at 256^3).  With it the kernel
// issues 61-63 warp instructions per cell and stage instead of 84-86 (825-834 FP64 operations per cell
// instead of 1006-1016): 256^3 stage 1 / 2 2.04 / 2.15 -> 1.64 / 1.77 ms, and 2.31 / 2.44 ms with the former
// tile split; field-free HLLC 203x117x161 0.538 / 0.586 -> 0.390 / 0.430 ms.
//
// The same formulas and the same wave-fan selection as riemann<double, NSTATE, false, false, true,
// true> in mhd_core.cuh (chlld, SET_Fortran_Cuda_MHD/Solvers.f90:1190-1855, face speed 0, n_disc 0),
// on states that carry b = B / sqrt(4 pi), with these differences, each exact in real arithmetic:
//   * fast speeds from cf^2 = (A + sqrt(D^2 + gamma p bt^2)) / rho, A, D = (gamma p +- |b|^2)/2,
//     bt the tangential field: the discriminant is a sum of squares (no cancellation; sqrt_ratio for p <= 0), and
//     cf = S / sqrt(rho S) needs no reciprocal of rho: 22 FP64 operations a side instead of 31;
//   * products the star states, contact speed and total pressure share (rho (S - u)) formed once;
//   * the wave-fan region from the sign of SM and the selected side's speeds: with ordered speeds
//     the chain of :1722-1814 (last match wins) is  SM <= 0: FR if SR < 0, R* if SZR <= 0, else
//     R**;  SM > 0: L** if SZL <= 0, L* if SL <= 0, else FL  (|bn| <= epsb sets SZL = SZR = SM);
//   * both single-star states are formed wherever a star region is selected (no nested branches),
//     the double-star differences vanish for rho and rho vn and are not formed, and the double
//     star is formed relative to the single stars (four FMAs a component);
//   * the B fluxes are returned in units of b (the caller's update scales by sqrt(4 pi) once).
#pragma once
#include "mhd_core.cuh"

namespace sb {

// Approximate 1/sqrt(x) (relative error ~1e-6), refined by the callers with one third-order step
// (see rs_rsqrt).
__device__ __forceinline__ double rsqrt_seed(double x) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    return y;
}
// a / sqrt(x) for x > 0: five FP64 operations more than the seed.  With a = x it is sqrt(x).
__device__ __forceinline__ double over_sqrt(double a, double x) {
    const double y = rsqrt_seed(x);
    const double e = fma(-x * y, y, 1.0);
    const double g = a * y;
    return fma(g * e, fma(0.375, e, 0.5), g);
}
// sqrt(x / y) for y > 0, and 0 for an x below about 2e-99, zero and negative too: a pressure that its
// recovery rounded below zero (kinetic energy above ~1e9 times the floor) is taken as none, as riemann()'s
// clamped square roots do.  A side without pressure and field has a speed of exactly 0: the faces between
// such sides at rest, which have no region, are told by it.  A NaN of either sign stays one, so the faces
// of an invalid state are found.  Below the line the reciprocal square root gets 2^-328 (a finite seed; its
// low word is that of 0, so the numerator costs one select more: 256^3 Heun 20.91 ms for six steps,
// 20.80 without).
__device__ __forceinline__ double sqrt_ratio(double x, double y) {
    const bool none = x < 0x1p-328;
    return over_sqrt(none ? 0.0 : x, y * (none ? 0x1p-328 : x));
}
__device__ __forceinline__ double pick(double l, double r, bool right) { return right ? r : l; }

// MUSCL-minmod slope halves: q = t_c +- h m with m the argument of smaller magnitude and h = 1/2, or
// 0 where the signs differ (one selected word instead of two; minmod() of mhd_core.cuh otherwise).
// One FP64 compare instead of minmod's 64-bit integer compare: two issue slots fewer, and a slope
// is used for both of its faces' values where a caller has both.  An a that is no
// number gives b (the far cell's difference comes first); a b that is none stays (face_values_bad).
__device__ __forceinline__ double slope(double a, double b, double& h) {
    h = (__double2hiint(a) ^ __double2hiint(b)) < 0 ? 0.0 : 0.5;
    return fabs(a) < fabs(b) ? a : b;
}

// Whether a pair of face states needs its cells' values: a negative density or pressure
// (cuf_solvers.cuf:394-406), or a neighbour that is no valid state (a cell's pressure is NaN where any of
// its conserved variables is, so the pressures show it).
__device__ __forceinline__ bool face_values_bad(double r1, double p1, double r2, double p2) {
    const unsigned r = max((unsigned)__double2hiint(r1), (unsigned)__double2hiint(r2));
    const unsigned p = max((unsigned)__double2hiint(p1), (unsigned)__double2hiint(p2));
    return max(r, p) >= 0x7ff00000u;   // the sign bit, or the exponent of infinities and NaNs
}
// Component v (0 density, 4 pressure) of such a state: the cell's value c instead of x.
__device__ __forceinline__ double mend_face_value(int v, double x, double c) {
    return (v == 0 || v == 4 ? x >= 0.0 : x == x) ? x : c;
}

// Face states from the 4-cell stencil (face-frame order; reconstruct() of mhd_core.cuh): second
// order in rho, v, p with the positivity fallback of cuf_solvers.cuf:394-406, B first order.  cell(s, v)
// gives component v of the left (s = 0) or right cell once more.
template <int ORDER, typename Cell>
__device__ __forceinline__ void reconstruct_fp64(const double* qLL, const double* qL, const double* qR,
                                                 const double* qRR, double* q1, double* q2, Cell cell) {
#pragma unroll
    for (int v = 0; v < 8; v++) {
        q1[v] = qL[v];
        q2[v] = qR[v];
    }
    if (ORDER == 2) {
#pragma unroll
        for (int v = 0; v < 5; v++) {
            const double d = qR[v] - qL[v];
            double h;
            const double m1 = slope(qL[v] - qLL[v], d, h);
            q1[v] = fma(h, m1, qL[v]);
            const double m2 = slope(qRR[v] - qR[v], d, h);
            q2[v] = fma(-h, m2, qR[v]);
        }
        if (face_values_bad(q1[0], q1[4], q2[0], q2[4])) {
#pragma unroll
            for (int v = 0; v < 5; v++) {
                q1[v] = mend_face_value(v, q1[v], cell(0, v));
                q2[v] = mend_face_value(v, q2[v], cell(1, v));
            }
        }
    }
}

// x, or about 1e-200 where x is below that (zero and negative too).  It keeps the seed of a reciprocal
// square root finite where the discriminant is zero, by one integer maximum of the high word, for an x
// whose NaN the caller's result shows by another operand: a NaN with its sign bit set counts as negative
// here.
__device__ __forceinline__ double at_least_tiny_bits(double x) {
    return __hiloint2double(max(__double2hiint(x), 0x16687e92), __double2loint(x));
}

// Fast magnetosonic speed, total pressure pt = p + |b|^2/2.
__device__ __forceinline__ double fast_speed(const double* q, double& pt) {
    const double bt2 = fma(q[7], q[7], q[6] * q[6]);
    const double b2 = fma(q[5], q[5], bt2);
    const double hp = (0.5 * kGamma) * q[4];
    const double A = fma(0.5, b2, hp), D = fma(-0.5, b2, hp);
    const double disc = at_least_tiny_bits(fma(2.0, hp * bt2, D * D));
    pt = fma(0.5, b2, q[4]);
    return sqrt_ratio(A + over_sqrt(disc, disc), q[0]);   // A is NaN where p or the field is
}

// Physical flux of a state with energy e and total pressure pt (no normal-field component).
__device__ __forceinline__ void phys_flux(double r, double u, double v, double w, double bx, double by, double bz,
                                          double e, double pt, double sbv, double* F) {
    const double m = r * u;
    F[0] = m;
    F[1] = fma(m, u, fma(-bx, bx, pt));
    F[2] = fma(m, v, -(bx * by));
    F[3] = fma(m, w, -(bx * bz));
    F[4] = fma(e + pt, u, -(bx * sbv));
    F[6] = fma(u, by, -(v * bx));
    F[7] = fma(u, bz, -(w * bx));
}

// Face-frame states q = (rho, vn, vt1, vt2, p, bn, bt1, bt2); F in the same order with the field
// components in units of b; SL, SR as chlld's dsl, dsp.  Returns true when no wave-fan region
// matched (a NaN state).
__device__ __forceinline__ bool hlld_fp64(const double* q1, const double* q2, double* F, double& SLo, double& SRo) {
    const double r1 = q1[0], u1 = q1[1], v1 = q1[2], w1 = q1[3], p1 = q1[4], bx1 = q1[5], by1 = q1[6], bz1 = q1[7];
    const double r2 = q2[0], u2 = q2[1], v2 = q2[2], w2 = q2[3], p2 = q2[4], bx2 = q2[5], by2 = q2[6], bz2 = q2[7];
    double pt1, pt2;
    const double cf1 = fast_speed(q1, pt1), cf2 = fast_speed(q2, pt2);
    const double SL = sb_min(u1 - cf1, u2 - cf2), SR = sb_max(u1 + cf1, u2 + cf2);
    SLo = SL;
    SRo = SR;
    F[5] = -sb_max(sb_abs(SL), sb_abs(SR)) * (bx2 - bx1);   // :1828-1839
    if (SR < 0.0) {   // FR, the last match of the region chain, reads nothing else
        const double e = fma(0.5 * r2, fma(w2, w2, fma(v2, v2, u2 * u2)), fma(0.5, p2, pt2));
        phys_flux(r2, u2, v2, w2, bx2, by2, bz2, e, pt2, fma(w2, bz2, fma(v2, by2, u2 * bx2)), F);
        return false;
    }
    const double su1 = SL - u1, su2 = SR - u2;
    const double rs1 = r1 * su1, rs2 = r2 * su2;
    const double idd = rs_rcp(rs2 - rs1);
    const double SM = fma(rs2, u2, fma(-rs1, u1, pt1 - pt2)) * idd;   // :1344-1348
    const double bn = fma(SR, bx2, -(SL * bx1)) * rs_rcp(SR - SL);    // UZ(6), :1406-1408
    const double d1 = SL - SM, d2 = SR - SM;
    const double i1 = rs_rcp(d1), i2 = rs_rcp(d2);
    const double rz1 = rs1 * i1, rz2 = rs2 * i2;                      // star densities
    const double is1 = rs_rsqrt(rz1), is2 = rs_rsqrt(rz2);
    const double abn = sb_abs(bn) > kEpsB ? sb_abs(bn) : 0.0;
    // Alfven speeds, :1660-1676; selected, as 0 * is1 is no number where a cold side recedes (rho* = 0)
    const double SZ1 = abn > 0.0 ? fma(-abn, is1, SM) : SM, SZ2 = abn > 0.0 ? fma(abn, is2, SM) : SM;
    const bool right = SM <= 0.0;   // a NaN SM (two cold sides that recede) is left: FL where SL > 0
    const double S1 = pick(SL, SR, right), S2 = pick(SZ1, SZ2, right);
    // the selected side: energy, physical flux (:1368-1404)
    const double r = pick(r1, r2, right), u = pick(u1, u2, right), v = pick(v1, v2, right), w = pick(w1, w2, right);
    const double p = pick(p1, p2, right), pt = pick(pt1, pt2, right);
    const double bx = pick(bx1, bx2, right), by = pick(by1, by2, right), bz = pick(bz1, bz2, right);
    const double e = fma(0.5 * r, fma(w, w, fma(v, v, u * u)), fma(0.5, p, pt));
    const double sbv = fma(w, bz, fma(v, by, u * bx));
    phys_flux(r, u, v, w, bx, by, bz, e, pt, sbv, F);
    // double star where the Alfven wave lies beyond the face, single star where the face lies
    // between it and the outer wave
    const bool use2 = right ? S2 > 0.0 : S2 <= 0.0;
    const bool use1 = use2 || right || S1 <= 0.0;
    if (use1) {
        const double bn2 = bn * bn;
        const double ptz = fma(rs1 * rs2, u2 - u1, fma(rs2, pt1, -(rs1 * pt2))) * idd;
        const double tt1 = fma(rs1, d1, -bn2), tt2 = fma(rs2, d2, -bn2);   // :1622-1640
        const double it1 = sb_abs(tt1) <= kTtEps ? 0.0 : rs_rcp(tt1), it2 = sb_abs(tt2) <= kTtEps ? 0.0 : rs_rcp(tt2);
        const double c1 = bn * ((SM - u1) * it1), c2 = bn * ((SM - u2) * it2);
        const double k1 = fma(rs1, su1, -bn2) * it1, k2 = fma(rs2, su2, -bn2) * it2;
        const double vy1 = fma(-c1, by1, v1), vz1 = fma(-c1, bz1, w1), vy2 = fma(-c2, by2, v2), vz2 = fma(-c2, bz2, w2);
        const double ty1 = by1 * k1, tz1 = bz1 * k1, ty2 = by2 * k2, tz2 = bz2 * k2;
        // the selected side's star state and energy (:1650-1656)
        const double su = pick(su1, su2, right), i = pick(i1, i2, right), rz = pick(rz1, rz2, right);
        const double vy = pick(vy1, vy2, right), vz = pick(vz1, vz2, right);
        const double ty = pick(ty1, ty2, right), tz = pick(tz1, tz2, right);
        const double sbs = fma(tz, vz, fma(ty, vy, bn * SM));
        const double ez = fma(bn, sbv - sbs, fma(ptz, SM, fma(-pt, u, e * su))) * i;
        F[0] = fma(S1, rz - r, F[0]);
        F[1] = fma(S1, fma(rz, SM, -(r * u)), F[1]);
        F[2] = fma(S1, fma(rz, vy, -(r * v)), F[2]);
        F[3] = fma(S1, fma(rz, vz, -(r * w)), F[3]);
        F[4] = fma(S1, ez - e, F[4]);
        F[6] = fma(S1, ty - by, F[6]);
        F[7] = fma(S1, tz - bz, F[7]);
        if (use2) {   // :1684-1718
            const double q_1 = rz1 * is1, q_2 = rz2 * is2;   // sqrt(rho*)
            const double is = rs_rcp(q_1 + q_2);
            const double sg = copysign(is, bn);              // sign(bn) / (sqrt(rho1*) + sqrt(rho2*))
            const double a2 = q_2 * is, sp = (q_1 * q_2) * sg;
            const double dvy = vy2 - vy1, dvz = vz2 - vz1, dty = ty2 - ty1, dtz = tz2 - tz1;
            const double vyd = fma(a2, dvy, fma(sg, dty, vy1)), vzd = fma(a2, dvz, fma(sg, dtz, vz1));
            const double tyd = fma(-a2, dty, fma(sp, dvy, ty2)), tzd = fma(-a2, dtz, fma(sp, dvz, tz2));
            const double sbd = fma(tzd, vzd, fma(tyd, vyd, bn * SM));
            const double sq = copysign(pick(q_1, q_2, right), (__double2hiint(bn) < 0) == right ? -1.0 : 1.0);
            const double S2r = S2 * rz;
            F[2] = fma(S2r, vyd - vy, F[2]);
            F[3] = fma(S2r, vzd - vz, F[3]);
            F[4] = fma(S2 * sq, sbs - sbd, F[4]);
            F[6] = fma(S2, tyd - ty, F[6]);
            F[7] = fma(S2, tzd - tz, F[7]);
        }
    }
    return !(S2 <= 0.0) && !(S2 > 0.0) && !(SL > 0.0);
}

// HLLC with no magnetic field on either side (:1465-1567 with bn = 0) from density, normal velocity and
// pressure: one sound speed a side, the star state of the selected side alone.
struct HydroFan {
    double SL, SR, SM, ptz;
    double r, u, p, su, rs, S;   // the selected side: state, S - u, rho (S - u), outer speed
    bool right, none;            // none: no region matched
    double F0, F1;               // mass and normal momentum flux
};
__device__ __forceinline__ void hllc_hydro_fan(double r1, double u1, double p1, double r2, double u2, double p2,
                                               HydroFan& f) {
    const double c1 = sqrt_ratio(kGamma * p1, r1), c2 = sqrt_ratio(kGamma * p2, r2);
    f.SL = sb_min(u1 - c1, u2 - c2);
    f.SR = sb_max(u1 + c1, u2 + c2);
    const double su1 = f.SL - u1, su2 = f.SR - u2;
    const double rs1 = r1 * su1, rs2 = r2 * su2;
    f.SM = fma(rs2, u2, fma(-rs1, u1, p1 - p2)) * rs_rcp(rs2 - rs1);
    f.ptz = 0.5 * (fma(rs2, f.SM - u2, p2) + fma(rs1, f.SM - u1, p1));
    // Two cold sides that recede have no contact speed, nor has a face beside an invalid state.  A face
    // outside the fan reads none: any finite contact speed on the far side of the outer wave and any
    // finite star pressure keep the terms that are multiplied by 0 there finite.
    if ((__double2hiint(f.SM) & 0x7ff00000) == 0x7ff00000) {
        if (f.SR < 0.0) {
            f.SM = f.SR - 1.0;
            f.ptz = 0.0;
        } else if (f.SL > 0.0 && !(f.SM <= 0.0)) {
            f.SM = f.SL + 1.0;
            f.ptz = 0.0;
        }
    }
    f.right = f.SM <= 0.0 || f.SR < 0.0;
    f.r = pick(r1, r2, f.right);
    f.u = pick(u1, u2, f.right);
    f.p = pick(p1, p2, f.right);
    f.S = pick(f.SL, f.SR, f.right);
    f.su = pick(su1, su2, f.right);
    f.rs = pick(rs1, rs2, f.right);
    f.none = !(f.SM <= 0.0) && !(f.SM > 0.0) && !(f.SL > 0.0) && !(f.SR < 0.0);
}
// Mass, normal momentum and energy flux; v2 = |v|^2 of the selected side.  The tangential momentum
// flux is F0 times the selected side's tangential velocity (m v + S (rho* - rho) v).
__device__ __forceinline__ double hllc_hydro_flux(HydroFan& f, double v2) {
    const double Ss = (f.right ? f.SR >= 0.0 : f.SL <= 0.0) ? f.S : 0.0;   // 0 outside the fan
    const double i = rs_rcp(f.S - f.SM);
    const double rz = f.rs * i;
    const double m = f.r * f.u;
    const double e = fma(0.5 * f.r, v2, 1.5 * f.p);
    const double ez = fma(f.ptz, f.SM, fma(-f.p, f.u, e * f.su)) * i;
    f.F0 = fma(Ss, rz - f.r, m);
    f.F1 = fma(Ss, fma(rz, f.SM, -m), fma(m, f.u, f.p));
    return fma(Ss, ez - e, (e + f.p) * f.u);
}
__device__ __forceinline__ bool hllc_hydro_fp64(const double* q1, const double* q2, double* F, double& SLo,
                                                double& SRo) {
    HydroFan f;
    hllc_hydro_fan(q1[0], q1[1], q1[4], q2[0], q2[1], q2[4], f);
    SLo = f.SL;
    SRo = f.SR;
    const double v = pick(q1[2], q2[2], f.right), w = pick(q1[3], q2[3], f.right);
    F[4] = hllc_hydro_flux(f, fma(w, w, fma(v, v, f.u * f.u)));
    F[0] = f.F0;
    F[1] = f.F1;
    F[2] = f.F0 * v;
    F[3] = f.F0 * w;
    F[5] = F[6] = F[7] = 0.0;
    return f.none;
}

// Whether any of the six field components of the two states is nonzero.
__device__ __forceinline__ bool has_field(const double* q1, const double* q2) {
    unsigned long long b = 0;
#pragma unroll
    for (int v = 5; v < 8; v++)
        b |= (unsigned long long)__double_as_longlong(q1[v]) | (unsigned long long)__double_as_longlong(q2[v]);
    return (b << 1) != 0;
}

// The plain form's face flux for n_disc 0 (HLLC / HLLD).  HLLC takes the field-free path for a face with
// no field on either side: by the face and not by its warp, as the two paths round differently and a
// face on the seam of two tiles is computed in both.  A warp pays for both paths only where it has faces
// of both kinds.
template <int NSTATE>
__device__ __forceinline__ bool flux_fp64(const double* q1, const double* q2, double* F, double& SL, double& SR) {
    static_assert(NSTATE == 2 || NSTATE == 3, "HLLC or HLLD");
    if constexpr (NSTATE == 3) {
        return hlld_fp64(q1, q2, F, SL, SR);
    } else {
        if (!has_field(q1, q2)) return hllc_hydro_fp64(q1, q2, F, SL, SR);
        double SM;
        const int fl = riemann<double, 2, false, false, true, true>(q1, q2, 0.0, 0, F, SL, SR, SM);
#pragma unroll
        for (int v = 5; v < 8; v++) F[v] *= kInvSpi4;
        return (fl & kFlagWave) != 0;
    }
}

// Unit tangents (e2, e3) completing a unit normal to an orthonormal frame (T. Duff et al., "Building
// an Orthonormal Basis, Revisited", JCGT 6(1), 2017).  The flux does not depend on which tangents are
// taken: every formula treats the two tangential components as a 2-vector.
__device__ __forceinline__ void tangent_frame(const double* n, double* e2, double* e3) {
    const double s = copysign(1.0, n[2]);
    const double a = -rs_rcp(s + n[2]);
    const double b = n[0] * n[1] * a;
    e2[0] = fma(s * n[0] * n[0], a, 1.0);
    e2[1] = s * b;
    e2[2] = -s * n[0];
    e3[0] = b;
    e3[1] = fma(n[1] * n[1], a, s);
    e3[2] = -n[1];
}
__device__ __forceinline__ double dot3(const double* a, double x, double y, double z) {
    return fma(a[2], z, fma(a[1], y, a[0] * x));
}

// The flux at a face of unit normal n (at rest) between lab states q (rho, u, v, w, p, b): F in lab
// components, field fluxes in units of b.  NSTATE as riemann().  FAST: HLLC / HLLD for n_disc 0 by the
// solvers above; otherwise riemann().
// reload(m) gives the normal once more.
template <int NSTATE, bool FAST, typename Reload>
__device__ __forceinline__ bool flux_normal_fp64(const double* n, Reload reload, const double* q1, const double* q2,
                                                 int n_disc, double* F, double& SL, double& SR) {
    if constexpr (NSTATE == 2 && FAST) {
        if (!has_field(q1, q2)) {   // by the face, as in flux_fp64: its flux is the same in any numbering
            HydroFan f;
            const double u1 = dot3(n, q1[1], q1[2], q1[3]), u2 = dot3(n, q2[1], q2[2], q2[3]);
            hllc_hydro_fan(q1[0], u1, q1[4], q2[0], u2, q2[4], f);
            SL = f.SL;
            SR = f.SR;
            double v[3];
#pragma unroll
            for (int c = 0; c < 3; c++) v[c] = pick(q1[1 + c], q2[1 + c], f.right);
            F[4] = hllc_hydro_flux(f, fma(v[2], v[2], fma(v[1], v[1], v[0] * v[0])));
            F[0] = f.F0;
            const double fn = fma(-f.F0, f.u, f.F1);   // n F1 + F0 (v - u n)
#pragma unroll
            for (int c = 0; c < 3; c++) {
                F[1 + c] = fma(fn, n[c], f.F0 * v[c]);
                F[5 + c] = 0.0;
            }
            return f.none;
        }
    }
    double e2[3], e3[3], a[8], b[8], G[8];
    tangent_frame(n, e2, e3);
    a[0] = q1[0];
    a[4] = q1[4];
    b[0] = q2[0];
    b[4] = q2[4];
#pragma unroll
    for (int o = 1; o < 8; o += 4) {
        a[o] = dot3(n, q1[o], q1[o + 1], q1[o + 2]);
        a[o + 1] = dot3(e2, q1[o], q1[o + 1], q1[o + 2]);
        a[o + 2] = dot3(e3, q1[o], q1[o + 1], q1[o + 2]);
        b[o] = dot3(n, q2[o], q2[o + 1], q2[o + 2]);
        b[o + 1] = dot3(e2, q2[o], q2[o + 1], q2[o + 2]);
        b[o + 2] = dot3(e3, q2[o], q2[o + 1], q2[o + 2]);
    }
    bool none;
    if constexpr (NSTATE == 3 && FAST) {
        none = hlld_fp64(a, b, G, SL, SR);
    } else {
        double SM;
        none = (riemann<double, NSTATE, false, false, true, true>(a, b, 0.0, n_disc, G, SL, SR, SM) & kFlagWave) != 0;
#pragma unroll
        for (int v = 5; v < 8; v++) G[v] *= kInvSpi4;
    }
    F[0] = G[0];
    F[4] = G[4];
    // the normal read again and the frame formed again: fewer registers across the solver than
    // keeping nine doubles
    double m[3];
    reload(m);
    tangent_frame(m, e2, e3);
#pragma unroll
    for (int c = 0; c < 3; c++) {
        F[1 + c] = fma(m[c], G[1], fma(e2[c], G[2], e3[c] * G[3]));
        F[5 + c] = fma(m[c], G[5], fma(e2[c], G[6], e3[c] * G[7]));
    }
    return none;
}

}  // namespace sb
