// Barbot, Moore & Lambert (2017) vertical cuboid strain volume, device side:
// stress at a receiver due to the six unit anelastic eigenstrains of one
// cuboid, all at once.
//
// Follows computeStressVerticalStrainVolume (fortran/3d/src/strainvolume.f90:
// 1042-1140): rotate the receiver into the cuboid frame, form the displacement
// gradient, remove the eigenstrain inside the cuboid (1124-1131), Hooke with
// lambda = 2 G nu / (1 - 2 nu).  The strain is the derivative of the published
// displacement integrals (bml17_disp.h) summed over the eight corners, written
// out below; the displacement itself (observation points) evaluates the
// integrals as published.
#pragma once
#include <cuda_runtime.h>
#include "rows.cuh"

// scalar hooks of bml17_disp.h for plain doubles, declared in the integrals'
// namespace so that the unqualified calls there find them
namespace bml17 {
__host__ __device__ __forceinline__ double sv_sqrt(double a) { return sqrt(a); }
__host__ __device__ __forceinline__ double sv_log(double a) { return log(a); }
__host__ __device__ __forceinline__ double sv_atan(double a) { return atan(a); }
__host__ __device__ __forceinline__ double sv_atan2(double y, double x) { return atan2(y, x); }
__host__ __device__ __forceinline__ double sv_val(double a) { return a; }
}  // namespace bml17

#include "bml17_disp.h"

namespace ucg {

constexpr bool kVolumesBuilt = true;

enum : int { SV_Q1 = 0, SV_Q2, SV_Q3, SV_L, SV_T, SV_W, SV_C, SV_S, SV_SIZE };

struct SvRec {
    const double *__restrict__ base;
    long stride;
    __device__ __forceinline__ double operator[](int f) const { return __ldg(base + (long)f * stride); }
};

inline void sv_prepare(const double *x, double L, double T, double W, double strike, double *r)
{
    r[SV_Q1] = x[0]; r[SV_Q2] = x[1]; r[SV_Q3] = x[2];
    r[SV_L] = L; r[SV_T] = T; r[SV_W] = W;
    r[SV_C] = cos(strike); r[SV_S] = sin(strike);
}

// boxcar functions of strainvolume.f90:53-84
__device__ __forceinline__ double sv_heaviside(double x) { return (0.0 < x) ? 1.0 : 0.0; }
__device__ __forceinline__ double sv_omega(double x) { return sv_heaviside(x + 0.5) - sv_heaviside(x - 0.5); }
__device__ __forceinline__ double sv_s(double x) { return sv_omega(x - 0.5); }

// a gradient
struct SvG {
    double x, y, z;
};
__device__ __forceinline__ SvG operator+(SvG a, SvG b) { return {a.x + b.x, a.y + b.y, a.z + b.z}; }
__device__ __forceinline__ SvG operator-(SvG a, SvG b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ __forceinline__ SvG operator*(double c, SvG a) { return {c * a.x, c * a.y, c * a.z}; }

// a sum of angles atan2(y, x), kept as a complex product and a count of turns
struct SvAngle {
    double x, y;
    int turns;
    // add (or, with y negated, subtract) the angle of (bx, by)
    __device__ __forceinline__ void add(double bx, double by)
    {
        const double nx = x * bx - y * by, ny = x * by + y * bx;
        const bool a = signbit(y), b = signbit(by), n = signbit(ny);
        turns += (!a && !b && n) - (a && b && !n);
        x = nx;
        y = ny;
    }
    __device__ __forceinline__ double value() const { return atan2(y, x) + 6.283185307179586476925286766559 * turns; }
};

// log(r + d) over corners: factors of the numerator and the denominator; lat2 = r^2 - d^2
__device__ __forceinline__ void sv_log_factor(bool plus, double r, double d, double lat2, double &num, double &den)
{
    const double s = r + fabs(d);
    const bool neg = d < 0.0;   // log(r + d) = log(lat2) - log(r - d)
    const double up = neg ? lat2 : s, dn = neg ? s : 1.0;
    num *= plus ? up : dn;
    den *= plus ? dn : up;
}

// Strain (11, 2 12, 2 13, 22, 2 23, 33, over c = 1 / (16 pi (1 - nu) G)) of the six
// combinations of the integrals that the unit eigenstrains need, summed over the
// corners with their signs: with J_ijk as in bml17_disp.h, for i = 1, 2, 3
//   E[0] J_i123,  E[1] J_i213,  E[2] J_i312,
//   E[3] J_i223 + J_i113,  E[4] J_i323 + J_i112,  E[5] J_i212 + J_i313.
//
// With d1 = x1 - y1, d2 = x2 - y2, dm = x3 - y3, dp = x3 + y3, r1, r2 the distances
// to the corner and its image, l1..l3 = ln(r1 + d1, d2, dm), m1..m3 = ln(r2 + d1, d2,
// dp), t1..t3 the angles of (r1 dm, d1 d2), (r1 d2, d1 dm), (r1 d1, d2 dm), u1..u3 the
// same of r2 and dp, e = 2 x3 y3 / r2, P1 = e d1 d2 / s13, P2 = e d1 d2 / s23,
// P3 = e d2 dp / s13, P4 = e d1 dp / s23 and Rk = dk (2 Bq / (r2 s12)) (s12, s13, s23, Bq
// as there), and because a term that does not depend on one of y1, y2, y3 cancels
// in the corner sum (so ln(r2 - d1) counts as -m1, the arctangents of multiples of
// x and y count nothing), the 27 integrals merge into, for instance,
//   J_1323 + J_1112 = 2 P1 - 8 (nu - 1) x3 u3 - 4 (nu - 1) (dm t1 + dp u1)
//                     - 2 (2 nu - 1) d1 (l2 - m2) - 4 (nu - 1) d2 (l1 + m1)
//   J_3323 + J_3112 = 2 P3 - 4 (nu - 1) (d1 (t3 - u3) + d2 (l3 - m3)) - 2 (2 nu - 1) dm (l2 - m2)
// The derivative of a coefficient (d1, dm, x3, ...) is the same at every corner, so
// the logarithms and angles themselves enter only as corner sums: six logarithms of
// products and six angles of complex products a pair, instead of one of each per
// term and corner.  Their gradients are rational in r and d.
//
// On the line through a vertical edge s12 vanishes: there Rk and the gradients of
// u2 and u3 grow as 1 / s12 and 1 / sqrt(s12), and cancel between the edge's two
// ends.  That part, which has no y3 (kap = (nu - 1)(2 nu - 1)),
//   Rk: dk 2 (1 - kap) x3^2 / s12,   u2: atan2(d2, d1),   u3: atan2(d1, d2),
// is left out before it is formed, with r2 - dp = s12 / (r2 + dp) and, in a3 and b3,
// the term in kap dp of the angle of (d1, d2) (J_3123, J_3213) that goes with it.
// Cuboid of 3,100 x 2,300 x 1,700 m, above and below it, against the surface forces on its
// faces: 1e-14 of the stress 1 m and 1 um from the line, where the sum over the
// corners had 1e-7 and 1e5.
//
// Per pair: 112 reciprocals, 32 square roots and about 5,200 other FP64
// instructions, against 130,174 flops on duals of the 27 integrals.
__device__ __forceinline__ void sv_strain(double x1, double x2, double x3, double q3, double L, double T, double W,
                                          double nu, double E[6][6])
{
    const double nm = nu - 1.0, n2 = 2.0 * nu - 1.0, n43 = 4.0 * nu - 3.0;
    const double k1 = (4.0 * nu - 2.0) * nu - 1.0, k3 = (4.0 * nu - 6.0) * nu + 3.0;
    const double k5 = (8.0 * nu - 12.0) * nu + 5.0;
    const double k7 = (8.0 * nu - 16.0) * nu + 7.0, k8 = 8.0 * nm * nu + 1.0, kap = nm * n2;
#pragma unroll
    for (int a = 0; a < 36; a++) E[a / 6][a % 6] = 0.0;
    // pass 1: values
    double ln[6] = {1, 1, 1, 1, 1, 1}, ld[6] = {1, 1, 1, 1, 1, 1};
    SvAngle an[6] = {{1, 0, 0}, {1, 0, 0}, {1, 0, 0}, {1, 0, 0}, {1, 0, 0}, {1, 0, 0}};
#pragma unroll 1
    for (int k = 0; k < 8; k++) {
        const double d1 = x1 - ((k & 4) ? 0.0 : L), d2 = x2 - ((k & 2) ? -0.5 * T : 0.5 * T);
        const double y3 = (k & 1) ? q3 : q3 + W;
        const bool plus = !(((k >> 2) ^ (k >> 1) ^ k) & 1);
        const double dm = x3 - y3, dp = x3 + y3;
        const double d11 = d1 * d1, d22 = d2 * d2, dmm = dm * dm, dpp = dp * dp;
        const double r1 = sqrt(d11 + d22 + dmm), r2 = sqrt(d11 + d22 + dpp);
        sv_log_factor(plus, r1, d1, d22 + dmm, ln[0], ld[0]);
        sv_log_factor(plus, r1, d2, d11 + dmm, ln[1], ld[1]);
        sv_log_factor(plus, r1, dm, d11 + d22, ln[2], ld[2]);
        sv_log_factor(plus, r2, d1, d22 + dpp, ln[3], ld[3]);
        sv_log_factor(plus, r2, d2, d11 + dpp, ln[4], ld[4]);
        sv_log_factor(plus, r2, dp, d11 + d22, ln[5], ld[5]);
        const double s = plus ? 1.0 : -1.0;
        an[0].add(d1 * d2, s * (r1 * dm));
        an[1].add(d1 * dm, s * (r1 * d2));
        an[2].add(d2 * dm, s * (r1 * d1));
        an[3].add(d1 * d2, s * (r2 * dp));
        an[4].add(d1 * dp, s * (r2 * d2));
        an[5].add(d2 * dp, s * (r2 * d1));
    }
    const double l1 = log(ln[0] / ld[0]), l2 = log(ln[1] / ld[1]), l3 = log(ln[2] / ld[2]);
    const double m1 = log(ln[3] / ld[3]), m2 = log(ln[4] / ld[4]), m3 = log(ln[5] / ld[5]);
    const double t1 = an[0].value(), t2 = an[1].value(), t3 = an[2].value();
    const double u1 = an[3].value(), u2 = an[4].value(), u3 = an[5].value();
    auto put = [&](double *e, SvG g1, SvG g2, SvG g3) {
        e[0] += g1.x;
        e[1] += g1.y + g2.x;
        e[2] += g1.z + g3.x;
        e[3] += g2.y;
        e[4] += g2.z + g3.y;
        e[5] += g3.z;
    };
    // the values' part: derivative of the coefficients
    put(E[0], SvG{-2 * n2 * (t3 + n2 * u3), -n43 * l3 - k3 * m3, (2 - k5) * m2 - n43 * l2}, SvG{-k1 * m3 - l3, 0, 0},
        SvG{k8 * m2 - l2, 0, -4 * n2 * nu * u3});
    put(E[1], SvG{0, -k1 * m3 - l3, 0}, SvG{-n43 * l3 - k3 * m3, -2 * n2 * (t2 + n2 * u2), (2 - k5) * m1 - n43 * l1},
        SvG{0, k8 * m1 - l1, -4 * n2 * nu * u2});
    put(E[2], SvG{-4 * kap * u3, -4 * kap * m3, -l2 - k7 * m2}, SvG{-4 * kap * m3, -4 * kap * u2, -l1 - k7 * m1},
        SvG{k5 * m2 - n43 * l2, k5 * m1 - n43 * l1, 2 * n2 * (n2 * u1 - t1)});
    const double dd = -2 * n2 * (l3 + n2 * m3);
    put(E[3], SvG{dd, -4 * nm * (t2 - u2), -4 * nm * (l1 - m1)}, SvG{-4 * nm * (t3 - u3), dd, -4 * nm * (l2 - m2)},
        SvG{0, 0, (8 * nu - 16 * nu * nu) * m3});
    put(E[4], SvG{-2 * n2 * (l2 - m2), -4 * nm * (l1 + m1), -4 * nm * (2 * u3 + t1 + u1)}, SvG{0, 0, -8 * nm * m3},
        SvG{-4 * nm * (t3 - u3), -4 * nm * (l3 - m3), -2 * n2 * (l2 - m2)});
    put(E[5], SvG{0, 0, -8 * nm * m3}, SvG{-4 * nm * (l2 + m2), -2 * n2 * (l1 - m1), -4 * nm * (2 * u2 + t1 + u1)},
        SvG{-4 * nm * (l3 - m3), -4 * nm * (t2 - u2), -2 * n2 * (l1 - m1)});
    // pass 2: gradients of the functions
#pragma unroll 1
    for (int k = 0; k < 8; k++) {
        const double d1 = x1 - ((k & 4) ? 0.0 : L), d2 = x2 - ((k & 2) ? -0.5 * T : 0.5 * T);
        const double y3 = (k & 1) ? q3 : q3 + W;
        const double sg = (((k >> 2) ^ (k >> 1) ^ k) & 1) ? -1.0 : 1.0;
        const double dm = x3 - y3, dp = x3 + y3;
        const double d11 = d1 * d1, d22 = d2 * d2, dmm = dm * dm, dpp = dp * dp, s12 = d11 + d22;
        const double r1 = sqrt(s12 + dmm), r2 = sqrt(s12 + dpp), ir1 = 1.0 / r1, ir2 = 1.0 / r2;
        const double i12 = 1.0 / s12, j13 = 1.0 / (d11 + dmm), j23 = 1.0 / (d22 + dmm), i13 = 1.0 / (d11 + dpp),
                     i23 = 1.0 / (d22 + dpp);
        // 1 / (r (r + d)) without cancellation where d < 0
        auto inv = [](double r, double ir, double d, double ilat2) {
            const double s = r + fabs(d);
            return d < 0.0 ? s * ilat2 * ir : ir / s;
        };
        const double v1 = inv(r1, ir1, d1, j23), v2 = inv(r1, ir1, d2, j13), v3 = inv(r1, ir1, dm, i12);
        const double w1 = inv(r2, ir2, d1, i23), w2 = inv(r2, ir2, d2, i13), w3 = inv(r2, ir2, dp, i12);
        const SvG L1{ir1, d2 * v1, dm * v1}, L2{d1 * v2, ir1, dm * v2}, L3{d1 * v3, d2 * v3, ir1};
        const SvG M1{ir2, d2 * w1, dp * w1}, M2{d1 * w2, ir2, dp * w2}, M3{d1 * w3, d2 * w3, ir2};
        // atan2(r1 dm, d1 d2) and the like
        const double ra = r1 * r1, rb = r2 * r2;
        const SvG T1{-d2 * dm * ir1 * j13, -d1 * dm * ir1 * j23, d1 * d2 * (ra + dmm) * ir1 * j13 * j23};
        const SvG T2{-d2 * dm * ir1 * i12, d1 * dm * (ra + d22) * ir1 * i12 * j23, -d1 * d2 * ir1 * j23};
        const SvG T3{d2 * dm * (ra + d11) * ir1 * i12 * j13, -d1 * dm * ir1 * i12, -d1 * d2 * ir1 * j13};
        const SvG U1{-d2 * dp * ir2 * i13, -d1 * dp * ir2 * i23, d1 * d2 * (rb + dpp) * ir2 * i13 * i23};
        // of u2 - atan2(d2, d1) and u3 - atan2(d1, d2): the angles' own part in 1 / s12
        // has no y3 under its coefficients and cancels between a vertical edge's ends
        const double ip = 1.0 / (r2 + dp);   // (r2 - dp) / s12
        const SvG U2{d2 * ir2 * ip, d1 * ir2 * (dp * i23 - ip), -d1 * d2 * ir2 * i23};
        const SvG U3{d2 * ir2 * (dp * i13 - ip), d1 * ir2 * ip, -d1 * d2 * ir2 * i13};
        // rational terms
        const double ir3 = ir2 * ir2;
        const double ev = 2.0 * ir2 * x3 * y3;
        const SvG E3{-ev * ir3 * d1, -ev * ir3 * d2, 2.0 * ir2 * y3 - ev * ir3 * dp};
        const double a13 = ev * i13, a23 = ev * i23;
        const SvG A13{i13 * (E3.x - 2.0 * a13 * d1), i13 * E3.y, i13 * (E3.z - 2.0 * a13 * dp)};
        const SvG A23{i23 * E3.x, i23 * (E3.y - 2.0 * a23 * d2), i23 * (E3.z - 2.0 * a23 * dp)};
        const double d12 = d1 * d2, d2p = d2 * dp, d1p = d1 * dp;
        const SvG P1{d12 * A13.x + a13 * d2, d12 * A13.y + a13 * d1, d12 * A13.z};
        const SvG P2{d12 * A23.x + a23 * d2, d12 * A23.y + a23 * d1, d12 * A23.z};
        const SvG P3{d2p * A13.x, d2p * A13.y + a13 * dp, d2p * A13.z + a13 * d2};
        const SvG P4{d1p * A23.x + a23 * dp, d1p * A23.y, d1p * A23.z + a23 * d1};
        // (2 / r2) (Bq - (1 - kap) x3^2 r2) / s12, less its part that cancels likewise
        const double bw = (kap * r2 * dp + x3 * x3) * ip;
        const double rv = 2.0 * ir2 * (x3 - bw);
        const double bx = 2.0 * ir3 * ip * (bw - kap * dp) - rv * ir3;   // over d1, d2
        const double bz = 1.0 - ip * (kap * (dpp * ir2 + r2) + 2.0 * x3 - bw * (1.0 + dp * ir2));
        const SvG Rb{d1 * bx, d2 * bx, 2.0 * ir2 * bz - rv * ir3 * dp};
        const SvG R1{d1 * Rb.x + rv, d1 * Rb.y, d1 * Rb.z}, R2{d2 * Rb.x, d2 * Rb.y + rv, d2 * Rb.z};
        const SvG N1{d1 * ir1, d2 * ir1, dm * ir1}, N2{d1 * ir2, d2 * ir2, dp * ir2};   // of r1 and r2
        const SvG a2 = R1 - (k1 * d1) * M3 - d1 * L3, b1 = R2 - (k1 * d2) * M3 - d2 * L3;
        const double xm = 2.0 * x3 - k5 * dp, xn = 4.0 * n2 * (nu * x3 + nm * y3), xk = k7 * x3 + k8 * y3;
        const SvG a1 = P3 - R2 - (2.0 * n2 * d1) * (T3 + n2 * U3) + xm * M2 - (n43 * d2) * L3 - (k3 * d2) * M3 -
                       (n43 * dm) * L2;
        const SvG b2 = P4 - R1 - (2.0 * n2 * d2) * (T2 + n2 * U2) + xm * M1 - (n43 * d1) * L3 - (k3 * d1) * M3 -
                       (n43 * dm) * L1;
        const SvG a3 = (k8 * d1) * M2 - d1 * L2 - P1 - xn * U3;
        const SvG b3 = (k8 * d2) * M1 - d2 * L1 - P2 - xn * U2;
        const SvG c1 = (-4.0 * kap) * (d1 * U3 + d2 * M3) - P3 - dm * L2 - xk * M2;
        const SvG c2 = (-4.0 * kap) * (d2 * U2 + d1 * M3) - P4 - dm * L1 - xk * M1;
        const SvG c3 = P1 + P2 + (2.0 * n2) * ((n2 * dp) * U1 - dm * T1) - n43 * (d1 * L2 + d2 * L1) +
                       k5 * (d1 * M2 + d2 * M1);
        const double m4 = -4.0 * nm, m2n = -2.0 * n2;
        const SvG q1 = 2.0 * R1 + (m2n * d1) * (L3 + n2 * M3) + m4 * (d2 * (T2 - U2) + dm * L1 - dp * M1);
        const SvG q2 = 2.0 * R2 + (m2n * d2) * (L3 + n2 * M3) + m4 * (d1 * (T3 - U3) + dm * L2 - dp * M2);
        const double kc = 4.0 * y3 - 4.0 * nu * x3 - 12.0 * nu * y3 + 8.0 * nu * nu * dp;
        const SvG q3v = -2.0 * (N1 - k8 * N2 - E3 + kc * M3);
        const SvG tt = m4 * (dm * T1 + dp * U1);
        const SvG e1 = 2.0 * P1 + (2.0 * m4 * x3) * U3 + tt + (m2n * d1) * (L2 - M2) + (m4 * d2) * (L1 + M1);
        const SvG f2 = 2.0 * P2 + (2.0 * m4 * x3) * U2 + tt + (m2n * d2) * (L1 - M1) + (m4 * d1) * (L2 + M2);
        const SvG e2 = (8.0 * nu - 6.0) * N2 - 2.0 * (N1 + E3) + (2.0 * m4 * x3) * M3;
        const SvG e3 = 2.0 * P3 + (m4 * d1) * (T3 - U3) + (m4 * d2) * (L3 - M3) + (m2n * dm) * (L2 - M2);
        const SvG f3 = 2.0 * P4 + (m4 * d2) * (T2 - U2) + (m4 * d1) * (L3 - M3) + (m2n * dm) * (L1 - M1);
        put(E[0], sg * a1, sg * a2, sg * a3);
        put(E[1], sg * b1, sg * b2, sg * b3);
        put(E[2], sg * c1, sg * c2, sg * c3);
        put(E[3], sg * q1, sg * q2, sg * q3v);
        put(E[4], sg * e1, sg * e2, sg * e3);
        put(E[5], sg * e2, sg * f2, sg * f3);
    }
}

// The rows that a receiver (record rc, NED) takes for unit eigenstrain q (11, 12,
// 13, 22, 23, 33 in the cuboid frame): out[q][row]
template <int NR>
__device__ __forceinline__ void sv_pair_rows(const double *rc, const SvRec &R, double mu, double nu,
                                             double out[6][NR])
{
    const double ct = R[SV_C], st = R[SV_S];
    const double x1 = rc[0] - R[SV_Q1], x2 = rc[1] - R[SV_Q2], x3 = rc[2];
    const double x1p = x1 * ct + x2 * st, x2p = -x1 * st + x2 * ct;
    double E[6][6];
    sv_strain(x1p, x2p, x3, R[SV_Q3], R[SV_L], R[SV_T], R[SV_W], nu, E);
    const double lambda = mu * 2.0 * nu / (1.0 - 2.0 * nu);
    const double inside = sv_s(x1p / R[SV_L]) * sv_omega(x2p / R[SV_T]) * sv_s((x3 - R[SV_Q3]) / R[SV_W]);
    // the receiver's unit vectors in the cuboid frame
    double v[3][3];
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const double *w = rc + 3 + 3 * k;
        v[k][0] = w[0] * ct + w[1] * st;
        v[k][1] = w[1] * ct - w[0] * st;
        v[k][2] = w[2];
    }
    const double c = 1.0 / 16.0 / (1.0 - nu) / 3.141592653589793115997963468544185161 / mu;
    const double cl = c * lambda, cg = 2.0 * c * mu;
#pragma unroll
    for (int q = 0; q < 6; q++) {
        double e[6];
#pragma unroll
        for (int k = 0; k < 6; k++) {
            const double s = cl * (E[0][k] + E[1][k] + E[2][k]);
            e[k] = q == 0 ? s + cg * E[0][k] : q == 3 ? s + cg * E[1][k] : q == 5 ? s + cg * E[2][k]
                 : cg * E[q == 1 ? 3 : q == 2 ? 4 : 5][k];
        }
        // the eigenstrain inside (a shear component counts twice here)
        e[q] -= (q == 0 || q == 3 || q == 5) ? inside : 2.0 * inside;
        const double tr = lambda * (e[0] + e[3] + e[5]);
        receiver_rows<NR>(v[0], v[1], v[2], tr + 2.0 * mu * e[0], mu * e[1], mu * e[2], tr + 2.0 * mu * e[3],
                          mu * e[4], tr + 2.0 * mu * e[5], out[q]);
    }
}

// Displacement (north, east, down) at xr (NED) for the six unit eigenstrains
// of one cuboid (computeDisplacementVerticalStrainVolume, strainvolume.f90:
// 215-991): the receiver rotated into the cuboid frame, the 8-corner sum of
// the displacement integrals, the horizontal components rotated back.
__device__ inline void sv_pair_disp(const double xr[3], const SvRec &R, double mu, double nu, double u[6][3])
{
    const double ct = R[SV_C], st = R[SV_S];
    const double x1p = (xr[0] - R[SV_Q1]) * ct + (xr[1] - R[SV_Q2]) * st;
    const double x2p = -(xr[0] - R[SV_Q1]) * st + (xr[1] - R[SV_Q2]) * ct;
    double up[6][3];
    bml17::displacement<-1, double>(x1p, x2p, xr[2], R[SV_Q3], R[SV_L], R[SV_T], R[SV_W], nu, mu, up);
#pragma unroll
    for (int q = 0; q < 6; q++) {
        u[q][0] = up[q][0] * ct - up[q][1] * st;
        u[q][1] = up[q][0] * st + up[q][1] * ct;
        u[q][2] = up[q][2];
    }
}

}  // namespace ucg
