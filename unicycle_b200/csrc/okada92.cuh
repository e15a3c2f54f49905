// Okada (1992) displacement gradient of a rectangular dislocation in an elastic
// half-space, evaluated on the device for unit strike slip and unit dip slip at
// once.  Follows Okada's finite-source solution as coded in DC3D
// (fortran/3d/src/dc3d.f:1-198, parts A/B/C at dc3d.f:200-507, the geometry
// constants at dc3d.f:509-544 and 596-665):
//   - real source: part A; image source: parts A + B + z*C;
//   - the 2x2 corner sum with the sign rule of dc3d.f:103-106;
//   - the EPS = 1e-6 snapping of xi, eta, q and the singular-edge rejection
//     (result zero) of dc3d.f:65-87;
//   - the DCCON2 call keeps the reference's index pairing (KXI(K), KET(J)).
// Only the nine derivative outputs are formed (the displacement itself is not
// needed for stress), and the corner geometry, logs and arctangents are shared
// by the two slip components instead of being recomputed per DC3D call.
//
// R32 = true reproduces the reference's REAL*4 interface (okada92.f90:121-160):
// the caller rounds the inputs to binary32, the two REAL*4 differences are taken
// in binary32, the REAL*4 EPS is used in DC3D, and the outputs are rounded to
// binary32.
#pragma once
#include <cuda_runtime.h>

namespace ucg {

struct OkDip {           // DCCON0 (dc3d.f:509-544)
    double sd, cd, sdsd, cdcd, sdcd;
    double icd;              // 1 / cd where cd is not 0
};

struct OkMed {           // medium constants alp1..alp5
    double alp1, alp2, alp3, alp4, alp5;
};

struct OkCorner {        // DCCON2 outputs (dc3d.f:596-665)
    double xi, et, q;
    double xi2, et2, q2, r, r2, y, d, x11, y11, x32, y32;
    double ir, ir2, ir3, ir5;   // reciprocal powers of r
    double ey, ez, fy, fz, gy, gz, hy, hz;
};

__host__ __device__ inline OkDip ok_dip(double dip_deg)
{
    const double p18 = 6.283185307179586 / 360.0;
    OkDip c;
    c.sd = sin(dip_deg * p18);
    c.cd = cos(dip_deg * p18);
    if (fabs(c.cd) < 1.0e-6) {
        c.cd = 0.0;
        if (c.sd > 0.0) c.sd = 1.0;
        if (c.sd < 0.0) c.sd = -1.0;
    }
    c.sdsd = c.sd * c.sd;
    c.cdcd = c.cd * c.cd;
    c.sdcd = c.sd * c.cd;
    c.icd = c.cd != 0.0 ? 1.0 / c.cd : 0.0;
    return c;
}

__host__ __device__ inline OkMed ok_med(double alpha)
{
    OkMed m;
    m.alp1 = (1.0 - alpha) / 2.0;
    m.alp2 = alpha / 2.0;
    m.alp3 = (1.0 - alpha) / alpha;
    m.alp4 = 1.0 - alpha;
    m.alp5 = alpha;
    return m;
}

// Corner geometry.  xi, et, q are snapped in place (the reference passes them
// by reference).  Returns false when r == 0 (unreachable after edge rejection).
__device__ inline bool ok_corner(double &xi, double &et, double &q, const OkDip &dp, int kxi,
                                 int ket, OkCorner &c)
{
    const double eps = 1.0e-6;
    if (fabs(xi) < eps) xi = 0.0;
    if (fabs(et) < eps) et = 0.0;
    if (fabs(q) < eps) q = 0.0;
    c.xi = xi; c.et = et; c.q = q;
    c.xi2 = xi * xi;
    c.et2 = et * et;
    c.q2 = q * q;
    c.r2 = c.xi2 + c.et2 + c.q2;
    c.r = sqrt(c.r2);
    if (c.r == 0.0) return false;
    c.ir = 1.0 / c.r;
    c.ir2 = c.ir * c.ir;
    c.ir3 = c.ir * c.ir2;
    c.ir5 = c.ir3 * c.ir2;
    c.y = et * dp.cd + q * dp.sd;
    c.d = et * dp.sd - q * dp.cd;
    // tt, alx and ale enter only the displacement entries of parts A/B/C, which the
    // gradient does not use; the flags still select the x11/x32, y11/y32 forms.
    if (kxi == 1) {
        c.x11 = 0.0;
        c.x32 = 0.0;
    } else {
        double rxi = c.r + xi;
        c.x11 = 1.0 / (c.r * rxi);
        c.x32 = (c.r + rxi) * c.x11 * c.x11 * c.ir;
    }
    if (ket == 1) {
        c.y11 = 0.0;
        c.y32 = 0.0;
    } else {
        double ret = c.r + et;
        c.y11 = 1.0 / (c.r * ret);
        c.y32 = (c.r + ret) * c.y11 * c.y11 * c.ir;
    }
    c.ey = dp.sd * c.ir - c.y * q * c.ir3;
    c.ez = dp.cd * c.ir + c.d * q * c.ir3;
    c.fy = c.d * c.ir3 + c.xi2 * c.y32 * dp.sd;
    c.fz = c.y * c.ir3 + c.xi2 * c.y32 * dp.cd;
    c.gy = 2.0 * c.x11 * dp.sd - c.y * q * c.x32;
    c.gz = 2.0 * c.x11 * dp.cd + c.d * q * c.x32;
    c.hy = c.d * q * c.x32 + xi * q * c.y32 * dp.sd;
    c.hz = c.y * q * c.x32 + xi * q * c.y32 * dp.cd;
    return true;
}

// The parts leave out the common factor 1 / (2 pi); the sums apply it once.
// Gradient entries g[0..8] correspond to DC3D's U(4..12):
// uxx, uyx, uzx, uxy, uyy, uzy, uxz, uyz, uzz.
#define OK_K (1.0 / 6.283185307179586)

// Part A (dc3d.f:200-282), strike (s) and dip (d) slip, gradient entries only.
// With a2 = alp2 and h = 1/2 it is the real source's.  Part B (dc3d.f:284-400)
// repeats its terms without the medium constants and with the halves negated, so
// that A + B of the image source is this with a2 = alp2 - 1 and h = -1/2 plus what
// ok_part_b adds.
__device__ inline void ok_part_a(const OkCorner &c, const OkDip &dp, double a1, double a2, double h, double s[9],
                                 double d[9])
{
    const double xi = c.xi, et = c.et, q = c.q;
    const double xy = xi * c.y11, qy = q * c.y11, a1xy = a1 * xy, a1qy = a1 * qy, hxy = h * xy;
    const double xr = a2 * xi, qr = a2 * q, er = a2 * et, qq = qr * q, q3 = qr * c.ir3;
    const double a1r = a1 * c.ir, hx = h * c.x11, a1x = a1 * c.x11;
    s[0] = -a1qy - qr * c.xi2 * c.y32;
    s[1] = -xi * q3;
    s[2] = a1xy + qq * xi * c.y32;
    s[3] = a1xy * dp.sd + xr * c.fy + c.d * hx;
    s[4] = a2 * c.ey;
    s[5] = a1r * dp.cd + a1qy * dp.sd - qr * c.fy;
    s[6] = a1xy * dp.cd + xr * c.fz + c.y * hx;
    s[7] = a2 * c.ez;
    s[8] = a1qy * dp.cd - a1r * dp.sd - qr * c.fz;

    d[0] = s[1];
    d[1] = -h * qy - et * q3;
    d[2] = a1r + q * q3;
    d[3] = s[4];
    d[4] = c.d * a1x + hxy * dp.sd + er * c.gy;
    d[5] = c.y * a1x - qr * c.gy;
    d[6] = s[7];
    d[7] = c.y * a1x + hxy * dp.cd + er * c.gz;
    d[8] = -c.d * a1x - qr * c.gz;
}

// Part B (dc3d.f:284-400) less what ok_part_a covers, added to s and d.
__device__ inline void ok_part_b(const OkCorner &c, const OkDip &dp, double a3, double s[9], double d[9])
{
    const double xi = c.xi, q = c.q, Y = c.y, D = c.d;
    const double ird = 1.0 / (c.r + D);
    const double d11 = c.ir * ird, yd = Y * ird;
    const double aj2 = xi * yd * d11;
    const double aj5 = -(D + Y * yd) * d11;
    // ai1..ai4 enter only the displacement entries and are not formed.
    double ak1, ak3, aj3, aj6;
    if (dp.cd != 0.0) {
        ak1 = xi * (d11 - c.y11 * dp.sd) * dp.icd;
        ak3 = (q * c.y11 - Y * d11) * dp.icd;
        aj3 = (ak1 - aj2 * dp.sd) * dp.icd;
        aj6 = (ak3 - aj5 * dp.sd) * dp.icd;
    } else {
        const double ird2 = ird * ird;
        ak1 = xi * q * ird * d11;
        ak3 = dp.sd * ird * (c.xi2 * d11 - 1.0);
        aj3 = -xi * ird2 * (c.q2 * d11 - 0.5);
        aj6 = -Y * ird2 * (c.xi2 * d11 - 0.5);
    }
    const double xy = xi * c.y11;
    const double ak2 = c.ir + ak3 * dp.sd;
    const double ak4 = xy * dp.cd - ak1 * dp.sd;
    const double aj1 = aj5 * dp.cd - aj6 * dp.sd;
    const double aj4 = -xy - aj2 * dp.cd + aj3 * dp.sd;
    const double as = a3 * dp.sd, ac = a3 * dp.sdcd;
    s[0] -= as * aj1;
    s[1] -= as * aj2;
    s[2] -= as * aj3;
    s[3] += as * (xy + aj4);
    s[4] += as * (c.ir + aj5);
    s[5] -= as * (q * c.y11 - aj6);
    s[6] += as * ak1;
    s[7] += as * (Y * d11);
    s[8] += as * ak2;
    d[0] += ac * aj4;
    d[1] += ac * aj5;
    d[2] += ac * aj6;
    d[3] += ac * aj1;
    d[4] += ac * aj2;
    d[5] += ac * aj3;
    d[6] -= ac * ak3;
    d[7] -= ac * (xi * d11);
    d[8] -= ac * ak4;
}

// Part C (dc3d.f:402-507).  Also returns the displacement entries 1..3 of part C
// (cs for strike, cdp for dip), which the image sum adds to the z-derivatives.
__device__ inline void ok_part_c(const OkCorner &c, const OkDip &dp, const OkMed &m, double Z,
                                 double s[9], double d[9], double cs[3], double cdp[3])
{
    const double xi = c.xi, et = c.et, q = c.q, Y = c.y, D = c.d, sd = dp.sd, cd = dp.cd;
    const double a4 = m.alp4, a5 = m.alp5, X11 = c.x11, X32 = c.x32, Y32 = c.y32;
    const double C = D + Z, aC = a5 * C;
    const double x53 = (8.0 * c.r2 + 9.0 * c.r * xi + 3.0 * c.xi2) * X11 * X11 * X11 * c.ir2;
    const double y53 = (8.0 * c.r2 + 9.0 * c.r * et + 3.0 * c.et2) * c.y11 * c.y11 * c.y11 * c.ir2;
    const double r3 = c.ir3, t5 = 3.0 * c.ir5;
    const double qR = q * r3, yR = Y * r3, dR = D * r3, eR = et * r3, sR = sd * r3, cR = cd * r3;
    const double h = q * cd - Z, qY = q * Y32;
    const double z32 = sR - h * Y32;
    const double z53 = sd * t5 - h * y53;
    const double y0 = c.y11 - c.xi2 * Y32;
    const double z0 = z32 - c.xi2 * z53;
    const double ppy = cR + qY * sd;
    const double ppz = sR - qY * cd;
    const double qq = Z * Y32 + z32 + z0;
    const double Ct = C * t5;
    const double qqy = Ct * D - qq * sd;
    const double qqz = Ct * Y - qq * cd + qY;
    const double xy = xi * c.y11, qy = q * c.y11;
    const double ar = a5 * Ct * q;             // a5 C qr
    const double acdr = a5 * (C + D) * r3;     // a5 cdr
    const double yy0 = yR - y0 * cd, qz0 = q * z0;
    const double w1 = acdr * sd - ar * Y, w2 = acdr * cd + ar * D;
    const double eq = et * q, aCq = aC * qR;

    cs[0] = xi * (a4 * c.y11 * cd - a5 * q * z32);
    cs[1] = a4 * (cd * c.ir + 2.0 * qy * sd) - aCq;
    cs[2] = a4 * qy * cd - aC * eR + a5 * (Z * c.y11 - c.xi2 * z32);
    s[0] = a4 * y0 * cd - a5 * qz0;
    s[1] = xi * (ar - a4 * (cR + 2.0 * qY * sd));
    s[2] = xi * (a5 * (Ct * et - qq) - a4 * qY * cd);
    s[3] = -xi * (a4 * ppy * cd + a5 * qqy);
    s[4] = a4 * 2.0 * (dR - y0 * sd) * sd - yR * cd - w1 + a5 * eR;
    s[5] = yy0 * sd - a4 * qR + w2 - a5 * sd * (y0 * cd + qz0);
    s[6] = xi * (a4 * ppz * cd - a5 * qqz);
    s[7] = a4 * 2.0 * (yR - y0 * cd) * sd + dR * cd - w2;
    s[8] = yy0 * cd - w1 + a5 * (y0 * dp.sdsd - qz0 * cd);

    const double xe = eq * x53, xq = c.q2 * x53, q2c = 2.0 * q * cd, q2s = 2.0 * q * sd;
    cdp[0] = a4 * cd * c.ir - qy * sd - aCq;
    cdp[1] = a4 * Y * X11 - aC * eq * X32;
    cdp[2] = -D * X11 - xy * sd - aC * (X11 - c.q2 * X32);
    d[0] = xi * (ar - a4 * cR + qY * sd);
    d[1] = ar * et - a4 * yR;
    d[2] = dR - y0 * sd + aC * r3 * (1.0 - 3.0 * c.q2 * c.ir2);
    d[3] = y0 * dp.sdsd - a4 * eR - w1;
    d[4] = a4 * (X11 - Y * Y * X32) - aC * ((D + q2c) * X32 - Y * xe);
    d[5] = xi * ppy * sd + Y * D * X32 + aC * ((Y + q2s) * X32 - Y * xq);
    d[6] = y0 * dp.sdcd - qR - w2;
    d[7] = a4 * Y * D * X32 - aC * ((Y - q2s) * X32 + D * xe);
    d[8] = X11 - xi * ppz * sd - D * D * X32 - aC * ((D - q2c) * X32 - D * xq);
}

// Part C's displacement entries are the same statements as DU(1..3) of UC.

// Singular-edge rejection and negative-extension flags (dc3d.f:70-87).
__device__ inline bool ok_edges(const double xi[2], const double et[2], double q, double eps,
                                int kxi[2], int ket[2])
{
    if (q == 0.0 && ((xi[0] * xi[1] <= 0.0 && et[0] * et[1] == 0.0) ||
                     (et[0] * et[1] <= 0.0 && xi[0] * xi[1] == 0.0)))
        return true;
    double r12 = sqrt(xi[0] * xi[0] + et[1] * et[1] + q * q);
    double r21 = sqrt(xi[1] * xi[1] + et[0] * et[0] + q * q);
    double r22 = sqrt(xi[1] * xi[1] + et[1] * et[1] + q * q);
    kxi[0] = (xi[0] < 0.0 && r21 + xi[1] < eps);
    kxi[1] = (xi[0] < 0.0 && r22 + xi[1] < eps);
    ket[0] = (et[0] < 0.0 && r12 + et[1] < eps);
    ket[1] = (et[0] < 0.0 && r22 + et[1] < eps);
    return false;
}

// Displacement gradient for unit strike slip (gs) and unit dip slip (gd) of a
// source at (depth, dip) spanning x in [0, al2] and eta in [aw1, 0], observed at
// (x, y, z) in the DC3D frame (x along strike, z up).  Returns false on the
// singular edge (gradients zero).
template <bool R32>
__device__ inline bool ok_dc3d_grad(const OkMed &m, const OkDip &dp, double x, double y, double z,
                                    double depth, double al2, double aw1, double gs[9],
                                    double gd[9])
{
    const double eps = R32 ? (double)1.0e-6f : 1.0e-6;
#pragma unroll
    for (int i = 0; i < 9; i++) { gs[i] = 0.0; gd[i] = 0.0; }
    double xi[2], et[2];
    if (R32) {
        xi[0] = (double)((float)x - 0.0f);
        xi[1] = (double)((float)x - (float)al2);
    } else {
        xi[0] = x;
        xi[1] = x - al2;
    }
    if (fabs(xi[0]) < eps) xi[0] = 0.0;
    if (fabs(xi[1]) < eps) xi[1] = 0.0;
    int kxi[2], ket[2];
    OkCorner c;
    double as[9], ad[9];

    // real source
    {
        double D = R32 ? (double)((float)depth + (float)z) : depth + z;
        double p = y * dp.cd + D * dp.sd;
        double q = y * dp.sd - D * dp.cd;
        et[0] = p - aw1;
        et[1] = p;
        if (fabs(q) < eps) q = 0.0;
        if (fabs(et[0]) < eps) et[0] = 0.0;
        if (fabs(et[1]) < eps) et[1] = 0.0;
        if (ok_edges(xi, et, q, eps, kxi, ket)) goto singular;
#pragma unroll 1
        for (int kk = 0; kk < 4; kk++) {
            const int k = kk >> 1, j = kk & 1;
            ok_corner(xi[j], et[k], q, dp, kxi[k], ket[j], c);
            ok_part_a(c, dp, m.alp1, m.alp2, 0.5, as, ad);
            const double sg = (j + k != 1) ? 1.0 : -1.0;
#pragma unroll
            for (int i = 0; i < 9; i++) {
                gs[i] += sg * as[i];
                gd[i] += sg * ad[i];
            }
        }
        // rows 1..3 of DC3D's 4x3 block rotation; the z-derivative row is negated
#pragma unroll
        for (int t = 0; t < 2; t++) {
            double *g = t ? gd : gs;
#pragma unroll
            for (int r = 0; r < 9; r += 3) {
                const double f = r == 6 ? 1.0 : -1.0, a1 = g[r + 1], a2 = g[r + 2];
                g[r] = f * g[r];
                g[r + 1] = f * (a1 * dp.cd - a2 * dp.sd);
                g[r + 2] = f * (a1 * dp.sd + a2 * dp.cd);
            }
        }
    }
    // image source
    {
        double D = R32 ? (double)((float)depth - (float)z) : depth - z;
        double p = y * dp.cd + D * dp.sd;
        double q = y * dp.sd - D * dp.cd;
        et[0] = p - aw1;
        et[1] = p;
        if (fabs(q) < eps) q = 0.0;
        if (fabs(et[0]) < eps) et[0] = 0.0;
        if (fabs(et[1]) < eps) et[1] = 0.0;
        if (ok_edges(xi, et, q, eps, kxi, ket)) goto singular;
#pragma unroll 1
        for (int kk = 0; kk < 4; kk++) {
            const int k = kk >> 1, j = kk & 1;
            ok_corner(xi[j], et[k], q, dp, kxi[k], ket[j], c);
            double cs9[9], cd9[9], c0s[3], c0d[3];
            ok_part_a(c, dp, m.alp1, m.alp2 - 1.0, -0.5, as, ad);
            ok_part_b(c, dp, m.alp3, as, ad);
            ok_part_c(c, dp, m, z, cs9, cd9, c0s, c0d);
            const double sg = (j + k != 1) ? 1.0 : -1.0;
#pragma unroll
            for (int t = 0; t < 2; t++) {
                const double *a = t ? ad : as;
                const double *cc = t ? cd9 : cs9;
                const double *c0 = t ? c0d : c0s;
                double *g = t ? gd : gs;
                double du[9];
#pragma unroll
                for (int r = 0; r < 3; r++) {
                    const int i = 3 * r;
                    du[i] = a[i] + z * cc[i];
                    du[i + 1] = (a[i + 1] + z * cc[i + 1]) * dp.cd - (a[i + 2] + z * cc[i + 2]) * dp.sd;
                    du[i + 2] = (a[i + 1] - z * cc[i + 1]) * dp.sd + (a[i + 2] - z * cc[i + 2]) * dp.cd;
                }
                du[6] = du[6] + c0[0];
                du[7] = du[7] + c0[1] * dp.cd - c0[2] * dp.sd;
                du[8] = du[8] - c0[1] * dp.sd - c0[2] * dp.cd;
#pragma unroll
                for (int i = 0; i < 9; i++) g[i] += sg * du[i];
            }
        }
    }
#pragma unroll
    for (int i = 0; i < 9; i++) {
        gs[i] *= OK_K;
        gd[i] *= OK_K;
        if (R32) {
            gs[i] = (double)__double2float_rn(gs[i]);
            gd[i] = (double)__double2float_rn(gd[i]);
        }
    }
    return true;
singular:
#pragma unroll
    for (int i = 0; i < 9; i++) { gs[i] = 0.0; gd[i] = 0.0; }
    return false;
}

// ---- displacement (observation points) ------------------------------------------

// The displacement entries DU(1..3) of parts A/B/C need three more corner
// quantities of DCCON2 (dc3d.f:596-665): TT, ALX, ALE.
struct OkLogs {
    double tt, alx, ale;
};

__device__ inline OkLogs ok_logs(const OkCorner &c, int kxi, int ket)
{
    OkLogs l;
    l.tt = (c.q == 0.0) ? 0.0 : atan(c.xi * c.et / (c.q * c.r));
    l.alx = (kxi == 1) ? -log(c.r - c.xi) : log(c.r + c.xi);
    l.ale = (ket == 1) ? -log(c.r - c.et) : log(c.r + c.et);
    return l;
}

// Part A (dc3d.f:200-282) DU(1..3), strike (s) and dip (d) slip.
__device__ inline void ok_part_a_disp(const OkCorner &c, const OkLogs &l, const OkMed &m, double s[3],
                                      double d[3])
{
    const double qx = c.q * c.x11, qy = c.q * c.y11;
    s[0] = OK_K * (l.tt / 2.0 + m.alp2 * c.xi * qy);
    s[1] = OK_K * (m.alp2 * c.q / c.r);
    s[2] = OK_K * (m.alp1 * l.ale - m.alp2 * c.q * qy);
    d[0] = OK_K * (m.alp2 * c.q / c.r);
    d[1] = OK_K * (l.tt / 2.0 + m.alp2 * c.et * qx);
    d[2] = OK_K * (m.alp1 * l.alx - m.alp2 * c.q * qx);
}

// Part B (dc3d.f:284-400) DU(1..3), with the I1..I4 terms the gradient does not use.
__device__ inline void ok_part_b_disp(const OkCorner &c, const OkLogs &l, const OkDip &dp, const OkMed &m,
                                      double s[3], double d[3])
{
    const double xi = c.xi, et = c.et, q = c.q, R = c.r, Y = c.y;
    const double rd = R + c.d;
    double ai3, ai4;
    if (dp.cd != 0.0) {
        if (xi == 0.0) {
            ai4 = 0.0;
        } else {
            const double x = sqrt(c.xi2 + c.q2);
            ai4 = 1.0 / dp.cdcd * (xi / rd * dp.sdcd +
                  2.0 * atan((et * (x + q * dp.cd) + x * (R + x) * dp.sd) / (xi * (R + x) * dp.cd)));
        }
        ai3 = (Y * dp.cd / rd - l.ale + dp.sd * log(rd)) / dp.cdcd;
    } else {
        const double rd2 = rd * rd;
        ai3 = (et / rd + Y * q / rd2 - l.ale) / 2.0;
        ai4 = xi * Y / rd2 / 2.0;
    }
    const double ai1 = -xi / rd * dp.cd - ai4 * dp.sd;
    const double ai2 = log(rd) + ai3 * dp.sd;
    const double qx = q * c.x11, qy = q * c.y11, a3 = m.alp3;
    s[0] = OK_K * (-xi * qy - l.tt - a3 * ai1 * dp.sd);
    s[1] = OK_K * (-q / R + a3 * Y / rd * dp.sd);
    s[2] = OK_K * (q * qy - a3 * ai2 * dp.sd);
    d[0] = OK_K * (-q / R + a3 * ai3 * dp.sdcd);
    d[1] = OK_K * (-et * qx - l.tt - a3 * xi / rd * dp.sdcd);
    d[2] = OK_K * (q * qx + a3 * ai4 * dp.sdcd);
}

// Displacement (ux, uy, uz in the DC3D frame) for unit strike slip (us) and
// unit dip slip (ud): DC3D's U(1..3) (dc3d.f:1-198) with the same corner
// loop, snapping, edge rejection and REAL*4 handling as ok_dc3d_grad.
template <bool R32>
__device__ inline bool ok_dc3d_disp(const OkMed &m, const OkDip &dp, double x, double y, double z,
                                    double depth, double al2, double aw1, double us[3], double ud[3])
{
    const double eps = R32 ? (double)1.0e-6f : 1.0e-6;
    for (int i = 0; i < 3; i++) { us[i] = 0.0; ud[i] = 0.0; }
    double xi[2], et[2];
    if (R32) {
        xi[0] = (double)((float)x - 0.0f);
        xi[1] = (double)((float)x - (float)al2);
    } else {
        xi[0] = x;
        xi[1] = x - al2;
    }
    if (fabs(xi[0]) < eps) xi[0] = 0.0;
    if (fabs(xi[1]) < eps) xi[1] = 0.0;
    int kxi[2], ket[2];
    OkCorner c;
#pragma unroll 1
    for (int img = 0; img < 2; img++) {
        const double D = R32 ? (double)(img ? (float)depth - (float)z : (float)depth + (float)z)
                             : (img ? depth - z : depth + z);
        const double p = y * dp.cd + D * dp.sd;
        double q = y * dp.sd - D * dp.cd;
        et[0] = p - aw1;
        et[1] = p;
        if (fabs(q) < eps) q = 0.0;
        if (fabs(et[0]) < eps) et[0] = 0.0;
        if (fabs(et[1]) < eps) et[1] = 0.0;
        if (ok_edges(xi, et, q, eps, kxi, ket)) {
            for (int i = 0; i < 3; i++) { us[i] = 0.0; ud[i] = 0.0; }
            return false;
        }
#pragma unroll 1
        for (int kk = 0; kk < 4; kk++) {
            const int k = kk >> 1, j = kk & 1;
            ok_corner(xi[j], et[k], q, dp, kxi[k], ket[j], c);
            const OkLogs l = ok_logs(c, kxi[k], ket[j]);
            double as[3], ad[3];
            ok_part_a_disp(c, l, m, as, ad);
            const double sg = (j + k != 1) ? 1.0 : -1.0;
            if (!img) {
#pragma unroll
                for (int t = 0; t < 2; t++) {
                    const double *a = t ? ad : as;
                    double *u = t ? ud : us;
                    const double du0 = -a[0];
                    const double du1 = -a[1] * dp.cd + a[2] * dp.sd;
                    const double du2 = -a[1] * dp.sd - a[2] * dp.cd;
                    u[0] = (sg > 0.0) ? u[0] + du0 : u[0] - du0;
                    u[1] = (sg > 0.0) ? u[1] + du1 : u[1] - du1;
                    u[2] = (sg > 0.0) ? u[2] + du2 : u[2] - du2;
                }
            } else {
                double bs[3], bd[3], cs9[9], cd9[9], c0s[3], c0d[3];
                ok_part_b_disp(c, l, dp, m, bs, bd);
                ok_part_c(c, dp, m, z, cs9, cd9, c0s, c0d);
#pragma unroll
                for (int t = 0; t < 2; t++) {
                    const double *a = t ? ad : as;
                    const double *b = t ? bd : bs;
                    const double *cc = t ? c0d : c0s;
                    double *u = t ? ud : us;
                    const double zk = z * OK_K;
                    const double du0 = a[0] + b[0] + zk * cc[0];
                    const double du1 = (a[1] + b[1] + zk * cc[1]) * dp.cd - (a[2] + b[2] + zk * cc[2]) * dp.sd;
                    const double du2 = (a[1] + b[1] - zk * cc[1]) * dp.sd + (a[2] + b[2] - zk * cc[2]) * dp.cd;
                    u[0] = (sg > 0.0) ? u[0] + du0 : u[0] - du0;
                    u[1] = (sg > 0.0) ? u[1] + du1 : u[1] - du1;
                    u[2] = (sg > 0.0) ? u[2] + du2 : u[2] - du2;
                }
            }
        }
    }
    if (R32) {
        for (int i = 0; i < 3; i++) {
            us[i] = (double)__double2float_rn(us[i]);
            ud[i] = (double)__double2float_rn(ud[i]);
        }
    }
    return true;
}

#undef OK_K

}  // namespace ucg
