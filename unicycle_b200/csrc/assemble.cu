// Assembly of the stress-interaction matrix K on the device.
//
// K is row-major with m rows (receiver force DOFs) and n columns (source DOFs);
// row k of K is column k of the reference's G(n,m) (fortran/3d/src/greens.f90:
// 73-275), so the reference layout is a plain copy:
//   rows:    patches 3 per element (ts, td, tn), volumes 6 (s11'..s33'),
//            elements ordered rectangles, triangles, volumes;
//   columns: rectangles 2 per source (strike, dip slip), triangles 2, volumes 6
//            (unit eigenstrain 11, 12, 13, 22, 23, 33), component fastest.
//
// One thread per (receiver, source) pair computes every unit component of the
// source at once, sharing the pair geometry, and writes them as contiguous
// columns: a warp covers 32 consecutive sources of one receiver, so each of its
// row stores is one coalesced 512-byte (patches) segment.  Per-source constants are
// formed once and read through the read-only path: the rectangles' (frames, the
// REAL*4-rounded DC3D inputs) and the cuboids' on the host, the triangles' records and
// their mesh edges' by a kernel from the vertices.
#include <algorithm>
#include <cmath>
#include <cstring>
#include "ucg_internal.cuh"
#include "okada92.cuh"
#include "nikkhoo15.cuh"
#include "strainvolume.cuh"
#include "blocks.cuh"

namespace ucg {

// ---- receivers -----------------------------------------------------------------

// receiver record: xc[3], sv[3], dv[3], nv[3]
enum { RC_X = 0, RC_S = 3, RC_D = 6, RC_N = 9, RC_SIZE = 12 };

// the NR rows of a receiver record from a stress (s11, s12, s13, s22, s23, s33)
template <int NR>
__device__ __forceinline__ void ned_rows(const double *r, const double s[6], double o[NR])
{
    receiver_rows<NR>(r + RC_S, r + RC_D, r + RC_N, s[0], s[1], s[2], s[3], s[4], s[5], o);
}

// ---- rectangles (Okada 1992) -------------------------------------------------

enum { RS_Q1 = 0, RS_Q2, RS_CS, RS_SS, RS_DEPTH, RS_AL2, RS_AW1, RS_SD, RS_CD, RS_SDSD, RS_CDCD,
       RS_SDCD, RS_ICD, RS_SIZE };

// Stress (s11, s12, s13, s22, s23, s33 for strike and dip slip) at receiver
// point (x1, x2, x3) of one rectangle record sr (okada92.f90:121-205).
template <bool R32>
__device__ __forceinline__ void rect_pair_sig(const double sr[RS_SIZE], const OkDip &dp, double x1, double x2,
                                              double x3, const OkMed &med, double mu, double lambda,
                                              double sig[2][6])
{
    const double csst = sr[RS_CS], ssst = sr[RS_SS];
    double x = (x1 - sr[RS_Q1]) * csst + (x2 - sr[RS_Q2]) * ssst;
    double y = (x1 - sr[RS_Q1]) * ssst - (x2 - sr[RS_Q2]) * csst;
    double z = -x3;
    if (R32) {
        x = (double)__double2float_rn(x);
        y = (double)__double2float_rn(y);
        z = (double)__double2float_rn(z);
    }
    double gs[9], gd[9];
    ok_dc3d_grad<R32>(med, dp, x, y, z, sr[RS_DEPTH], sr[RS_AL2], sr[RS_AW1], gs, gd);
#pragma unroll
    for (int t = 0; t < 2; t++) {
        const double *g = t ? gd : gs;
        // okada92.f90:165-205: rotate the gradient back from the strike frame
        const double uxx = g[0], uyx = g[1], uzx = g[2], uxy = g[3], uyy = g[4], uzy = g[5];
        const double uxz = g[6], uyz = g[7], uzz = g[8];
        const double uxxr = (csst * uxx + ssst * uyx) * csst - (-csst * uxy - ssst * uyy) * ssst;
        const double uxyr = (csst * uxx + ssst * uyx) * ssst + (-csst * uxy - ssst * uyy) * csst;
        const double uxzr = -csst * uxz + ssst * uyz;
        const double uyxr = (ssst * uxx - csst * uyx) * csst - (-ssst * uxy + csst * uyy) * ssst;
        const double uyyr = (ssst * uxx - csst * uyx) * ssst + (-ssst * uxy + csst * uyy) * csst;
        const double uyzr = -ssst * uxz + csst * uyz;
        const double uzxr = -csst * uzx - ssst * uzy;
        const double uzyr = -ssst * uzx + csst * uzy;
        const double e11 = uxxr, e12 = (uxyr + uyxr) / 2.0, e13 = (uxzr + uzxr) / 2.0;
        const double e22 = uyyr, e23 = (uyzr + uzyr) / 2.0, e33 = uzz;
        const double ekk = e11 + e22 + e33;
        sig[t][0] = lambda * ekk + 2.0 * mu * e11;
        sig[t][1] = 2.0 * mu * e12;
        sig[t][2] = 2.0 * mu * e13;
        sig[t][3] = lambda * ekk + 2.0 * mu * e22;
        sig[t][4] = 2.0 * mu * e23;
        sig[t][5] = lambda * ekk + 2.0 * mu * e33;
    }
}

__device__ __forceinline__ void rect_record(const double *__restrict__ src, int ns, int j, double sr[RS_SIZE],
                                            OkDip &dp)
{
#pragma unroll
    for (int f = 0; f < RS_SIZE; f++) sr[f] = __ldg(src + (long)f * ns + j);
    dp.sd = sr[RS_SD]; dp.cd = sr[RS_CD]; dp.sdsd = sr[RS_SDSD]; dp.cdcd = sr[RS_CDCD];
    dp.sdcd = sr[RS_SDCD];
    dp.icd = sr[RS_ICD];
}

// Bound by the FP64 pipe.  Divisions were 60 of a corner's operations and each is
// a sequence of its own with a branch, which kept the warps waiting (28 % of the
// pipe's cycles); four reciprocals a corner are left, parts A and B of the image
// share their terms and the real source is rotated once, after its corner sum.
// 2,048 rectangles on as many receivers: 3.21 -> 0.93 ms (65 % of the pipe, 240
// registers, 8 warps an SM).
template <bool R32, int NR>
__global__ void __launch_bounds__(128) k_assemble_rect(double *__restrict__ K, long n, long row0,
        const double *__restrict__ rcv, int r0, int r1, const double *__restrict__ src, int ns, OkMed med, double mu,
        double lambda)
{
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= ns) return;
    double sr[RS_SIZE];
    OkDip dp;
    rect_record(src, ns, j, sr, dp);
    for (int e = r0 + blockIdx.y; e < r1; e += gridDim.y) {
        const double *rc = rcv + (long)e * RC_SIZE;
        double sig[2][6], rloc[RC_SIZE], oS[NR], oD[NR];
        rect_pair_sig<R32>(sr, dp, __ldg(rc + 0), __ldg(rc + 1), __ldg(rc + 2), med, mu, lambda, sig);
#pragma unroll
        for (int f = 0; f < RC_SIZE; f++) rloc[f] = __ldg(rc + f);
        ned_rows<NR>(rloc, sig[0], oS);
        ned_rows<NR>(rloc, sig[1], oD);
#pragma unroll
        for (int c = 0; c < NR; c++)
            *reinterpret_cast<double2 *>(K + (row0 + (long)NR * (e - r0) + c) * n + 2L * j) = make_double2(oS[c], oD[c]);
    }
}

// ---- triangles (Nikkhoo & Walter 2015) -----------------------------------------
//
// Two kernels per batch of receivers.  k_tri_edges forms the free-surface term
// of every mesh edge for unit slip along east, north and up (9 or 18 values per
// receiver) into a scratch small enough to stay in L2; k_assemble_tri adds, for
// every triangle, its main and image dislocations and its three edges times its
// slip directions, and writes K once.  A mesh of N triangles has about 1.5 N
// edges against 3 N sides.
//
// Bound by the FP64 pipe: 74 % active in k_tri_edges (254 registers, 8 warps an
// SM), 58 % in k_assemble_tri (164 registers, 12 warps; the rest waits on record
// loads and the scratch).  FP64 instructions per pair: 970 for the triangle's own
// dislocations and 1,150 per edge, against 12,050 for the free-surface term of a
// pair on single-direction duals, one side at a time.  N = 5,000: 68 -> 8.5 ms,
// N = 20,000: 893 -> 132 ms (3 % of it the HBM writes of K).  Triangles in one
// pass instead of three also drops the two re-reads of K.

// position and unit vectors of a receiver, NED -> ENU
__device__ __forceinline__ void enu_receiver(const double *rc, double X[3], double vs[3], double vd[3], double vn[3])
{
    const double *v[4] = {rc + RC_X, rc + RC_S, rc + RC_D, rc + RC_N};
    double *o[4] = {X, vs, vd, vn};
#pragma unroll
    for (int k = 0; k < 4; k++) {
        o[k][0] = __ldg(v[k] + 1);
        o[k][1] = __ldg(v[k]);
        o[k][2] = -__ldg(v[k] + 2);
    }
}

__device__ __forceinline__ void load_edge(const TriTables &t, int j, double e[NE_SIZE])
{
#pragma unroll
    for (int f = 0; f < NE_SIZE; f++) e[f] = __ldg(t.ed + (long)f * t.ne + j);
}

template <int NR>
__global__ void __launch_bounds__(128) k_tri_edges(double *__restrict__ sc, const double *__restrict__ rcv, int r0,
        int r1, TriTables tab, NwConst cst)
{
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= tab.ne) return;
    double ed[NE_SIZE];
    load_edge(tab, j, ed);
    for (int e = r0 + blockIdx.y; e < r1; e += gridDim.y) {
        double X[3], vs[3], vd[3], vn[3], o[NR][3];
        enu_receiver(rcv + (long)e * RC_SIZE, X, vs, vd, vn);
        nw_edge_rows<NR>(X, vs, vd, vn, ed, cst, o);
        double *p = sc + (long)(e - r0) * (3 * NR) * tab.ne + j;
#pragma unroll
        for (int q = 0; q < NR; q++)
#pragma unroll
            for (int x = 0; x < 3; x++) p[(long)(3 * q + x) * tab.ne] = o[q][x];
    }
}

// slip of the strike and dip modes (ENU): the strike axis and minus the dip
// axis of the TD frame (nikkhoo15.f90:140)
__device__ __forceinline__ void tri_slip(const NwRec &R, double bS[3], double bD[3])
{
#pragma unroll
    for (int k = 0; k < 3; k++) {
        bS[k] = R[NW_MAIN + TD_S + k];
        bD[k] = -R[NW_MAIN + TD_D + k];
    }
}

// main and image dislocation of triangle j (R), summed into oS, oD
template <int NR>
__device__ __forceinline__ void tri_rows(const double X[3], const double vs[3], const double vd[3],
                                         const double vn[3], const NwRec &R, const NwConst &cst, double oS[NR],
                                         double oD[NR])
{
#pragma unroll
    for (int q = 0; q < NR; q++) oS[q] = oD[q] = 0.0;
#pragma unroll 1
    for (int part = 0; part < 2; part++) {
        const bool flip = part && R[NW_SURF] != 0.0;
        if (!nw_td_rows<NR>(X, vs, vd, vn, R, part ? NW_IMG : NW_MAIN, flip, cst, oS, oD)) {
#pragma unroll
            for (int q = 0; q < NR; q++) oS[q] = oD[q] = nan("");
        }
    }
}

template <int NR>
__global__ void __launch_bounds__(128) k_assemble_tri(double *__restrict__ K, long n, long col0, long row0,
        const double *__restrict__ sc, const double *__restrict__ rcv, int r0, int r1, TriTables tab, NwConst cst)
{
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= tab.ns) return;
    const NwRec R{tab.rec + j, (long)tab.ns};
    for (int e = r0 + blockIdx.y; e < r1; e += gridDim.y) {
        double X[3], vs[3], vd[3], vn[3], oS[NR], oD[NR], bS[3], bD[3];
        enu_receiver(rcv + (long)e * RC_SIZE, X, vs, vd, vn);
        tri_rows<NR>(X, vs, vd, vn, R, cst, oS, oD);
        tri_slip(R, bS, bD);
#pragma unroll
        for (int side = 0; side < 3; side++) {
            const int id = __ldg(tab.edge + (long)side * tab.ns + j);
            const double sg = (id & 1) ? -1.0 : 1.0;
            const double *p = sc + (long)(e - r0) * (3 * NR) * tab.ne + (id >> 1);
#pragma unroll
            for (int q = 0; q < NR; q++) {
                const double a = p[(long)(3 * q) * tab.ne], b = p[(long)(3 * q + 1) * tab.ne],
                             c = p[(long)(3 * q + 2) * tab.ne];
                oS[q] += sg * (a * bS[0] + b * bS[1] + c * bS[2]);
                oD[q] += sg * (a * bD[0] + b * bD[1] + c * bD[2]);
            }
        }
#pragma unroll
        for (int q = 0; q < NR; q++)
            *reinterpret_cast<double2 *>(K + (row0 + (long)NR * (e - r0) + q) * n + col0 + 2L * j) =
                make_double2(oS[q], oD[q]);
    }
}

// source records from the vertices (north, east, down): one thread per triangle
// and per edge
__global__ void k_tri_prepare(const double *__restrict__ vert, const int *__restrict__ id, int ns,
                              double *__restrict__ rec)
{
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= ns) return;
    double P[3][3], r[NW_SIZE];
    for (int k = 0; k < 3; k++) {
        // NED -> ENU (nikkhoo15.f90:143-146)
        const double *v = vert + 3L * id[(long)k * ns + j];
        P[k][0] = v[1]; P[k][1] = v[0]; P[k][2] = -v[2];
    }
    nw_prepare(P[0], P[1], P[2], r);
    for (int f = 0; f < NW_SIZE; f++) rec[(long)f * ns + j] = r[f];
}

__global__ void k_edge_prepare(const double *__restrict__ vert, const int2 *__restrict__ ends, int ne,
                               double *__restrict__ ed)
{
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= ne) return;
    const double *a = vert + 3L * ends[j].x, *b = vert + 3L * ends[j].y;
    const double PA[3] = {a[1], a[0], -a[2]}, PB[3] = {b[1], b[0], -b[2]};
    double r[NE_SIZE];
    nw_prepare_edge(PA, PB, r);
    for (int f = 0; f < NE_SIZE; f++) ed[(long)f * ne + j] = r[f];
}

// ---- strain volumes (Barbot, Moore & Lambert 2017) -------------------------------
//
// Bound by the FP64 pipe and its divisions (sv_strain; 254 registers, 8 warps an
// SM).  1,024 cuboids on 2,048 receivers: 38.3 -> 1.46 ms (0.70 ns a pair) after the
// 27 dual-number integrals a corner gave way to their corner sums; patch and volume
// receivers are separate launches so that their row counts are known at compile time.

template <int NR>
__global__ void __launch_bounds__(128) k_assemble_vol(double *__restrict__ K, long n, long col0, long row0,
        const double *__restrict__ rcv, int r0, int r1, const double *__restrict__ rec, int ns, double mu, double nu)
{
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= ns) return;
    const SvRec R{rec + j, (long)ns};
    for (int e = r0 + blockIdx.y; e < r1; e += gridDim.y) {
        const double *rc = rcv + (long)e * RC_SIZE;
        double rloc[RC_SIZE], o[6][NR];
#pragma unroll
        for (int f = 0; f < RC_SIZE; f++) rloc[f] = __ldg(rc + f);
        sv_pair_rows<NR>(rloc, R, mu, nu, o);
#pragma unroll
        for (int c = 0; c < NR; c++) {
            double2 *p = reinterpret_cast<double2 *>(K + (row0 + (long)NR * (e - r0) + c) * n + col0 + 6L * j);
            p[0] = make_double2(o[0][c], o[1][c]);
            p[1] = make_double2(o[2][c], o[3][c]);
            p[2] = make_double2(o[4][c], o[5][c]);
        }
    }
}

// ---- dense blocks of K for the hierarchical approximation -------------------------
//
// Many blocks in one launch.  A CTA takes one tile, BLOCK_TILE consecutive
// (receiver, source) pairs of one block in row-major order, so that its threads
// read the same few source records (kept in the permuted order) from L1 and write
// consecutive columns.  Patches only: 3 traction rows a receiver, 2 slip columns
// a source.  One launch per block and pass, as before, left the device waiting
// for launches: 7,500 blocks at N = 7,200 (build 223 -> 70 ms, 26 ms of it these kernels;
// N = 20,000: 3.6 s with the old pair kernels -> 0.47 s).

constexpr int BLOCK_TILE = 512;

template <bool R32>
__global__ void __launch_bounds__(128) k_blocks_rect(const BlockJob *__restrict__ jobs, const int2 *__restrict__ tiles,
        const int *__restrict__ perm, const double *__restrict__ rcv, const double *__restrict__ src, int ns,
        OkMed med, double mu, double lambda)
{
    const int2 tile = tiles[blockIdx.x];
    const BlockJob J = jobs[tile.x];
    const int pairs = J.nr * J.ns, last = min(pairs, tile.y + BLOCK_TILE);
    const long ld = 2L * J.ns;
    for (int p = tile.y + threadIdx.x; p < last; p += blockDim.x) {
        const int ii = p / J.ns, jj = p - ii * J.ns;
        double sr[RS_SIZE], rloc[RC_SIZE], sig[2][6], tS[3], tD[3];
        OkDip dp;
        rect_record(src, ns, J.s0 + jj, sr, dp);
        const double *rc = rcv + (long)__ldg(perm + J.r0 + ii) * RC_SIZE;
#pragma unroll
        for (int f = 0; f < RC_SIZE; f++) rloc[f] = __ldg(rc + f);
        rect_pair_sig<R32>(sr, dp, rloc[0], rloc[1], rloc[2], med, mu, lambda, sig);
        ned_rows<3>(rloc, sig[0], tS);
        ned_rows<3>(rloc, sig[1], tD);
#pragma unroll
        for (int c = 0; c < 3; c++)
            *reinterpret_cast<double2 *>(J.out + (3L * ii + c) * ld + 2L * jj) = make_double2(tS[c], tD[c]);
    }
}

__global__ void __launch_bounds__(128) k_blocks_tri(const BlockJob *__restrict__ jobs, const int2 *__restrict__ tiles,
        const int *__restrict__ perm, const double *__restrict__ rcv, TriTables tab, NwConst cst)
{
    const int2 tile = tiles[blockIdx.x];
    const BlockJob J = jobs[tile.x];
    const int pairs = J.nr * J.ns, last = min(pairs, tile.y + BLOCK_TILE);
    const long ld = 2L * J.ns;
    for (int p = tile.y + threadIdx.x; p < last; p += blockDim.x) {
        const int ii = p / J.ns, jj = p - ii * J.ns, j = J.s0 + jj;
        const NwRec R{tab.rec + j, (long)tab.ns};
        double X[3], vs[3], vd[3], vn[3], oS[3], oD[3], bS[3], bD[3];
        enu_receiver(rcv + (long)__ldg(perm + J.r0 + ii) * RC_SIZE, X, vs, vd, vn);
        tri_rows<3>(X, vs, vd, vn, R, cst, oS, oD);
        tri_slip(R, bS, bD);
#pragma unroll 1
        for (int side = 0; side < 3; side++) {
            const int id = __ldg(tab.edge + (long)side * tab.ns + j);
            const double sg = (id & 1) ? -1.0 : 1.0;
            double ed[NE_SIZE], o[3][3];
            load_edge(tab, id >> 1, ed);
            nw_edge_rows<3>(X, vs, vd, vn, ed, cst, o);
#pragma unroll
            for (int q = 0; q < 3; q++) {
                oS[q] += sg * (o[q][0] * bS[0] + o[q][1] * bS[1] + o[q][2] * bS[2]);
                oD[q] += sg * (o[q][0] * bD[0] + o[q][1] * bD[1] + o[q][2] * bD[2]);
            }
        }
#pragma unroll
        for (int c = 0; c < 3; c++)
            *reinterpret_cast<double2 *>(J.out + (3L * ii + c) * ld + 2L * jj) = make_double2(oS[c], oD[c]);
    }
}

// ---- observation points: the displacement kernels O (buildO) ---------------------
//
// O is row-major with 3 nobs rows (north, east, down per point) and n columns
// (the source DOFs of K); row 3k + c is column (k, c) of the reference's
// O(n, 3 nobs) (fortran/3d/src/greens.f90:302-462).  Same launch shape as K:
// one thread per source, the grid's y dimension strides over points, and each
// row store of a warp is one coalesced segment.

template <bool R32>
__global__ void __launch_bounds__(128) k_observe_rect(double *__restrict__ O, long n, long col0,
        const double *__restrict__ obs, int nobs, const double *__restrict__ src, int ns, OkMed med)
{
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= ns) return;
    double sr[RS_SIZE];
#pragma unroll
    for (int f = 0; f < RS_SIZE; f++) sr[f] = __ldg(src + (long)f * ns + j);
    OkDip dp;
    dp.sd = sr[RS_SD]; dp.cd = sr[RS_CD]; dp.sdsd = sr[RS_SDSD]; dp.cdcd = sr[RS_CDCD];
    dp.sdcd = sr[RS_SDCD];
    dp.icd = sr[RS_ICD];
    const double csst = sr[RS_CS], ssst = sr[RS_SS];
    for (int k = blockIdx.y; k < nobs; k += gridDim.y) {
        const double x1 = __ldg(obs + 3L * k), x2 = __ldg(obs + 3L * k + 1), x3 = __ldg(obs + 3L * k + 2);
        // okada92.f90:251-290
        double x = (x1 - sr[RS_Q1]) * csst + (x2 - sr[RS_Q2]) * ssst;
        double y = (x1 - sr[RS_Q1]) * ssst - (x2 - sr[RS_Q2]) * csst;
        double z = -x3;
        if (R32) {
            x = (double)__double2float_rn(x);
            y = (double)__double2float_rn(y);
            z = (double)__double2float_rn(z);
        }
        double us[3], ud[3];
        ok_dc3d_disp<R32>(med, dp, x, y, z, sr[RS_DEPTH], sr[RS_AL2], sr[RS_AW1], us, ud);
        const double oS[3] = {us[0] * csst + us[1] * ssst, us[0] * ssst - us[1] * csst, -us[2]};
        const double oD[3] = {ud[0] * csst + ud[1] * ssst, ud[0] * ssst - ud[1] * csst, -ud[2]};
#pragma unroll
        for (int c = 0; c < 3; c++)
            *reinterpret_cast<double2 *>(O + (3L * k + c) * n + col0 + 2L * j) = make_double2(oS[c], oD[c]);
    }
}

__global__ void __launch_bounds__(128) k_observe_tri(double *__restrict__ O, long n, long col0,
        const double *__restrict__ obs, int nobs, const double *__restrict__ rec, int ns, double nu)
{
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= ns) return;
    NwRec R{rec + j, (long)ns};
    for (int k = blockIdx.y; k < nobs; k += gridDim.y) {
        const double xr[3] = {__ldg(obs + 3L * k), __ldg(obs + 3L * k + 1), __ldg(obs + 3L * k + 2)};
        double uS[3], uD[3];
        nw_pair_disp(xr, R, nu, uS, uD);
#pragma unroll
        for (int c = 0; c < 3; c++)
            *reinterpret_cast<double2 *>(O + (3L * k + c) * n + col0 + 2L * j) = make_double2(uS[c], uD[c]);
    }
}

__global__ void __launch_bounds__(128) k_observe_vol(double *__restrict__ O, long n, long col0,
        const double *__restrict__ obs, int nobs, const double *__restrict__ rec, int ns, double mu, double nu)
{
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= ns) return;
    SvRec R{rec + j, (long)ns};
    for (int k = blockIdx.y; k < nobs; k += gridDim.y) {
        const double xr[3] = {__ldg(obs + 3L * k), __ldg(obs + 3L * k + 1), __ldg(obs + 3L * k + 2)};
        double u[6][3];
        sv_pair_disp(xr, R, mu, nu, u);
#pragma unroll
        for (int c = 0; c < 3; c++) {
            double2 *p = reinterpret_cast<double2 *>(O + (3L * k + c) * n + col0 + 6L * j);
            p[0] = make_double2(u[0][c], u[1][c]);
            p[1] = make_double2(u[2][c], u[3][c]);
            p[2] = make_double2(u[4][c], u[5][c]);
        }
    }
}

// ---- host side -----------------------------------------------------------------

static float f32(double v) { return (float)v; }

// receiver frames and centres: okada92.f90:59-87, nikkhoo15.f90:50-101,
// strainvolume.f90:135-163
static void build_receivers(ucg_ctx *c, std::vector<double> &r)
{
    const int ne = c->nr + c->nt + c->nv;
    r.assign((size_t)ne * RC_SIZE, 0.0);
    for (int i = 0; i < c->nr; i++) {
        double *q = &r[(size_t)i * RC_SIZE];
        const double st = c->rstrike[i], dp = c->rdip[i];
        double sv[3] = {cos(st), sin(st), 0.0};
        double dv[3] = {+sin(st) * cos(dp), -cos(st) * cos(dp), -sin(dp)};
        double nv[3] = {-sin(st) * sin(dp), +cos(st) * sin(dp), -cos(dp)};
        for (int k = 0; k < 3; k++) {
            q[RC_X + k] = c->rx[3 * i + k] + c->rL[i] / 2 * sv[k] - c->rW[i] / 2 * dv[k];
            q[RC_S + k] = sv[k]; q[RC_D + k] = dv[k]; q[RC_N + k] = nv[k];
        }
    }
    for (int j = 0; j < c->nt; j++) {
        double *q = &r[(size_t)(c->nr + j) * RC_SIZE];
        const double *A = &c->tvert[3L * (c->ti1[j] - 1)];
        const double *B = &c->tvert[3L * (c->ti2[j] - 1)];
        const double *C = &c->tvert[3L * (c->ti3[j] - 1)];
        double n[3];
        n[0] = (B[1] - A[1]) * (C[2] - A[2]) - (B[2] - A[2]) * (C[1] - A[1]);
        n[1] = (B[2] - A[2]) * (C[0] - A[0]) - (B[0] - A[0]) * (C[2] - A[2]);
        n[2] = (B[0] - A[0]) * (C[1] - A[1]) - (B[1] - A[1]) * (C[0] - A[0]);
        double norm = sqrt(n[0] * n[0] + n[1] * n[1] + n[2] * n[2]);
        for (int k = 0; k < 3; k++) n[k] = n[k] / norm;
        if (0.0 < n[2]) for (int k = 0; k < 3; k++) n[k] = -n[k];
        double s[3] = {cos(atan2(n[0], n[1])), -sin(atan2(n[0], n[1])), 0.0};
        double d[3] = {n[1] * s[2] - n[2] * s[1], n[2] * s[0] - n[0] * s[2], n[0] * s[1] - n[1] * s[0]};
        for (int k = 0; k < 3; k++) {
            q[RC_X + k] = (A[k] + B[k] + C[k]) / 3.0;
            q[RC_S + k] = s[k]; q[RC_D + k] = d[k]; q[RC_N + k] = n[k];
        }
    }
    for (int i = 0; i < c->nv; i++) {
        double *q = &r[(size_t)(c->nr + c->nt + i) * RC_SIZE];
        const double st = c->vstrike[i];
        double sv[3] = {cos(st), sin(st), 0.0};
        double dv[3] = {0.0, 0.0, -1.0};
        double nv[3] = {-sin(st), +cos(st), -0.0};
        for (int k = 0; k < 3; k++) {
            q[RC_X + k] = c->vx[3 * i + k] + c->vL[i] / 2 * sv[k] - c->vW[i] / 2 * dv[k];
            q[RC_S + k] = sv[k]; q[RC_D + k] = dv[k]; q[RC_N + k] = nv[k];
        }
    }
}

static void build_rect_sources(ucg_ctx *c, int mode, std::vector<double> &s)
{
    const int ns = c->nr;
    const bool r32 = (mode == UCG_OKADA_REF32IO);
    const double RAD2DEG = 57.29577951308232;
    s.assign((size_t)ns * RS_SIZE, 0.0);
    auto put = [&](int f, int j, double v) { s[(size_t)f * ns + j] = v; };
    for (int j = 0; j < ns; j++) {
        double dip = c->rdip[j] * RAD2DEG;
        double depth = c->rx[3 * j + 2], L = c->rL[j], W = c->rW[j];
        if (r32) { dip = f32(dip); depth = f32(depth); L = f32(L); W = f32(W); }
        OkDip dp = ok_dip(dip);
        put(RS_Q1, j, c->rx[3 * j + 0]);
        put(RS_Q2, j, c->rx[3 * j + 1]);
        put(RS_CS, j, cos(c->rstrike[j]));
        put(RS_SS, j, sin(c->rstrike[j]));
        put(RS_DEPTH, j, depth);
        put(RS_AL2, j, L);
        put(RS_AW1, j, -W);
        put(RS_SD, j, dp.sd);
        put(RS_CD, j, dp.cd);
        put(RS_SDSD, j, dp.sdsd);
        put(RS_CDCD, j, dp.cdcd);
        put(RS_SDCD, j, dp.sdcd);
        put(RS_ICD, j, dp.icd);
    }
}

// the receiver table of every element
static int upload_receivers(ucg_ctx *c)
{
    std::vector<double> r;
    build_receivers(c, r);
    if (c->rcv_len != r.size()) {
        if (c->rcv) cudaFree(c->rcv);
        c->rcv = nullptr;
        c->rcv_len = 0;
        UCG_CUDA(cudaMalloc(&c->rcv, sizeof(double) * r.size()));
        c->rcv_len = r.size();
    }
    UCG_CUDA(cudaMemcpyAsync(c->rcv, r.data(), sizeof(double) * r.size(), cudaMemcpyHostToDevice, c->stream));
    return UCG_OK;
}

// device tables of the triangles (in the order perm, or the mesh's); with edges,
// the unique edges of the mesh by vertex pair, oriented as their first triangle
// runs along them, numbered in triangle order so that neighbours stay close
static int tri_tables_build(ucg_ctx *c, bool edges, const int *perm, TriTables *t)
{
    const int ns = c->nt, nve = c->nve;
    *t = TriTables{};
    t->ns = ns;
    std::vector<int> id((size_t)3 * ns);
    const std::vector<int> *ti[3] = {&c->ti1, &c->ti2, &c->ti3};
    for (int k = 0; k < 3; k++)
        for (int j = 0; j < ns; j++) id[(size_t)k * ns + j] = (*ti[k])[perm ? perm[j] : j] - 1;
    std::vector<int> side((size_t)3 * ns);
    std::vector<int2> ends;
    if (edges) {
        std::vector<int> head(nve, -1), next;   // edges chained by their smaller vertex
        ends.reserve((size_t)ns * 2);
        next.reserve((size_t)ns * 2);
        for (int j = 0; j < ns; j++)
            for (int k = 0; k < 3; k++) {
                const int a = id[(size_t)k * ns + j], b = id[(size_t)((k + 1) % 3) * ns + j];
                const int lo = a < b ? a : b;
                int e = head[lo];
                while (e >= 0 && !((ends[e].x == a && ends[e].y == b) || (ends[e].x == b && ends[e].y == a))) e = next[e];
                if (e < 0) {
                    e = (int)ends.size();
                    ends.push_back(make_int2(a, b));
                    next.push_back(head[lo]);
                    head[lo] = e;
                }
                side[(size_t)k * ns + j] = 2 * e + (ends[e].x == a ? 0 : 1);
            }
    }
    t->ne = (int)ends.size();
    double *vert, *rec, *ed;
    int *idd, *sd;
    int2 *endd;
    int rc;
    if ((rc = workspace_upload(c, WS_VERT, c->tvert, &vert)) || (rc = workspace_upload(c, WS_ID, id, &idd)) ||
        (rc = workspace(c, WS_SRC, sizeof(double) * (size_t)NW_SIZE * ns, &rec)))
        return rc;
    t->rec = rec;
    k_tri_prepare<<<(ns + 127) / 128, 128, 0, c->stream>>>(vert, idd, ns, rec);
    c->launches.count++;
    if (edges) {
        if ((rc = workspace_upload(c, WS_SIDE, side, &sd)) || (rc = workspace_upload(c, WS_ENDS, ends, &endd)) ||
            (rc = workspace(c, WS_EDGE, sizeof(double) * (size_t)NE_SIZE * t->ne, &ed)))
            return rc;
        t->edge = sd;
        t->ed = ed;
        k_edge_prepare<<<(t->ne + 127) / 128, 128, 0, c->stream>>>(vert, endd, t->ne, ed);
        c->launches.count++;
    }
    UCG_CUDA(cudaGetLastError());
    return UCG_OK;
}

static void build_vol_sources(ucg_ctx *c, std::vector<double> &s)
{
    const int ns = c->nv;
    s.assign((size_t)ns * SV_SIZE, 0.0);
    std::vector<double> r(SV_SIZE);
    for (int j = 0; j < ns; j++) {
        sv_prepare(&c->vx[3 * j], c->vL[j], c->vT[j], c->vW[j], c->vstrike[j], r.data());
        for (int f = 0; f < SV_SIZE; f++) s[(size_t)f * ns + j] = r[f];
    }
}

// gridDim.y of a pair kernel: up to 8 receivers per thread, so that a thread's
// source record is read from L1 after the first, while about 16 CTAs per SM are left
static int receiver_grid(const ucg_ctx *c, int xblocks, int receivers)
{
    long per = (long)xblocks * receivers / (16L * c->sms);
    per = per < 1 ? 1 : per > 8 ? 8 : per;
    const long gy = (receivers + per - 1) / per;
    return (int)(gy < 65535 ? gy : 65535);
}

// rows of receivers [e0, e1) (NR each, the first at row0) against all triangles,
// in batches whose edge scratch stays in L2
template <int NR>
static int assemble_tri_rows(ucg_ctx *c, long n, int e0, int e1, long row0, const TriTables &tab, const NwConst &cst)
{
    if (e1 <= e0) return UCG_OK;
    const size_t SCRATCH = (size_t)96 << 20;
    const size_t per = sizeof(double) * 3 * NR * (size_t)tab.ne;
    const int batch = (int)std::max<size_t>(1, std::min<size_t>(SCRATCH / per, (size_t)(e1 - e0)));
    double *sc;
    const int rc = workspace(c, WS_SCRATCH, per * batch, &sc);
    if (rc) return rc;
    const int TPB = 128, xe = (tab.ne + TPB - 1) / TPB, xt = (tab.ns + TPB - 1) / TPB;
    for (int r0 = e0; r0 < e1; r0 += batch) {
        const int r1 = std::min(e1, r0 + batch);
        k_tri_edges<NR><<<dim3(xe, receiver_grid(c, xe, r1 - r0)), TPB, 0, c->stream>>>(sc, c->rcv, r0, r1, tab, cst);
        k_assemble_tri<NR><<<dim3(xt, receiver_grid(c, xt, r1 - r0)), TPB, 0, c->stream>>>(
            c->K, n, 2L * c->nr, row0 + (long)NR * (r0 - e0), sc, c->rcv, r0, r1, tab, cst);
        c->launches.count += 2;
    }
    UCG_CUDA(cudaGetLastError());
    return UCG_OK;
}

int assemble_matrix(ucg_ctx *c, int okada_mode)
{
    const int ne = c->nr + c->nt + c->nv;
    const int np = c->nr + c->nt;
    const long n = 2L * np + 6L * c->nv;
    const long m = 3L * np + 6L * c->nv;
    if (ne == 0) return UCG_E_BADARG;
    UCG_CUDA(cudaSetDevice(c->device));
    c->assembled = false;   // until all of K is
    if (c->K && (c->n != n || c->m != m)) {
        cudaFree(c->K);
        c->K = nullptr;
    }
    if (!c->K) {
        cudaError_t e = cudaMalloc(&c->K, sizeof(double) * (size_t)n * (size_t)m);
        if (e != cudaSuccess) {
            c->K = nullptr;
            cuda_fail(c, e, "cudaMalloc(K)");
            return UCG_E_OOM;
        }
    }
    c->n = n;
    c->m = m;
    int rc = upload_receivers(c);
    if (rc) return rc;

    const int TPB = 128;
    double *dsrc = nullptr;
    // device time of each family's launches (ucg_assembly_times)
    cudaEvent_t ev[6];
    for (cudaEvent_t &e : ev) UCG_CUDA(cudaEventCreate(&e));
    for (double &t : c->asm_ms) t = 0.0;
    // load the kernels' code before the first event: under lazy module loading
    // a first launch would otherwise count the load in its family's time
    cudaFuncAttributes fa;
    if (c->nr) {
        const bool r32 = okada_mode == UCG_OKADA_REF32IO;
        UCG_CUDA(cudaFuncGetAttributes(&fa, r32 ? k_assemble_rect<true, 3> : k_assemble_rect<false, 3>));
        if (c->nv) UCG_CUDA(cudaFuncGetAttributes(&fa, r32 ? k_assemble_rect<true, 6> : k_assemble_rect<false, 6>));
    }
    if (c->nt) {
        UCG_CUDA(cudaFuncGetAttributes(&fa, k_tri_edges<3>));
        UCG_CUDA(cudaFuncGetAttributes(&fa, k_assemble_tri<3>));
        if (c->nv) {
            UCG_CUDA(cudaFuncGetAttributes(&fa, k_tri_edges<6>));
            UCG_CUDA(cudaFuncGetAttributes(&fa, k_assemble_tri<6>));
        }
    }
    if (c->nv) {
        UCG_CUDA(cudaFuncGetAttributes(&fa, k_assemble_vol<3>));
        UCG_CUDA(cudaFuncGetAttributes(&fa, k_assemble_vol<6>));
    }
    if (c->nr) {
        std::vector<double> s;
        build_rect_sources(c, okada_mode, s);
        if ((rc = workspace_upload(c, WS_SRC, s, &dsrc))) return rc;
        UCG_CUDA(cudaEventRecord(ev[0], c->stream));
        const double alpha_d = (c->lambda + c->mu) / (c->lambda + 2.0 * c->mu);
        const double alpha = okada_mode == UCG_OKADA_REF32IO ? (double)f32(alpha_d) : alpha_d;
        const int xb = (c->nr + TPB - 1) / TPB;
        const OkMed med = ok_med(alpha);
        auto rows = [&](auto kern, int e0, int e1, long row0) {
            kern<<<dim3(xb, receiver_grid(c, xb, e1 - e0)), TPB, 0, c->stream>>>(c->K, n, row0, c->rcv, e0, e1, dsrc,
                                                                                c->nr, med, c->mu, c->lambda);
            c->launches.count++;
        };
        const bool r32 = okada_mode == UCG_OKADA_REF32IO;
        rows(r32 ? k_assemble_rect<true, 3> : k_assemble_rect<false, 3>, 0, np, 0);
        if (c->nv) rows(r32 ? k_assemble_rect<true, 6> : k_assemble_rect<false, 6>, np, ne, 3L * np);
        UCG_CUDA(cudaGetLastError());
        UCG_CUDA(cudaEventRecord(ev[1], c->stream));
    }
    if (c->nt) {
        TriTables tab;
        if ((rc = tri_tables_build(c, true, nullptr, &tab))) return rc;
        UCG_CUDA(cudaEventRecord(ev[2], c->stream));
        const NwConst cst{c->lambda / (c->lambda + c->mu) / 2.0, c->mu, c->lambda};
        rc = assemble_tri_rows<3>(c, n, 0, np, 0, tab, cst);
        if (!rc && c->nv) rc = assemble_tri_rows<6>(c, n, np, ne, 3L * np, tab, cst);
        if (rc) return rc;
        UCG_CUDA(cudaEventRecord(ev[3], c->stream));
    }
    if (c->nv) {
        std::vector<double> s;
        build_vol_sources(c, s);
        if ((rc = workspace_upload(c, WS_SRC, s, &dsrc))) return rc;
        UCG_CUDA(cudaEventRecord(ev[4], c->stream));
        const double nu = c->lambda / (c->lambda + c->mu) / 2.0;
        const int xb = (c->nv + TPB - 1) / TPB;
        if (np) {
            k_assemble_vol<3><<<dim3(xb, receiver_grid(c, xb, np)), TPB, 0, c->stream>>>(
                c->K, n, 2L * np, 0, c->rcv, 0, np, dsrc, c->nv, c->mu, nu);
            c->launches.count++;
        }
        k_assemble_vol<6><<<dim3(xb, receiver_grid(c, xb, c->nv)), TPB, 0, c->stream>>>(
            c->K, n, 2L * np, 3L * np, c->rcv, np, ne, dsrc, c->nv, c->mu, nu);
        c->launches.count++;
        UCG_CUDA(cudaGetLastError());
        UCG_CUDA(cudaEventRecord(ev[5], c->stream));
    }
    UCG_CUDA(cudaStreamSynchronize(c->stream));
    const int have[3] = {c->nr > 0, c->nt > 0, c->nv > 0};
    for (int f = 0; f < 3; f++) {
        float ms = 0.0f;
        if (have[f] && cudaEventElapsedTime(&ms, ev[2 * f], ev[2 * f + 1]) == cudaSuccess) c->asm_ms[f] = ms;
    }
    for (cudaEvent_t &e : ev) cudaEventDestroy(e);
    c->okada_mode = okada_mode;
    c->assembled = true;
    return UCG_OK;
}

int assemble_observation(ucg_ctx *c, int okada_mode)
{
    const int np = c->nr + c->nt;
    const long n = 2L * np + 6L * c->nv;
    const int nobs = (int)(c->obs_x.size() / 3);
    if (np + c->nv == 0 || nobs == 0) return UCG_E_BADARG;
    UCG_CUDA(cudaSetDevice(c->device));
    const size_t bytes = sizeof(double) * (size_t)n * 3 * (size_t)nobs;
    if (c->O && c->O_bytes != bytes) {
        cudaFree(c->O);
        c->O = nullptr;
    }
    if (!c->O) {
        cudaError_t e = cudaMalloc(&c->O, bytes);
        if (e != cudaSuccess) {
            c->O = nullptr;
            return cuda_fail(c, e, "cudaMalloc(O)");
        }
        c->O_bytes = bytes;
    }
    if (c->obs_dev) cudaFree(c->obs_dev);
    c->obs_dev = nullptr;
    UCG_CUDA(cudaMalloc(&c->obs_dev, sizeof(double) * c->obs_x.size()));
    UCG_CUDA(cudaMemcpyAsync(c->obs_dev, c->obs_x.data(), sizeof(double) * c->obs_x.size(),
                             cudaMemcpyHostToDevice, c->stream));
    const int TPB = 128;
    const int gy = nobs < 65535 ? nobs : 65535;
    double *dsrc = nullptr;
    int rc;
    cudaEvent_t ev[2];
    for (cudaEvent_t &e : ev) UCG_CUDA(cudaEventCreate(&e));
    UCG_CUDA(cudaEventRecord(ev[0], c->stream));
    if (c->nr) {
        std::vector<double> s;
        build_rect_sources(c, okada_mode, s);
        if ((rc = workspace_upload(c, WS_SRC, s, &dsrc))) return rc;
        const double alpha_d = (c->lambda + c->mu) / (c->lambda + 2.0 * c->mu);
        const double alpha = okada_mode == UCG_OKADA_REF32IO ? (double)f32(alpha_d) : alpha_d;
        dim3 grid((c->nr + TPB - 1) / TPB, gy);
        if (okada_mode == UCG_OKADA_REF32IO)
            k_observe_rect<true><<<grid, TPB, 0, c->stream>>>(c->O, n, 0, c->obs_dev, nobs, dsrc, c->nr, ok_med(alpha));
        else
            k_observe_rect<false><<<grid, TPB, 0, c->stream>>>(c->O, n, 0, c->obs_dev, nobs, dsrc, c->nr, ok_med(alpha));
        c->launches.count++;
        UCG_CUDA(cudaGetLastError());
    }
    if (c->nt) {
        TriTables tab;
        if ((rc = tri_tables_build(c, false, nullptr, &tab))) return rc;
        dim3 grid((c->nt + TPB - 1) / TPB, gy);
        k_observe_tri<<<grid, TPB, 0, c->stream>>>(c->O, n, 2L * c->nr, c->obs_dev, nobs, tab.rec, c->nt,
                                                   c->lambda / (c->lambda + c->mu) / 2.0);
        c->launches.count++;
        UCG_CUDA(cudaGetLastError());
    }
    if (c->nv) {
        std::vector<double> s;
        build_vol_sources(c, s);
        if ((rc = workspace_upload(c, WS_SRC, s, &dsrc))) return rc;
        dim3 grid((c->nv + TPB - 1) / TPB, gy);
        k_observe_vol<<<grid, TPB, 0, c->stream>>>(c->O, n, 2L * np, c->obs_dev, nobs, dsrc, c->nv, c->mu,
                                                   c->lambda / (c->lambda + c->mu) / 2.0);
        c->launches.count++;
        UCG_CUDA(cudaGetLastError());
    }
    UCG_CUDA(cudaEventRecord(ev[1], c->stream));
    UCG_CUDA(cudaStreamSynchronize(c->stream));
    float ms = 0.0f;
    if (cudaEventElapsedTime(&ms, ev[0], ev[1]) == cudaSuccess) c->obs_ms = ms;
    for (cudaEvent_t &e : ev) cudaEventDestroy(e);
    c->O_ready = true;
    return UCG_OK;
}

// ---- block sources (hierarchical approximation) -----------------------------------

int block_family(const ucg_ctx *c)
{
    return (c->nr > 0) == (c->nt > 0) || c->nv > 0 ? UCG_E_UNSUPPORTED : UCG_OK;
}

int block_sources_build(ucg_ctx *c, int okada_mode, const std::vector<int> &perm, BlockSources *bs)
{
    int rc = block_family(c);
    if (rc) return rc;
    UCG_CUDA(cudaSetDevice(c->device));
    if ((rc = upload_receivers(c))) return rc;
    bs->family = c->nr > 0 ? 0 : 1;
    bs->okada_mode = okada_mode;
    if (bs->family == 1) {
        bs->ns = c->nt;
        bs->cst = NwConst{c->lambda / (c->lambda + c->mu) / 2.0, c->mu, c->lambda};
        return tri_tables_build(c, true, perm.data(), &bs->tri);
    }
    std::vector<double> s, sp;
    build_rect_sources(c, okada_mode, s);
    bs->ns = c->nr;
    sp.resize(s.size());
    for (int f = 0; f < RS_SIZE; f++)
        for (int j = 0; j < c->nr; j++) sp[(size_t)f * c->nr + j] = s[(size_t)f * c->nr + perm[j]];
    const double alpha_d = (c->lambda + c->mu) / (c->lambda + 2.0 * c->mu);
    bs->med = ok_med(okada_mode == UCG_OKADA_REF32IO ? (double)f32(alpha_d) : alpha_d);
    double *src;
    if ((rc = workspace_upload(c, WS_SRC, sp, &src))) return rc;
    bs->src = src;
    return UCG_OK;
}

int assemble_blocks(ucg_ctx *c, const BlockSources &bs, const int *perm_d, const std::vector<BlockJob> &jobs)
{
    if (jobs.empty()) return UCG_OK;
    std::vector<int2> tiles;
    for (size_t q = 0; q < jobs.size(); q++) {
        const int pairs = jobs[q].nr * jobs[q].ns;
        for (int p = 0; p < pairs; p += BLOCK_TILE) tiles.push_back(make_int2((int)q, p));
    }
    BlockJob *jd;
    int2 *td;
    int rc;
    if ((rc = workspace_upload(c, WS_JOBS, jobs, &jd)) || (rc = workspace_upload(c, WS_TILES, tiles, &td))) return rc;
    const int grid = (int)tiles.size(), TPB = 128;
    if (bs.family == 1)
        k_blocks_tri<<<grid, TPB, 0, c->stream>>>(jd, td, perm_d, c->rcv, bs.tri, bs.cst);
    else if (bs.okada_mode == UCG_OKADA_REF32IO)
        k_blocks_rect<true><<<grid, TPB, 0, c->stream>>>(jd, td, perm_d, c->rcv, bs.src, bs.ns, bs.med, c->mu, c->lambda);
    else
        k_blocks_rect<false><<<grid, TPB, 0, c->stream>>>(jd, td, perm_d, c->rcv, bs.src, bs.ns, bs.med, c->mu, c->lambda);
    c->launches.count++;
    UCG_CUDA(cudaGetLastError());
    return UCG_OK;
}

// element bounding boxes (lo[3], hi[3] per element, patches in K's order) and centres
void element_boxes(const ucg_ctx *c, std::vector<double> &box, std::vector<double> &ctr)
{
    const int np = c->nr + c->nt;
    box.assign(6L * np, 0.0);
    ctr.assign(3L * np, 0.0);
    for (int i = 0; i < np; i++) {
        double p[4][3];
        int nv;
        if (i < c->nr) {
            const double st = c->rstrike[i], dp = c->rdip[i];
            const double sv[3] = {cos(st), sin(st), 0.0};
            const double dv[3] = {+sin(st) * cos(dp), -cos(st) * cos(dp), -sin(dp)};
            for (int k = 0; k < 3; k++) {
                const double x = c->rx[3 * i + k];
                p[0][k] = x;
                p[1][k] = x + c->rL[i] * sv[k];
                p[2][k] = x + c->rL[i] * sv[k] - c->rW[i] * dv[k];
                p[3][k] = x - c->rW[i] * dv[k];
            }
            nv = 4;
        } else {
            const int j = i - c->nr;
            const int id[3] = {c->ti1[j] - 1, c->ti2[j] - 1, c->ti3[j] - 1};
            for (int q = 0; q < 3; q++)
                for (int k = 0; k < 3; k++) p[q][k] = c->tvert[3L * id[q] + k];
            nv = 3;
        }
        for (int k = 0; k < 3; k++) {
            double lo = p[0][k], hi = p[0][k], s = 0.0;
            for (int q = 0; q < nv; q++) {
                lo = std::fmin(lo, p[q][k]);
                hi = std::fmax(hi, p[q][k]);
                s += p[q][k];
            }
            box[6L * i + k] = lo;
            box[6L * i + 3 + k] = hi;
            ctr[3L * i + k] = s / nv;
        }
    }
}

}  // namespace ucg
