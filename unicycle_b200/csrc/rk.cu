// Right-hand side and Cash-Karp RK4(5) stepping on the device.
//
// One attempt of RKQSm (fortran/3d/src/ode45.f90:51-108) is six launches, one per
// stage, captured once into a CUDA graph.  The launch of stage s
//
//   multiplies    t = K v_s (k_traction; hierarchical K: its two product launches
//                 leave partial sums, which k_hm_stage adds up)
//   and then, element by element as the row sums arrive,
//   evaluates     k_s = f(y_s) (rate-state / Maxwell epilogue),
//   and forms     s < 6: y_{s+1} = y + h sum_j b_sj k_j (BLAS-1 order of RKCKm) and
//                        the source rates v_{s+1} of the next launch;
//                 s = 6: ycand, yerr, max|yerr/yscal| (ordered-bit atomicMax) and the
//                        source rates of ycand.
//
// The last CTA of stage 6 decides: accept/reject, step size, time, counters.  All of
// an element's stage vectors are local to it, so nothing but v crosses elements; v
// alternates between two buffers.  Stage 1 of the next attempt commits an accepted
// candidate into y; after a rejection it only forms y_2 again for the new h.
//
// Every kernel of this file looks at the control block and does nothing when the
// integration is inactive (k_traction has asked for its first block of K by then), so
// the same graph serves accepted and rejected attempts and many attempts can be
// queued without host round trips.  The hierarchical product does not look: an idle
// attempt moves its matrix six times all the same (tens of thousands of CTAs that
// read one word: one reading each took 1.5 % of a live attempt at 7,200 triangles).
// Separate kernels for the stage state, the error norm and the decision (14 launches
// an attempt) cost 67 us a step at N = 512, where each launch is latency alone.
//
// The stage combinations, yout and yerr follow the reference's operation order
// with explicit round-to-nearest multiplies and adds (no FMA contraction), so
// they round exactly as the oracle's restatement of RKCKm.
//
// With the split-BF16 matrix the stages are anchored: stage 1 of a step keeps
// v1 = v(y) and t1 = K v1, and stages 2-6 multiply only the increment,
// t_s = t1 + K (v_s - v1).  The product's rounding (about 1e-5 of |K| |v|)
// then cancels from the embedded error estimate (its weights sum to zero)
// instead of dominating it on components whose state and rate are near zero,
// which at rtol 1e-8 would reject nearly every attempt.  The FP64 path keeps
// the reference's plain form.
#include <utility>
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include "ucg_internal.cuh"

namespace ucg {

__device__ __constant__ double c_B[6][5] = {
    {0, 0, 0, 0, 0},
    {0.2, 0, 0, 0, 0},
    {3.0 / 40.0, 9.0 / 40.0, 0, 0, 0},
    {0.3, -0.9, 1.2, 0, 0},
    {-11.0 / 54.0, 2.5, -70.0 / 27.0, 35.0 / 27.0, 0},
    {1631.0 / 55296.0, 175.0 / 512.0, 575.0 / 13824.0, 44275.0 / 110592.0, 253.0 / 4096.0}};

#define C1 (37.0 / 378.0)
#define C3 (250.0 / 621.0)
#define C4 (125.0 / 594.0)
#define C6 (512.0 / 1771.0)
#define DC1 (C1 - 2825.0 / 27648.0)
#define DC3 (C3 - 18575.0 / 48384.0)
#define DC4 (C4 - 13525.0 / 55296.0)
#define DC5 (-277.0 / 14336.0)
#define DC6 (C6 - 0.25)

static const double LG10 = 2.302585092994045684017991454684364208;

struct StageArgs {
    double *y;             // state at the start of the step
    double *ys;            // state of the stages after the first
    double *k[6];
    double *ks;            // k of this stage
    const double *v;       // source rates of this stage
    double *vn;            // source rates of the next one
    const int *perm;       // hierarchical K: vn is in the order perm (position -> element)
    int next;              // form the next stage's state (0: only k_s)
    double *ycand, *yerr, *yscal;
    double *v1, *t1;       // stage-1 anchor (split-BF16 matrix only)
    int anchored;
    Friction fr;
    Rheology rh;
    int np, nvol;
    long len;
};

__device__ __forceinline__ bool ctl_live(const Ctl *c) { return c->active && c->status == 0; }
// the same while the launch in front may still change it: a hint, nothing to decide by
__device__ __forceinline__ bool ctl_hint(const Ctl *c) { return *(const volatile int *)&c->active != 0; }

// Programmatic dependent launch.  The kernels of an attempt are launched with
// programmatic stream serialization: each may be scheduled while its
// predecessor in the stream still runs, waits here (griddepcontrol.wait) until
// that predecessor has completed and its writes are visible, and at once lets
// its own successor be scheduled.  So the launch latency of every kernel of an
// attempt overlaps the previous kernel instead of adding to it (it dominates
// at small N).  Without a programmatic predecessor the wait returns at once.
__device__ __forceinline__ void pdl_enter()
{
    pdl_wait();
    pdl_launch();
}

__device__ __forceinline__ void atomic_max_pos(unsigned long long *p, double x)
{
    // non-negative doubles order like their bit patterns
    atomicMax(p, (unsigned long long)__double_as_longlong(x));
}

// ---- one element of a stage -------------------------------------------------------
//
// A patch takes 8 lanes of a warp, a volume 16; lane c holds component c of the
// element's state (7 and 12), so that the stage vectors are read as short runs and
// the combination of a component is one lane's work.  What does not depend on the
// product (the state, the sums over the earlier stages, the friction terms of f) is
// loaded and formed before the row sums arrive: the next launch waits for what
// comes after them.

struct LaneState {
    double y;             // the step's initial state
    double r, e;          // the combination and (stage 6) the error over the stages so far
    double cs;            // coefficient of this stage in the next one's combination
    double yscal;         // stage 6
    bool on;              // the lane holds a component
};

// state of stage S + 1 with the reference BLAS-1 order, ks = k_S being its last term
__device__ __forceinline__ double stage_comb(int S, const LaneState &st, double ks, double h)
{
    if (S == 1) return __dadd_rn(st.y, __dmul_rn(__dmul_rn(h, c_B[1][0]), ks));
    return __dadd_rn(st.y, __dmul_rn(h, __dadd_rn(st.r, __dmul_rn(st.cs, ks))));
}

// x / d where rd = 1 / d is at hand before x: the quotient's residual corrects it
// once (Markstein, IBM J. Res. Dev. 34, 1990), which rounds like the division for
// normal quotients; three dependent operations instead of a division's sequence.
// (x, d and the quotient finite)
__device__ __forceinline__ double div_by(double x, double d, double rd)
{
    const double q = x * rd;
    return fma(fma(-d, q, x), rd, q);
}

// where one of them may be infinite the correction is NaN, and the product x rd (or a
// chain of them) is already the quotient (an infinite L is a fault without state
// evolution)
__device__ __forceinline__ double or_product(double quotient, double product)
{
    return isnan(quotient) ? product : quotient;
}

constexpr double INV_LG10 = 0.434294481903251827651128918916605082;   // 1 / ln 10

// slip velocity and the cosine and sine of the rake atan2(td, ts)
// (ratestate.f90:682-690); where the sum of squares is of no use the angle itself
__device__ __forceinline__ void patch_slip(double ts, double td, double lv, double &vel, double &cr, double &sr)
{
    vel = exp(lv * LG10);
    const double h2 = ts * ts + td * td;
    if (h2 > 1.0e-280 && h2 < 1.0e280) {
        // the square root from its reciprocal by the same correction, then the quotients
        const double ih = rsqrt(h2), g = h2 * ih, hy = fma(fma(-g, g, h2), 0.5 * ih, g);
        cr = div_by(ts, hy, ih);
        sr = div_by(td, hy, ih);
    } else {
        const double rake = atan2(td, ts);
        cr = cos(rake);
        sr = sin(rake);
    }
}

// Maxwell strain rate of component q of a volume with stresses s11 .. s33
// (viscouscycles.f90:938-995)
__device__ __forceinline__ double volume_rate(const Rheology &rh, int iv, int q, double s11, double s12, double s13,
                                              double s22, double s23, double s33)
{
    if (!rh.nonlinear) return 0.0;
    const double p = (s11 + s22 + s33) / 3.0;
    s11 = s11 - p; s22 = s22 - p; s33 = s33 - p;
    const double sII = sqrt((s11 * s11 + 2.0 * s12 * s12 + 2.0 * s13 * s13 + s22 * s22 + 2.0 * s23 * s23 + s33 * s33) /
                            2.0);
    const double eII = rh.gd0[iv] * pow(sII, rh.npow[iv] - 1);
    return eII * (q == 0 ? s11 : q == 1 ? s12 : q == 2 ? s13 : q == 3 ? s22 : q == 4 ? s23 : s33);
}

// state of stage S in the lane (commits an accepted candidate at stage 1), and the
// sums over the earlier stages
__device__ __forceinline__ double lane_load(int S, const StageArgs &a, const Ctl *ctl, long i, bool on, LaneState &st)
{
    st = LaneState{0.0, 0.0, 0.0, 0.0, 1.0, on};
    if (!on) return 0.0;
    st.y = a.y[i];
    if (S == 1) {
        if (!a.next) return st.y;
        const double yc = a.ycand[i];
        if (ctl->pending) a.y[i] = st.y = yc;
        return st.y;
    }
    const double ys = a.ys[i];
    if (!a.next) return ys;
    double k[5];
#pragma unroll
    for (int j = 0; j < 5; j++) k[j] = j < S - 1 ? a.k[j][i] : 0.0;
    if (S < 6) {
        double r = __dmul_rn(c_B[S][0], k[0]);
#pragma unroll
        for (int j = 1; j < 4; j++)
            if (j < S - 1) r = __dadd_rn(r, __dmul_rn(c_B[S][j], k[j]));
        st.r = r;
        st.cs = c_B[S][S - 1];
        return ys;
    }
    st.yscal = a.yscal[i];
    // ode45.f90:184-200
    double r = __dmul_rn(C1, k[0]);
    r = __dadd_rn(r, __dmul_rn(C3, k[2]));
    st.r = __dadd_rn(r, __dmul_rn(C4, k[3]));
    double e = __dmul_rn(DC1, k[0]);
    e = __dadd_rn(e, __dmul_rn(DC3, k[2]));
    e = __dadd_rn(e, __dmul_rn(DC4, k[3]));
    st.e = __dadd_rn(e, __dmul_rn(DC5, k[4]));
    return ys;
}

// the lane's rate ks at stage S known: store it, then the next stage's component,
// or at stage 6 the candidate and its error.  Returns the new component.
__device__ __forceinline__ double lane_advance(int S, const StageArgs &a, long i, double h, const LaneState &st,
                                               double ks, double &mx, bool &bad)
{
    if (!st.on) return 0.0;
    a.ks[i] = ks;
    if (!a.next) return 0.0;
    if (S < 6) {
        const double yn = stage_comb(S, st, ks, h);
        a.ys[i] = yn;
        if (S == 1) a.yscal[i] = fabs(st.y) + fabs(h * ks) + 1.0e-30;   // ratestate.f90:315; h == dt_try here
        return yn;
    }
    const double yc = __dadd_rn(st.y, __dmul_rn(h, __dadd_rn(st.r, __dmul_rn(C6, ks))));
    const double e = __dmul_rn(h, __dadd_rn(st.e, __dmul_rn(DC6, ks)));
    a.ycand[i] = yc;
    a.yerr[i] = e;
    // MAXVAL semantics: a NaN ratio (0/0) does not raise the maximum; an
    // infinite one does and drives the step to underflow as in the
    // reference.  A non-finite candidate state is reported as such.
    if (!isfinite(yc)) bad = true;
    mx = fmax(mx, fabs(e / st.yscal));
    return yc;
}

// source rate of column j (at jn of the buffer) of the next stage.  Anchored forms multiply increments
// over stage 1 in the stages 2-6; vs: this stage's own rate (stage 1: the anchor)
__device__ __forceinline__ void store_rate(int S, const StageArgs &a, long j, long jn, double vnext, double vs)
{
    if (a.anchored) {
        if (S == 1) a.v1[j] = vs;
        if (S < 6) vnext -= S == 1 ? vs : a.v1[j];
    }
    if (a.next) a.vn[jn] = vnext;
}

// friction of a patch, and of its terms in f what the state gives
// (ratestate.f90:731-776)
struct PatchFriction {
    double sig, a, b, eta, L, iL, vpl;
};
struct PatchTerms {
    double vel, cr, sr, dth, q, den, rden, ev, vpl;
};

__device__ __forceinline__ PatchFriction patch_friction(const StageArgs &a, int e, int c, bool on)
{
    if (!on) return PatchFriction{1, 1, 0, 0, 1, 1, 0};
    const double L = a.fr.L[e];
    return PatchFriction{a.fr.sig[e], a.fr.a[e], a.fr.b[e], a.fr.damping[e], L, 1.0 / L,
                         c == 0 ? a.fr.vpl_c[e] : c == 1 ? a.fr.vpl_s[e] : 0.0};
}

__device__ __forceinline__ PatchTerms patch_terms(int S, Ctl *ctl, const PatchFriction &f, int c, bool on, double ys)
{
    PatchTerms p;
    const double ts = __shfl_sync(~0u, ys, 2, 8), td = __shfl_sync(~0u, ys, 3, 8);
    const double th = __shfl_sync(~0u, ys, 5, 8), lv = __shfl_sync(~0u, ys, 6, 8);
    patch_slip(ts, td, lv, p.vel, p.cr, p.sr);
    p.den = f.a * f.sig + f.eta * p.vel;
    p.rden = 1.0 / p.den;
    const double rate = exp(-th * LG10) - or_product(div_by(p.vel, f.L, f.iL), p.vel * f.iL);
    p.dth = or_product(div_by(rate, LG10, INV_LG10), rate * INV_LG10);
    p.q = f.b * f.sig * p.dth * LG10;
    p.ev = f.eta * p.vel;
    p.vpl = f.vpl;
    if (S == 1 && on && c == 0) {
        atomic_max_pos((unsigned long long *)&ctl->vmax, p.vel);
        if (!isfinite(p.vel) || !isfinite(p.cr) || !isfinite(p.sr)) ctl->nonfinite = 1;
    }
    return p;
}

// patch e: rates from its tractions t, then the next stage
__device__ __forceinline__ void patch_finish(int S, const StageArgs &a, Ctl *ctl, int e, int pos, int c, double h,
                                             const LaneState &st, const PatchTerms &p, double t0, double t1,
                                             double t2, double &mx, bool &bad)
{
    const double dtau = t0 * p.cr + t1 * p.sr - p.q;
    const double dv = or_product(div_by(div_by(dtau, p.den, p.rden), LG10, INV_LG10), dtau * p.rden * INV_LG10);
    const double corr = p.ev * dv * LG10;
    const double vs = p.vel * (c == 0 ? p.cr : p.sr);
    const double ks = c < 2 ? vs : c == 2 ? t0 - corr * p.cr : c == 3 ? t1 - corr * p.sr : c == 4 ? t2
                    : c == 5 ? p.dth : dv;
    const double yn = lane_advance(S, a, 7L * e + c, h, st, ks, mx, bad);
    const double ts = __shfl_sync(~0u, yn, 2, 8), td = __shfl_sync(~0u, yn, 3, 8), lv = __shfl_sync(~0u, yn, 6, 8);
    if (!st.on || c > 1) return;
    double vel = 0.0, cr = 1.0, sr = 0.0;
    if (a.next) {
        patch_slip(ts, td, lv, vel, cr, sr);
        // (of a candidate only once it is accepted, at the next stage 1)
        if (S < 6 && (!isfinite(vel) || !isfinite(cr) || !isfinite(sr))) ctl->nonfinite = 1;
    }
    store_rate(S, a, 2L * e + c, 2L * pos + c, vel * (c == 0 ? cr : sr) - p.vpl, vs - p.vpl);
}

// volume iv: rates from its stress rate t (its own row for the lanes 6..11;
// viscouscycles.f90:1072-1080), then the next stage.  ev: the lane's strain rate
__device__ __forceinline__ void volume_finish(int S, const StageArgs &a, int iv, int c, double h, const LaneState &st,
                                              double ev, double t, double &mx, bool &bad)
{
    const long o = 7L * a.np + 12L * iv;
    const double yn = lane_advance(S, a, o + c, h, st, c < 6 ? ev : t, mx, bad);
    double s[6];
#pragma unroll
    for (int q = 0; q < 6; q++) s[q] = __shfl_sync(~0u, yn, 6 + q, 16);
    if (!st.on || c > 5) return;
    const double ebg = a.rh.ebg[6L * iv + c];
    const double en = a.next ? volume_rate(a.rh, iv, c, s[0], s[1], s[2], s[3], s[4], s[5]) : 0.0;
    const long j = 2L * a.np + 6L * iv + c;
    store_rate(S, a, j, j, en - ebg, ev - ebg);
}

// source rates of the state y (before the first stage of a run; the attempts form
// them as they go)
__global__ void k_begin(StageArgs a, const Ctl *ctl, double *__restrict__ v)
{
    pdl_enter();
    if (!ctl_live(ctl) || !ctl->need_stage1) return;
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= a.np + a.nvol) return;
    if (p < a.np) {
        const int e = a.perm ? a.perm[p] : p;
        const double *y = a.y + 7L * e;
        double vel, cr, sr;
        patch_slip(y[2], y[3], y[6], vel, cr, sr);
        v[2L * p] = vel * cr - a.fr.vpl_c[e];
        v[2L * p + 1] = vel * sr - a.fr.vpl_s[e];
    } else {
        const int iv = p - a.np;
        const double *s = a.y + 7L * a.np + 12L * iv + 6;
        for (int q = 0; q < 6; q++)
            v[2L * a.np + 6L * iv + q] = volume_rate(a.rh, iv, q, s[0], s[1], s[2], s[3], s[4], s[5]) -
                                         a.rh.ebg[6L * iv + q];
    }
}

// ---- control: RKQSm decision ---------------------------------------------------

// by one thread, once every element's error is in
__device__ void decide(Ctl *ctl)
{
    const double SAFETY = 0.7, PGROW = -0.2, PSHRNK = -0.15, ERRCON = 1.89e-4;
    double errmax = __longlong_as_double((long long)ctl->errbits);
    ctl->errbits = 0ull;
    if (ctl->status) return;
    if (ctl->nonfinite) {
        ctl->status = UCG_E_NONFINITE;
        ctl->active = 0;
        return;
    }
    errmax = errmax / ctl->epsilon;
    double h = ctl->h;
    if (errmax > 1.0) {
        h = h * SAFETY * pow(errmax, PSHRNK);
        if (h < 0.5 * h) h = 0.5 * h;   // never taken (ode45.f90:83)
        ctl->h = h;
        ctl->clamped = 0;   // a shrunk step stays short of t_stop
        ctl->rejected += 1;
        ctl->need_stage1 = 0;
        ctl->pending = 0;
        const double tnew = 0.0 + h;     // the main loop passes t0 = 0 (ratestate.f90:317)
        if (tnew == 0.0) {
            ctl->status = UCG_E_STEP_UNDERFLOW;
            ctl->active = 0;
        }
    } else {
        double hnext;
        if (errmax > ERRCON) hnext = SAFETY * h * pow(errmax, PGROW);
        else hnext = 10.0 * h;
        if (hnext > ctl->hmax) hnext = ctl->hmax;
        ctl->hdid = h;
        ctl->time = ctl->clamped ? ctl->t_stop : ctl->time + h;
        ctl->dt_next = hnext;
        ctl->h = hnext;
        ctl->clamped = 0;
        if (ctl->stop_on && ctl->time < ctl->t_stop && ctl->time + hnext > ctl->t_stop) {
            ctl->h = ctl->t_stop - ctl->time;
            ctl->clamped = 1;
        }
        ctl->accepted += 1;
        ctl->pending = 1;
        ctl->vmax = 0.0;
        ctl->need_stage1 = 1;
        if (ctl->time >= ctl->t_end || ctl->accepted >= ctl->step_target) ctl->active = 0;
    }
}

// End of stage 6 in one warp of every CTA that takes part: its largest error, and
// the decision by the CTA that comes last.
__device__ __forceinline__ void attempt_end(Ctl *ctl, double mx, bool bad)
{
    for (int off = 16; off > 0; off >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, off));
    bad = __any_sync(0xffffffffu, bad);
    if ((threadIdx.x & 31) == 0) {
        if (mx > 0.0) atomic_max_pos(&ctl->errbits, mx);
        if (bad) ctl->nonfinite = 1;
        __threadfence();
        if (atomicAdd(&ctl->ticket, 1) == (int)(gridDim.x * gridDim.y) - 1) {
            __threadfence();
            ctl->ticket = 0;
            decide(ctl);
        }
    }
}

// a rejected attempt repeats with a smaller step from the same k_1: stage 2 of a
// patch for the new h
__device__ __forceinline__ void retry_stage2(const StageArgs &a, Ctl *ctl, int e, int pos, int c, bool on, double h)
{
    const long i = 7L * e + c;
    double yn = 0.0;
    if (on) {
        yn = stage_comb(1, LaneState{a.y[i], 0, 0, 0, 1, true}, a.k[0][i], h);
        a.ys[i] = yn;
    }
    const double ts = __shfl_sync(~0u, yn, 2, 8), td = __shfl_sync(~0u, yn, 3, 8), lv = __shfl_sync(~0u, yn, 6, 8);
    if (!on || c > 1) return;
    double vel, cr, sr;
    patch_slip(ts, td, lv, vel, cr, sr);
    if (!isfinite(vel) || !isfinite(cr) || !isfinite(sr)) ctl->nonfinite = 1;
    double v = vel * (c == 0 ? cr : sr) - (c == 0 ? a.fr.vpl_c[e] : a.fr.vpl_s[e]);
    if (a.anchored) v -= a.v1[2L * e + c];
    a.vn[2L * pos + c] = v;
}

// and of a volume
__device__ __forceinline__ void retry_stage2_volume(const StageArgs &a, int iv, int c, bool on, double h)
{
    const long i = 7L * a.np + 12L * iv + c;
    double yn = 0.0;
    if (on) {
        yn = stage_comb(1, LaneState{a.y[i], 0, 0, 0, 1, true}, a.k[0][i], h);
        a.ys[i] = yn;
    }
    double s[6];
#pragma unroll
    for (int q = 0; q < 6; q++) s[q] = __shfl_sync(~0u, yn, 6 + q, 16);
    if (!on || c > 5) return;
    const long j = 2L * a.np + 6L * iv + c;
    double v = volume_rate(a.rh, iv, c, s[0], s[1], s[2], s[3], s[4], s[5]) - a.rh.ebg[6L * iv + c];
    if (a.anchored) v -= a.v1[j];
    a.vn[j] = v;
}

// ---- traction product fused with the right-hand side ----------------------------
//
// K (m x n, row-major) times v.  A CTA owns an equal share of the patches and of
// the volumes (to one element), taken in blocks of at most 12 rows in FP64, 4
// patches (3 rows each) or 2 volumes (6 rows each), and 24 in the split forms.  Its
// 8 warps sweep interleaved column slices of a block's rows, so every v element
// loaded feeds all of them; K is streamed once.  The row sums are reduced across
// lanes and warps, and a warp of its own runs the block's elements through the
// stage (patch_finish, volume_finish) while the others are at the next block.

constexpr int MV_WARPS = 8;

// Stage S on the hierarchical K: a CTA takes HS_P patches of a row leaf, adds up
// their rows over the leaf's chunks (HS_G groups of threads each every HS_G-th
// chunk, then the groups in order) and runs them through the stage, their source
// rates straight into the product's permuted input.  As separate kernels (gather,
// reduction, right-hand side, stage state) these took 24 more launches an attempt.
// One CTA for a whole leaf (225 of 1,024 threads at N = 7,200) left two uneven
// waves: 32 us against 16 with eight patches a CTA (both cold).
constexpr int HS_P = 8, HS_ROWS = 3 * HS_P, HS_G = 8, HS_EL = 8 * HS_P, HS_THREADS = HS_EL + HS_ROWS * HS_G;

__global__ void __launch_bounds__(HS_THREADS, 4) k_hm_stage(int S, StageArgs a, Ctl *ctl, HmParts hp)
{
    __shared__ double sh[HS_G][HS_ROWS];
    __shared__ double tt[HS_ROWS];
    pdl_enter();
    if (!ctl_live(ctl)) return;
    const double h = ctl->h;
    const int L = blockIdx.x, p0 = blockIdx.y * HS_P, e0 = hp.leaf_e0[L] + p0;
    const int nel = min(HS_P, hp.leaf_e0[L + 1] - e0), rows = 3 * nel;   // nel <= 0: a short leaf
    // the first two warps take the patches, the others the sums
    const int c = threadIdx.x & 7, q = threadIdx.x >> 3, pos = e0 + q;
    const bool elem = threadIdx.x < HS_EL, on = elem && q < nel && c < 7;
    const int e = on ? hp.perm[pos] : 0;
    double mx = 0.0;
    bool bad = false;
    if (S == 1 && !ctl->need_stage1) {
        if (elem) retry_stage2(a, ctl, e, pos, c, on, h);
        return;
    }
    LaneState st;
    PatchTerms p;
    if (elem) {
        const double ys = lane_load(S, a, ctl, 7L * e + c, on, st);
        p = patch_terms(S, ctl, patch_friction(a, e, c, on), c, on, ys);
    }
    const int c0 = hp.leaf_chunk[L], c1 = hp.leaf_chunk[L + 1];
    if (!elem) {
        const int g = (threadIdx.x - HS_EL) / HS_ROWS, i = (threadIdx.x - HS_EL) % HS_ROWS;
        double s[8] = {};
        if (i < rows) {
            const double *part = hp.part + 3 * p0 + i;
            int k = c0 + g;
            for (; k + 7 * HS_G < c1; k += 8 * HS_G) {
                double v[8];
#pragma unroll
                for (int u = 0; u < 8; u++) v[u] = part[(long)(k + u * HS_G) * hp.rows_max];
#pragma unroll
                for (int u = 0; u < 8; u++) s[u] += v[u];
            }
#pragma unroll
            for (int u = 0; u < 8; u++)
                if (k + u * HS_G < c1) s[u] += part[(long)(k + u * HS_G) * hp.rows_max];
        }
        sh[g][i] = ((s[0] + s[1]) + (s[2] + s[3])) + ((s[4] + s[5]) + (s[6] + s[7]));
    }
    __syncthreads();
    if (threadIdx.x < HS_ROWS) {
        const int i = threadIdx.x;
        double t = 0.0;
        for (int k = 0; k < HS_G; k++) t += sh[k][i];
        if (a.anchored && i < rows) {
            // anchored stages: stage 1 keeps t1 = K v1, the others add K (v - v1) to it
            double *t1 = a.t1 + 3L * hp.perm[e0 + i / 3] + i % 3;
            if (S == 1) *t1 = t;
            else t += *t1;
        }
        tt[i] = t;
    }
    __syncthreads();
    if (!elem) return;
    patch_finish(S, a, ctl, e, pos, c, h, st, p, tt[3 * q], tt[3 * q + 1], tt[3 * q + 2], mx, bad);
    if (S == 6 && a.next) {
        __shared__ double smx;
        __shared__ int sbad;
        for (int off = 16; off > 0; off >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, off));
        bad = __any_sync(0xffffffffu, bad);
        if (threadIdx.x == 32) {
            smx = mx;
            sbad = bad;
        }
        asm volatile("bar.sync 1, 64;" ::: "memory");   // the two warps of the patches
        if (threadIdx.x < 32) attempt_end(ctl, fmax(mx, smx), bad || sbad);
    }
}

// ---- TMA bulk-copy pipeline ------------------------------------------------------
//
// The traction product streams K once per stage evaluation and is bound by HBM
// bandwidth.  Each persistent CTA (one per SM) owns a sequence of row blocks;
// a producer warp moves K into shared memory with cp.async.bulk row copies
// (192 KB in flight: 4 stages of 48 KB in FP64, 2 of 96 KB in the split forms;
// completion counted on mbarriers) while
// 8 consumer warps multiply by v and hand the stage back.  Consumer thread
// t = 32 w + l accumulates columns c = CH k + PER t .. (PER per thread) across
// chunks, so the per-row summation order is: per-thread fused multiply-adds
// along its columns, an xor butterfly across the 32 lanes, then the 8 warps in
// order (the oracle restates exactly this order).
//
// Every mbarrier wait is bounded (about 4 s of %globaltimer); a wait that runs
// out records UCG_E_TIMEOUT in the control block and the CTA stops.

constexpr unsigned long long TM_TIMEOUT_NS = 4000000000ull;

__device__ __forceinline__ uint32_t smem_u32(const void *p)
{
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t *bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try(uint64_t *bar, uint32_t parity)
{
    uint32_t ok;
    asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
                 " selp.u32 %0, 1, 0, p;\n}" : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
    return ok != 0;
}
__device__ __forceinline__ unsigned long long gtimer()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}
// bounded wait: false when `limit` ns pass or (abort != nullptr) another
// thread aborted
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity, volatile int *abort,
                                          unsigned long long limit = TM_TIMEOUT_NS)
{
    if (mbar_try(bar, parity)) return true;
    const unsigned long long t0 = gtimer();
    for (unsigned it = 1;; it++) {
        if (mbar_try(bar, parity)) return true;
        if ((it & 255u) == 0u) {
            if (abort && *abort) return false;
            if (gtimer() - t0 > limit) return false;
        }
    }
}
__device__ __forceinline__ void bulk_g2s(void *dst, const void *src, uint32_t bytes, uint64_t *bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(smem_u32(dst)), "l"(src), "r"(bytes), "r"(smem_u32(bar)) : "memory");
}

// element traits: FP64 K (2 columns per thread) or split-BF16 pairs (4 per thread)
template <class KT> struct TmTraits;
// ROWS per block: 12 (4 patches or 2 volumes) in FP64; the split forms take
// 24 rows (8 patches or 4 volumes) in two 96 KB stages, which halves the
// per-block reduction and epilogue per K byte where a chunk holds 2-4 times
// more columns
template <> struct TmTraits<double> {
    static constexpr int PER = 2, CH = 512, ROWS = 12, STAGES = 4;
    using Acc = double;
};
template <> struct TmTraits<float> {   // the anchor of the split form: K/s in FP32, FP64 sums
    static constexpr int PER = 4, CH = 1024, ROWS = 24, STAGES = 2;
    using Acc = double;
};
template <> struct TmTraits<__half> {   // the fp16 plane (anchored stages 2-6): FP32 products
    static constexpr int PER = 8, CH = 2048, ROWS = 24, STAGES = 2;   // and 8-term sums, FP64 across
    using Acc = double;
};
template <class KT>
constexpr size_t tm_smem_bytes()
{
    return (size_t)TmTraits<KT>::STAGES * TmTraits<KT>::ROWS * TmTraits<KT>::CH * sizeof(KT);
}
// the thread's PER values of v for one chunk, loaded once and used for all the
// rows of the stage; then one row's contribution
template <class KT> struct TmV;
template <> struct TmV<double> { double2 x; };
template <> struct TmV<float> { double x[4]; };
template <> struct TmV<__half> { float x[8]; };   // v in FP32: the plane itself carries 2^-12
// v as loaded (one chunk ahead): the fp16 form keeps the doubles and converts
// them when the chunk is used, so that no instruction waits on the loads early
template <class KT> struct TmVRaw { TmV<KT> v; };
template <> struct TmVRaw<__half> { double x[8]; };

template <class KT>
__device__ __forceinline__ void tm_load_v(const double *v, long c, long n, TmV<KT> &vr);
template <>
__device__ __forceinline__ void tm_load_v<double>(const double *v, long c, long n, TmV<double> &vr)
{
    (void)n;
    vr.x = *reinterpret_cast<const double2 *>(v + c);
}
// c is a multiple of the values per thread (4 or 8), so away from the ragged
// end the thread's values are 16-byte aligned pairs.  Plain loads: the launch in
// front may still be writing v when this one starts, and the read-only path asks for
// memory that nobody writes while the kernel runs (same time)
template <>
__device__ __forceinline__ void tm_load_v<float>(const double *v, long c, long n, TmV<float> &vr)
{
    if (c + 4 <= n) {
        const double2 a = *reinterpret_cast<const double2 *>(v + c);
        const double2 b = *reinterpret_cast<const double2 *>(v + c + 2);
        vr.x[0] = a.x; vr.x[1] = a.y; vr.x[2] = b.x; vr.x[3] = b.y;
        return;
    }
#pragma unroll
    for (int q = 0; q < 4; q++) vr.x[q] = (c + q < n) ? v[c + q] : 0.0;
}
// the raw loads of one chunk's v (every form) and their conversion when used
template <class KT>
__device__ __forceinline__ void tm_load_raw(const double *v, long c, long n, TmVRaw<KT> &raw)
{
    tm_load_v<KT>(v, c, n, raw.v);
}
template <>
__device__ __forceinline__ void tm_load_raw<__half>(const double *v, long c, long n, TmVRaw<__half> &raw)
{
    if (c + 8 <= n) {
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const double2 a = *reinterpret_cast<const double2 *>(v + c + 2 * q);
            raw.x[2 * q] = a.x;
            raw.x[2 * q + 1] = a.y;
        }
        return;
    }
#pragma unroll
    for (int q = 0; q < 8; q++) raw.x[q] = (c + q < n) ? v[c + q] : 0.0;
}
template <class KT>
__device__ __forceinline__ void tm_cook(const TmVRaw<KT> &raw, TmV<KT> &vr)
{
    vr = raw.v;
}
template <>
__device__ __forceinline__ void tm_cook<__half>(const TmVRaw<__half> &raw, TmV<__half> &vr)
{
#pragma unroll
    for (int q = 0; q < 8; q++) vr.x[q] = __double2float_rn(raw.x[q]);
}

template <class KT>
__device__ __forceinline__ void tm_accumulate(const KT *srow, int cl, const TmV<KT> &vr,
                                              typename TmTraits<KT>::Acc &acc);
template <>
__device__ __forceinline__ void tm_accumulate<double>(const double *srow, int cl, const TmV<double> &vr, double &acc)
{
    const double2 kv = *reinterpret_cast<const double2 *>(srow + cl);
    acc = fma(kv.y, vr.x.y, fma(kv.x, vr.x.x, acc));
}
template <>
__device__ __forceinline__ void tm_accumulate<float>(const float *srow, int cl, const TmV<float> &vr, double &acc)
{
    const float4 kv = *reinterpret_cast<const float4 *>(srow + cl);
    acc = fma((double)kv.x, vr.x[0], acc);
    acc = fma((double)kv.y, vr.x[1], acc);
    acc = fma((double)kv.z, vr.x[2], acc);
    acc = fma((double)kv.w, vr.x[3], acc);
}
// the thread's 8 products of the row in FP32 (each rounded once, 2^-24: far
// below the plane's own 2^-12), their sum added to the FP64 row sum: one
// conversion to FP64 per 8 entries instead of one per entry
template <>
__device__ __forceinline__ void tm_accumulate<__half>(const __half *srow, int cl, const TmV<__half> &vr, double &acc)
{
    const uint4 raw = *reinterpret_cast<const uint4 *>(srow + cl);
    const uint32_t w4[4] = {raw.x, raw.y, raw.z, raw.w};
    float p = 0.0f;
#pragma unroll
    for (int q = 0; q < 4; q++) {
        const float2 f = __half22float2(*reinterpret_cast<const __half2 *>(&w4[q]));
        p = __fmaf_rn(f.x, vr.x[2 * q], p);
        p = __fmaf_rn(f.y, vr.x[2 * q + 1], p);
    }
    acc += (double)p;
}

// Sums of ROWS values over the lanes of a warp, row by row, each the xor butterfly
// with offsets 16, 8, 4, 2, 1.  Instead of 5 exchanges a row, each step sends half
// of the rows a lane still holds to its partner and keeps the other half (13
// exchanges and adds for 12 rows instead of 60: 1.38 -> 0.3 us of a launch at N = 512).  Lane
// l ends up with the sum of row warp_row(l).
template <int ROWS>
struct RowHalves {
    static constexpr int n1 = ROWS / 2, n2 = (n1 + 1) / 2, n3 = (n2 + 1) / 2, n4 = (n3 + 1) / 2,
                         n5 = (n4 + 1) / 2;
};
template <int N, int H>
__device__ __forceinline__ void fold_rows(double *x, int lane, int off)
{
    const bool up = lane & off;
#pragma unroll
    for (int i = 0; i < H; i++) {
        const double hi = H + i < N ? x[H + i] : 0.0;
        const double keep = up ? hi : x[i], give = up ? x[i] : hi;
        x[i] = keep + __shfl_xor_sync(0xffffffffu, give, off);
    }
}
template <int ROWS>
__device__ __forceinline__ double warp_row_sums(double *x, int lane)
{
    using R = RowHalves<ROWS>;
    fold_rows<ROWS, R::n1>(x, lane, 16);
    fold_rows<R::n1, R::n2>(x, lane, 8);
    fold_rows<R::n2, R::n3>(x, lane, 4);
    fold_rows<R::n3, R::n4>(x, lane, 2);
    fold_rows<R::n4, R::n5>(x, lane, 1);
    static_assert(R::n5 == 1, "at most 32 rows");
    return x[0];
}
// the row of a lane's sum, ROWS where it has none
template <int ROWS>
__device__ __forceinline__ int warp_row(int lane)
{
    using R = RowHalves<ROWS>;
    int n = ROWS, row = 0;
    const int h[5] = {R::n1, R::n2, R::n3, R::n4, R::n5};
#pragma unroll
    for (int s = 0; s < 5; s++) {
        const bool up = lane & (16 >> s);
        row += up ? h[s] : 0;
        n = up ? n - h[s] : n < h[s] ? n : h[s];
    }
    return n > 0 ? row : ROWS;
}

// the blocks of a CTA: its patches, then its volumes, each share in blocks of
// nearly equal size
template <class KT>
struct Share {
    static constexpr int PB = TmTraits<KT>::ROWS / 3, VB = TmTraits<KT>::ROWS / 6;   // patches, volumes per block
    int p0, np, v0, nv;     // this CTA's patches and volumes
    int bp, bv;             // their blocks
    long prows;             // rows of all patches

    __device__ __forceinline__ Share(int npatch, int nvol, int cta, int ctas)
    {
        // the first `more` CTAs take one element above the quotient
        const int qp = npatch / ctas, mp = npatch - qp * ctas, qv = nvol / ctas, mv = nvol - qv * ctas;
        p0 = qp * cta + min(cta, mp);
        np = qp + (cta < mp);
        v0 = qv * cta + min(cta, mv);
        nv = qv + (cta < mv);
        bp = (np + PB - 1) / PB;
        bv = (nv + VB - 1) / VB;
        prows = 3L * npatch;
    }
    __device__ __forceinline__ int blocks() const { return bp + bv; }
    // first row and rows of block b, its first element and their number
    __device__ __forceinline__ bool block(int b, long &row0, int &nrows, int &e0, int &nel) const
    {
        const bool patch = b < bp;
        if (patch) {
            const int lo = np * b / bp;
            nel = np * (b + 1) / bp - lo;
            e0 = p0 + lo;
            row0 = 3L * e0;
            nrows = 3 * nel;
        } else {
            const int q = b - bp, lo = nv * q / bv;
            nel = nv * (q + 1) / bv - lo;
            e0 = v0 + lo;
            row0 = prows + 6L * e0;
            nrows = 6 * nel;
        }
        return patch;
    }
};

constexpr int TM_THREADS = (MV_WARPS + 2) * 32;   // consumers, producer, epilogue

// named barriers between the consumers and the epilogue warp: buffer b of the row
// sums is full (1 + b), or read and free again (3 + b)
__device__ __forceinline__ void bar_arrive(int id) { asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(MV_WARPS * 32 + 32) : "memory"); }
__device__ __forceinline__ void bar_wait(int id) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(MV_WARPS * 32 + 32) : "memory"); }

// What a CTA of k_traction takes from the control block, read once and handed to all
// its warps: another CTA may end the run (a wait that ran out) between two reads, and
// a warp that left by itself would keep the others waiting at the barriers above.  The
// consumers and the epilogue warp meet at a barrier, the producer's one lane waits for
// `read` (a producer warp kept whole for the barrier took 1.5 % of 8 steps of 7,200
// triangles, split pair: 10.13 ms against 9.95).
struct TmHead {
    double h;
    unsigned long long wait_ns;
    int live, first;       // first: the product is wanted (stage 1 of a rejected attempt repeats nothing)
};
__device__ __forceinline__ TmHead tm_head(int S, const Ctl *ctl, TmHead &sh, uint64_t *read, bool reader)
{
    if (reader) {
        sh = TmHead{ctl->h, ctl->wait_ns, ctl_live(ctl), S > 1 || ctl->need_stage1};
        mbar_arrive(read);
    }
    asm volatile("bar.sync 5, %0;" ::"n"(MV_WARPS * 32 + 32) : "memory");
    return sh;
}

// The stage number is an argument: the six launches of an attempt run the same
// code, which then stays in the instruction caches.
template <class KT>
__global__ void __launch_bounds__(TM_THREADS, 1) k_traction(int S, const KT *__restrict__ K, long n,
        long ldk, const float *__restrict__ scale, StageArgs a, Ctl *ctl)
{
    using Tr = TmTraits<KT>;
    using Acc = typename Tr::Acc;
    constexpr int CH = Tr::CH, PER = Tr::PER, ROWS = Tr::ROWS, stages = Tr::STAGES;
    extern __shared__ __align__(128) unsigned char tm_smem[];
    KT *stage = reinterpret_cast<KT *>(tm_smem);
    __shared__ __align__(8) uint64_t full[Tr::STAGES], empty[Tr::STAGES], head_read;
    __shared__ double red[2][MV_WARPS][ROWS];
    __shared__ int abort_flag;
    __shared__ TmHead head;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // the next launch may come as soon as there is room: before its own wait it only
    // reads K and the friction, which no launch changes
    pdl_launch();
    const Share<KT> share(a.np, a.nvol, blockIdx.x, gridDim.x);
    const int nblk = share.blocks();
    const int nch = (int)((n + CH - 1) / CH);
    if (threadIdx.x == 0) {
        for (int s = 0; s < stages; s++) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], MV_WARPS);
        }
        mbar_init(&head_read, 1);
        abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();

    if (warp == MV_WARPS) {
        // producer: one lane issues the row copies of each (block, chunk) item.  K does
        // not depend on the launches before, so the first stages are filled before
        // the wait for them.  The first goes out blind; the others once the control
        // block does not say that the run has ended (a value that is out of date costs
        // nothing but these copies, or their lead).  With all of them blind the 31 attempts
        // that may be queued behind a run's end took 701 us (7,200 triangles), now 448, in a
        // run of 16 x 16 rectangles and 128 cuboids 572 and 379; with none, a step of
        // 512 rectangles takes 7 % longer.
        if (lane != 0) return;
        int item = 0, s = 0, ph = 0, b = 0, ch = 0, nrows = 0, e0, nel;
        long row0 = 0;
        const int total = nblk * nch;
        auto issue = [&]() {
            if (ch == 0) share.block(b, row0, nrows, e0, nel);
            const long c0 = (long)ch * CH;
            const long w = min((long)CH, ldk - c0);
            const uint32_t rowbytes = (uint32_t)(w * sizeof(KT));
            mbar_expect_tx(&full[s], rowbytes * nrows);
            KT *dst = stage + (size_t)s * ROWS * CH;
            for (int r = 0; r < nrows; r++)
                bulk_g2s(dst + (size_t)r * CH, K + (row0 + r) * ldk + c0, rowbytes, &full[s]);
            item++;
            if (++ch == nch) { ch = 0; b++; }
            if (++s == stages) { s = 0; ph ^= 1; }
        };
        // (test_hold: the first CTA issues nothing, its consumers' waits run out)
        const bool hold = blockIdx.x == 0 && *(volatile int *)&ctl->test_hold;
        if (!hold && total > 0) {
            issue();
            if (ctl_hint(ctl))
                while (item < total && item < stages) issue();
        }
        pdl_wait();
        const bool go = mbar_wait(&head_read, 0, nullptr) && head.live && head.first;
        if (!hold && go) {
            while (item < total && !*(volatile int *)&abort_flag) {
                if (!mbar_wait(&empty[s], ph ^ 1, &abort_flag)) {
                    abort_flag = 1;
                    ctl->status = UCG_E_TIMEOUT;
                    break;
                }
                issue();
            }
        }
        // items are issued in order, so the last copies into each stage are those
        // of the last items: they land before the CTA may exit, also when the
        // consumers gave up on them or never started (bounded at the normal limit)
        for (int i = item > stages ? item - stages : 0; i < item; i++)
            mbar_wait(&full[i % stages], (uint32_t)((i / stages) & 1), nullptr);
        return;
    }

    if (warp == MV_WARPS + 1) {
        // epilogue: the elements of one block after the other.  The first patches'
        // friction is asked for before the wait for the launches before.
        PatchFriction fr{1, 1, 0, 0, 1, 1, 0};
        {
            long row0;
            int nrows, e0, nel;
            if (nblk > 0 && share.block(0, row0, nrows, e0, nel))
                fr = patch_friction(a, e0 + (lane >> 3), lane & 7, (lane >> 3) < nel && (lane & 7) < 7);
        }
        pdl_wait();
        const TmHead hd = tm_head(S, ctl, head, &head_read, lane == 0);
        if (!hd.live) return;
        const double h = hd.h;
        const bool first = hd.first;
        double mx = 0.0;
        bool bad = false;
        for (int b = 0; b < nblk; b++) {
            long row0;
            int nrows, e0, nel;
            const bool patch = share.block(b, row0, nrows, e0, nel);
            const int per = patch ? 4 : 2, c = patch ? lane & 7 : lane & 15, nc = patch ? 7 : 12;
            const int sub = patch ? lane >> 3 : lane >> 4;
            for (int q0 = 0; q0 < nel; q0 += per) {
                const int q = q0 + sub, e = e0 + q;
                const bool on = q < nel && c < nc;
                if (!first) {
                    if (patch) retry_stage2(a, ctl, e, e, c, on, h);
                    else retry_stage2_volume(a, e, c, on, h);
                    continue;
                }
                // rows of the element that this lane adds up over the warps: a patch's
                // three in its lanes 0..2, a volume's six in 6..11
                const int r = patch ? 3 * q + c : 6 * q + c - 6;
                const bool sum = on && (patch ? c < 3 : c > 5);
                if (patch) {
                    LaneState st;
                    const double ys = lane_load(S, a, ctl, 7L * e + c, on, st);
                    if (b + q0 > 0) fr = patch_friction(a, e, c, on);
                    const PatchTerms p = patch_terms(S, ctl, fr, c, on, ys);
                    if (q0 == 0) bar_wait(1 + (b & 1));
                    double t = 0.0;
                    if (sum) {
                        for (int w = 0; w < MV_WARPS; w++) t += red[b & 1][w][r];
                        if (scale) t = t * (double)scale[row0 + r];
                        if (a.anchored) {
                            if (S == 1) a.t1[row0 + r] = t;
                            else t += a.t1[row0 + r];
                        }
                    }
                    const double t0 = __shfl_sync(~0u, t, 0, 8), t1 = __shfl_sync(~0u, t, 1, 8),
                                 t2 = __shfl_sync(~0u, t, 2, 8);
                    if (!abort_flag) patch_finish(S, a, ctl, e, e, c, h, st, p, t0, t1, t2, mx, bad);
                } else {
                    LaneState st;
                    const double ys = lane_load(S, a, ctl, 7L * a.np + 12L * e + c, on, st);
                    double sv[6];
#pragma unroll
                    for (int k = 0; k < 6; k++) sv[k] = __shfl_sync(~0u, ys, 6 + k, 16);
                    const double ev = on && c < 6 ? volume_rate(a.rh, e, c, sv[0], sv[1], sv[2], sv[3], sv[4], sv[5])
                                                  : 0.0;
                    if (q0 == 0) bar_wait(1 + (b & 1));
                    double t = 0.0;
                    if (sum) {
                        for (int w = 0; w < MV_WARPS; w++) t += red[b & 1][w][r];
                        if (scale) t = t * (double)scale[row0 + r];
                        if (a.anchored) {
                            if (S == 1) a.t1[row0 + r] = t;
                            else t += a.t1[row0 + r];
                        }
                    }
                    if (!abort_flag) volume_finish(S, a, e, c, h, st, ev, t, mx, bad);
                }
            }
            // the buffer comes round again two blocks later
            if (first && b + 2 < nblk) bar_arrive(3 + (b & 1));
        }
        if (S == 6 && a.next) attempt_end(ctl, mx, bad);
        return;
    }

    // consumers.  The first v values are on their way while the control block is read.
    const int t = threadIdx.x, cl = PER * t;
    pdl_wait();
    TmVRaw<KT> vn;
    if (cl < n) tm_load_raw<KT>(a.v, cl, n, vn);
    const TmHead hd = tm_head(S, ctl, head, &head_read, false);
    if (!hd.live || !hd.first) return;
    const unsigned long long wait_ns = hd.wait_ns;
    int s = 0, ph = 0;
    for (int b = 0; b < nblk; b++) {
        long row0;
        int nrows, e0, nel;
        share.block(b, row0, nrows, e0, nel);
        Acc acc[ROWS];
#pragma unroll
        for (int r = 0; r < ROWS; r++) acc[r] = Acc(0);
        // v does not depend on the stage: each chunk's values are loaded one
        // chunk ahead, so their latency overlaps the previous chunk's products
        for (int ch = 0; ch < nch; ch++) {
            // on a timed-out wait every consumer keeps walking the same item
            // sequence without computing, so all of them reach each named barrier
            const long c = (long)ch * CH + cl;
            TmV<KT> vr;
            if (c < n) tm_cook<KT>(vn, vr);
            const long cn = ch + 1 < nch ? c + CH : cl;   // the next block starts at its first chunk
            if (cn < n) tm_load_raw<KT>(a.v, cn, n, vn);
            const bool ready = !abort_flag && (mbar_try(&full[s], ph) ||
                                               mbar_wait(&full[s], ph, &abort_flag, wait_ns ? wait_ns : TM_TIMEOUT_NS));
            if (!ready && !abort_flag) {
                abort_flag = 1;
                ctl->status = UCG_E_TIMEOUT;
            }
            const KT *src = stage + (size_t)s * ROWS * CH;
            if (ready && c < n) {
#pragma unroll
                for (int r = 0; r < ROWS; r++)
                    if (r < nrows) tm_accumulate<KT>(src + (size_t)r * CH, cl, vr, acc[r]);
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&empty[s]);
            if (++s == stages) { s = 0; ph ^= 1; }
        }
        const double x = warp_row_sums<ROWS>(acc, lane);
        if (b > 1) bar_wait(3 + (b & 1));
        const int row = warp_row<ROWS>(lane);
        if (row < ROWS) red[b & 1][warp][row] = x;
        __syncwarp();
        bar_arrive(1 + (b & 1));
    }
}

// one output record at the start of a step (after stage 1: y and its rate k1)
__global__ void k_record(StageArgs a, const Ctl *ctl, Rec *rec)
{
    pdl_enter();
    if (!rec->enabled || !ctl_live(ctl) || !ctl->need_stage1) return;
    const long long step = ctl->accepted - rec->base;
    if (step < 0 || step % rec->every) return;
    const long long idx = step / rec->every;
    double *r = rec->buf + (idx % rec->cap) * rec->len;
    const int t = blockIdx.x * blockDim.x + threadIdx.x, nt = gridDim.x * blockDim.x;
    if (t == 0) {
        r[0] = ctl->time;
        r[1] = ctl->hdid;
        r[2] = ctl->vmax;
        r[3] = (double)ctl->accepted;
    }
    // listed elements: state then rate, 7 per patch / 12 per volume, in a slot of 24
    for (int j = t; j < rec->nelem * 24; j += nt) {
        const int e = rec->elem[j / 24], q = j % 24;
        const bool patch = e < a.np;
        const int w = patch ? 7 : 12;
        const long o = patch ? 7L * e : 7L * a.np + 12L * (e - a.np);
        double v = 0.0;
        if (q < w) v = a.y[o + q];
        else if (q >= 12 && q - 12 < w) v = a.k[0][o + q - 12];
        r[4 + j] = v;
    }
    // observation-point displacements: row k of O against the slip (patches)
    // and the strain (volumes) of the state, one warp per row
    const int warp = t >> 5, nw = nt >> 5;
    double *ro = r + 4 + 24 * rec->nelem;
    for (int k = warp; k < 3 * rec->nobs; k += nw) {
        double sf, sl;
        observe_row(rec->O + (long)k * (2L * a.np + 6L * a.nvol), a.np, a.nvol, a.y, sf, sl);
        if ((t & 31) == 0) {
            const int p = k / 3, c = k % 3;
            if (rec->per_point == 3) {
                ro[3 * p + c] = sf + sl;
            } else {
                double d, df, dl;
                observe_split(c, sf, sl, d, df, dl);
                ro[9 * p + c] = d;
                ro[9 * p + 3 + c] = df;
                ro[9 * p + 6 + c] = dl;
            }
        }
    }
    if (t == 0) rec->written = idx + 1;
}

__global__ void k_commit(StageArgs a, Ctl *ctl)
{
    pdl_enter();
    if (ctl_live(ctl) || !ctl->pending) return;      // the same in every block: the last one out clears it
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < a.len; i += (long)gridDim.x * blockDim.x)
        a.y[i] = a.ycand[i];
    __syncthreads();
    if (threadIdx.x == 0 && atomicAdd(&ctl->committed, 1) == (int)gridDim.x - 1) {
        ctl->committed = 0;
        ctl->pending = 0;
    }
}

// ---- host side -----------------------------------------------------------------

bool rk_anchored(const ucg_ctx *c)
{
    return ((c->precision == UCG_PREC_SPLIT_BF16 || c->precision == UCG_PREC_SPLIT_PAIR) && c->Ksp != nullptr) ||
           c->precision == UCG_PREC_HMATRIX_SPLIT;
}

// the attempt graph holds device addresses of the matrix and parameter arrays;
// whoever frees or replaces one of them drops the graph first
void rk_drop_graph(ucg_ctx *c)
{
    if (!c->attempt_graph) return;
    cudaStreamSynchronize(c->stream);
    cudaGraphExecDestroy(c->attempt_graph);
    c->attempt_graph = nullptr;
}

static bool rk_hierarchical(const ucg_ctx *c)
{
    return c->precision == UCG_PREC_HMATRIX || c->precision == UCG_PREC_HMATRIX_SPLIT;
}

// stage s reads its source rates from buffer s & 1 and writes the next stage's
// into the other (hierarchical K: one buffer, the product's permuted input)
static StageArgs stage_args(ucg_ctx *c, int s, int next)
{
    StageArgs a;
    a.y = c->st.y;
    a.ys = c->st.ytmp;
    for (int j = 0; j < 6; j++) a.k[j] = c->st.k[j];
    a.ks = c->st.k[s - 1];
    a.v = c->st.v[s & 1];
    a.vn = c->st.v[(s + 1) & 1];
    a.perm = nullptr;
    if (rk_hierarchical(c)) {
        const HmParts hp = hmatrix_parts(c);
        a.vn = hp.xp;
        a.perm = hp.perm;
    }
    a.next = next;
    a.ycand = c->st.ycand;
    a.yerr = c->st.yerr;
    a.yscal = c->st.yscal;
    a.v1 = c->st.v1;
    a.t1 = c->st.t1;
    a.anchored = rk_anchored(c) ? 1 : 0;
    a.fr = c->fr;
    a.rh = c->rh;
    a.np = c->nr + c->nt;
    a.nvol = c->nv;
    a.len = c->state_len;
    return a;
}

int rk_alloc(ucg_ctx *c)
{
    rk_free(c);
    const long len = c->state_len;
    double **bufs[] = {&c->st.y, &c->st.ycand, &c->st.ytmp, &c->st.yerr, &c->st.yscal,
                       &c->st.k[0], &c->st.k[1], &c->st.k[2], &c->st.k[3], &c->st.k[4], &c->st.k[5]};
    for (double **b : bufs) {
        if (cudaMalloc(b, sizeof(double) * (len + 2)) != cudaSuccess) return UCG_E_OOM;
        cudaMemsetAsync(*b, 0, sizeof(double) * (len + 2), c->stream);
    }
    for (double *&v : c->st.v)
        if (cudaMalloc(&v, sizeof(double) * (c->n + 2)) != cudaSuccess) return UCG_E_OOM;
    if (cudaMalloc(&c->st.v1, sizeof(double) * (c->n + 2)) != cudaSuccess) return UCG_E_OOM;
    if (cudaMalloc(&c->st.t1, sizeof(double) * (c->m + 2)) != cudaSuccess) return UCG_E_OOM;
    if (cudaMalloc(&c->ctl, sizeof(Ctl)) != cudaSuccess) return UCG_E_OOM;
    if (cudaMalloc(&c->rec, sizeof(Rec)) != cudaSuccess) return UCG_E_OOM;
    {
        Rec off{};
        UCG_CUDA(cudaMemcpyAsync(c->rec, &off, sizeof(Rec), cudaMemcpyHostToDevice, c->stream));
        c->rec_host = off;
    }
    if (cudaMallocHost(&c->ctl_host, sizeof(Ctl)) != cudaSuccess) return UCG_E_OOM;
    if (cudaMallocHost(&c->pin, sizeof(double) * (2 * len + 8)) != cudaSuccess) return UCG_E_OOM;
    memset(c->ctl_host, 0, sizeof(Ctl));
    c->ctl_host->epsilon = c->epsilon;
    c->ctl_host->hmax = c->hmax;
    UCG_CUDA(cudaMemcpyAsync(c->ctl, c->ctl_host, sizeof(Ctl), cudaMemcpyHostToDevice, c->stream));
    return UCG_OK;
}

void rk_free(ucg_ctx *c)
{
    double **bufs[] = {&c->st.y, &c->st.ycand, &c->st.ytmp, &c->st.yerr, &c->st.yscal,
                       &c->st.k[0], &c->st.k[1], &c->st.k[2], &c->st.k[3], &c->st.k[4], &c->st.k[5],
                       &c->st.v[0], &c->st.v[1], &c->st.v1, &c->st.t1};
    for (double **b : bufs) {
        if (*b) cudaFree(*b);
        *b = nullptr;
    }
    if (c->ctl) cudaFree(c->ctl);
    c->ctl = nullptr;
    if (c->rec) cudaFree(c->rec);
    c->rec = nullptr;
    if (c->rec_buf) cudaFree(c->rec_buf);
    c->rec_buf = nullptr;
    if (c->rec_elem) cudaFree(c->rec_elem);
    c->rec_elem = nullptr;
    c->rec_host = Rec{};
    c->rec_drained = 0;
    if (c->pert) cudaFree(c->pert);
    c->pert = nullptr;
    if (c->ctl_host) cudaFreeHost(c->ctl_host);
    c->ctl_host = nullptr;
    if (c->pin) cudaFreeHost(c->pin);
    c->pin = nullptr;
    if (c->attempt_graph) cudaGraphExecDestroy(c->attempt_graph);
    c->attempt_graph = nullptr;
}

template <class KT>
static cudaError_t launch_traction_t(ucg_ctx *c, int S, const StageArgs &a, const KT *K, long ldk, const float *scale)
{
    const int ne = a.np + a.nvol, grid = ne < c->sms ? ne : c->sms;
    const size_t smem = tm_smem_bytes<KT>();
    auto kfn = k_traction<KT>;
    const cudaError_t e = cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    return launch_pdl(kfn, dim3(grid), dim3(TM_THREADS), smem, c->stream, S, K, c->n, ldk, scale, a, c->ctl);
}

static cudaError_t launch_traction(ucg_ctx *c, int S, const StageArgs &a)
{
    if (S > 1 && c->precision == UCG_PREC_SPLIT_BF16 && rk_anchored(c) && c->Khi_plane) {
        // anchored stages multiply the increments by the fp16 plane
        return launch_traction_t<__half>(c, S, a, c->Khi_plane, c->ldk_split, c->Kscale);
    } else if ((c->precision == UCG_PREC_SPLIT_BF16 || c->precision == UCG_PREC_SPLIT_PAIR) && c->Ksp) {
        return launch_traction_t<float>(c, S, a, c->Ksp, c->ldk_split, c->Kscale);
    }
    return launch_traction_t<double>(c, S, a, c->K, c->n, nullptr);
}

static cudaError_t enqueue_stage(ucg_ctx *c, int S, int next)
{
    const StageArgs a = stage_args(c, S, next);
    c->launches.count += 1;
    if (!rk_hierarchical(c)) return launch_traction(c, S, a);
    const cudaError_t e = hmatrix_products(c, c->precision == UCG_PREC_HMATRIX_SPLIT);
    if (e != cudaSuccess) return e;
    const HmParts hp = hmatrix_parts(c);
    return launch_pdl(k_hm_stage, dim3(hp.n_leaves, (hp.rows_max + HS_ROWS - 1) / HS_ROWS), dim3(HS_THREADS), 0,
                      c->stream, S, a, c->ctl, hp);
}

// source rates of the state y, before a run's first attempt
cudaError_t rk_enqueue_begin(ucg_ctx *c)
{
    const StageArgs a = stage_args(c, 1, 0);
    const int ne = a.np + a.nvol;
    c->launches.count += 1;
    return launch_pdl(k_begin, dim3((ne + 127) / 128), dim3(128), 0, c->stream, a, c->ctl,
                      a.perm ? a.vn : c->st.v[1]);
}

static cudaError_t enqueue_attempt_raw(ucg_ctx *c)
{
    cudaError_t e = enqueue_stage(c, 1, 1);
    // the recorder joins the attempt (and its graph) only while recording is on
    if (e == cudaSuccess && c->rec_host.enabled) {
        e = launch_pdl(k_record, dim3(c->sms), dim3(256), 0, c->stream, stage_args(c, 1, 0), c->ctl, c->rec);
        c->launches.count += 1;
    }
    for (int s = 2; s <= 6 && e == cudaSuccess; s++) e = enqueue_stage(c, s, 1);
    return e;
}

cudaError_t rk_enqueue_attempt(ucg_ctx *c)
{
    if (!c->attempt_graph || c->graph_precision != c->precision) {
        if (c->attempt_graph) cudaGraphExecDestroy(c->attempt_graph);
        c->attempt_graph = nullptr;
        cudaGraph_t g;
        long before = c->launches.count;
        cudaError_t refused = cudaSuccess;
        if (cudaStreamBeginCapture(c->stream, cudaStreamCaptureModeThreadLocal) == cudaSuccess) {
            refused = enqueue_attempt_raw(c);
            c->graph_launches = c->launches.count - before;
            if (cudaStreamEndCapture(c->stream, &g) == cudaSuccess) {
                // (an attempt without one of its kernels is no attempt)
                if (refused != cudaSuccess || cudaGraphInstantiate(&c->attempt_graph, g, 0) != cudaSuccess)
                    c->attempt_graph = nullptr;
                cudaGraphDestroy(g);
            }
        }
        c->launches.count = before;
        c->graph_precision = c->precision;
        cudaGetLastError();
    }
    // without a graph the attempt is launched kernel by kernel, and says what refuses it
    if (!c->attempt_graph) return enqueue_attempt_raw(c);
    c->launches.count += c->graph_launches;
    return cudaGraphLaunch(c->attempt_graph, c->stream);
}

cudaError_t rk_enqueue_commit(ucg_ctx *c)
{
    const StageArgs a = stage_args(c, 1, 0);
    c->launches.count += 1;
    return launch_pdl(k_commit, dim3((unsigned)((c->state_len + 255) / 256)), dim3(256), 0, c->stream, a, c->ctl);
}

// Mean device time of the stage-2 traction launch (the dominant kernel), timed
// with events on the context stream.  The control block is made live for the
// measurement and restored afterwards.
int rk_profile_traction(ucg_ctx *c, int reps, double *ms)
{
    Ctl *h = c->ctl_host;
    UCG_CUDA(cudaMemcpyAsync(h, c->ctl, sizeof(Ctl), cudaMemcpyDeviceToHost, c->stream));
    UCG_CUDA(cudaStreamSynchronize(c->stream));
    Ctl saved = *h;
    h->active = 1;
    h->status = 0;
    UCG_CUDA(cudaMemcpyAsync(c->ctl, h, sizeof(Ctl), cudaMemcpyHostToDevice, c->stream));
    StageArgs a = stage_args(c, 2, 0);
    cudaEvent_t e0, e1;
    UCG_CUDA(cudaEventCreate(&e0));
    UCG_CUDA(cudaEventCreate(&e1));
    UCG_CUDA(cudaEventRecord(e0, c->stream));
    cudaError_t le = cudaSuccess;
    for (int r = 0; r < reps && le == cudaSuccess; r++) le = launch_traction(c, 2, a);
    c->launches.count += reps;
    UCG_CUDA(cudaEventRecord(e1, c->stream));
    UCG_CUDA(cudaEventSynchronize(e1));
    float t = 0.0f;
    UCG_CUDA(cudaEventElapsedTime(&t, e0, e1));
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    *ms = (double)t / reps;
    *h = saved;
    UCG_CUDA(cudaMemcpyAsync(c->ctl, h, sizeof(Ctl), cudaMemcpyHostToDevice, c->stream));
    UCG_CUDA(cudaStreamSynchronize(c->stream));
    return le == cudaSuccess ? UCG_OK : cuda_fail(c, le, "traction launch");
}

// A coseismic perturbation of the state: slip (2 per patch) and eigenstrain
// (6 per volume) increments u, and the stress they cause, K u, added to the
// tractions (3 per patch) and stresses (6 per volume).  One warp per row of K.
__global__ void k_perturb(const double *__restrict__ K, long m, long n, int np, const double *__restrict__ u,
                          double *__restrict__ y)
{
    const long t = (long)blockIdx.x * blockDim.x + threadIdx.x, nt = (long)gridDim.x * blockDim.x;
    const int lane = threadIdx.x & 31;
    for (long r = t >> 5; r < m; r += nt >> 5) {
        const double *Kr = K + r * n;
        double s = 0.0;
        for (long c = lane; c < n; c += 32) s = fma(Kr[c], u[c], s);
        for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
        if (lane == 0) {
            const long i = r < 3L * np ? 7L * (r / 3) + 2 + r % 3
                                       : 7L * np + 12L * ((r - 3L * np) / 6) + 6 + (r - 3L * np) % 6;
            y[i] += s;
        }
    }
    for (long c = t; c < n; c += nt) {
        const long i = c < 2L * np ? 7L * (c >> 1) + (c & 1) : 7L * np + 12L * ((c - 2L * np) / 6) + (c - 2L * np) % 6;
        y[i] += u[c];
    }
}

// the same with the stress change t = H u already formed (hierarchical matrix)
__global__ void k_perturb_t(long m, long n, int np, const double *__restrict__ t, const double *__restrict__ u,
                            double *__restrict__ y)
{
    const long i0 = (long)blockIdx.x * blockDim.x + threadIdx.x, nt = (long)gridDim.x * blockDim.x;
    for (long r = i0; r < m; r += nt) y[7L * (r / 3) + 2 + r % 3] += t[r];
    for (long c = i0; c < n; c += nt) y[7L * (c >> 1) + (c & 1)] += u[c];
}

int rk_perturb(ucg_ctx *c, const double *u)
{
    if (!c->K && !(c->hm && c->nv == 0)) return UCG_E_STATE;
    if (!c->pert) UCG_CUDA(cudaMalloc(&c->pert, sizeof(double) * c->n));
    UCG_CUDA(cudaMemcpyAsync(c->pert, u, sizeof(double) * c->n, cudaMemcpyHostToDevice, c->stream));
    const int blocks = (int)std::min<long>((c->m + 7) / 8, 8L * c->sms);
    if (c->K) {
        k_perturb<<<blocks, 256, 0, c->stream>>>(c->K, c->m, c->n, c->nr + c->nt, c->pert, c->st.y);
    } else {
        double *t = hmatrix_t(c);
        UCG_CUDA(hmatrix_apply(c, c->pert, t));
        k_perturb_t<<<blocks, 256, 0, c->stream>>>(c->m, c->n, c->nr + c->nt, t, c->pert, c->st.y);
    }
    c->launches.count++;
    UCG_CUDA(cudaGetLastError());
    UCG_CUDA(cudaStreamSynchronize(c->stream));
    return UCG_OK;
}

// f(y) for the state currently in st.y into st.k[0]
int rk_odefun(ucg_ctx *c)
{
    Ctl *h = c->ctl_host;
    UCG_CUDA(cudaMemcpyAsync(h, c->ctl, sizeof(Ctl), cudaMemcpyDeviceToHost, c->stream));
    UCG_CUDA(cudaStreamSynchronize(c->stream));
    h->active = 1;
    h->status = 0;
    h->need_stage1 = 1;
    h->pending = 0;
    h->vmax = 0.0;
    h->nonfinite = 0;
    h->ticket = 0;
    UCG_CUDA(cudaMemcpyAsync(c->ctl, h, sizeof(Ctl), cudaMemcpyHostToDevice, c->stream));
    UCG_CUDA(rk_enqueue_begin(c));
    UCG_CUDA(enqueue_stage(c, 1, 0));
    UCG_CUDA(cudaGetLastError());
    UCG_CUDA(cudaMemcpyAsync(h, c->ctl, sizeof(Ctl), cudaMemcpyDeviceToHost, c->stream));
    UCG_CUDA(cudaStreamSynchronize(c->stream));
    if (h->status) return h->status;
    return h->nonfinite ? UCG_E_NONFINITE : UCG_OK;
}

// fault injection for the tests of the bounded waits
int rk_test_wait_timeout(ucg_ctx *c, unsigned long long wait_ns, int hold)
{
    Ctl *h = c->ctl_host;
    UCG_CUDA(cudaMemcpyAsync(h, c->ctl, sizeof(Ctl), cudaMemcpyDeviceToHost, c->stream));
    UCG_CUDA(cudaStreamSynchronize(c->stream));
    h->wait_ns = wait_ns;
    h->test_hold = hold;
    h->status = 0;
    UCG_CUDA(cudaMemcpyAsync(c->ctl, h, sizeof(Ctl), cudaMemcpyHostToDevice, c->stream));
    UCG_CUDA(cudaStreamSynchronize(c->stream));
    return UCG_OK;
}

// ---- allocation-free right-hand side --------------------------------------------
//
// ucg_odefun_noalloc evaluates dydt = f(y) for a fault model whose matrix, state,
// friction parameters and output all live in caller-owned device memory, for
// callers that cannot allocate device memory at the point of the call (code
// running under an external memory manager or an allocation-free real-time
// loop, which must not call cudaMalloc or pull in an allocating library).  The
// only working storage it needs -- the source velocity vector v and the control
// block the kernels read -- lives in the fixed array below.  The array is part
// of the loaded library: every GPU that loads libucg.so holds its 8 MB until
// the process exits.  Calls share it, so calls that overlap on the GPU (on
// different streams without ordering) race on v; the array keeps the last
// call's contents, and the control block is reset at the start of every call.

namespace {

constexpr long NOALLOC_MAX_N = 1L << 20;                // source DOFs (2 per patch)
constexpr long NOALLOC_CTL_DOUBLES = (sizeof(Ctl) + sizeof(double) - 1) / sizeof(double);

static __device__ __align__(256) double g_noalloc_scratch[NOALLOC_MAX_N + NOALLOC_CTL_DOUBLES];

__global__ void k_noalloc_ctl_reset(Ctl *ctl)
{
    Ctl z;
    memset(&z, 0, sizeof z);
    z.active = 1;
    z.need_stage1 = 1;
    z.step_target = 1;
    z.t_end = 1.0e300;
    *ctl = z;
}

// the call's outcome into the caller's status word, after the other kernels:
// a wait that gave up (UCG_E_TIMEOUT), a NaN/Inf met on the way, or UCG_OK
__global__ void k_noalloc_status(const Ctl *ctl, int *status)
{
    *status = ctl->status ? ctl->status : (ctl->nonfinite ? UCG_E_NONFINITE : UCG_OK);
}

inline bool aligned_to(const void *p, uintptr_t a) { return (reinterpret_cast<uintptr_t>(p) & (a - 1)) == 0; }

}  // namespace

}  // namespace ucg

extern "C" int ucg_odefun_noalloc(const double *K, long n, long m, int np, const double *y,
                                  const double *Vpl_cos_rake, const double *Vpl_sin_rake,
                                  const double *a, const double *b, const double *sig, const double *L,
                                  const double *damping, double *dydt, void *stream, int *status)
{
    using namespace ucg;
    const double *dp[] = {y, dydt, Vpl_cos_rake, Vpl_sin_rake, a, b, sig, L, damping};
    if (!K) return UCG_E_BADARG;
    for (const double *p : dp)
        if (!p || !aligned_to(p, sizeof(double))) return UCG_E_BADARG;
    // K's rows go to shared memory by bulk copies, whose source must sit on a
    // 16-byte boundary (n is even, so every row then does)
    if (!aligned_to(K, 16)) return UCG_E_BADARG;
    if (status && !aligned_to(status, sizeof(int))) return UCG_E_BADARG;
    if (np <= 0 || n != 2L * np || m != 3L * np) return UCG_E_BADARG;
    if (n > NOALLOC_MAX_N) return UCG_E_BADARG;   // beyond the fixed scratch: 2^20 source DOFs
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return UCG_E_NODEVICE;
    // the host-side name of the array is not a device address: resolve it on
    // every call with the calling device current (no allocation; the first call
    // on a device may load the module)
    void *p = nullptr;
    if (cudaGetSymbolAddress(&p, g_noalloc_scratch) != cudaSuccess || !p) return UCG_E_CUDA;
    double *v = static_cast<double *>(p);
    Ctl *ctl = reinterpret_cast<Ctl *>(v + NOALLOC_MAX_N);
    cudaStream_t st = static_cast<cudaStream_t>(stream);

    StageArgs sa{};
    sa.y = const_cast<double *>(y);   // stage 1 without a pending candidate reads y only
    sa.ys = sa.y;
    sa.ks = dydt;
    sa.v = v;
    sa.fr.vpl_c = const_cast<double *>(Vpl_cos_rake);
    sa.fr.vpl_s = const_cast<double *>(Vpl_sin_rake);
    sa.fr.a = const_cast<double *>(a);
    sa.fr.b = const_cast<double *>(b);
    sa.fr.sig = const_cast<double *>(sig);
    sa.fr.L = const_cast<double *>(L);
    sa.fr.damping = const_cast<double *>(damping);
    sa.np = np;
    sa.nvol = 0;
    sa.len = 7L * np;

    int dcount = 0;
    if (cudaDeviceGetAttribute(&dcount, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || dcount <= 0)
        return UCG_E_CUDA;
    const int grid = np < dcount ? np : dcount;
    const size_t smem = tm_smem_bytes<double>();
    auto kfn = k_traction<double>;
    if (cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
        return UCG_E_CUDA;
    k_noalloc_ctl_reset<<<1, 1, 0, st>>>(ctl);
    k_begin<<<(np + 127) / 128, 128, 0, st>>>(sa, ctl, v);
    kfn<<<grid, TM_THREADS, smem, st>>>(1, K, n, n, nullptr, sa, ctl);
    if (status) k_noalloc_status<<<1, 1, 0, st>>>(ctl, status);
    return cudaGetLastError() == cudaSuccess ? UCG_OK : UCG_E_CUDA;
}
