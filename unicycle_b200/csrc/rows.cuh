// The rows of K that one receiver takes from a stress tensor: the 3 tractions
// (ts, td, tn) of a patch or the 6 stresses (s11, s12, s13, s22, s23, s33 in the
// element's frame) of a volume.  The stress and the receiver's unit vectors along
// strike, dip and normal may be given in any one frame.
#pragma once
#include <cuda_runtime.h>

namespace ucg {

template <int NR>
__device__ __forceinline__ void receiver_rows(const double vs[3], const double vd[3], const double vn[3], double sxx,
                                        double sxy, double sxz, double syy, double syz, double szz, double o[NR])
{
    const double t0 = sxx * vn[0] + sxy * vn[1] + sxz * vn[2];
    const double t1 = sxy * vn[0] + syy * vn[1] + syz * vn[2];
    const double t2 = sxz * vn[0] + syz * vn[1] + szz * vn[2];
    if (NR == 3) {
        // okada92.f90:390-398
        o[0] = t0 * vs[0] + t1 * vs[1] + t2 * vs[2];
        o[1] = t0 * vd[0] + t1 * vd[1] + t2 * vd[2];
        o[2] = t0 * vn[0] + t1 * vn[1] + t2 * vn[2];
    } else {
        // okada92.f90:445-462 (the third axis is the dip vector negated)
        const double a0 = sxx * vs[0] + sxy * vs[1] + sxz * vs[2];
        const double a1 = sxy * vs[0] + syy * vs[1] + syz * vs[2];
        const double a2 = sxz * vs[0] + syz * vs[1] + szz * vs[2];
        const double b0 = sxx * vd[0] + sxy * vd[1] + sxz * vd[2];
        const double b1 = sxy * vd[0] + syy * vd[1] + syz * vd[2];
        const double b2 = sxz * vd[0] + syz * vd[1] + szz * vd[2];
        o[0] = a0 * vs[0] + a1 * vs[1] + a2 * vs[2];
        o[1] = t0 * vs[0] + t1 * vs[1] + t2 * vs[2];
        o[2 % NR] = -(b0 * vs[0] + b1 * vs[1] + b2 * vs[2]);
        o[3 % NR] = t0 * vn[0] + t1 * vn[1] + t2 * vn[2];
        o[4 % NR] = -(t0 * vd[0] + t1 * vd[1] + t2 * vd[2]);
        o[5 % NR] = b0 * vd[0] + b1 * vd[1] + b2 * vd[2];
    }
}

}  // namespace ucg
