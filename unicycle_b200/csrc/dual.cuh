// Forward-mode dual numbers for device code: a value and its gradient with
// respect to the three observation coordinates.  Evaluating a closed-form
// displacement field on these yields its exact displacement gradient (to
// rounding), from which strain and stress follow.
#pragma once
#include <cuda_runtime.h>

namespace ucg {

struct Dd {
    double v, x, y, z;
    Dd() = default;
    __host__ __device__ constexpr Dd(double c) : v(c), x(0.0), y(0.0), z(0.0) {}
    __host__ __device__ constexpr Dd(double c, double a, double b, double e) : v(c), x(a), y(b), z(e) {}
};

__device__ __forceinline__ Dd dd(double c) { return Dd{c, 0.0, 0.0, 0.0}; }
__device__ __forceinline__ Dd operator+(Dd a, Dd b) { return Dd{a.v + b.v, a.x + b.x, a.y + b.y, a.z + b.z}; }
__device__ __forceinline__ Dd operator-(Dd a, Dd b) { return Dd{a.v - b.v, a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ __forceinline__ Dd operator-(Dd a) { return Dd{-a.v, -a.x, -a.y, -a.z}; }
__device__ __forceinline__ Dd operator*(Dd a, Dd b)
{
    return Dd{a.v * b.v, a.x * b.v + a.v * b.x, a.y * b.v + a.v * b.y, a.z * b.v + a.v * b.z};
}
__device__ __forceinline__ Dd operator+(Dd a, double c) { return Dd{a.v + c, a.x, a.y, a.z}; }
__device__ __forceinline__ Dd operator+(double c, Dd a) { return Dd{a.v + c, a.x, a.y, a.z}; }
__device__ __forceinline__ Dd operator-(Dd a, double c) { return Dd{a.v - c, a.x, a.y, a.z}; }
__device__ __forceinline__ Dd operator-(double c, Dd a) { return Dd{c - a.v, -a.x, -a.y, -a.z}; }
__device__ __forceinline__ Dd operator*(Dd a, double c) { return Dd{a.v * c, a.x * c, a.y * c, a.z * c}; }
__device__ __forceinline__ Dd operator*(double c, Dd a) { return Dd{a.v * c, a.x * c, a.y * c, a.z * c}; }
// Plain value: closed forms written for any scalar type, evaluated for the
// displacement itself (observation-point displacements).
struct Dv {
    double v;
    Dv() = default;
    __host__ __device__ constexpr Dv(double c) : v(c) {}
};
__device__ __forceinline__ Dv operator+(Dv a, Dv b) { return Dv{a.v + b.v}; }
__device__ __forceinline__ Dv operator-(Dv a, Dv b) { return Dv{a.v - b.v}; }
__device__ __forceinline__ Dv operator-(Dv a) { return Dv{-a.v}; }
__device__ __forceinline__ Dv operator*(Dv a, Dv b) { return Dv{a.v * b.v}; }
__device__ __forceinline__ Dv operator+(Dv a, double c) { return Dv{a.v + c}; }
__device__ __forceinline__ Dv operator+(double c, Dv a) { return Dv{c + a.v}; }
__device__ __forceinline__ Dv operator-(Dv a, double c) { return Dv{a.v - c}; }
__device__ __forceinline__ Dv operator-(double c, Dv a) { return Dv{c - a.v}; }
__device__ __forceinline__ Dv operator*(Dv a, double c) { return Dv{a.v * c}; }
__device__ __forceinline__ Dv operator*(double c, Dv a) { return Dv{c * a.v}; }
__device__ __forceinline__ Dv rcp(Dv a) { return Dv{1.0 / a.v}; }
__device__ __forceinline__ Dv operator/(Dv a, Dv b) { return Dv{a.v / b.v}; }
__device__ __forceinline__ Dv operator/(Dv a, double c) { return Dv{a.v / c}; }
__device__ __forceinline__ Dv operator/(double c, Dv a) { return Dv{c / a.v}; }
__device__ __forceinline__ Dv dsqrt(Dv a) { return Dv{sqrt(a.v)}; }
__device__ __forceinline__ Dv datan2_g(Dv y, Dv x) { return Dv{atan2(y.v, x.v)}; }

// the square root and its reciprocal, the logarithm, and the arctangent of the
// quotient as written (not atan2: the value keeps the closed form's branch)
__device__ __forceinline__ void dsqrt_inv(Dv a, Dv &s, Dv &is)
{
    s = Dv{sqrt(a.v)};
    is = Dv{1.0 / s.v};
}
__device__ __forceinline__ Dv dlog_gi(Dv a, Dv) { return Dv{log(a.v)}; }
__device__ __forceinline__ Dv datan_q_g(Dv n, Dv d) { return Dv{atan(n.v / d.v)}; }

}  // namespace ucg
