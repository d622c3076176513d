// uns_tan.cuh -- forward-mode tangent numbers for the discrete adjoint.
//
// Tan carries a value and one directional derivative.  The physics functions
// of uns_phys.cuh are templates on their arithmetic type, so instantiating
// them on Tan and seeding one input direction at a time gives one column of
// their exact local Jacobian (no finite-difference step).  Branches
// (comparisons, fabs, the min/max of the limiter and the fluxes) follow the
// value, so the Jacobian is the one of the branch the forward pass took.
#pragma once
#include <cuda_runtime.h>

#include <cmath>

#include "uns_fp64.cuh"

namespace uns {
// A namespace of its own, so that sqrt/fabs/pow of Tan are found only by
// argument-dependent lookup and never hide ::sqrt for doubles in namespace uns.
namespace ad {

struct Tan {
    double v, d;
    __host__ __device__ Tan() : v(0.0), d(0.0) {}
    __host__ __device__ Tan(double x) : v(x), d(0.0) {}
    __host__ __device__ Tan(double x, double dx) : v(x), d(dx) {}
};

// (Register FMAs and divisions on the integer pipe: the IEEE results,
// uns_fp64.cuh.  Not its products: a seed's derivatives are mostly zero, which
// the integer route hands to a call.)
typedef F64 N;
__device__ __forceinline__ Tan operator+(Tan a, Tan b) { return Tan((N(a.v) + b.v).v, (N(a.d) + b.d).v); }
__device__ __forceinline__ Tan operator-(Tan a, Tan b) { return Tan((N(a.v) - b.v).v, (N(a.d) - b.d).v); }
__device__ __forceinline__ Tan operator-(Tan a) { return Tan(neg64(a.v), neg64(a.d)); }
__device__ __forceinline__ Tan operator*(Tan a, Tan b) {
    return Tan((N(a.v) * b.v).v, (N(a.d) * b.v + N(a.v) * b.d).v);
}
__device__ __forceinline__ Tan operator/(Tan a, Tan b) {
    const N q = N(a.v) / b.v;
    return Tan(q.v, ((N(a.d) - q * b.d) / b.v).v);
}
__device__ __forceinline__ Tan operator+(Tan a, double b) { return Tan((N(a.v) + b).v, a.d); }
__device__ __forceinline__ Tan operator+(double a, Tan b) { return Tan((N(a) + b.v).v, b.d); }
__device__ __forceinline__ Tan operator-(Tan a, double b) { return Tan((N(a.v) - b).v, a.d); }
__device__ __forceinline__ Tan operator-(double a, Tan b) { return Tan((N(a) - b.v).v, neg64(b.d)); }
__device__ __forceinline__ Tan operator*(Tan a, double b) { return Tan((N(a.v) * b).v, (N(a.d) * b).v); }
__device__ __forceinline__ Tan operator*(double a, Tan b) { return Tan((N(a) * b.v).v, (N(a) * b.d).v); }
__device__ __forceinline__ Tan operator/(Tan a, double b) { return Tan((N(a.v) / b).v, (N(a.d) / b).v); }
__device__ __forceinline__ Tan operator/(double a, Tan b) {
    const N q = N(a) / b.v;
    return Tan(q.v, (-q * b.d / b.v).v);
}
__device__ __forceinline__ Tan& operator+=(Tan& a, Tan b) { a = a + b; return a; }
__device__ __forceinline__ Tan& operator-=(Tan& a, Tan b) { a = a - b; return a; }
__device__ __forceinline__ Tan& operator*=(Tan& a, Tan b) { a = a * b; return a; }

__host__ __device__ __forceinline__ bool operator<(Tan a, Tan b) { return a.v < b.v; }
__host__ __device__ __forceinline__ bool operator>(Tan a, Tan b) { return a.v > b.v; }
__host__ __device__ __forceinline__ bool operator<=(Tan a, Tan b) { return a.v <= b.v; }
__host__ __device__ __forceinline__ bool operator>=(Tan a, Tan b) { return a.v >= b.v; }

__device__ __forceinline__ Tan sqrt(Tan a) {
    const double r = sqrt_digits(a.v);
    return Tan(r, (N(a.d) / (N(2.0) * r)).v);
}
__device__ __forceinline__ Tan fabs(Tan a) { return a.v < 0.0 ? -a : a; }
// a^b for a > 0: d(a^b) = a^b (b' ln a + b a'/a).
__host__ __device__ __forceinline__ Tan pow(Tan a, Tan b) {
    double p = ::pow(a.v, b.v);
    double dd = b.v * a.d / a.v;
    if (b.d != 0.0) dd = dd + b.d * ::log(a.v);
    return Tan(p, p * dd);
}
__host__ __device__ __forceinline__ Tan pow(Tan a, double b) {
    double p = ::pow(a.v, b);
    return Tan(p, p * b * a.d / a.v);
}

}  // namespace ad
using ad::Tan;

// Value of a double or a Tan, for the few places that need the plain number.
__host__ __device__ __forceinline__ double val(double x) { return x; }
__host__ __device__ __forceinline__ double val(Tan x) { return x.v; }
__host__ __device__ __forceinline__ double der(Tan x) { return x.d; }

}  // namespace uns
