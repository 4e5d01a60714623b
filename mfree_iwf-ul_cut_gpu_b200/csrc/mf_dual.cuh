// Forward-mode dual numbers for the tangent (differentiable) step: a value and one directional
// derivative, with the chain rule of every operation the step uses. The functions the
// reference evaluates in float on double arguments (sqrtf, atan2f, cosf, sinf, fmaxf) keep
// that value here; their derivative is the one of the exact function (the float rounding is
// piecewise constant and has none).
#pragma once

#include <cmath>

namespace mf {

struct __align__(16) dual {
  double v, d;
};

__host__ __device__ __forceinline__ dual dconst(double v) { return dual{v, 0.}; }

// r = f(x): value f, derivative scale fp
__device__ __forceinline__ dual dchain(double f, double fp, const dual &x) { return dual{f, fp * x.d}; }

__device__ __forceinline__ dual operator+(const dual &a, const dual &b) { return dual{a.v + b.v, a.d + b.d}; }
__device__ __forceinline__ dual operator-(const dual &a, const dual &b) { return dual{a.v - b.v, a.d - b.d}; }
__device__ __forceinline__ dual operator*(const dual &a, const dual &b) {
  return dual{a.v * b.v, a.d * b.v + a.v * b.d};
}
__device__ __forceinline__ dual operator/(const dual &a, const dual &b) {
  return dual{a.v / b.v, (a.d * b.v - a.v * b.d) / (b.v * b.v)};
}
__device__ __forceinline__ dual operator-(const dual &a) { return dual{-a.v, -a.d}; }
__device__ __forceinline__ dual operator+(const dual &a, double b) { return dual{a.v + b, a.d}; }
__device__ __forceinline__ dual operator+(double a, const dual &b) { return dual{a + b.v, b.d}; }
__device__ __forceinline__ dual operator-(const dual &a, double b) { return dual{a.v - b, a.d}; }
__device__ __forceinline__ dual operator-(double a, const dual &b) { return dual{a - b.v, -b.d}; }
__device__ __forceinline__ dual operator*(const dual &a, double b) { return dual{a.v * b, a.d * b}; }
__device__ __forceinline__ dual operator*(double a, const dual &b) { return dual{a * b.v, a * b.d}; }
__device__ __forceinline__ dual operator/(const dual &a, double b) { return dual{a.v / b, a.d / b}; }
__device__ __forceinline__ dual operator/(double a, const dual &b) {
  return dual{a / b.v, -(a * b.d) / (b.v * b.v)};
}
__device__ __forceinline__ dual &operator+=(dual &a, const dual &b) { return a = a + b; }
__device__ __forceinline__ dual &operator+=(dual &a, double b) {
  a.v += b;
  return a;
}

__device__ __forceinline__ dual dsqrt(const dual &x) {
  const double s = sqrt(x.v);
  return dchain(s, s > 0. ? 0.5 / s : 0., x);
}

// (double)sqrtf((float)x): the reference's float-rounded root
__device__ __forceinline__ dual dsqrtf_narrow(const dual &x) {
  const double s = (double)sqrtf((float)x.v);
  const double se = sqrt(x.v);
  return dchain(s, se > 0. ? 0.5 / se : 0., x);
}

__device__ __forceinline__ dual dlog(const dual &x) { return dchain(log(x.v), 1. / x.v, x); }

// x^y with both operands carrying derivatives: d = x^y (y' ln x + y x'/x); at x = 0 the
// value is pow's and the derivative is taken as 0 (the limit of the y' term for y > 0)
__device__ __forceinline__ dual dpow(const dual &x, const dual &y) {
  dual r = dconst(pow(x.v, y.v));
  if (x.v > 0.) {  // (a direction carries one parameter: most exponents and many bases have no derivative)
    double s = 0.;
    if (y.d != 0.) s = y.d * log(x.v);
    if (x.d != 0.) s += y.v * x.d / x.v;
    r.d = r.v * s;
  }
  return r;
}

__device__ __forceinline__ dual dfmax0(const dual &x) {  // fmax(x, 0)
  return x.v > 0. ? x : dconst(fmax(x.v, 0.));
}

// (double)atan2f((float)y, (float)x)
__device__ __forceinline__ dual datan2f_narrow(const dual &y, const dual &x) {
  const double den = x.v * x.v + y.v * y.v;
  return dual{(double)atan2f((float)y.v, (float)x.v), den > 0. ? (x.v * y.d - y.v * x.d) / den : 0.};
}

__device__ __forceinline__ dual dcosf_narrow(const dual &x) { return dchain((double)cosf((float)x.v), -sin(x.v), x); }
__device__ __forceinline__ dual dsinf_narrow(const dual &x) { return dchain((double)sinf((float)x.v), cos(x.v), x); }

}  // namespace mf
