// Generated by gen_obc_series.py; do not edit.
//
// FP64 polynomials of the energy path: the OBC far-field series V(u) on the
// value tiers of pb2_obc_series.cuh, and 2^-g on [-1/2, 1/2].  In exact
// arithmetic each is within 3.2e-16 relative of its function.
#pragma once

namespace pb2 {

template <int TIER>
struct ObcPoly64;

// V(u), u <= 0.0075: 6 terms, relative error 1.9e-16
template <>
struct ObcPoly64<0> {
  __device__ __forceinline__ static double eval(double u) {
  double p = 0.4721890744691199;
  p = fma(p, u, 0.4544551766836329);
  p = fma(p, u, 0.4444447962803791);
  p = fma(p, u, 0.4285714279522711);
  p = fma(p, u, 0.40000000000039826);
  p = fma(p, u, 0.3333333333333333);
  return p;
  }
};

// V(u), u <= 0.036: 8 terms, relative error 2.2e-16
template <>
struct ObcPoly64<1> {
  __device__ __forceinline__ static double eval(double u) {
  double p = 0.5450756274331202;
  p = fma(p, u, 0.46218471591939103);
  p = fma(p, u, 0.46167686051756734);
  p = fma(p, u, 0.454543100921073);
  p = fma(p, u, 0.4444444661135055);
  p = fma(p, u, 0.4285714284736442);
  p = fma(p, u, 0.4000000000001679);
  p = fma(p, u, 0.33333333333333326);
  return p;
  }
};

// V(u), u <= 0.089: 10 terms, relative error 2.2e-16
template <>
struct ObcPoly64<2> {
  __device__ __forceinline__ static double eval(double u) {
  double p = 0.7562977366004668;
  p = fma(p, u, 0.41608176115407697);
  p = fma(p, u, 0.4768711224707585);
  p = fma(p, u, 0.4662595213072118);
  p = fma(p, u, 0.4615546502723991);
  p = fma(p, u, 0.45454506468454803);
  p = fma(p, u, 0.4444444498187205);
  p = fma(p, u, 0.4285714285339005);
  p = fma(p, u, 0.40000000000010144);
  p = fma(p, u, 0.3333333333333333);
  return p;
  }
};

// V(u), u <= 0.16: 12 terms, relative error 2.1e-16
template <>
struct ObcPoly64<3> {
  __device__ __forceinline__ static double eval(double u) {
  double p = 1.3397247599196342;
  p = fma(p, u, 0.04944419001773069);
  p = fma(p, u, 0.5887244460496047);
  p = fma(p, u, 0.45558504439508096);
  p = fma(p, u, 0.472478012964598);
  p = fma(p, u, 0.46653636681535476);
  p = fma(p, u, 0.4615443366575405);
  p = fma(p, u, 0.45454528739805267);
  p = fma(p, u, 0.4444444472402044);
  p = fma(p, u, 0.4285714285473392);
  p = fma(p, u, 0.40000000000008107);
  p = fma(p, u, 0.3333333333333333);
  return p;
  }
};

// 2^-g, |g| <= 1/2: 11 terms, relative error 3.1e-16
__device__ __forceinline__ double exp2neg_poly(double g) {
  double p = 7.072585949269223e-09;
  p = fma(p, g, -1.0208690299958306e-07);
  p = fma(p, g, 1.321544258792169e-06);
  p = fma(p, g, -1.5252657260200837e-05);
  p = fma(p, g, 0.0001540353044173605);
  p = fma(p, g, -0.0013333558230164974);
  p = fma(p, g, 0.009618129107606888);
  p = fma(p, g, -0.05550410866444772);
  p = fma(p, g, 0.24022650695910097);
  p = fma(p, g, -0.69314718055995);
  p = fma(p, g, 1.0);
  return p;
}

}  // namespace pb2
