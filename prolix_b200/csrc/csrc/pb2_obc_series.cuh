// Generated by gen_obc_series.py; do not edit.
//
// Minimax (relative error) polynomials in u = (s/r)^2 for the OBC far-field
// series V(u) (descreening) and D(u) (its radial derivative), one per tier
// of tiles sorted by the largest u of their pairs.  In exact arithmetic each
// is within 2e-08 relative of the full series on its tier.
#pragma once

namespace pb2 {

constexpr double kValueTierU[4] = {0.0075, 0.036, 0.089, 0.16};  // u_max of each tier
constexpr int kValueTierTerms[4] = {3, 4, 5, 6};
constexpr double kDerivTierU[4] = {0.027, 0.07, 0.129, 0.16};  // u_max of each tier
constexpr int kDerivTierTerms[4] = {4, 5, 6, 7};

template <bool DER, int TIER>
struct ObcPoly;

// V(u), u <= 0.0075: 3 terms, relative error 1.78e-08
template <>
struct ObcPoly<false, 0> {
  static constexpr int kTerms = 3;
  __device__ __forceinline__ static float2 eval2(float2 u) {
    float2 p = make_float2(4.336143434e-01f, 4.336143434e-01f);
    p = __ffma2_rn(p, u, make_float2(3.999857903e-01f, 3.999857903e-01f));
    p = __ffma2_rn(p, u, make_float2(3.333333433e-01f, 3.333333433e-01f));
    return p;
  }
};

// V(u), u <= 0.036: 4 terms, relative error 1.92e-08
template <>
struct ObcPoly<false, 1> {
  static constexpr int kTerms = 4;
  __device__ __forceinline__ static float2 eval2(float2 u) {
    float2 p = make_float2(4.788752198e-01f, 4.788752198e-01f);
    p = __ffma2_rn(p, u, make_float2(4.277850091e-01f, 4.277850091e-01f));
    p = __ffma2_rn(p, u, make_float2(4.000056982e-01f, 4.000056982e-01f));
    p = __ffma2_rn(p, u, make_float2(3.333333135e-01f, 3.333333135e-01f));
    return p;
  }
};

// V(u), u <= 0.089: 5 terms, relative error 1.89e-08
template <>
struct ObcPoly<false, 2> {
  static constexpr int kTerms = 5;
  __device__ __forceinline__ static float2 eval2(float2 u) {
    float2 p = make_float2(5.741708279e-01f, 5.741708279e-01f);
    p = __ffma2_rn(p, u, make_float2(4.346917272e-01f, 4.346917272e-01f));
    p = __ffma2_rn(p, u, make_float2(4.288875163e-01f, 4.288875163e-01f));
    p = __ffma2_rn(p, u, make_float2(3.999964595e-01f, 3.999964595e-01f));
    p = __ffma2_rn(p, u, make_float2(3.333333433e-01f, 3.333333433e-01f));
    return p;
  }
};

// V(u), u <= 0.16: 6 terms, relative error 1.89e-08
template <>
struct ObcPoly<false, 3> {
  static constexpr int kTerms = 6;
  __device__ __forceinline__ static float2 eval2(float2 u) {
    float2 p = make_float2(7.736505270e-01f, 7.736505270e-01f);
    p = __ffma2_rn(p, u, make_float2(3.926562965e-01f, 3.926562965e-01f));
    p = __ffma2_rn(p, u, make_float2(4.498088360e-01f, 4.498088360e-01f));
    p = __ffma2_rn(p, u, make_float2(4.283659160e-01f, 4.283659160e-01f));
    p = __ffma2_rn(p, u, make_float2(4.000028372e-01f, 4.000028372e-01f));
    p = __ffma2_rn(p, u, make_float2(3.333333135e-01f, 3.333333135e-01f));
    return p;
  }
};

// D(u), u <= 0.027: 4 terms, relative error 1.80e-08
template <>
struct ObcPoly<true, 0> {
  static constexpr int kTerms = 4;
  __device__ __forceinline__ static float2 eval2(float2 u) {
    float2 p = make_float2(4.752100945e+00f, 4.752100945e+00f);
    p = __ffma2_rn(p, u, make_float2(3.423316240e+00f, 3.423316240e+00f));
    p = __ffma2_rn(p, u, make_float2(2.400028467e+00f, 2.400028467e+00f));
    p = __ffma2_rn(p, u, make_float2(1.333333254e+00f, 1.333333254e+00f));
    return p;
  }
};

// D(u), u <= 0.07: 5 terms, relative error 1.91e-08
template <>
struct ObcPoly<true, 1> {
  static constexpr int kTerms = 5;
  __device__ __forceinline__ static float2 eval2(float2 u) {
    float2 p = make_float2(6.748081684e+00f, 6.748081684e+00f);
    p = __ffma2_rn(p, u, make_float2(4.362066746e+00f, 4.362066746e+00f));
    p = __ffma2_rn(p, u, make_float2(3.430661440e+00f, 3.430661440e+00f));
    p = __ffma2_rn(p, u, make_float2(2.399981737e+00f, 2.399981737e+00f));
    p = __ffma2_rn(p, u, make_float2(1.333333373e+00f, 1.333333373e+00f));
    return p;
  }
};

// D(u), u <= 0.129: 6 terms, relative error 1.91e-08
template <>
struct ObcPoly<true, 2> {
  static constexpr int kTerms = 6;
  __device__ __forceinline__ static float2 eval2(float2 u) {
    float2 p = make_float2(1.033754539e+01f, 1.033754539e+01f);
    p = __ffma2_rn(p, u, make_float2(4.842800617e+00f, 4.842800617e+00f));
    p = __ffma2_rn(p, u, make_float2(4.486836910e+00f, 4.486836910e+00f));
    p = __ffma2_rn(p, u, make_float2(3.427271605e+00f, 3.427271605e+00f));
    p = __ffma2_rn(p, u, make_float2(2.400014400e+00f, 2.400014400e+00f));
    p = __ffma2_rn(p, u, make_float2(1.333333254e+00f, 1.333333254e+00f));
    return p;
  }
};

// D(u), u <= 0.16: 7 terms, relative error 3.82e-09
template <>
struct ObcPoly<true, 3> {
  static constexpr int kTerms = 7;
  __device__ __forceinline__ static float2 eval2(float2 u) {
    float2 p = make_float2(1.468234348e+01f, 1.468234348e+01f);
    p = __ffma2_rn(p, u, make_float2(4.675673962e+00f, 4.675673962e+00f));
    p = __ffma2_rn(p, u, make_float2(5.659827709e+00f, 5.659827709e+00f));
    p = __ffma2_rn(p, u, make_float2(4.432657719e+00f, 4.432657719e+00f));
    p = __ffma2_rn(p, u, make_float2(3.428888798e+00f, 3.428888798e+00f));
    p = __ffma2_rn(p, u, make_float2(2.399996758e+00f, 2.399996758e+00f));
    p = __ffma2_rn(p, u, make_float2(1.333333373e+00f, 1.333333373e+00f));
    return p;
  }
};

}  // namespace pb2
