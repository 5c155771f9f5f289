"""Writes pb2_obc_series.cuh: minimax polynomials for the OBC far-field series.

In the far field (r - s >= rho~, t = s/r) the OBC descreening integral and its
radial derivative are

    I      =  (t^3 / r)   V(u),  V(u) = sum_{k>=1} k/(2k+1) u^(k-1),
    dI/dr  = -(t^3 / r^2) D(u),  D(u) = sum_{k>=1} 2k(k+1)/(2k+1) u^(k-1),

with u = t^2 (prolix physics/generalized_born.py:211-263 in closed form).
The pair kernels sort tiles into tiers by the largest u any of their pairs
can have, and evaluate V or D there by a polynomial of a few terms.  Instead
of the truncated Taylor series, each tier uses the polynomial of its degree
that minimises the largest RELATIVE error on [0, u_max] (Remez exchange),
which needs far fewer terms for the same bound: 6 terms reach 2e-8 up to
u = 0.16 where the Taylor series needs 10.

The FP64 energy path evaluates V in the same tiers, and 2^-g on
[-1/2, 1/2], in double precision: there each polynomial interpolates at the
Chebyshev nodes of its interval (within a few units of the minimax error at
these degrees), solved in rational arithmetic so that the coefficients carry
no rounding but their own (pb2_series64.cuh).

Run:  python prolix_b200/csrc/gen_obc_series.py   (rewrites both headers)
"""

from __future__ import annotations

import decimal
import math
import os
from fractions import Fraction

import numpy as np

# Tiers: (terms, u_max).  The bound on every tier is a relative error of 2e-8
# in exact arithmetic (a third of a float32 ulp); the last tier of each
# series is the near-tile domain, whose pairs are tested one by one
# against u <= 0.16.
VALUE_TIERS = ((3, 0.0075), (4, 0.036), (5, 0.089), (6, 0.16))
DERIV_TIERS = ((4, 0.027), (5, 0.07), (6, 0.129), (7, 0.16))
REL_BOUND = 2e-8
# FP64: terms of V on each value tier and of 2^-g; the bound is 1.5 ulp
VALUE_TERMS64 = (6, 8, 10, 12)
EXP2_TERMS64 = 11
REL_BOUND64 = 3.2e-16


def exact(u, der: bool, n_terms: int = 300) -> np.ndarray:
  """V(u) or D(u) summed to convergence in FP64 (u <= 0.5)."""
  u = np.asarray(u, np.float64)
  k = np.arange(1, n_terms + 1, dtype=np.float64)[:, None]
  c = 2.0 * k * (k + 1) / (2 * k + 1) if der else k / (2 * k + 1)
  return (c * u[None, :] ** (k - 1)).sum(0)


def remez(u_max: float, n_terms: int, der: bool, iters: int = 40):
  """Coefficients (ascending powers of u) of the relative-error minimax
  polynomial with n_terms terms on [0, u_max], and its error."""
  deg = n_terms - 1
  m = deg + 2
  x = 0.5 * (1.0 - np.cos(np.pi * np.arange(m) / (m - 1)))  # on [0, 1]
  grid = np.linspace(0.0, 1.0, 40001)
  fg = exact(grid * u_max, der)
  coef = None
  err_max = np.inf
  for _ in range(iters):
    f = exact(x * u_max, der)
    a = np.zeros((m, m))
    for j in range(deg + 1):
      a[:, j] = x ** j
    a[:, deg + 1] = (-1.0) ** np.arange(m) * f
    sol = np.linalg.solve(a, f)
    coef = sol[:deg + 1]
    err = (np.polyval(coef[::-1], grid) - fg) / fg
    err_max = float(np.max(np.abs(err)))
    cuts = np.where(np.diff(np.sign(err)) != 0)[0] + 1
    ext = [seg[np.argmax(np.abs(err[seg]))] for seg in np.split(np.arange(grid.size), cuts)]
    if len(ext) < m:
      break
    best = max(range(len(ext) - m + 1), key=lambda s: np.min(np.abs(err[ext[s:s + m]])))
    x = grid[ext[best:best + m]]
  return coef / u_max ** np.arange(deg + 1), err_max


def header() -> str:
  out = [
      "// Generated by gen_obc_series.py; do not edit.",
      "//",
      "// Minimax (relative error) polynomials in u = (s/r)^2 for the OBC far-field",
      "// series V(u) (descreening) and D(u) (its radial derivative), one per tier",
      "// of tiles sorted by the largest u of their pairs.  In exact arithmetic each",
      f"// is within {REL_BOUND:.0e} relative of the full series on its tier.",
      "#pragma once",
      "",
      "namespace pb2 {",
      "",
  ]
  for name, tiers in (("Value", VALUE_TIERS), ("Deriv", DERIV_TIERS)):
    us = ", ".join(f"{u!r}" for _, u in tiers)
    ks = ", ".join(str(k) for k, _ in tiers)
    out.append(f"constexpr double k{name}TierU[4] = {{{us}}};  // u_max of each tier")
    out.append(f"constexpr int k{name}TierTerms[4] = {{{ks}}};")
  out += ["", "template <bool DER, int TIER>", "struct ObcPoly;", ""]
  for der, tiers in ((False, VALUE_TIERS), (True, DERIV_TIERS)):
    for tier, (k, u_max) in enumerate(tiers):
      coef, err = remez(u_max, k, der)
      if err > REL_BOUND:
        raise SystemExit(f"tier {tier} ({'D' if der else 'V'}): {err:.3e} > {REL_BOUND}")
      c32 = [float(np.float32(c)) for c in coef]
      out.append(f"// {'D' if der else 'V'}(u), u <= {u_max}: {k} terms, relative error {err:.2e}")
      out.append("template <>")
      out.append(f"struct ObcPoly<{'true' if der else 'false'}, {tier}> {{")
      out.append(f"  static constexpr int kTerms = {k};")
      out.append("  __device__ __forceinline__ static float2 eval2(float2 u) {")
      out.append(f"    float2 p = make_float2({c32[-1]:.9e}f, {c32[-1]:.9e}f);")
      for c in reversed(c32[:-1]):
        out.append(f"    p = __ffma2_rn(p, u, make_float2({c:.9e}f, {c:.9e}f));")
      out.append("    return p;")
      out.append("  }")
      out.append("};")
      out.append("")
  out.append("}  // namespace pb2")
  return "\n".join(out) + "\n"


def _value_exact(u: Fraction) -> Fraction:
  """V(u) to 1e-30 (u <= 0.16)."""
  return sum(Fraction(k, 2 * k + 1) * u ** (k - 1) for k in range(1, 42))


def _exp2neg_exact(g: Fraction) -> Fraction:
  with decimal.localcontext() as c:
    c.prec = 50
    x = decimal.Decimal(g.numerator) / decimal.Decimal(g.denominator)
    return Fraction((-x * decimal.Decimal(2).ln()).exp())


def interpolant(f, lo: float, hi: float, n_terms: int):
  """Coefficients (ascending powers, as FP64) of the polynomial through f at
  the n_terms Chebyshev nodes of [lo, hi], and the largest relative error of
  the exact polynomial with the rounded coefficients on a grid."""
  nodes = [Fraction(0.5 * (lo + hi) + 0.5 * (hi - lo) * math.cos(math.pi * (2 * k + 1) / (2 * n_terms)))
           for k in range(n_terms)]
  d = [f(x) for x in nodes]  # divided differences
  for j in range(1, n_terms):
    for k in range(n_terms - 1, j - 1, -1):
      d[k] = (d[k] - d[k - 1]) / (nodes[k] - nodes[k - j])
  c = [Fraction(0)] * n_terms  # Newton form to powers
  for k in range(n_terms - 1, -1, -1):
    c = [d[k] - nodes[k] * c[0]] + [c[j - 1] - nodes[k] * c[j] for j in range(1, n_terms)]
  c = [float(v) for v in c]
  worst = 0.0
  for t in range(201):
    x = Fraction(lo + (hi - lo) * t / 200)
    p = Fraction(0)
    for v in reversed(c):
      p = p * x + Fraction(v)
    y = f(x)
    worst = max(worst, abs(float((p - y) / y)))
  return c, worst


def header64() -> str:
  out = [
      "// Generated by gen_obc_series.py; do not edit.",
      "//",
      "// FP64 polynomials of the energy path: the OBC far-field series V(u) on the",
      "// value tiers of pb2_obc_series.cuh, and 2^-g on [-1/2, 1/2].  In exact",
      f"// arithmetic each is within {REL_BOUND64:.1e} relative of its function.",
      "#pragma once",
      "",
      "namespace pb2 {",
      "",
      "template <int TIER>",
      "struct ObcPoly64;",
      "",
  ]

  def body(arg, coef):
    out.append(f"  double p = {coef[-1]!r};")
    for c in reversed(coef[:-1]):
      out.append(f"  p = fma(p, {arg}, {c!r});")
    out.append("  return p;")

  for tier, ((_, u_max), n) in enumerate(zip(VALUE_TIERS, VALUE_TERMS64)):
    coef, err = interpolant(_value_exact, 0.0, u_max, n)
    if err > REL_BOUND64:
      raise SystemExit(f"FP64 tier {tier}: {err:.3e} > {REL_BOUND64}")
    out.append(f"// V(u), u <= {u_max}: {n} terms, relative error {err:.1e}")
    out += ["template <>", f"struct ObcPoly64<{tier}> {{", "  __device__ __forceinline__ static double eval(double u) {"]
    body("u", coef)
    out += ["  }", "};", ""]
  coef, err = interpolant(_exp2neg_exact, -0.5, 0.5, EXP2_TERMS64)
  if err > REL_BOUND64:
    raise SystemExit(f"FP64 2^-g: {err:.3e} > {REL_BOUND64}")
  out.append(f"// 2^-g, |g| <= 1/2: {EXP2_TERMS64} terms, relative error {err:.1e}")
  out.append("__device__ __forceinline__ double exp2neg_poly(double g) {")
  body("g", coef)
  out += ["}", "", "}  // namespace pb2"]
  return "\n".join(out) + "\n"


if __name__ == "__main__":
  for name, text in (("pb2_obc_series.cuh", header), ("pb2_series64.cuh", header64)):
    path = os.path.join(os.path.dirname(os.path.abspath(__file__)), name)
    with open(path, "w") as f:
      f.write(text())
    print("wrote", path)
