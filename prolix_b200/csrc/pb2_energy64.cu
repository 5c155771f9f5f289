// FP64 energy evaluation (energy reporting, NVE drift checks; never part of
// an MD step, which needs forces only).
//
// Float32 coordinates bound the accuracy of a pair energy: a Lennard-Jones
// term moves by 12 dr/r for a coordinate rounding dr, about 1e-6 relative in
// a 20 A system, so per-term energies to 1e-6 need FP64 distances.  These
// kernels read the FP64 state and evaluate the same formulas as the force
// kernels in double:
//   born   : descreening sums (prolix physics/generalized_born.py:211-263);
//   energy : GB polar pair terms, Coulomb and LJ energies
//            (generalized_born.py:118-208, physics/optimization.py:21-297).
// The Born radii of this path come from its own FP64 sums (finalize64).
//
// Mapping: as in the force kernels, one warp per work item (system, i-blocks
// ib and ib + 1, range of j-blocks), lane l owning one atom of each i-block
// and meeting j-atom (l + k) mod 32 at step k; the j-block sits in shared
// memory (field-major, so a field's 32 reads are conflict-free) and serves
// both i atoms.  What bounds it is the FP64 pipe (16 lanes per SM quarter: a
// warp instruction takes two cycles), so the work is in its instruction
// count:
//  * descreening of tiles far enough apart (the force kernels' tiers by box
//    distance) by the far-field series in FP64, about 28 FP64 instructions
//    per pair for both directions, against two logarithms and a dozen
//    divisions of the closed form;
//  * pairs of near tiles outside the series' domain (about 1.3 %) go to a
//    queue in shared memory and take the closed form one pair per lane
//    (in place, one such lane made all 32 wait for it at nearly every step);
//  * 1/r^2, 1/r and 1/f from the hardware's 20-bit seeds by one third-order
//    step (Householder), and the exponential as 2^-w by a polynomial: no
//    divisions, and no calls in the loop.
// N = 20,000, all pairs: the two passes 3.85 + 2.19 -> 0.48 + 0.78 ms (the
// FP64 instructions counted above take 0.30 + 0.49 at full rate); N = 166:
// 73 + 47 -> 8.3 + 6.3 us.
#include "pb2_common.cuh"
#include "pb2_kernels.cuh"
#include "pb2_obc_series.cuh"
#include "pb2_pairmath.cuh"
#include "pb2_series64.cuh"

namespace pb2 {

constexpr int kE64Threads = 128;
constexpr int kE64Warps = kE64Threads / 32;
constexpr int kE64Queue = 128;  // queued closed-form pairs per warp (1 KB)
// r^2 at which a masked pair is evaluated: its 1/r^4 (1e-60) vanishes beside
// any descreening sum, and it is never sent to the closed form.
constexpr double kFarR2d = 1e30;

__device__ __forceinline__ double warp_sum_d(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
  return v;
}

__device__ __forceinline__ double obc_integral_d(double r, double rho, double s) {
  if (!(r + s > rho)) return 0.0;
  const double L = fmax(fmax(rho, fabs(r - s)), 1e-4);
  const double U = fmax(r + s, 1e-4);
  const double rs = fmax(r, 1e-4);
  const double il = 1.0 / L, iu = 1.0 / U;
  return 0.5 * (il - iu) + 0.25 * log(L / U) / rs + 0.125 * (r - s * s / rs) * (iu * iu - il * il);
}

// 1/a and 1/sqrt(a) from the hardware's seed (at least 20 bits) by one
// third-order Householder step: the relative error e of the seed becomes
// O(e^3) < 1e-17.  Outside [2^-1000, 2^1000] (zero, infinity, NaN) the seed
// itself is the answer (1/0 = inf, 1/inf = 0).
__device__ __forceinline__ bool mid_range(double a) {  // by the high word: positive, exponent within +-1000
  return (unsigned)(__double2hiint(a) - 0x01700000) < 0x7d000000u;
}
__device__ __forceinline__ double rcp_d(double a) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(a));
  const double e = fma(-a, y, 1.0);
  const double z = fma(y, fma(e, e, e), y);
  return mid_range(a) ? z : y;
}
__device__ __forceinline__ double rsqrt_d(double a) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(a));
  const double e = fma(-(a * y), y, 1.0);
  const double z = fma(y * e, fma(0.375, e, 0.5), y);
  return mid_range(a) ? z : y;
}

// 2^-w: w = n + g with integer n, 2^-g by its polynomial, and n off the
// exponent; zero from w = 1000 on.  SIGNED: w may be negative (one Born radius
// of a pair is, where an atom's radius is below the dielectric offset), and
// from -1000 down the answer is infinity.  A NaN takes any of these: the
// caller's r^2 or Born radii carry it on.
template <bool SIGNED>
__device__ __forceinline__ double exp2neg_d(double w) {
  const double magic = 6755399441055744.0;  // 1.5 * 2^52: rounds to an integer
  const double t = w + magic;
  const double p = exp2neg_poly(w - (t - magic));
  const double v = __hiloint2double(__double2hiint(p) - (__double2loint(t) << 20), __double2loint(p));
  const int hi = __double2hiint(w);
  if (!SIGNED) return (unsigned)hi < 0x408f4000u ? v : 0.0;
  if ((hi & 0x7fffffff) < 0x408f4000) return v;
  return hi < 0 ? __hiloint2double(0x7ff00000, 0) : 0.0;
}

// The warp's closed-form queue: (i, j) batch atom indices.
struct E64Queue {
  int2 *q;
  int n;  // warp-uniform
};

__device__ __forceinline__ void e64_drain(const Energy64Args &a, E64Queue &Q, int lane) {
  __syncwarp();
  for (int e = lane; e < Q.n; e += 32) {
    const int2 p = Q.q[e];
    const double dx = a.x[p.x] - a.x[p.y], dy = a.y[p.x] - a.y[p.y], dz = a.z[p.x] - a.z[p.y];
    const double r = sqrt(fma(dx, dx, fma(dy, dy, dz * dz)) + 1e-12);
    atomic_add_fix(&a.born_acc[p.x], to_fix(obc_integral_d(r, a.ro[p.x], a.sr[p.y]), kBornScale));
    atomic_add_fix(&a.born_acc[p.y], to_fix(obc_integral_d(r, a.ro[p.y], a.sr[p.x]), kBornScale));
  }
  __syncwarp();
  Q.n = 0;
}

// (x, y, z, s^2, s^3, t^2) of the descreening pass, t = max(s / 0.4, s +
// rho~_max): pairs with r >= both t are in the series' domain; (x, y, z, q,
// sigma/2, sqrt(eps), B, sqrt(log2(e)/4)/B) of the energy pass.
typedef double E64Tile[8][32];

struct E64Born {
  double x, y, z, s2, s3, t2;
};
struct E64Pair {
  double x, y, z, q, hs, se, B, iB;
};

__device__ __forceinline__ E64Born load_born64(const Energy64Args &a, int g, double ro_max) {
  const double s = a.sr[g], t = fmax(2.5 * s, s + ro_max);  // 2.5 = 1 / sqrt(kSeriesUNear)
  return E64Born{a.x[g], a.y[g], a.z[g], s * s, s * s * s, t * t};
}
// No position (a NaN, or an infinity): the closed form takes a NaN's pairs as
// nothing, the series would carry it into the other atom's sum.  By the
// exponents, off the FP64 pipe.
__device__ __forceinline__ bool lost(const E64Born &A) {
  const int m = 0x7ff00000;
  return (__double2hiint(A.x) & m) == m || (__double2hiint(A.y) & m) == m || (__double2hiint(A.z) & m) == m;
}


// One tile of the descreening pass, steps k0 .. k0 + kn - 1.  FAR: both
// tiles in the series' domain; FULL: every pair exists and no cutoff.
struct E64Tests {
  uint32_t V0, V1;  // bit k: the lane's pair of step k exists
  double bcut2;
  int ig0, ig1, jg0;
};
template <bool FAR, bool FULL, int TIER>
__device__ __forceinline__ void born64_tile(const Energy64Args &a, const E64Born &I0, const E64Born &I1,
                                            const E64Tile &T, int k0, int kn, int lane, const E64Tests &M,
                                            double &acc0, double &acc1, double &accj, E64Queue &Q) {
#pragma unroll 1
  for (int k = k0; k < k0 + kn; ++k) {
    const int c = (lane + k) & 31;
    const double xj = T[0][c], yj = T[1][c], zj = T[2][c], s2j = T[3][c], s3j = T[4][c];
    const double dx0 = I0.x - xj, dy0 = I0.y - yj, dz0 = I0.z - zj;
    const double dx1 = I1.x - xj, dy1 = I1.y - yj, dz1 = I1.z - zj;
    double r20 = fma(dx0, dx0, fma(dy0, dy0, fma(dz0, dz0, 1e-12)));
    double r21 = fma(dx1, dx1, fma(dy1, dy1, fma(dz1, dz1, 1e-12)));
    if (!FULL) {
      bool in0 = (M.V0 >> k) & 1u, in1 = (M.V1 >> k) & 1u;
      if (M.bcut2 > 0.0) {  // by r^2 itself: 1e-12 cannot be taken off again exactly
        in0 = in0 && fma(dx0, dx0, fma(dy0, dy0, dz0 * dz0)) < M.bcut2;
        in1 = in1 && fma(dx1, dx1, fma(dy1, dy1, dz1 * dz1)) < M.bcut2;
      }
      if (!in0) r20 = kFarR2d;
      if (!in1) r21 = kFarR2d;
    }
    if (!FAR) {
      const double t2j = T[5][c];
      const bool n0 = !(r20 >= I0.t2 && r20 >= t2j), n1 = !(r21 >= I1.t2 && r21 >= t2j);
      const unsigned b0 = __ballot_sync(kFull, n0), b1 = __ballot_sync(kFull, n1);
      if (b0 | b1) {  // warp-uniform
        const int c0 = __popc(b0), cnt = c0 + __popc(b1);
        if (Q.n + cnt > kE64Queue) e64_drain(a, Q, lane);
        const unsigned lt = (1u << lane) - 1u;
        if (n0) {
          Q.q[Q.n + __popc(b0 & lt)] = make_int2(M.ig0, M.jg0 + c);
          r20 = kFarR2d;
        }
        if (n1) {
          Q.q[Q.n + c0 + __popc(b1 & lt)] = make_int2(M.ig1, M.jg0 + c);
          r21 = kFarR2d;
        }
        Q.n += cnt;
      }
    }
    const double w0 = rcp_d(r20), w1 = rcp_d(r21);
    const double f0 = w0 * w0, f1 = w1 * w1;
    const double vj0 = s3j * ObcPoly64<TIER>::eval(s2j * w0), vj1 = s3j * ObcPoly64<TIER>::eval(s2j * w1);
    const double vi0 = I0.s3 * ObcPoly64<TIER>::eval(I0.s2 * w0), vi1 = I1.s3 * ObcPoly64<TIER>::eval(I1.s2 * w1);
    acc0 = fma(vj0, f0, acc0);
    acc1 = fma(vj1, f1, acc1);
    accj = fma(vi0, f0, fma(vi1, f1, accj));
    accj = __shfl_sync(kFull, accj, (lane + 1) & 31);
  }
}

// One tile of the energy pass.  FULL: every pair exists, no exclusion, no
// cutoff, all three terms.  SIGNED: a Born radius may be negative.
struct E64Masks {
  uint32_t V0, V1, E0, E1, S0, S1;  // bit k: the pair of step k exists / excluded / 1-4
  double cut2, gcut2, lj14, coul14;
  bool use_gb, use_lj, use_coul;
};
struct E64Sums {
  double gb, coul, lj;
};
template <bool FULL, bool SIGNED>
__device__ __forceinline__ void pair64(const E64Pair &I, double dx, double dy, double dz, double qj, double hsj,
                                       double sej, double Bj, double iBj, bool ok, bool ex, bool s14,
                                       const E64Masks &M, E64Sums &E) {
  double r2 = fma(dx, dx, fma(dy, dy, dz * dz));
  const double qq = I.q * qj;
  if (FULL || M.use_gb) {
    const double rg2 = r2 + 1e-12, e = exp2neg_d<SIGNED>(rg2 * (I.iB * iBj));
    double f2 = fma(I.B * Bj, e, rg2), qg = qq;
    if (!FULL && !(ok && (M.gcut2 == 0.0 || r2 < M.gcut2))) {
      f2 = 1.0;  // a masked pair's own may have no root (a negative Born radius)
      qg = 0.0;
    }
    E.gb = fma(qg, rsqrt_d(f2), E.gb);
  }
  if (FULL || M.use_coul || M.use_lj) {
    double fc = 1.0, fl = 1.0;
    if (!FULL) {
      if (!(ok && !ex && (M.cut2 == 0.0 || r2 < M.cut2))) {
        r2 = 1.0;
        fc = fl = 0.0;
      } else if (s14) {
        fc = M.coul14;
        fl = M.lj14;
      }
    }
    const double inv_r = rsqrt_d(r2);
    if (FULL || M.use_coul) E.coul = fma(FULL ? qq : qq * fc, inv_r, E.coul);
    if (FULL || M.use_lj) {
      const double t = (I.hs + hsj) * inv_r;
      const double t2 = t * t, s6 = t2 * t2 * t2;
      const double eps = I.se * sej;
      E.lj = fma(FULL ? eps : eps * fl, fma(s6, s6, -s6), E.lj);
    }
  }
}

template <bool FULL, bool SIGNED>
__device__ __forceinline__ void pair64_tile(const E64Pair &I0, const E64Pair &I1, const E64Tile &T, int k0, int kn,
                                            int lane, const E64Masks &M, E64Sums &E0, E64Sums &E1) {
#pragma unroll 1
  for (int k = k0; k < k0 + kn; ++k) {
    const int c = (lane + k) & 31;
    const double xj = T[0][c], yj = T[1][c], zj = T[2][c], qj = T[3][c], hsj = T[4][c], sej = T[5][c],
                 Bj = T[6][c], iBj = T[7][c];
    pair64<FULL, SIGNED>(I0, I0.x - xj, I0.y - yj, I0.z - zj, qj, hsj, sej, Bj, iBj, (M.V0 >> k) & 1u, (M.E0 >> k) & 1u,
                 (M.S0 >> k) & 1u, M, E0);
    pair64<FULL, SIGNED>(I1, I1.x - xj, I1.y - yj, I1.z - zj, qj, hsj, sej, Bj, iBj, (M.V1 >> k) & 1u, (M.E1 >> k) & 1u,
                 (M.S1 >> k) & 1u, M, E1);
  }
}

__device__ __forceinline__ uint32_t rotr_u32(uint32_t x, int s) { return __funnelshift_r(x, x, s); }

__device__ __forceinline__ double e64_box_dist2(const float4 *bbox, int a, int b) {
  const float4 alo = bbox[2 * a], ahi = bbox[2 * a + 1];
  const float4 blo = bbox[2 * b], bhi = bbox[2 * b + 1];
  const float dx = fmaxf(0.f, fmaxf(alo.x - bhi.x, blo.x - ahi.x));
  const float dy = fmaxf(0.f, fmaxf(alo.y - bhi.y, blo.y - ahi.y));
  const float dz = fmaxf(0.f, fmaxf(alo.z - bhi.z, blo.z - ahi.z));
  return (double)fmaf(dx, dx, fmaf(dy, dy, dz * dz));
}

// sqrt(log2(e) / 4): exp(-r^2 / (4 B_i B_j)) = 2^-(r^2 iB_i iB_j)
constexpr double kSqrtQuarterLog2eD = 0.60056120439322491;

__device__ __forceinline__ E64Sums warp_sums(const E64Sums &E) {
  return E64Sums{warp_sum_d(E.gb), warp_sum_d(E.coul), warp_sum_d(E.lj)};
}

// An i-block's sums of one item, added to its system's accumulators.
__device__ __forceinline__ void add_energy64(const Energy64Args &a, int sys, const E64Sums &E) {
  const SysInfo &S = a.sys[sys];
  long long *e = a.energy + (size_t)sys * PB2_NTERMS;
  atomic_add_fix(&e[PB2_TERM_GB], to_fix(2.0 * S.pref_d * E.gb, kEnergyScale));
  atomic_add_fix(&e[PB2_TERM_COULOMB], to_fix(S.kcoul_d * E.coul, kEnergyScale));
  atomic_add_fix(&e[PB2_TERM_LJ], to_fix(4.0 * E.lj, kEnergyScale));
}

__device__ __forceinline__ E64Pair load_pair64(const Energy64Args &a, int g, bool use_gb) {
  E64Pair P{a.x[g], a.y[g], a.z[g], a.q[g], a.hs[g], a.se[g], 1.0, 1.0};
  if (use_gb) {
    P.B = a.born64[g];
    P.iB = a.iborn64[g];
  }
  return P;
}
__device__ __forceinline__ void store_pair64(E64Tile &T, int lane, const E64Pair &J) {
  T[0][lane] = J.x; T[1][lane] = J.y; T[2][lane] = J.z; T[3][lane] = J.q;
  T[4][lane] = J.hs; T[5][lane] = J.se; T[6][lane] = J.B; T[7][lane] = J.iB;
}

// Pairs of lane i with j-lane c that exist: both atoms do, j > i on a diagonal.
struct E64Valid {
  uint32_t C0, C1;
};
__device__ __forceinline__ E64Valid valid64(int jb, int ib0, int n, bool iv0, bool iv1, int lane) {
  const int nj = n - jb * 32;
  const uint32_t jmask = nj >= 32 ? 0xffffffffu : ((1u << nj) - 1u);
  const uint32_t diag_mask = lane == 31 ? 0u : (0xffffffffu << (lane + 1));
  E64Valid v{iv0 ? jmask : 0u, iv1 ? jmask : 0u};
  if (jb == ib0) {
    v.C0 &= diag_mask;
    v.C1 = 0u;
  } else if (jb == ib0 + 1) {
    v.C1 &= diag_mask;
  }
  return v;
}

// No pair of the energy pass beyond its root (0: unbounded).
__device__ __forceinline__ double energy_reach2(const E64Masks &M) {
  const bool direct = M.use_lj || M.use_coul;
  if ((M.use_gb && !(M.gcut2 > 0.0)) || (direct && !(M.cut2 > 0.0))) return 0.0;
  return fmax(M.use_gb ? M.gcut2 : 0.0, direct ? M.cut2 : 0.0);
}

// The exclusion rows of a tile's two i-blocks; ent: lanes 0-15 hold block
// ib0's entries, 16-31 block ib0 + 1's.  True if the tile has any.
__device__ __forceinline__ bool excl64(const Energy64Args &a, int2 ent, int jb, int lane, ExclRow &r0, ExclRow &r1) {
  const unsigned hit = __ballot_sync(kFull, ent.x == jb);
  const unsigned hit0 = hit & 0xffffu, hit1 = hit & 0xffff0000u;
  r0 = r1 = ExclRow{0u, 0u};
  if (hit0) r0 = a.excl_rows[__shfl_sync(kFull, ent.y, __ffs(hit0) - 1) + lane];
  if (hit1) r1 = a.excl_rows[__shfl_sync(kFull, ent.y, __ffs(hit1) - 1) + lane];
  return hit != 0u;
}

// Steps k0 .. k0 + kn - 1 of a tile's pair energies.
__device__ __forceinline__ void pair64_steps(const E64Pair &P0, const E64Pair &P1, const E64Tile &T, int k0, int kn,
                                             int lane, bool plain, const E64Valid &v, const ExclRow &r0,
                                             const ExclRow &r1, E64Masks &M, E64Sums &E0, E64Sums &E1) {
  const int signs = __double2hiint(P0.iB) | __double2hiint(P1.iB) | __double2hiint(T[7][lane]);
  const bool negative = __any_sync(kFull, signs < 0);
  if (plain && !negative) {
    pair64_tile<true, false>(P0, P1, T, k0, kn, lane, M, E0, E1);
    return;
  }
  M.V0 = rotr_u32(v.C0, lane); M.V1 = rotr_u32(v.C1, lane);
  M.E0 = rotr_u32(r0.excl, lane); M.E1 = rotr_u32(r1.excl, lane);
  M.S0 = rotr_u32(r0.s14, lane); M.S1 = rotr_u32(r1.s14, lane);
  if (negative) pair64_tile<false, true>(P0, P1, T, k0, kn, lane, M, E0, E1);
  else pair64_tile<false, false>(P0, P1, T, k0, kn, lane, M, E0, E1);
}

// PASS 0: descreening sums; PASS 1: pair energies.  The warps of one
// resident wave each start with an item of their own, spread over the SMs,
// and take further items from a counter (the last warp to finish resets it).
template <int PASS>
__global__ void __launch_bounds__(kE64Threads, PASS == 0 ? 4 : 3) energy64_kernel(const Energy64Args a) {
  __shared__ E64Tile s_tile[kE64Warps];
  __shared__ int2 s_q[PASS == 0 ? kE64Warps : 1][PASS == 0 ? kE64Queue : 1];
  const int lane = threadIdx.x & 31, wl = threadIdx.x >> 5;
  const int nwarps = (int)gridDim.x * kE64Warps;
  E64Tile &T = s_tile[wl];
  E64Queue Q{s_q[PASS == 0 ? wl : 0], 0};
  E64Masks M;
  M.use_gb = (a.terms & PB2_USE_GB) != 0;
  M.use_lj = (a.terms & PB2_USE_LJ) != 0;
  M.use_coul = (a.terms & PB2_USE_COULOMB) != 0;
  const bool all_terms = M.use_gb && M.use_lj && M.use_coul;
  const bool one_wave = a.n_items <= nwarps;  // no warp asks the counter for another item
  pdl_wait();
  pdl_trigger();
  for (int it = wl * (int)gridDim.x + (int)blockIdx.x; it < a.n_items;) {
    const TileItem item = a.items[it];
    const ItemRange R = item_range(item);
    const SysInfo &S = a.sys[item.sys];
    const int n = S.n, off = S.off;
    M.cut2 = (double)S.cutoff2; M.gcut2 = (double)S.gb_cutoff2;
    M.lj14 = (double)S.lj14; M.coul14 = (double)S.coul14;
    const double bcut2 = (double)S.born_cut2;
    // no pair of this pass beyond reach2 (0: unbounded); the boxes are of
    // the float32 positions, so the test leaves a margin for their rounding
    const double reach2 = PASS == 0 ? bcut2 : energy_reach2(M);
    const double skip2 = reach2 * 1.001 + 0.01;
    const bool cut = PASS == 0 ? bcut2 > 0.0 : (M.cut2 > 0.0 || M.gcut2 > 0.0);
    const int ib0 = item.iblk, ib1 = ib0 + 1;
    const bool has1 = ib1 < S.nblk;
    const int gib0 = S.blk_base + ib0, gib1 = S.blk_base + (has1 ? ib1 : ib0);
    const int il0 = ib0 * 32 + lane, il1 = ib1 * 32 + lane;
    const bool iv0 = il0 < n, iv1 = il1 < n;  // il1 >= n whenever !has1
    const int ig0 = off + (iv0 ? il0 : n - 1), ig1 = off + (iv1 ? il1 : n - 1);
    E64Born A0{}, A1{};
    E64Pair P0{}, P1{};
    int2 ent = make_int2(-1, -1);
    if (PASS == 0) {
      A0 = load_born64(a, ig0, (double)S.ro_max);
      A1 = load_born64(a, ig1, (double)S.ro_max);
    } else {
      P0 = load_pair64(a, ig0, M.use_gb);
      P1 = load_pair64(a, ig1, M.use_gb);
      if (lane < kExclPerBlock) ent = a.excl_ent[gib0 * kExclPerBlock + lane];
      else if (has1) ent = a.excl_ent[gib1 * kExclPerBlock + lane - kExclPerBlock];
    }
    const bool lost_i = PASS == 0 && (lost(A0) || lost(A1));
    double acc0 = 0.0, acc1 = 0.0;
    E64Sums E0{0.0, 0.0, 0.0}, E1{0.0, 0.0, 0.0};
    for (int jb = R.jb0; jb < R.jb1; ++jb) {
      const int gjb = S.blk_base + jb;
      double d2 = 0.0;
      if (PASS == 0 || reach2 > 0.0) {
        d2 = e64_box_dist2(a.bbox, gib0, gjb);
        if (has1 && jb > ib0) d2 = fmin(d2, e64_box_dist2(a.bbox, gib1, gjb));
        if (reach2 > 0.0 && d2 >= skip2) continue;
      }
      const int jl0 = jb * 32, jl = jl0 + lane;
      const int jg = off + (jl < n ? jl : n - 1);
      bool series = true;  // every pair may take the series
      __syncwarp();  // every lane is done with the previous tile
      if (PASS == 0) {
        const E64Born J = load_born64(a, jg, (double)S.ro_max);
        T[0][lane] = J.x; T[1][lane] = J.y; T[2][lane] = J.z;
        T[3][lane] = J.s2; T[4][lane] = J.s3; T[5][lane] = J.t2;
        series = !__any_sync(kFull, lost_i || lost(J));
      } else {
        store_pair64(T, lane, load_pair64(a, jg, M.use_gb));
      }
      __syncwarp();
      const E64Valid v = valid64(jb, ib0, n, iv0, iv1, lane);
      const bool full = __all_sync(kFull, (v.C0 & v.C1) == 0xffffffffu) && !cut;
      if (PASS == 0) {
        const E64Tests K{rotr_u32(v.C0, lane), rotr_u32(v.C1, lane), bcut2, ig0, ig1, off + jl0};
        const float *tier2 = S.tier2[0];
        const int k0 = R.k0, kn = R.kn;
        double accj = 0.0;
        if (full && series) {
          if (d2 >= tier2[0]) born64_tile<true, true, 0>(a, A0, A1, T, k0, kn, lane, K, acc0, acc1, accj, Q);
          else if (d2 >= tier2[1]) born64_tile<true, true, 1>(a, A0, A1, T, k0, kn, lane, K, acc0, acc1, accj, Q);
          else if (d2 >= tier2[2]) born64_tile<true, true, 2>(a, A0, A1, T, k0, kn, lane, K, acc0, acc1, accj, Q);
          else if (d2 >= S.far2) born64_tile<true, true, 3>(a, A0, A1, T, k0, kn, lane, K, acc0, acc1, accj, Q);
          else born64_tile<false, true, 3>(a, A0, A1, T, k0, kn, lane, K, acc0, acc1, accj, Q);
        } else if (d2 >= S.far2 && series) {
          born64_tile<true, false, 3>(a, A0, A1, T, k0, kn, lane, K, acc0, acc1, accj, Q);
        } else {
          born64_tile<false, false, 3>(a, A0, A1, T, k0, kn, lane, K, acc0, acc1, accj, Q);
        }
        if (Q.n >= 32) e64_drain(a, Q, lane);
        // lane l holds the sum of j-atom (l + k0 + kn) mod 32
        const int jc = jl0 + ((lane + k0 + kn) & 31);
        if (jc < n && accj != 0.0) atomic_add_fix(&a.born_acc[off + jc], to_fix(accj, kBornScale));
      } else {
        ExclRow r0, r1;
        const bool hit = excl64(a, ent, jb, lane, r0, r1);
        pair64_steps(P0, P1, T, R.k0, R.kn, lane, full && !hit && all_terms, v, r0, r1, M, E0, E1);
      }
    }
    if (PASS == 0) {
      if (iv0 && acc0 != 0.0) atomic_add_fix(&a.born_acc[ig0], to_fix(acc0, kBornScale));
      if (iv1 && acc1 != 0.0) atomic_add_fix(&a.born_acc[ig1], to_fix(acc1, kBornScale));
    } else {
      E0 = warp_sums(E0);
      E1 = warp_sums(E1);
      if (lane == 0) {
        add_energy64(a, item.sys, E0);
        add_energy64(a, item.sys, E1);
      }
    }
    if (one_wave) break;
    int next = 0;
    if (lane == 0) next = nwarps + atomicAdd(&a.sched[0], 1);
    it = __shfl_sync(kFull, next, 0);
  }
  if (PASS == 0 && Q.n > 0) e64_drain(a, Q, lane);
  if (!one_wave && lane == 0 && atomicAdd(&a.sched[1], 1) == nwarps - 1) {
    // every warp has stopped taking items: reset for the next launch
    a.sched[0] = 0;
    a.sched[1] = 0;
  }
}

// Pair energies of the small systems (a.tiles): a thread block per tile, its
// warps sharing the 32 steps.  The warps' sums meet in shared memory in warp
// order and a tile's sums go to fixed point once per i-block: rounding each
// warp's share by itself left the total of a 166-atom system 2e-9 off.
constexpr int kTileWarps = 8;
__global__ void __launch_bounds__(32 * kTileWarps) energy64_tile_kernel(const Energy64Args a) {
  __shared__ E64Tile T;
  __shared__ E64Sums s_e[2][kTileWarps];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  constexpr int kn = 32 / kTileWarps;
  E64Masks M;
  M.use_gb = (a.terms & PB2_USE_GB) != 0;
  M.use_lj = (a.terms & PB2_USE_LJ) != 0;
  M.use_coul = (a.terms & PB2_USE_COULOMB) != 0;
  pdl_wait();
  pdl_trigger();
  for (int u = (int)blockIdx.x; u < a.n_tiles; u += (int)gridDim.x) {
    const TileItem item = a.tiles[u];
    const SysInfo &S = a.sys[item.sys];
    const int n = S.n, off = S.off, jb = item.jb0;
    M.cut2 = (double)S.cutoff2; M.gcut2 = (double)S.gb_cutoff2;
    M.lj14 = (double)S.lj14; M.coul14 = (double)S.coul14;
    const int ib0 = item.iblk;
    const bool has1 = ib0 + 1 < S.nblk;
    const int gib0 = S.blk_base + ib0, gib1 = gib0 + (has1 ? 1 : 0);
    const int il0 = ib0 * 32 + lane, il1 = il0 + 32, jl = jb * 32 + lane;
    const bool iv0 = il0 < n, iv1 = il1 < n;
    const double reach2 = energy_reach2(M);
    if (reach2 > 0.0) {  // as energy64_kernel
      double d2 = e64_box_dist2(a.bbox, gib0, S.blk_base + jb);
      if (has1 && jb > ib0) d2 = fmin(d2, e64_box_dist2(a.bbox, gib1, S.blk_base + jb));
      if (d2 >= reach2 * 1.001 + 0.01) continue;  // block-uniform
    }
    const E64Pair P0 = load_pair64(a, off + (iv0 ? il0 : n - 1), M.use_gb);
    const E64Pair P1 = load_pair64(a, off + (iv1 ? il1 : n - 1), M.use_gb);
    int2 ent = make_int2(-1, -1);
    if (lane < kExclPerBlock) ent = a.excl_ent[gib0 * kExclPerBlock + lane];
    else if (has1) ent = a.excl_ent[gib1 * kExclPerBlock + lane - kExclPerBlock];
    ExclRow r0, r1;
    const bool hit = excl64(a, ent, jb, lane, r0, r1);
    const E64Valid v = valid64(jb, ib0, n, iv0, iv1, lane);
    const bool plain = __all_sync(kFull, (v.C0 & v.C1) == 0xffffffffu) && !hit && M.use_gb && M.use_lj &&
                       M.use_coul && !(M.cut2 > 0.0 || M.gcut2 > 0.0);
    if (w == 0) store_pair64(T, lane, load_pair64(a, off + (jl < n ? jl : n - 1), M.use_gb));
    __syncthreads();
    E64Sums E0{0.0, 0.0, 0.0}, E1{0.0, 0.0, 0.0};
    pair64_steps(P0, P1, T, w * kn, kn, lane, plain, v, r0, r1, M, E0, E1);
    E0 = warp_sums(E0);
    E1 = warp_sums(E1);
    if (lane == 0) {
      s_e[0][w] = E0;
      s_e[1][w] = E1;
    }
    __syncthreads();
    if (threadIdx.x < 2) {
      E64Sums t = s_e[threadIdx.x][0];
      for (int k = 1; k < kTileWarps; ++k) {
        const E64Sums &v = s_e[threadIdx.x][k];
        t.gb += v.gb; t.coul += v.coul; t.lj += v.lj;
      }
      add_energy64(a, item.sys, t);
    }
  }
}

cudaError_t launch_energy64_tiles(const Energy64Args &a, int grid, cudaStream_t st) {
  if (a.n_tiles <= 0) return cudaSuccess;
  return launch_after(energy64_tile_kernel, grid, 32 * kTileWarps, st, a);
}
int energy64_tile_occupancy() {
  int blocks = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, energy64_tile_kernel, 32 * kTileWarps, 0);
  return blocks > 0 ? blocks : 1;
}

// FP64 Born radii from the descreening sums (cleared for the next
// evaluation), the GB self terms and ACE: one warp per 32-atom block, whose
// atoms belong to one system, so a block adds its two energies once (one
// addition per atom queued 2 n atomics on one address).  The sums are of the
// same fixed-point values in either order.
__device__ __forceinline__ long long warp_sum_ll(long long v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
  return v;
}
__global__ void __launch_bounds__(128) finalize64_kernel(const Energy64Args a) {
  const int lane = threadIdx.x & 31;
  const int nw = (int)((gridDim.x * blockDim.x) >> 5);
  pdl_wait();
  pdl_trigger();
  for (int b = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5); b < a.n_blocks; b += nw) {
    const int s = a.blk_sys[b];
    const SysInfo &S = a.sys[s];
    const int l = (b - S.blk_base) * 32 + lane;
    long long e_gb = 0, e_ace = 0;
    if (l < S.n) {
      const int i = S.off + l;
      const double isum = (double)a.born_acc[i] * kBornInv;
      a.born_acc[i] = 0;
      const double r_in = a.radius[i], q = a.q[i];
      const BornRadius R = born_radius(isum, r_in, S.clamp != 0);
      a.born64[i] = R.B;
      a.iborn64[i] = kSqrtQuarterLog2eD / R.B;
      e_gb = to_fix(S.pref_d * q * q * R.inv_b, kEnergyScale);
      e_ace = to_fix(ace_energy(r_in, R.B), kEnergyScale);
    }
    e_gb = warp_sum_ll(e_gb);
    e_ace = warp_sum_ll(e_ace);
    if (lane == 0) {
      atomic_add_fix(&a.energy[(size_t)s * PB2_NTERMS + PB2_TERM_GB], e_gb);
      atomic_add_fix(&a.energy[(size_t)s * PB2_NTERMS + PB2_TERM_NONPOLAR], e_ace);
    }
  }
}

cudaError_t launch_finalize64(const Energy64Args &a, cudaStream_t st) {
  if (a.n_blocks <= 0) return cudaSuccess;
  return launch_after(finalize64_kernel, (a.n_blocks + 3) / 4, 128, st, a);
}

cudaError_t launch_energy64(int pass, const Energy64Args &a, int grid, cudaStream_t st) {
  if (a.n_items <= 0) return cudaSuccess;
  return launch_after(pass == 0 ? energy64_kernel<0> : energy64_kernel<1>, grid, kE64Threads, st, a);
}

int energy64_occupancy(int pass) {
  int blocks = 0;
  if (pass == 0) cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, energy64_kernel<0>, kE64Threads, 0);
  else cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, energy64_kernel<1>, kE64Threads, 0);
  return blocks > 0 ? blocks : 1;
}

}  // namespace pb2
