// Batched energy minimisation: restrained steepest descent and FIRE, all
// systems of the batch at once (prolix batched_simulate.py:682-960,
// `batched_minimize`).
//
// Forces come from the same force kernels as the MD step (fixed-point
// accumulators F); the minimiser adds a harmonic position restraint
//   E = k/2 sum_i m_i |r_i - r0_i|^2   (batched_simulate.py:675-679)
// on a per-atom selection m (all atoms, heavy atoms or backbone atoms) and
// zeroes non-finite force components (the reference's NaN guard).
//
// Steepest descent (batched_simulate.py:748-791): dr = F dt, |dr| capped at
// max_dx per atom, r += dr.
//
// FIRE (Bitzek et al., PRL 97, 170201 (2006), as jax_md 0.2.27
// minimize.fire_descent applies it; the reference calls it at
// batched_simulate.py:818-878): a velocity-Verlet step on momenta
//   p += dt/2 F; r += dt p / m; F = force(r); p += dt/2 F,
// then per system, with P = sum F.p, |F| = sqrt(sum F^2 + 1e-6), |p|:
//   p = p + alpha (F |p| / |F| - p);
//   P >= 0: n_pos += 1, else n_pos = 0;
//   P > 0 and n_pos > 5: dt = min(1.1 dt, dt_max), alpha *= 0.99;
//   P < 0: dt *= 0.5, alpha = 0.1, p = 0.
// The reference then caps each atom's displacement of the step at max_disp
// (0.1 A), scales its momentum by the same factor, keeps the force of the
// uncapped position, and returns the positions of the lowest force RMS seen
// at the start of an iteration.  The same order is kept here.
//
// An iteration is two launches around the force kernels: min_fire_move (the
// mixing and cap that close the last iteration, the lowest-RMS snapshot, the
// half kick and drift) and min_fire_close (the second half kick and the
// system's sums).  Both run one thread block per 256 atoms; a system's sums
// are added chunk by chunk in a fixed order by its last block to finish, so
// the trajectory does not depend on scheduling or on the batch.  (One block
// per system and four launches took 55 of an iteration's 155 us for 16
// systems of 150 to 4,000 atoms; these take 9, and an iteration 110.)
#include "pb2_common.cuh"
#include "pb2_kernels.cuh"

namespace pb2 {

constexpr int kMinThreads = 256;

__device__ __forceinline__ double fix_d(long long v) { return (double)v * kForceInv; }

// Restraint selection of atom i for the kind in par[kMinKind].
__device__ __forceinline__ bool selected(const MinArgs &a, int i) {
  const int kind = (int)a.par[kMinKind];
  if (kind == 0) return true;
  return ((a.sel[i] >> (kind - 1)) & 1u) != 0;
}

// F (physical, fixed point) + restraint force at the current position.
__device__ __forceinline__ void total_force(const MinArgs &a, int i, double f[3]) {
  const double k = a.par[kMinK];
  const bool m = k != 0.0 && selected(a, i);
  const size_t N = a.n_total;
  f[0] = fix_d(a.fx[i]);
  f[1] = fix_d(a.fy[i]);
  f[2] = fix_d(a.fz[i]);
  if (m) {
    f[0] -= k * (a.x[i] - a.x0[i]);
    f[1] -= k * (a.y[i] - a.x0[N + i]);
    f[2] -= k * (a.z[i] - a.x0[2 * N + i]);
  }
#pragma unroll
  for (int c = 0; c < 3; ++c)
    if (!isfinite(f[c])) f[c] = 0.0;
}

// The float32 copy of atom i's new position (returned for its block's box);
// raises the pair list's rebuild flag when it is past half the skin.
__device__ __forceinline__ float4 place_atom(const MinArgs &a, int i, const SysInfo &S, double x, double y, double z) {
  const float4 q = make_float4((float)(x - S.ox), (float)(y - S.oy), (float)(z - S.oz), (float)a.charge[i]);
  if (a.pl_ref) {
    const float4 r = a.pl_ref[i];
    const float dx = q.x - r.x, dy = q.y - r.y, dz = q.z - r.z;
    if ((double)fmaf(dx, dx, fmaf(dy, dy, dz * dz)) > S.skin_half2) atomicOr(&a.pl_ctl[PL_DIRTY], 1);
  }
  a.posq[i] = q;
  return q;
}

__device__ __forceinline__ void put_posq(const MinArgs &a, int i) {
  const SysInfo &S = a.sys[a.atom_sys[i]];
  a.posq[i] = make_float4((float)(a.x[i] - S.ox), (float)(a.y[i] - S.oy), (float)(a.z[i] - S.oz),
                          (float)a.charge[i]);
}

// Block-wide sums of up to three values (fixed order: deterministic).
__device__ __forceinline__ void block_sum3(double &v0, double &v1, double &v2) {
  __shared__ double sh[3][kMinThreads / 32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    v0 += __shfl_down_sync(kFull, v0, o);
    v1 += __shfl_down_sync(kFull, v1, o);
    v2 += __shfl_down_sync(kFull, v2, o);
  }
  if (lane == 0) { sh[0][w] = v0; sh[1][w] = v1; sh[2][w] = v2; }
  __syncthreads();
  if (threadIdx.x == 0) {
    double s0 = 0.0, s1 = 0.0, s2 = 0.0;
    for (int k = 0; k < kMinThreads / 32; ++k) { s0 += sh[0][k]; s1 += sh[1][k]; s2 += sh[2][k]; }
    sh[0][0] = s0; sh[1][0] = s1; sh[2][0] = s2;
  }
  __syncthreads();
  v0 = sh[0][0]; v1 = sh[1][0]; v2 = sh[2][0];
  __syncthreads();
}

// The thread's atom: thread block c is chunk c (system, first 32-atom block
// of eight), warp w its block w, lane l the block's atom l.
struct MinAtom {
  int s, b, i;        // system, batch-wide block, atom
  bool block, valid;  // the block exists; the atom exists
};
__device__ __forceinline__ MinAtom min_atom(const MinArgs &a) {
  const int2 ch = a.chunks[blockIdx.x];
  const SysInfo &S = a.sys[ch.x];
  const int lb = ch.y + (int)(threadIdx.x >> 5);
  const int l = lb * 32 + (int)(threadIdx.x & 31);
  return MinAtom{ch.x, S.blk_base + lb, S.off + l, lb < S.nblk, l < S.n};
}

// Adds the chunk's three sums to its system's; the system's last chunk to
// arrive gets true in every thread, and the totals, summed in chunk order.
__device__ __forceinline__ bool sys_sum3(const MinArgs &a, int s, double &v0, double &v1, double &v2) {
  __shared__ int last;
  block_sum3(v0, v1, v2);
  const int c0 = a.chunk0[s], nc = a.chunk0[s + 1] - c0;
  if (nc == 1) return true;
  if (threadIdx.x == 0) {
    double *p = a.part + 3 * (size_t)blockIdx.x;
    p[0] = v0; p[1] = v1; p[2] = v2;
    __threadfence();
    last = atomicAdd(&a.sys_done[s], 1) == nc - 1;
    if (last) a.sys_done[s] = 0;
  }
  __syncthreads();
  if (!last) return false;
  __threadfence();
  v0 = v1 = v2 = 0.0;
  for (int c = threadIdx.x; c < nc; c += blockDim.x) {
    const double *p = a.part + 3 * (size_t)(c0 + c);
    v0 += __ldcg(p); v1 += __ldcg(p + 1); v2 += __ldcg(p + 2);
  }
  block_sum3(v0, v1, v2);
  return true;
}

// ----------------------------------------------------------- steepest descent

// One warp per 32-atom block, which also writes the block's box.  (By the
// batch's blocks, not by a system's chunks of eight: a batch of 8,000 systems
// of one block each has 1,000 thread blocks instead of 8,000, and an iteration
// of them takes 152.5 us instead of 157.9.)
__global__ void __launch_bounds__(kMinThreads) min_sd_kernel(const MinArgs a) {
  pdl_wait();
  pdl_trigger();
  const double dt = a.par[kMinSdDt], max_dx = a.par[kMinMaxDx];
  const int b = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
  if (b >= a.n_blocks) return;
  const int4 info = a.blk_info[b];  // system, first atom, atoms
  const bool valid = lane < info.z;
  float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
  if (valid) {
    const int i = info.y + lane;
    double f[3];
    total_force(a, i, f);
    double d[3] = {f[0] * dt, f[1] * dt, f[2] * dt};
    const double dm = sqrt(d[0] * d[0] + d[1] * d[1] + d[2] * d[2] + 1e-30);
    const double sc = fmin(1.0, max_dx / dm);
    const double x = a.x[i] + d[0] * sc, y = a.y[i] + d[1] * sc, z = a.z[i] + d[2] * sc;
    a.x[i] = x; a.y[i] = y; a.z[i] = z;
    a.fx[i] = 0; a.fy[i] = 0; a.fz[i] = 0;
    q = place_atom(a, i, a.sys[info.x], x, y, z);
  }
  block_box(a.bbox, b, lane, valid, q);
}

// A system with any non-finite coordinate goes back to its reference
// positions (the reference's rollback after SD and after FIRE).
__global__ void min_rollback_kernel(const MinArgs a) {
  __shared__ int bad;
  const size_t N = a.n_total;
  for (int s = blockIdx.x; s < a.n_sys; s += gridDim.x) {
    const SysInfo &S = a.sys[s];
    if (threadIdx.x == 0) bad = 0;
    __syncthreads();
    for (int i = S.off + threadIdx.x; i < S.off + S.n; i += blockDim.x)
      if (!(isfinite(a.x[i]) && isfinite(a.y[i]) && isfinite(a.z[i]))) bad = 1;
    __syncthreads();
    if (bad) {
      for (int i = S.off + threadIdx.x; i < S.off + S.n; i += blockDim.x) {
        a.x[i] = a.x0[i]; a.y[i] = a.x0[N + i]; a.z[i] = a.x0[2 * N + i];
        put_posq(a, i);
      }
      if (threadIdx.x == 0) atomicOr(&a.status[s], (uint32_t)PB2_STATUS_NONFINITE);
    }
    __syncthreads();
  }
}

// --------------------------------------------------------------------- FIRE

// Scalars that close an iteration, read by the next min_fire_move: p <- p +
// (mix_f F - mix_p p), or zero; and whether the state force's RMS is the
// lowest so far.
enum { kFireZeroP = 1, kFireBetter = 2 };

__device__ __forceinline__ bool rms_is_lowest(const MinArgs &a, int s, double f2) {
  const double rms = sqrt(f2 / (double)a.sys[s].n);
  const bool better = rms < a.sys_best[s];
  if (better) a.sys_best[s] = rms;
  return better;
}

// p = 0, state force = F + restraint, per-system scalars reset (a mixing that
// changes nothing pending).
__global__ void __launch_bounds__(kMinThreads) min_fire_init_kernel(const MinArgs a) {
  const size_t N = a.n_total;
  const MinAtom m = min_atom(a);
  double f2 = 0.0, z0 = 0.0, z1 = 0.0;
  if (m.valid) {
    const int i = m.i;
    double f[3];
    total_force(a, i, f);
    a.ft[i] = f[0]; a.ft[N + i] = f[1]; a.ft[2 * N + i] = f[2];
    a.px[i] = 0.0; a.py[i] = 0.0; a.pz[i] = 0.0;
    const double x = a.x[i], y = a.y[i], z = a.z[i];
    a.best[i] = x; a.best[N + i] = y; a.best[2 * N + i] = z;
    a.xb[i] = x; a.xb[N + i] = y; a.xb[2 * N + i] = z;
    f2 = f[0] * f[0] + f[1] * f[1] + f[2] * f[2];
  }
  if (sys_sum3(a, m.s, f2, z0, z1) && threadIdx.x == 0) {
    a.sys_dt[m.s] = a.par[kMinDtStart];
    a.sys_alpha[m.s] = kFireAlphaStart;
    a.sys_npos[m.s] = 0;
    a.sys_best[m.s] = 1e10;
    a.mix_f[m.s] = 0.0;
    a.mix_p[m.s] = 0.0;
    a.sys_flags[m.s] = rms_is_lowest(a, m.s, f2) ? kFireBetter : 0;
  }
}

// The mixing and the displacement cap that close the last iteration.
__device__ __forceinline__ void close_iteration(const MinArgs &a, int i, int s, int flags, double x[3], double p[3],
                                                const double f[3]) {
  const size_t N = a.n_total;
  const double max_disp = a.par[kMinMaxDisp], mf = a.mix_f[s], mp = a.mix_p[s];
#pragma unroll
  for (int c = 0; c < 3; ++c) p[c] = (flags & kFireZeroP) ? 0.0 : p[c] + (mf * f[c] - mp * p[c]);
  const double xb[3] = {a.xb[i], a.xb[N + i], a.xb[2 * N + i]};
  const double dx = x[0] - xb[0], dy = x[1] - xb[1], dz = x[2] - xb[2];
  const double dm = sqrt(dx * dx + dy * dy + dz * dz + 1e-30);
  const double sc = max_disp > 0.0 ? fmin(1.0, max_disp / dm) : 1.0;  // 0: no cap
  x[0] = xb[0] + dx * sc; x[1] = xb[1] + dy * sc; x[2] = xb[2] + dz * sc;
#pragma unroll
  for (int c = 0; c < 3; ++c) p[c] *= sc;
}

// Start of an iteration: closes the last one, keeps the positions if their
// force RMS is the lowest so far, then the first half kick and drift; the
// positions before are remembered for the displacement cap.  With a force cap
// (prolix simulate.py:613-621) the state force of each atom is scaled to at
// most that norm for this kick.  Also writes the blocks' boxes.
__global__ void __launch_bounds__(kMinThreads) min_fire_move_kernel(const MinArgs a) {
  pdl_wait();
  pdl_trigger();
  const size_t N = a.n_total;
  const MinAtom m = min_atom(a);
  if (!m.block) return;
  float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
  if (m.valid) {
    const int i = m.i;
    const int flags = a.sys_flags[m.s];
    const double cap = a.par[kMinForceCap], dt = a.sys_dt[m.s], h = 0.5 * dt, ms = a.mass[i];
    double f[3] = {a.ft[i], a.ft[N + i], a.ft[2 * N + i]};
    double x[3] = {a.x[i], a.y[i], a.z[i]}, p[3] = {a.px[i], a.py[i], a.pz[i]};
    close_iteration(a, i, m.s, flags, x, p, f);
    if (flags & kFireBetter) {
      a.best[i] = x[0]; a.best[N + i] = x[1]; a.best[2 * N + i] = x[2];
    }
    if (cap > 0.0) {
      const double sc = fmin(1.0, cap / (sqrt(f[0] * f[0] + f[1] * f[1] + f[2] * f[2]) + 1e-8));
      f[0] *= sc; f[1] *= sc; f[2] *= sc;
    }
    const double px = p[0] + h * f[0], py = p[1] + h * f[1], pz = p[2] + h * f[2];
    a.px[i] = px; a.py[i] = py; a.pz[i] = pz;
    a.xb[i] = x[0]; a.xb[N + i] = x[1]; a.xb[2 * N + i] = x[2];
    x[0] += dt * px / ms;
    x[1] += dt * py / ms;
    x[2] += dt * pz / ms;
    a.x[i] = x[0]; a.y[i] = x[1]; a.z[i] = x[2];
    a.fx[i] = 0; a.fy[i] = 0; a.fz[i] = 0;
    q = place_atom(a, i, a.sys[m.s], x[0], x[1], x[2]);
  }
  block_box(a.bbox, m.b, threadIdx.x & 31, m.valid, q);
}

// Second half kick with the new force, and the system's sums: the FIRE mixing
// factors and time-step control, and the RMS of the new state force.
__global__ void __launch_bounds__(kMinThreads) min_fire_close_kernel(const MinArgs a) {
  pdl_wait();
  pdl_trigger();
  const size_t N = a.n_total;
  const MinAtom m = min_atom(a);
  const int s = m.s;
  const double dt_max = a.par[kMinDtMax];
  double fp = 0.0, f2 = 0.0, p2 = 0.0;
  if (m.valid) {
    const int i = m.i;
    const double h = 0.5 * a.sys_dt[s];
    double f[3];
    total_force(a, i, f);
    a.ft[i] = f[0]; a.ft[N + i] = f[1]; a.ft[2 * N + i] = f[2];
    const double px = a.px[i] + h * f[0], py = a.py[i] + h * f[1], pz = a.pz[i] + h * f[2];
    a.px[i] = px; a.py[i] = py; a.pz[i] = pz;
    fp = f[0] * px + f[1] * py + f[2] * pz;
    f2 = f[0] * f[0] + f[1] * f[1] + f[2] * f[2];
    p2 = px * px + py * py + pz * pz;
  }
  if (!sys_sum3(a, s, fp, f2, p2) || threadIdx.x != 0) return;
  const double alpha = a.sys_alpha[s];
  a.mix_f[s] = alpha * sqrt(p2) / sqrt(f2 + 1e-6);
  a.mix_p[s] = alpha;
  const int npos = fp >= 0.0 ? a.sys_npos[s] + 1 : 0;
  double dt = a.sys_dt[s], al = alpha;
  if (fp > 0.0 && npos > kFireNmin) {
    dt = fmin(dt * kFireFinc, dt_max);
    al = al * kFireFalpha;
  }
  if (fp < 0.0) {
    dt = dt * kFireFdec;
    al = kFireAlphaStart;
  }
  a.sys_npos[s] = npos;
  a.sys_dt[s] = dt;
  a.sys_alpha[s] = al;
  a.sys_flags[s] = (fp < 0.0 ? kFireZeroP : 0) | (rms_is_lowest(a, s, f2) ? kFireBetter : 0);
}

// End of a FIRE stage: closes its last iteration.
__global__ void __launch_bounds__(kMinThreads) min_fire_end_kernel(const MinArgs a) {
  const size_t N = a.n_total;
  const MinAtom m = min_atom(a);
  if (!m.valid) return;
  const int i = m.i;
  const double f[3] = {a.ft[i], a.ft[N + i], a.ft[2 * N + i]};
  double x[3] = {a.x[i], a.y[i], a.z[i]}, p[3] = {a.px[i], a.py[i], a.pz[i]};
  close_iteration(a, i, m.s, a.sys_flags[m.s], x, p, f);
  a.x[i] = x[0]; a.y[i] = x[1]; a.z[i] = x[2];
  a.px[i] = p[0]; a.py[i] = p[1]; a.pz[i] = p[2];
}

// End of a FIRE stage: the best positions become the state.
__global__ void min_take_best_kernel(const MinArgs a) {
  const size_t N = a.n_total;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < a.n_total; i += gridDim.x * blockDim.x) {
    a.x[i] = a.best[i]; a.y[i] = a.best[N + i]; a.z[i] = a.best[2 * N + i];
    put_posq(a, i);
  }
}

// RMS over atoms of the physical force (unrestrained), per system.
__global__ void min_rms_kernel(const MinArgs a, double *out) {
  for (int s = blockIdx.x; s < a.n_sys; s += gridDim.x) {
    const SysInfo &S = a.sys[s];
    double f2 = 0.0, z0 = 0.0, z1 = 0.0;
    for (int i = S.off + threadIdx.x; i < S.off + S.n; i += blockDim.x) {
      const double f[3] = {fix_d(a.fx[i]), fix_d(a.fy[i]), fix_d(a.fz[i])};
      f2 += f[0] * f[0] + f[1] * f[1] + f[2] * f[2];
    }
    block_sum3(f2, z0, z1);
    if (threadIdx.x == 0) out[s] = sqrt(f2 / (double)S.n);
  }
}

// -------------------------------------------------------------------- L-BFGS
//
// Limited-memory BFGS (Nocedal & Wright, Numerical Optimization, alg. 7.4
// and 7.5) per system, the polish stage of the reference (jaxopt LBFGS,
// batched_simulate.py:885-936): history of the last m steps s = x' - x and
// gradient changes y = g' - g, two-loop recursion for d = -H g with
// H0 = (s.y / y.y) I of the newest pair, and a backtracking line search
// (x0 + t d, t from min(1, max_step) shrinking by 0.8: jaxopt's
// max_stepsize clips the step length) accepting the first t with
// E(t) <= E0 + 1e-4 t g.d and |g(t).d| <= 0.9 |g.d|, or the last of the
// trials.  The gradient is minus the force; energies come from the FP64
// energy path.

__device__ __forceinline__ double grad_c(const LbfgsArgs &a, int i, int c) {
  const long long *f = c == 0 ? a.m.fx : (c == 1 ? a.m.fy : a.m.fz);
  const double v = -fix_d(f[i]);
  return isfinite(v) ? v : 0.0;
}

// A block sums one product over the system's 3n coordinates.
__device__ __forceinline__ double sys_dot(const double *u, const double *v, const SysInfo &S, size_t N) {
  double acc = 0.0, z0 = 0.0, z1 = 0.0;
  for (int i = S.off + threadIdx.x; i < S.off + S.n; i += blockDim.x)
    acc += u[i] * v[i] + u[N + i] * v[N + i] + u[2 * N + i] * v[2 * N + i];
  block_sum3(acc, z0, z1);
  return acc;
}

// g <- gradient at the current positions, x0 <- positions, E0 <- energy,
// empty history.
__global__ void lbfgs_begin_kernel(const LbfgsArgs a) {
  const size_t N = a.m.n_total;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < a.m.n_total; i += gridDim.x * blockDim.x) {
    a.g[i] = grad_c(a, i, 0); a.g[N + i] = grad_c(a, i, 1); a.g[2 * N + i] = grad_c(a, i, 2);
    a.x0[i] = a.m.x[i]; a.x0[N + i] = a.m.y[i]; a.x0[2 * N + i] = a.m.z[i];
  }
  for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < a.m.n_sys; s += gridDim.x * blockDim.x) {
    a.e0[s] = a.energy[(size_t)s * PB2_NTERMS + PB2_TERM_TOTAL];
    a.count[s] = 0;
    a.head[s] = 0;
    a.flags[s] = 0;
  }
}

// Two-loop recursion: d = -H g; t = min(1, max_step); gd = g.d.
__global__ void lbfgs_direction_kernel(const LbfgsArgs a) {
  __shared__ double alpha[kLbfgsMaxHist];
  __shared__ double coef;
  const size_t N = a.m.n_total, H = 3 * N;
  for (int s = blockIdx.x; s < a.m.n_sys; s += gridDim.x) {
    const SysInfo &S = a.m.sys[s];
    if (a.flags[s] & kLbfgsDone) continue;  // uniform over the block
    const int cnt = a.count[s], head = a.head[s], m = a.hist;
    for (int i = S.off + threadIdx.x; i < S.off + S.n; i += blockDim.x) {
      a.d[i] = a.g[i]; a.d[N + i] = a.g[N + i]; a.d[2 * N + i] = a.g[2 * N + i];
    }
    __syncthreads();
    for (int k = 0; k < cnt; ++k) {  // newest to oldest
      const int h = (head - 1 - k + m) % m;
      const double *sh = a.hs + h * H, *yh = a.hy + h * H;
      const double al = a.rho[(size_t)h * a.m.n_sys + s] * sys_dot(sh, a.d, S, N);
      if (threadIdx.x == 0) alpha[k] = al;
      for (int i = S.off + threadIdx.x; i < S.off + S.n; i += blockDim.x) {
        a.d[i] -= al * yh[i]; a.d[N + i] -= al * yh[N + i]; a.d[2 * N + i] -= al * yh[2 * N + i];
      }
      __syncthreads();
    }
    double gamma = 1.0;
    if (cnt > 0) {
      const int h = (head - 1 + m) % m;
      const double sy = sys_dot(a.hs + h * H, a.hy + h * H, S, N);
      const double yy = sys_dot(a.hy + h * H, a.hy + h * H, S, N);
      if (yy > 0.0) gamma = sy / yy;
    }
    for (int i = S.off + threadIdx.x; i < S.off + S.n; i += blockDim.x) {
      a.d[i] *= gamma; a.d[N + i] *= gamma; a.d[2 * N + i] *= gamma;
    }
    __syncthreads();
    for (int k = cnt - 1; k >= 0; --k) {  // oldest to newest
      const int h = (head - 1 - k + m) % m;
      const double *sh = a.hs + h * H, *yh = a.hy + h * H;
      const double be = a.rho[(size_t)h * a.m.n_sys + s] * sys_dot(yh, a.d, S, N);
      const double c = alpha[k] - be;
      for (int i = S.off + threadIdx.x; i < S.off + S.n; i += blockDim.x) {
        a.d[i] += c * sh[i]; a.d[N + i] += c * sh[N + i]; a.d[2 * N + i] += c * sh[2 * N + i];
      }
      __syncthreads();
    }
    // d = -r; not a descent direction (or empty history start): steepest descent
    double gd = -sys_dot(a.g, a.d, S, N);
    if (threadIdx.x == 0) coef = (gd < 0.0) ? -1.0 : 0.0;
    __syncthreads();
    const bool sd = coef == 0.0;
    for (int i = S.off + threadIdx.x; i < S.off + S.n; i += blockDim.x) {
      for (int c = 0; c < 3; ++c) {
        double &dv = a.d[c * N + i];
        dv = sd ? -a.g[c * N + i] : -dv;
      }
    }
    __syncthreads();
    if (sd) gd = -sys_dot(a.g, a.g, S, N);
    if (threadIdx.x == 0) {
      if (sd) a.count[s] = 0;
      a.gd[s] = gd;
      a.t[s] = fmin(1.0, a.max_step);
      a.flags[s] &= ~kLbfgsAccepted;
    }
    __syncthreads();
  }
}

// Trial positions x0 + t d for the systems still searching.
__global__ void lbfgs_trial_kernel(const LbfgsArgs a) {
  const size_t N = a.m.n_total;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < a.m.n_total; i += gridDim.x * blockDim.x) {
    const int s = a.m.atom_sys[i];
    if (!(a.flags[s] & (kLbfgsDone | kLbfgsAccepted))) {
      const double t = a.t[s];
      a.m.x[i] = a.x0[i] + t * a.d[i];
      a.m.y[i] = a.x0[N + i] + t * a.d[N + i];
      a.m.z[i] = a.x0[2 * N + i] + t * a.d[2 * N + i];
    }
    a.m.fx[i] = 0; a.m.fy[i] = 0; a.m.fz[i] = 0;
    put_posq(a.m, i);
  }
}

// Line-search test; on acceptance (or the last trial) the history, gradient,
// energy and base positions advance and convergence is checked.
__global__ void lbfgs_check_kernel(const LbfgsArgs a, int last_trial) {
  __shared__ int take;
  const size_t N = a.m.n_total, H = 3 * N;
  for (int s = blockIdx.x; s < a.m.n_sys; s += gridDim.x) {
    const SysInfo &S = a.m.sys[s];
    if (a.flags[s] & (kLbfgsDone | kLbfgsAccepted)) continue;
    const double et = a.energy[(size_t)s * PB2_NTERMS + PB2_TERM_TOTAL];
    double gtd = 0.0, z0 = 0.0, z1 = 0.0;
    for (int i = S.off + threadIdx.x; i < S.off + S.n; i += blockDim.x)
      gtd += grad_c(a, i, 0) * a.d[i] + grad_c(a, i, 1) * a.d[N + i] + grad_c(a, i, 2) * a.d[2 * N + i];
    block_sum3(gtd, z0, z1);
    if (threadIdx.x == 0) {
      const double t = a.t[s], gd = a.gd[s];
      const bool ok = isfinite(et) && et <= a.e0[s] + 1e-4 * t * gd && fabs(gtd) <= 0.9 * fabs(gd);
      take = ok || last_trial;
      if (!take) a.t[s] = t * 0.8;
    }
    __syncthreads();
    if (take) {
      const int m = a.hist, h = a.head[s];
      double *sh = a.hs + h * H, *yh = a.hy + h * H;
      double sy = 0.0, g2 = 0.0, z2 = 0.0;
      for (int i = S.off + threadIdx.x; i < S.off + S.n; i += blockDim.x) {
        const double xn[3] = {a.m.x[i], a.m.y[i], a.m.z[i]};
        for (int c = 0; c < 3; ++c) {
          const size_t k = c * N + i;
          const double gn = grad_c(a, i, c);
          sh[k] = xn[c] - a.x0[k];
          yh[k] = gn - a.g[k];
          sy += sh[k] * yh[k];
          g2 += gn * gn;
          a.g[k] = gn;
          a.x0[k] = xn[c];
        }
      }
      block_sum3(sy, g2, z2);
      if (threadIdx.x == 0) {
        if (sy > 1e-12) {  // keep the pair only with positive curvature
          a.rho[(size_t)h * a.m.n_sys + s] = 1.0 / sy;
          a.head[s] = (h + 1) % m;
          a.count[s] = min(a.count[s] + 1, m);
        }
        a.e0[s] = et;
        a.flags[s] |= kLbfgsAccepted;
        if (sqrt(g2) < a.tol) a.flags[s] |= kLbfgsDone;
      }
    }
    __syncthreads();
  }
}

// ----------------------------------------------------------------- launchers

static int atom_grid(int n) {
  const int g = (n + kMinThreads - 1) / kMinThreads;
  return g < 1 ? 1 : (g > 8192 ? 8192 : g);
}

cudaError_t launch_min(int op, const MinArgs &a, double *out, cudaStream_t st) {
  if (a.n_total <= 0) return cudaSuccess;
  const int ga = atom_grid(a.n_total), gs = a.n_sys;
  switch (op) {
    case kMinOpSd:
      return launch_after(min_sd_kernel, (a.n_blocks + kMinThreads / 32 - 1) / (kMinThreads / 32), kMinThreads, st, a);
    case kMinOpRollback: min_rollback_kernel<<<gs, kMinThreads, 0, st>>>(a); break;
    case kMinOpFireInit: min_fire_init_kernel<<<a.n_chunks, kMinThreads, 0, st>>>(a); break;
    case kMinOpFireMove: return launch_after(min_fire_move_kernel, a.n_chunks, kMinThreads, st, a);
    case kMinOpFireClose: return launch_after(min_fire_close_kernel, a.n_chunks, kMinThreads, st, a);
    case kMinOpFireEnd: min_fire_end_kernel<<<a.n_chunks, kMinThreads, 0, st>>>(a); break;
    case kMinOpTakeBest: min_take_best_kernel<<<ga, kMinThreads, 0, st>>>(a); break;
    case kMinOpRms: min_rms_kernel<<<gs, kMinThreads, 0, st>>>(a, out); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

cudaError_t launch_lbfgs(int op, const LbfgsArgs &a, int last_trial, cudaStream_t st) {
  if (a.m.n_total <= 0) return cudaSuccess;
  const int ga = atom_grid(a.m.n_total), gs = a.m.n_sys;
  switch (op) {
    case kLbfgsOpBegin: lbfgs_begin_kernel<<<ga, kMinThreads, 0, st>>>(a); break;
    case kLbfgsOpDirection: lbfgs_direction_kernel<<<gs, kMinThreads, 0, st>>>(a); break;
    case kLbfgsOpTrial: lbfgs_trial_kernel<<<ga, kMinThreads, 0, st>>>(a); break;
    case kLbfgsOpCheck: lbfgs_check_kernel<<<gs, kMinThreads, 0, st>>>(a, last_trial); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

}  // namespace pb2
