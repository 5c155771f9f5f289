// Bonded terms: harmonic bonds, Urey-Bradley springs and angles, periodic
// torsions, periodic and harmonic impropers and CMAP, all systems of the
// batch in one launch, one thread per term.
//
// Reference: prolix physics/bonded.py:20-185 (bond via jax_md
// simple_spring_bond, E = k/2 (r - r0)^2, also for the Urey-Bradley 1-3
// springs of system.py:93-95; angle with the 1e-8 guard and the
// +-0.999999 clip; dihedral angle b0 = r_i - r_j, b1 = r_k - r_j,
// b2 = r_l - r_k, phi = atan2(y, x); torsion sum k (1 + cos(n phi - delta)),
// also for periodic impropers; harmonic impropers k d^2 with
// d = ((phi - phi0 + pi) mod 2 pi) - pi)
// and physics/cmap.py:316-376 (bicubic patch evaluation at angles mapped to
// [0, 2 pi); phi from row atoms 0-3, psi from 1-4, system.py:99-102), and the
// explicit 1-4 exception pairs of bonded.py:186-230.
//
// These terms are O(N) and stiff: a bond force k (r - r0) needs r - r0 to
// ~1e-7 A, which float32 coordinates cannot give, so the arithmetic is
// FP64 on the FP64 integrator positions.  Forces go to the same 2^32
// fixed-point accumulators as the pair kernels.
#include "pb2_bonded.cuh"

namespace pb2 {

// With energies wanted, a warp whose terms share one accumulator (nearly
// every warp: terms are ordered by kind and atom) adds their fixed-point sum
// once: the terms of a kind all meet at one address, and 80,000 atomics on
// four addresses took 38 of the kernel's 43 us at N = 20,000.
__global__ void bonded_kernel(const BondedArgs a) {
  // The terms read positions, which the launch before (a pair pass) does not
  // write, and add to accumulators: they need not wait for it.
  const int total = bonded_total(a);
  const int lane = threadIdx.x & 31;
  for (int t0 = blockIdx.x * blockDim.x + threadIdx.x - lane; t0 < total; t0 += gridDim.x * blockDim.x) {
    TermEnergy v{-1, 0};
    if (t0 + lane < total) v = bonded_term(a, t0 + lane);
    if (a.energy_mode) {  // uniform
      int same = 0;
      __match_all_sync(kFull, v.key, &same);
      if (same) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v.e += __shfl_xor_sync(kFull, v.e, o);
      }
      if (v.key >= 0 && (!same || lane == 0)) atomic_add_fix(&a.energy[v.key], v.e);
    }
  }
  pdl_wait();
}

cudaError_t launch_bonded(const BondedArgs &a, int grid_cap, cudaStream_t st) {
  const int total = a.n_bond + a.n_angle + a.n_tors + a.n_cmap + a.n_exc;
  if (total <= 0) return cudaSuccess;
  int grid = (total + 255) / 256;
  if (grid > grid_cap) grid = grid_cap;
  return launch_after(bonded_kernel, grid, 256, st, a);
}

}  // namespace pb2
