// Shared device-side definitions: batch layout in HBM, fixed-point
// accumulation, and launch helpers.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <tuple>

#include "prolix_b200.h"

namespace pb2 {

constexpr int kWarp = 32;
constexpr unsigned kFull = 0xffffffffu;

// Fixed-point scales.  Forces and dE/dB use 2^32 (range +-2.1e9, resolution
// 2.3e-10); the descreening sums use 2^40 (range +-8.4e6).
constexpr double kForceScale = 4294967296.0;
constexpr double kForceInv = 1.0 / 4294967296.0;
constexpr double kBornScale = 1099511627776.0;
constexpr double kBornInv = 1.0 / 1099511627776.0;
// Energies: 2^24 (range +-5.5e11 kcal/mol, resolution 6e-8 kcal/mol).
constexpr double kEnergyScale = 16777216.0;
constexpr double kEnergyInv = 1.0 / 16777216.0;
constexpr double kFixMax = 9.0e18;  // below 2^63: values beyond are flagged

// OBC II constants (prolix physics/generalized_born.py:18-21) and ACE
// constants (:628-647).
constexpr double kObcAlpha = 1.0, kObcBeta = 0.8, kObcGamma = 4.85;
constexpr double kDielOffset = 0.09;
constexpr double kAceCoeff = 28.3919551, kKjToKcal = 0.239006;

constexpr int kExclPerBlock = 16;  // distinct j-blocks with exclusions per i-block

// Per-system constants, one 168-byte record per system.  Pair kernels see
// positions relative to the system origin (its initial centroid), which keeps
// float32 coordinates small.
struct SysInfo {
  int32_t n;          // atoms
  int32_t off;        // first atom in the batch arrays
  int32_t nblk;       // 32-atom blocks
  int32_t blk_base;   // first block in the batch-wide block numbering
  float pref;         // P = -0.5 k_gb (1/eps_in - 1/eps_out)
  float kcoul;        // direct Coulomb constant
  float lj14, coul14; // 1-4 scales
  float cutoff2;      // LJ / Coulomb cutoff^2; 0: all pairs
  float far2;         // tiles at least this far apart (squared) take the far-field series
                      // of the widest tier; nearer tiles test each pair
  float gb_cutoff2;   // GB / descreening cutoff^2; 0: all pairs
  int32_t clamp;      // neighbour-list clamps on Born radii (GB cutoff set)
  float ro_max;       // largest rho~ = radius - offset of the system
  float born_cut2;    // descreening / chain-rule cutoff^2; 0: all pairs
  float tier2[2][3];  // [value, derivative][tier 0-2]: tiles at least this far apart
                      // (squared) evaluate that tier's series polynomial
  double kcoul_d;     // direct Coulomb constant in double (energy path)
  double pref_d;      // P in double (self / energy terms)
  double dt, half_dt; // tau
  double c1, c2;      // exp(-gamma dt), sqrt(1 - c1^2)
  double kT;
  double skin_half2;  // (skin/2)^2
  double ox, oy, oz;  // origin subtracted before the float32 pair kernels
};
static_assert(sizeof(SysInfo) == 168, "SysInfo layout");

// Work item of the tile kernels: tiles (iblk, jb) for jb in [jb0, jb1) of
// system sys.  Block indices are local to the system.  A tile's 32 steps can
// be shared between items: jb1 = part_code(k0, kn) < 0 stands for steps
// k0 .. k0 + kn - 1 of the one tile (iblk, jb0).
struct TileItem {
  int32_t sys, iblk, jb0, jb1;
};
struct ItemRange {
  int jb0, jb1, k0, kn;
};
__host__ __device__ __forceinline__ int32_t part_code(int k0, int kn) { return ~(k0 | (kn << 5)); }
__host__ __device__ __forceinline__ ItemRange item_range(const TileItem &t) {
  if (t.jb1 >= 0) return ItemRange{t.jb0, t.jb1, 0, 32};
  const int c = ~t.jb1;
  return ItemRange{t.jb0, t.jb0 + 1, c & 31, c >> 5};
}

// One row of the pair list: the even i-block iblk (with iblk + 1) of system
// sys; its live j-blocks are stored from pair_list_j[jbase], room for
// nblk - iblk of them.
struct PlRow {
  int32_t sys, iblk, jbase, pad;
};

// Exclusion masks of one (i-block, j-block) tile: per i row, bit c set when
// (row, col c) is excluded (1-2/1-3) or 1-4 scaled.
struct ExclRow {
  uint32_t excl, s14;
};

// Fixed-point helpers.  Conversion rounds to nearest; out-of-range values
// saturate in the hardware conversion and are flagged by the integrator.
__device__ __forceinline__ long long to_fix(double v, double scale) {
  return __double2ll_rn(v * scale);
}
__device__ __forceinline__ long long to_fix_f(float v, float scale) {
  return __float2ll_rn(v * scale);
}
__device__ __forceinline__ void atomic_add_fix(long long *addr, long long v) {
  atomicAdd(reinterpret_cast<unsigned long long *>(addr), static_cast<unsigned long long>(v));
}

// The bounding box of 32-atom block b, whose atom `lane` is at q (lanes past a
// system's last atom take the block's first).
__device__ __forceinline__ void block_box(float4 *bbox, int b, int lane, bool valid, float4 q) {
  const float4 q0 = make_float4(__shfl_sync(kFull, q.x, 0), __shfl_sync(kFull, q.y, 0),
                                __shfl_sync(kFull, q.z, 0), 0.f);
  if (!valid) q = q0;
  float lo[3] = {q.x, q.y, q.z}, hi[3] = {q.x, q.y, q.z};
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      lo[c] = fminf(lo[c], __shfl_xor_sync(kFull, lo[c], o));
      hi[c] = fmaxf(hi[c], __shfl_xor_sync(kFull, hi[c], o));
    }
  if (lane == 0) {
    bbox[2 * b] = make_float4(lo[0], lo[1], lo[2], 0.f);
    bbox[2 * b + 1] = make_float4(hi[0], hi[1], hi[2], 0.f);
  }
}

// Asynchronous global -> shared copies (cp.async): a thread's copies land in
// groups, in order; cp_async_wait<N>() waits until at most N groups are in
// flight.  Source and destination aligned to the copy's size.
__device__ __forceinline__ void cp_async16(void *smem, const void *gmem) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(sa), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async8(void *smem, const void *gmem) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(sa), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async4(void *smem, const void *gmem) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(sa), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Programmatic dependent launch.  A kernel launched with launch_after may
// start once every block of the launch before it in the stream has called
// pdl_trigger (or ended), while that launch still runs; pdl_wait returns when
// that launch has completed and its writes are visible.  Every kernel
// launched so calls pdl_wait in each of its blocks before the block ends, and
// triggers only after its wait: at most two launches of a chain overlap, and
// a completed launch implies that all before it are complete.  Before its
// wait a kernel reads only what no launch right before it writes.
// A chain of small launches then pays neither their start-up nor their first
// loads one after another (N = 166, before the kernels that share a tile: a
// step 41.2 -> 34.2 us, an energy and force evaluation 89 -> 53 us).
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// The launches of a chain ask for one split of the SM's memory, 72 % of the
// 228 KB as shared memory (the descreening pass's three blocks take 147 KB):
// an SM changes its split only when it is empty, so a kernel whose first
// blocks start beside one with a smaller share keeps that share, and with it
// fewer blocks, until it ends (256 systems of 800 atoms: 497 us per step with
// one split, 516 with each kernel's own, 504 at 100 %).
constexpr unsigned kSmemCarveout = 72;

// A chain of such launches as nodes of a graph instead, while a thread holds a
// chain: each depends on the one before as it would in a stream.  (Capturing a
// stream would do the same, but while any stream of the process is being
// captured, other threads' work on the default stream and waits for the device
// fail.)
struct GraphChain {
  cudaGraph_t graph;
  cudaGraphNode_t last = nullptr;
  cudaError_t add(const void *kernel, int grid, int block, void **params) {
    cudaKernelNodeParams p{};
    p.func = const_cast<void *>(kernel);
    p.gridDim = dim3((unsigned)grid);
    p.blockDim = dim3((unsigned)block);
    p.kernelParams = params;
    cudaGraphNode_t node;
    cudaError_t e = cudaGraphAddKernelNode(&node, graph, nullptr, 0, &p);
    cudaLaunchAttributeValue v{};
    v.sharedMemCarveout = kSmemCarveout;
    if (e == cudaSuccess) e = cudaGraphKernelNodeSetAttribute(node, cudaLaunchAttributePreferredSharedMemoryCarveout, &v);
    if (e == cudaSuccess && last) {
      cudaGraphEdgeData d{};
      d.from_port = cudaGraphKernelNodePortProgrammatic;
      d.type = cudaGraphDependencyTypeProgrammatic;
      e = cudaGraphAddDependencies_v2(graph, &last, &node, &d, 1);
    }
    last = node;
    return e;
  }
};
inline thread_local GraphChain *held_chain = nullptr;

template <class... P, class... A>
inline cudaError_t launch_after(void (*kernel)(P...), int grid, int block, cudaStream_t st, const A &...args) {
  if (held_chain) {
    std::tuple<P...> values{static_cast<P>(args)...};
    return std::apply(
        [&](auto &...v) {
          void *params[] = {const_cast<void *>(static_cast<const void *>(&v))...};
          return held_chain->add(reinterpret_cast<const void *>(kernel), grid, block, params);
        },
        values);
  }
  cudaLaunchAttribute at[2] = {};
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  at[1].id = cudaLaunchAttributePreferredSharedMemoryCarveout;
  at[1].val.sharedMemCarveout = kSmemCarveout;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3((unsigned)block);
  cfg.stream = st;
  cfg.attrs = at;
  cfg.numAttrs = 2;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

}  // namespace pb2
