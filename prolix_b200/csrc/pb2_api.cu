// C ABI of prolix_b200: context and batch management, force evaluation,
// Langevin runs (replayed as CUDA graphs), state access.
//
// Data layout in HBM (batch order = systems concatenated, atoms in input
// order within a system):
//   FP64 SoA state x, y, z, px, py, pz; int64 fixed-point forces fx, fy, fz;
//   float4 posq (x, y, z relative to the system origin, charge) and
//   float4 par (sigma/2, sqrt(eps), rho~, scaled radius) for the pair
//   kernels; float4 born (B, 1/B, dB/dI); int64 descreening and dE/dB sums;
//   per-system SysInfo records, keys (two buffers), step counters, status.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <map>
#include <memory>
#include <string>
#include <thread>
#include <vector>

#include "pb2_common.cuh"
#include "pb2_kernels.cuh"
#include "pb2_obc_series.cuh"


#include "pb2_internal.h"

using namespace pb2;

int pb2::set_error(pb2_ctx *ctx, int code, const char *msg) { return fail(ctx, code, msg); }

extern "C" int pb2_abi_version(void) { return PB2_ABI_VERSION; }

extern "C" int pb2_ctx_create(int device, pb2_ctx **out) {
  if (!out) return PB2_EINVAL;
  *out = nullptr;
  int n = 0;
  if (cudaGetDeviceCount(&n) != cudaSuccess || n <= device || device < 0) return PB2_ENODEV;
  cudaDeviceProp prop;
  if (cudaGetDeviceProperties(&prop, device) != cudaSuccess) return PB2_ENODEV;
  if (prop.major != 10) return PB2_ENODEV;  // built for sm_100a only
  if (cudaSetDevice(device) != cudaSuccess) return PB2_ENODEV;
  auto *c = new (std::nothrow) pb2_ctx;
  if (!c) return PB2_ENOMEM;
  c->device = device;
  c->sm_count = prop.multiProcessorCount;
  // keep memory freed by dropped batches in this process's pool (the
  // attribute belongs to this process's context and ends with it)
  cudaMemPool_t pool;
  if (cudaDeviceGetDefaultMemPool(&pool, device) == cudaSuccess) {
    uint64_t keep = UINT64_MAX;
    cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
  }
  *out = c;
  return PB2_OK;
}

extern "C" int pb2_ctx_destroy(pb2_ctx *ctx) {
  delete ctx;
  return PB2_OK;
}

extern "C" const char *pb2_last_error(const pb2_ctx *ctx) {
  return ctx ? ctx->err.c_str() : "null context";
}

// ------------------------------------------------------------ batch build

static PairArgs pair_args(pb2_batch *b) {
  PairArgs a;
  a.sys = b->sys;
  a.items = b->items2;
  a.n_items = b->n_items2;
  a.item_count = b->item_count;
  a.terms = b->params.terms;
  a.excl_ent = b->excl_ent;
  a.excl_rows = b->excl_rows;
  a.posq = b->posq;
  a.par = b->par;
  a.born = b->born;
  a.bbox = b->bbox;
  a.cut = b->cut ? 1 : 0;
  a.sched = b->sched;
  a.early = 0;
  a.heads = 0;
  a.born_acc = b->born_acc;
  a.dedb_acc = b->dedb_acc;
  a.fx = b->fx;
  a.fy = b->fy;
  a.fz = b->fz;
  a.energy = b->energy;
  a.pl_ctl = b->pl_on ? b->pl_ctl : nullptr;
  a.pl_items0 = b->pl_items[0];
  a.pl_items1 = b->pl_items[1];
  a.pl_jlist = b->pl_jlist;
  a.bonded = b->bonded;
  a.n_bonded_chunks = 0;
  a.sys_items = nullptr;
  a.sys_done = b->sys_done;
  a.fin = FinalizeArgs{};
  a.pl_sys_items0 = b->pl_sys_items[0];
  a.pl_sys_items1 = b->pl_sys_items[1];
  return a;
}

static PlArgs pl_args(pb2_batch *b) {
  PlArgs a;
  a.sys = b->sys;
  a.rows = b->pl_rows;
  a.n_rows = b->n_pl_rows;
  a.bbox = b->bbox;
  a.posq = b->posq;
  a.ref = b->pl_ref;
  a.jlist = b->pl_jlist;
  a.items0 = b->pl_items[0];
  a.items1 = b->pl_items[1];
  a.sys_items0 = b->pl_sys_items[0];
  a.sys_items1 = b->pl_sys_items[1];
  a.n_sys = b->n_sys;
  a.ctl = b->pl_ctl;
  a.reach2 = b->pl_reach2;
  a.seg = b->params.tile_segment;
  a.retired = b->retired;
  return a;
}

IntArgs int_args_for_nl(pb2_batch *b);

static IntArgs int_args(pb2_batch *b, int parity, int finish_prev) {
  IntArgs a;
  a.sys = b->sys;
  a.atom_sys = b->atom_sys;
  a.user = b->user;
  a.x = b->x; a.y = b->y; a.z = b->z;
  a.px = b->px; a.py = b->py; a.pz = b->pz;
  a.fx = b->fx; a.fy = b->fy; a.fz = b->fz;
  a.mass = b->mass;
  a.sigma = b->sigma;
  a.charge = b->charge;
  a.posq = b->posq;
  a.keys = b->keys;
  a.splits = b->key_splits;
  a.steps = b->steps;
  a.status = b->status;
  a.n_total = b->n_total;
  a.n_sys = b->n_sys;
  a.parity = parity;
  a.finish_prev = finish_prev;
  a.partitionable = b->params.partitionable_keys;
  a.vlimit = b->guard[0];
  a.max_dx = b->guard[1];
  a.force_cap = b->guard[2];
  a.guard_end = b->guard_end;
  a.warn_flags = b->warn_flags;
  a.warn_counts = b->warn_counts;
  a.blk_sys = b->blk_sys;
  a.bbox = b->bbox;
  a.n_blocks = b->n_blocks;
  a.pl_ref = b->pl_on ? b->pl_ref : nullptr;
  a.pl_ctl = b->pl_on ? b->pl_ctl : nullptr;
  a.retired = b->retired;
  a.blk_info = b->blk_info;
  return a;
}

// The force accumulators no longer hold a step's closing force (the state
// was set or moved outside a Langevin step): the next step applies them as
// they are, without the force cap.
static int forces_not_from_step(pb2_batch *b, cudaStream_t st) {
  CUDA_TRY(b->ctx, cudaMemsetAsync(b->guard_end, 0, sizeof(int32_t), st));
  return PB2_OK;
}

IntArgs int_args_for_nl(pb2_batch *b) { return int_args(b, b->key_parity, 0); }

// Spatial order of one system's atoms: recursive bisection of the input
// positions along the longest side of their bounding box, cut at a multiple
// of 32 atoms near the middle, so that every 32-atom block is a compact
// cluster (smaller block boxes: more tile pairs in the far field and beyond
// cutoffs).  Ties go by input index, so the order depends on the positions
// alone.  ord[l] = input index of the atom stored at l.  Non-finite
// positions keep the input order.
static void spatial_order(const double *pos, int n, std::vector<int> &ord) {
  ord.resize(n);
  for (int i = 0; i < n; ++i) ord[i] = i;
  for (int i = 0; i < 3 * n; ++i)
    if (!std::isfinite(pos[i])) return;
  struct At {
    double c[3];
    int i;
  };
  std::vector<At> at(n);  // positions travel with their indices (contiguous)
  for (int i = 0; i < n; ++i) at[i] = At{{pos[3 * i], pos[3 * i + 1], pos[3 * i + 2]}, i};
  std::vector<std::pair<int, int>> todo{{0, n}};
  while (!todo.empty()) {
    const auto [a, e] = todo.back();
    todo.pop_back();
    if (e - a <= 32) continue;
    double lo[3] = {at[a].c[0], at[a].c[1], at[a].c[2]};
    double hi[3] = {lo[0], lo[1], lo[2]};
    for (int k = a; k < e; ++k)
      for (int c = 0; c < 3; ++c) {
        lo[c] = std::min(lo[c], at[k].c[c]);
        hi[c] = std::max(hi[c], at[k].c[c]);
      }
    int ax = 0;
    for (int c = 1; c < 3; ++c)
      if (hi[c] - lo[c] > hi[ax] - lo[ax]) ax = c;
    const int half = (e - a) / 2;
    const int m = a + std::max(32, std::min((half + 16) / 32 * 32, (e - a - 1) / 32 * 32));
    // partition only: the atoms below the cut come first (a strict total
    // order, so the result is the same on every run)
    std::nth_element(at.begin() + a, at.begin() + m, at.begin() + e, [ax](const At &p, const At &q) {
      return p.c[ax] < q.c[ax] || (p.c[ax] == q.c[ax] && p.i < q.i);
    });
    todo.push_back({a, m});
    todo.push_back({m, e});
  }
  for (int l = 0; l < n; ++l) ord[l] = at[l].i;
  // within each block, input order
  for (int a = 0; a < n; a += 32) std::sort(ord.begin() + a, ord.begin() + std::min(n, a + 32));
}

// Stable sort by cost, longest first (a counting sort: a large batch has
// hundreds of thousands of items of a few costs).
static void longest_first(std::vector<TileItem> &items) {
  auto cost = [](const TileItem &t) {
    const ItemRange r = item_range(t);
    return (size_t)(r.jb1 - r.jb0) * r.kn;
  };
  size_t most = 0;
  for (const TileItem &t : items) most = std::max(most, cost(t));
  std::vector<size_t> at(most + 2, 0);  // at[c + 1]: items longer than most - c, then their next place
  for (const TileItem &t : items) ++at[most - cost(t) + 1];
  for (size_t c = 1; c < at.size(); ++c) at[c] += at[c - 1];
  std::vector<TileItem> out(items.size());
  for (const TileItem &t : items) out[at[most - cost(t)]++] = t;
  items.swap(out);
}

// Work items of the two-i-block kernels: even i-blocks ib (with ib + 1)
// against j-blocks [j0, j1), j0 >= ib, of at most seg tiles, longest first.
// Where few items are shorter than seg by nature (long rows), a sixth of each
// row's tiles are items of their own: handed out last, they fill the end of
// the pass, where the last warps' whole segments would leave the others idle
// (20,000 atoms, all pairs, seg 4: 825 -> 806 us per step; a ragged batch has
// its rows' short remainders for that, and 15 % more single tiles cost it 1 %).
static std::vector<TileItem> build_items2(const std::vector<SysInfo> &sinfo, int seg) {
  long long tiles = 0, rest = 0;  // all, and in the rows' last, shorter items
  for (const SysInfo &S : sinfo)
    for (int ib = 0; ib < S.nblk; ib += 2) {
      tiles += S.nblk - ib;
      rest += (S.nblk - ib) % seg;
    }
  const bool singles = 20 * rest < tiles;
  std::vector<TileItem> items;
  for (int s = 0; s < (int)sinfo.size(); ++s) {
    const int nblk = sinfo[s].nblk;
    for (int ib = 0; ib < nblk; ib += 2) {
      const int whole = singles ? ib + (nblk - ib) * 5 / 6 / seg * seg : nblk;  // seg tiles per item up to here
      for (int j0 = ib; j0 < nblk;) {
        const int j1 = std::min(j0 + (j0 < whole ? seg : 1), nblk);
        items.push_back(TileItem{s, ib, j0, j1});
        j0 = j1;
      }
    }
  }
  longest_first(items);
  return items;
}

// Items of `seg` tiles over all rows, tiles(s, ib) in the row of system s that
// begins at i-block ib.
template <class F>
static long long count_items(const std::vector<SysInfo> &sinfo, int seg, F &&tiles) {
  long long items = 0;
  for (int s = 0; s < (int)sinfo.size(); ++s)
    for (int ib = 0; ib < sinfo[s].nblk; ib += 2) items += (tiles(s, ib) + seg - 1) / seg;
  return items;
}

// Default length of those items: the longest (6, 4, 2 or 1 tiles, up to
// `most`) that still gives every resident warp of the force pass a few items,
// so a small batch spreads over the whole GPU.  us per step with 8, 6, 4, 2, 1:
// a ragged batch of 256 systems, all pairs, 1308, 1308, 1325, 1346, 1398;
// 20,000 atoms, all pairs, 817, 807, 806, 826, 891; with a direct cutoff of 9 A
// beside GB over all pairs 885, 868, 867, 884, 953.  Where a reach drops tiles
// whole, an item's cost varies and shorter ones even it out: without a pair
// list at most two tiles (64 systems of 1,500 atoms at 9 A 420, 404, 386, 369,
// 382; 20,000 atoms at 20 A 314, 289, 268, 284, 429).
static int default_segment(const std::vector<SysInfo> &sinfo, int most, int sm_count) {
  for (int cand : {6, 4, 2})
    if (cand <= most && count_items(sinfo, cand, [&](int s, int ib) { return sinfo[s].nblk - ib; }) >= 4LL * sm_count * 16)
      return cand;
  return 1;
}

// The same with a pair list, whose items come in no order: the longest (4, 2
// or 1 tiles) that gives every resident warp eight items of the tiles within
// reach of the initial positions.  us per step with 4, 2, 1 and the items of
// two tiles: 20,000 atoms at 20 A (7,800 items) 232, 201, 193; 40,000 at 20 A
// (16,900) 389, 367, 365; 32 systems of 2,500 atoms at 12 A (18,900) 451, 428,
// 432; 128 ragged systems at 12 A (22,200) 526, 507, 519; 256 of them at 12 A
// (53,900, of four tiles 28,100) 1138, 1144, 1188, at 20 A 1410, 1424, 1482.
static int listed_segment(const std::vector<SysInfo> &sinfo, const std::vector<float4> &posq, float reach2,
                          int sm_count) {
  std::vector<std::vector<int>> live(sinfo.size());
  std::vector<float> box[6];  // block boxes: low x, y, z, high x, y, z
  for (int s = 0; s < (int)sinfo.size(); ++s) {
    const SysInfo &S = sinfo[s];
    for (int c = 0; c < 6; ++c) box[c].assign(S.nblk + 1, c < 3 ? INFINITY : -INFINITY);
    for (int l = 0; l < S.n; ++l) {
      const float4 p = posq[S.off + l];
      const float x[3] = {p.x, p.y, p.z};
      for (int c = 0; c < 3; ++c) {
        box[c][l / 32] = std::min(box[c][l / 32], x[c]);
        box[3 + c][l / 32] = std::max(box[3 + c][l / 32], x[c]);
      }
    }
    const float *lx = box[0].data(), *ly = box[1].data(), *lz = box[2].data();
    const float *hx = box[3].data(), *hy = box[4].data(), *hz = box[5].data();
    auto dist2 = [&](int a, int b) {
      const float dx = std::max(0.f, std::max(lx[a] - hx[b], lx[b] - hx[a]));
      const float dy = std::max(0.f, std::max(ly[a] - hy[b], ly[b] - hy[a]));
      const float dz = std::max(0.f, std::max(lz[a] - hz[b], lz[b] - hz[a]));
      return dx * dx + dy * dy + dz * dz;
    };
    for (int ib = 0; ib < S.nblk; ib += 2) {  // (block nblk is an empty box, out of every reach)
      int n = 1;
      for (int jb = ib + 1; jb < S.nblk; ++jb) n += std::min(dist2(ib, jb), dist2(ib + 1, jb)) < reach2;
      live[s].push_back(n);
    }
  }
  for (int cand : {4, 2})
    if (count_items(sinfo, cand, [&](int s, int ib) { return live[s][ib / 2]; }) >= 8LL * sm_count * 16) return cand;
  return 1;
}

// Items of the FP64 energy kernels: pairs of i-blocks.  Each item's sums are
// rounded to fixed point once, so how a system is cut depends on its own size
// alone and its energies are the same in every batch.  A small system (up to
// 57 blocks, 841 tiles) waits for its longest item: its tiles' 32 steps are
// shared by 8, 4 or 2 items in the descreening pass (1,680 at 28 and at 40
// blocks, 1,682 at 57, of the 2,368 warps resident on 148 SMs), and by a
// thread block's warps in the energy pass (tiles).  A large one takes several
// tiles per item, which load their i atoms once.
struct E64Items {
  std::vector<TileItem> born, pair, tiles;
};
static E64Items build_items_e64(const std::vector<SysInfo> &sinfo) {
  E64Items out;
  for (int s = 0; s < (int)sinfo.size(); ++s) {
    const int nblk = sinfo[s].nblk;
    const int parts = nblk <= 28 ? 8 : nblk <= 40 ? 4 : nblk <= 57 ? 2 : 1;  // 210, 420, 841 tiles
    const int seg = nblk < 160 ? 1 : nblk < 256 ? 2 : nblk < 400 ? 4 : 8;
    const int kn = 32 / parts;
    for (int ib = 0; ib < nblk; ib += 2)
      for (int j0 = ib; j0 < nblk; j0 += seg) {
        const TileItem whole{s, ib, j0, std::min(j0 + seg, nblk)};
        for (int p = 0; p < parts; ++p)
          out.born.push_back(parts > 1 ? TileItem{s, ib, j0, part_code(p * kn, kn)} : whole);
        (parts > 1 ? out.tiles : out.pair).push_back(whole);
      }
  }
  longest_first(out.born);
  longest_first(out.pair);
  return out;
}

// Work items of the four-block force kernel: i-blocks ib, ib % 4 == 0 (with
// ib + 1 .. ib + 3), against j-blocks [j0, j1), j0 >= ib; sorted by cost.
static std::vector<TileItem> build_items4(const std::vector<SysInfo> &sinfo, int seg) {
  std::vector<TileItem> items;
  for (int s = 0; s < (int)sinfo.size(); ++s) {
    const int nblk = sinfo[s].nblk;
    for (int ib = 0; ib < nblk; ib += 4)
      for (int j0 = ib; j0 < nblk; j0 += seg) items.push_back(TileItem{s, ib, j0, std::min(j0 + seg, nblk)});
  }
  longest_first(items);
  return items;
}

static void set_force4_grid(pb2_batch *b) {
  const int cap = force4_occupancy(b->cut, b->shape4) * b->ctx->sm_count;
  int t = 0, m = 0;
  force4_shape(b->shape4, &t, &m);
  const int w = t / 32;
  b->grid4 = std::max(1, std::min(cap, (b->n_items4 + w - 1) / w));
}

// Grid of pair pass p for its block shape: one resident wave, no more thread
// blocks than units of work (items; for the chain pass the bonded chunks
// too, for the descreening pass the finalize chunks), of which few spread
// over the SMs.
static void set_pair_grid(pb2_batch *b, int p) {
  const int cap = tile_kernel_occupancy(p, b->cut, b->shape[p]) * b->ctx->sm_count;
  const BondedArgs &ba = b->bonded;
  const int bonded = ba.n_bond + ba.n_angle + ba.n_tors + ba.n_cmap + ba.n_exc;
  const int chunks = (bonded + kBondedChunk - 1) / kBondedChunk;
  const int units = b->n_units2 + (p == PASS_CHAIN ? chunks : p == PASS_BORN ? b->n_blocks : 0);
  b->grid_pair[p] = std::max(1, std::min(cap, units));
}

// Teams (a thread block of 8 or 4 warps per tile) for a batch of so few tiles
// that with one warp each the chip waits for single warps' steps.  The lines
// lie where the step times cross (us per step, one system, all pairs; none /
// 8 warps / 4 warps): 896 atoms, 210 tiles 36.9 / 22.5 / 24.9; 1,200, 380
// tiles 38.8 / 31.5 / 28.0; 1,500, 576 tiles 40.1 / 36.0 / 30.6; 1,800, 841
// tiles 40.1 / 45.7 / 41.8.  Never with a pair list (its smallest batch, one
// system of 64 blocks, has 1,056 tiles): the team kernels have no list.
static void set_team(pb2_batch *b, int seg) {
  const int n = b->n_units2;
  b->team = seg != 1 || b->pl_on ? 0 : n <= 296 ? 8 : n <= 640 ? 4 : 0;
  if (!b->team) return;
  const BondedArgs &ba = b->bonded;
  const int bonded = ba.n_bond + ba.n_angle + ba.n_tors + ba.n_cmap + ba.n_exc;
  for (int p = 0; p < 3; ++p) {
    const int units = n + (p == PASS_CHAIN ? (bonded + kBondedChunk * b->team - 1) / (kBondedChunk * b->team) : 0);
    b->grid_team[p] = std::max(1, std::min(team_occupancy(p, b->team, b->cut) * b->ctx->sm_count, units));
  }
}

// (Re)build the pair kernels' two-i-block work list and their grids (one
// resident wave each; warps take items dynamically).  The kernels read the
// live list: the full one without the items of retired systems.  With a pair
// list its items take their place, and these lists stay empty: at one tile
// per item they would hold 48 B per tile beside the list's 36 (40,000 atoms
// at 12 A: 1,335 B per atom with them, 866 without), and retiring a system
// would compact them.
static int setup_items2(pb2_batch *b, int seg) {
  pb2_ctx *ctx = b->ctx;
  std::vector<TileItem> items;
  if (!b->pl_on) items = build_items2(b->sys_host, seg);
  b->n_units2 = b->pl_on ? (int)count_items(b->sys_host, seg, [&](int s, int ib) { return b->sys_host[s].nblk - ib; })
                         : (int)items.size();
  b->dev.release(b->items2);
  b->dev.release(b->items2_all);
  b->items2 = b->dev.alloc<TileItem>(std::max<size_t>(items.size(), 1));
  b->items2_all = b->dev.alloc<TileItem>(std::max<size_t>(items.size(), 1));
  if (!b->items2 || !b->items2_all) return fail(ctx, PB2_ENOMEM, "work-item allocation failed");
  if (!items.empty())
    CUDA_TRY(ctx, cudaMemcpy(b->items2_all, items.data(), items.size() * sizeof(TileItem), cudaMemcpyHostToDevice));
  b->n_items2 = (int)items.size();
  if (!b->retired) {
    b->retired = b->dev.alloc<int8_t>(b->n_sys);
    b->item_count = b->dev.alloc<int32_t>(1);
    if (!b->retired || !b->item_count) return fail(ctx, PB2_ENOMEM, "work-item allocation failed");
    CUDA_TRY(ctx, cudaMemset(b->retired, 0, b->n_sys));
    b->retired_host.assign(b->n_sys, 0);
  }
  CUDA_TRY(ctx, launch_retire(-1, b->retired, b->items2_all, b->n_items2, b->items2, b->item_count, nullptr, nullptr));
  {
    std::vector<TileItem> items4;
    if (!b->pl_on) items4 = build_items4(b->sys_host, seg);
    b->dev.release(b->items4);
    b->dev.release(b->items4_all);
    b->items4 = b->dev.alloc<TileItem>(std::max<size_t>(items4.size(), 1));
    b->items4_all = b->dev.alloc<TileItem>(std::max<size_t>(items4.size(), 1));
    if (!b->item_count4) b->item_count4 = b->dev.alloc<int32_t>(1);
    if (!b->items4 || !b->items4_all || !b->item_count4) return fail(ctx, PB2_ENOMEM, "work-item allocation failed");
    if (!items4.empty())
      CUDA_TRY(ctx, cudaMemcpy(b->items4_all, items4.data(), items4.size() * sizeof(TileItem), cudaMemcpyHostToDevice));
    b->n_items4 = (int)items4.size();
    CUDA_TRY(ctx, launch_retire(-1, b->retired, b->items4_all, b->n_items4, b->items4, b->item_count4, nullptr, nullptr));
  }
  CUDA_TRY(ctx, cudaDeviceSynchronize());
  std::vector<int32_t> per_sys(b->n_sys, 0);
  for (const TileItem &t : items) ++per_sys[t.sys];
  if (!b->sys_items) {
    b->sys_items = b->dev.alloc<int32_t>(b->n_sys);
    b->sys_done = b->dev.alloc<int32_t>(b->n_sys);
    b->sys_fin = b->dev.alloc<int32_t>(b->n_sys);
    if (!b->sys_items || !b->sys_done || !b->sys_fin) return fail(ctx, PB2_ENOMEM, "work-item allocation failed");
    CUDA_TRY(ctx, cudaMemset(b->sys_done, 0, b->n_sys * sizeof(int32_t)));
    CUDA_TRY(ctx, cudaMemset(b->sys_fin, 0, b->n_sys * sizeof(int32_t)));
  }
  CUDA_TRY(ctx, cudaMemcpy(b->sys_items, per_sys.data(), per_sys.size() * sizeof(int32_t), cudaMemcpyHostToDevice));
  b->sys_items_host = per_sys;
  for (int p = 0; p < 3; ++p) set_pair_grid(b, p);
  set_team(b, seg);
  set_force4_grid(b);
  return PB2_OK;
}

// The pair list of a cutoff run (pb2_pairlist.cu): rows (one per pair of
// i-blocks), room for every j-block of each row, two item buffers sized for
// the segment, and the control words, with the rebuild flag set so that the
// first force evaluation builds it.
static int setup_pair_list(pb2_batch *b, int seg) {
  pb2_ctx *ctx = b->ctx;
  if (!b->pl_on) return PB2_OK;
  std::vector<PlRow> rows;
  size_t jcap = 0, icap = 0;
  for (int s = 0; s < b->n_sys; ++s) {
    const int nblk = b->sys_host[s].nblk;
    for (int ib = 0; ib < nblk; ib += 2) {
      rows.push_back(PlRow{s, ib, (int32_t)jcap, 0});
      jcap += (size_t)(nblk - ib);
      icap += (size_t)((nblk - ib + seg - 1) / seg);
    }
  }
  if (jcap > (size_t)INT32_MAX) return fail(ctx, PB2_EINVAL, "pair list too large");
  Dev &D = b->dev;
  if (!b->pl_rows) {
    b->pl_rows = D.alloc<PlRow>(rows.size());
    b->pl_jlist = D.alloc<int32_t>(std::max<size_t>(jcap, 1));
    b->pl_ctl = D.alloc<int32_t>(PL_WORDS);
    b->pl_ref = D.alloc<float4>(b->n_total);
    b->pl_sys_items[0] = D.alloc<int32_t>(b->n_sys);
    b->pl_sys_items[1] = D.alloc<int32_t>(b->n_sys);
    if (!b->pl_rows || !b->pl_jlist || !b->pl_ctl || !b->pl_ref || !b->pl_sys_items[0] ||
        !b->pl_sys_items[1])
      return fail(ctx, PB2_ENOMEM, "pair-list allocation failed");
    CUDA_TRY(ctx, cudaMemcpy(b->pl_rows, rows.data(), rows.size() * sizeof(PlRow), cudaMemcpyHostToDevice));
    b->n_pl_rows = (int)rows.size();
  }
  if (icap > b->pl_item_cap) {
    for (auto &p : b->pl_items) {
      D.release(p);
      p = D.alloc<TileItem>(icap);
      if (!p) return fail(ctx, PB2_ENOMEM, "pair-list item allocation failed");
    }
    b->pl_item_cap = icap;
  }
  const int32_t ctl[PL_WORDS] = {1, 0, 0, 0, 0, 0, 0, 0};  // dirty: rebuild at the next evaluation
  CUDA_TRY(ctx, cudaMemcpy(b->pl_ctl, ctl, sizeof ctl, cudaMemcpyHostToDevice));
  for (auto p : b->pl_sys_items) CUDA_TRY(ctx, cudaMemset(p, 0, b->n_sys * sizeof(int32_t)));
  b->grid_pl = std::max(1, std::min(8 * ctx->sm_count, (b->n_pl_rows + 7) / 8));
  return PB2_OK;
}

static int validate(pb2_ctx *ctx, const pb2_system_desc &d, int s) {
  char buf[256];
  auto bad = [&](const char *what) {
    snprintf(buf, sizeof buf, "system %d: %s", s, what);
    return fail(ctx, PB2_EINVAL, buf);
  };
  if (d.n_atoms <= 0) return bad("n_atoms must be > 0");
  if (!d.positions || !d.charges || !d.sigmas || !d.epsilons || !d.radii || !d.scaled_radii ||
      !d.masses)
    return bad("per-atom arrays must not be NULL");
  const int n = d.n_atoms;
  for (int i = 0; i < n; ++i) {
    if (!(d.masses[i] > 0.0)) return bad("masses must be > 0");
    if (!(d.radii[i] > 0.0)) return bad("radii must be > 0");
  }
  auto check_idx = [&](const int32_t *idx, int64_t count, const char *what) -> bool {
    for (int64_t k = 0; k < count; ++k)
      if (idx[k] < 0 || idx[k] >= n) {
        snprintf(buf, sizeof buf, "system %d: %s index %d out of range", s, what, idx[k]);
        return false;
      }
    return true;
  };
  if (d.n_bonds < 0 || d.n_angles < 0 || d.n_torsions < 0 || d.n_cmap < 0 || d.n_excl < 0 ||
      d.n_exceptions < 0 || d.n_impropers < 0 || d.n_urey_bradley < 0)
    return bad("negative term count");
  if (d.n_impropers && (!d.impropers || !d.improper_params || d.n_improper_terms <= 0 ||
                        (d.improper_form != 0 && d.improper_form != 1)))
    return bad("improper arrays missing or improper_form not 0 (periodic) / 1 (harmonic)");
  if (d.n_urey_bradley && (!d.urey_bradley_bonds || !d.urey_bradley_params))
    return bad("Urey-Bradley arrays missing");
  if (d.n_bonds && (!d.bonds || !d.bond_params)) return bad("bond arrays missing");
  if (d.n_angles && (!d.angles || !d.angle_params)) return bad("angle arrays missing");
  if (d.n_torsions && (!d.torsions || !d.torsion_params || d.n_torsion_terms <= 0))
    return bad("torsion arrays missing");
  if (d.n_cmap && (!d.cmap_rows || !d.cmap_map || !d.cmap_coeffs || d.n_cmap_maps <= 0 ||
                   d.cmap_grid <= 0))
    return bad("cmap arrays missing");
  if (d.n_excl && (!d.excl_pairs || !d.excl_kind)) return bad("exclusion arrays missing");
  if (d.n_exceptions && (!d.exception_pairs || !d.exception_params)) return bad("exception arrays missing");
  if (!check_idx(d.bonds, 2LL * d.n_bonds, "bond") ||
      !check_idx(d.angles, 3LL * d.n_angles, "angle") ||
      !check_idx(d.torsions, 4LL * d.n_torsions, "torsion") ||
      !check_idx(d.cmap_rows, 5LL * d.n_cmap, "cmap") ||
      !check_idx(d.excl_pairs, 2LL * d.n_excl, "exclusion") ||
      !check_idx(d.exception_pairs, 2LL * d.n_exceptions, "exception") ||
      !check_idx(d.impropers, 4LL * d.n_impropers, "improper") ||
      !check_idx(d.urey_bradley_bonds, 2LL * d.n_urey_bradley, "Urey-Bradley"))
    return fail(ctx, PB2_EINVAL, buf);
  for (int k = 0; k < d.n_cmap; ++k)
    if (d.cmap_map[k] < 0 || d.cmap_map[k] >= d.n_cmap_maps) return bad("cmap map index out of range");
  for (int k = 0; k < d.n_excl; ++k) {
    if (d.excl_pairs[2 * k] >= d.excl_pairs[2 * k + 1]) return bad("exclusion pairs need i < j");
    if (d.excl_kind[k] != 0 && d.excl_kind[k] != 1) return bad("exclusion kind must be 0 or 1");
  }
  if (!(d.dt > 0.0) || !(d.kT >= 0.0) || !(d.gamma >= 0.0)) return bad("dt > 0, kT >= 0, gamma >= 0");
  if (!(d.eps_in > 0.0) || !(d.eps_out > 0.0)) return bad("dielectrics must be > 0");
  return PB2_OK;
}

template <class T>
static int upload(pb2_ctx *ctx, T *dst, const std::vector<T> &src) {
  if (src.empty()) return PB2_OK;
  CUDA_TRY(ctx, cudaMemcpy(dst, src.data(), src.size() * sizeof(T), cudaMemcpyHostToDevice));
  return PB2_OK;
}

extern "C" int pb2_batch_create(pb2_ctx *ctx, int32_t n_systems, const pb2_system_desc *systems,
                                const pb2_run_params *params, pb2_batch **out) {
  if (!ctx || !out || !systems || !params || n_systems <= 0) return fail(ctx, PB2_EINVAL, "bad arguments");
  *out = nullptr;
  CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  for (int s = 0; s < n_systems; ++s) {
    int rc = validate(ctx, systems[s], s);
    if (rc) return rc;
  }
  std::unique_ptr<pb2_batch> b(new (std::nothrow) pb2_batch);
  if (!b) return fail(ctx, PB2_ENOMEM, "host allocation");
  b->ctx = ctx;
  b->params = *params;
  if (b->params.graph_chunk <= 0) b->params.graph_chunk = 50;
  b->n_sys = n_systems;
  const bool cutoff_mode = params->cutoff > 0.0;
  const double gb_cut = params->gb_cutoff < 0.0 ? (cutoff_mode ? params->cutoff : 0.0) : params->gb_cutoff;
  const bool gb_cut_mode = gb_cut > 0.0;
  const double born_cut = params->born_cutoff > 0.0 ? params->born_cutoff : gb_cut;
  const bool born_mode = born_cut > 0.0;  // Born radii from a cutoff: its clamps apply

  // --- stored atom order of each system (spatial unless asked to keep the
  // input order), computed for all systems at once on the host's cores
  std::vector<std::vector<int>> orders(n_systems);
  {
    auto work = [&](int s) {
      std::vector<int> &ord = orders[s];
      const int n = systems[s].n_atoms;
      if (params->keep_atom_order) {
        ord.resize(n);
        for (int i = 0; i < n; ++i) ord[i] = i;
      } else {
        spatial_order(systems[s].positions, n, ord);
      }
    };
    const int n_threads =
        std::max(1, std::min<int>(n_systems, std::min(16u, std::max(1u, std::thread::hardware_concurrency()))));
    std::atomic<int> next{0};
    auto worker = [&]() {
      for (int s; (s = next.fetch_add(1)) < n_systems;) work(s);
    };
    std::vector<std::thread> pool;
    for (int t = 1; t < n_threads; ++t) pool.emplace_back(worker);
    worker();
    for (auto &t : pool) t.join();
  }

  // --- per-atom host arrays
  int64_t total = 0;
  int blocks_total = 0;
  for (int s = 0; s < n_systems; ++s) {
    b->off.push_back((int)total);
    b->nat.push_back(systems[s].n_atoms);
    total += systems[s].n_atoms;
    blocks_total += (systems[s].n_atoms + 31) / 32;
  }
  if (total > (1LL << 30)) return fail(ctx, PB2_EINVAL, "too many atoms");
  const int N = (int)total;
  b->n_total = N;
  std::vector<double> hx(N), hy(N), hz(N), hm(N), hsig(N), hq(N), hrad(N);
  std::vector<float4> hposq(N), hpar(N);
  std::vector<double> hhs(N), hse(N), hro(N), hsr(N);
  std::vector<int32_t> hsys(N);
  b->user_host.resize(N);
  b->dev_host.resize(N);
  std::vector<std::vector<int>> inv_all(n_systems);  // per system: input index -> stored index
  std::vector<SysInfo> sinfo(n_systems);
  std::vector<uint32_t> hkeys(4 * (size_t)n_systems, 0u);
  std::vector<int2> hent((size_t)blocks_total * kExclPerBlock, make_int2(-1, -1));
  std::vector<int32_t> hblk_sys(blocks_total);
  std::vector<int4> hblk_info(blocks_total);
  std::vector<ExclRow> hrows;
  E64Items he64;
  int blk_base = 0;
  for (int s = 0; s < n_systems; ++s) {
    const pb2_system_desc &d = systems[s];
    const int n = d.n_atoms, o = b->off[s];
    SysInfo &S = sinfo[s];
    memset(&S, 0, sizeof S);
    S.n = n;
    S.off = o;
    S.nblk = (n + 31) / 32;
    S.blk_base = blk_base;
    const double pref = -0.5 * d.k_gb * (1.0 / d.eps_in - 1.0 / d.eps_out);
    S.pref = (float)pref;
    S.pref_d = pref;
    S.kcoul = (float)d.k_coulomb;
    S.kcoul_d = d.k_coulomb;
    S.lj14 = (float)d.lj14_scale;
    S.coul14 = (float)d.coul14_scale;
    S.cutoff2 = cutoff_mode ? (float)(params->cutoff * params->cutoff) : 0.f;
    S.gb_cutoff2 = gb_cut_mode ? (float)(gb_cut * gb_cut) : 0.f;
    S.born_cut2 = born_mode ? (float)(born_cut * born_cut) : 0.f;
    S.clamp = born_mode ? 1 : 0;
    b->gamma_host.push_back(d.gamma);
    S.dt = d.dt;
    S.half_dt = 0.5 * d.dt;
    S.c1 = std::exp(-d.gamma * d.dt);
    S.c2 = std::sqrt(1.0 - S.c1 * S.c1);
    S.kT = d.kT;
    S.skin_half2 = 0.25 * params->skin * params->skin;
    double cx = 0, cy = 0, cz = 0;
    for (int i = 0; i < n; ++i) {
      cx += d.positions[3 * i];
      cy += d.positions[3 * i + 1];
      cz += d.positions[3 * i + 2];
    }
    S.ox = std::round(cx / n);
    S.oy = std::round(cy / n);
    S.oz = std::round(cz / n);
    if (d.use_origin) {
      S.ox = d.origin[0];
      S.oy = d.origin[1];
      S.oz = d.origin[2];
    }
    // the stored atom order computed above, or the input order when that
    // one gives an i-block exclusion partners in more j-blocks than the
    // exclusion table holds
    std::vector<int> ord;
    std::vector<int> &inv = inv_all[s];
    inv.resize(n);
    const size_t rows_before = hrows.size();
    int2 *ent_sys = &hent[(size_t)blk_base * kExclPerBlock];
    auto build_excl = [&]() -> int {  // -1: fits; else the i-block that overflows
      for (size_t e = 0; e < (size_t)S.nblk * kExclPerBlock; ++e) ent_sys[e] = make_int2(-1, -1);
      hrows.resize(rows_before);
      for (int k = 0; k < d.n_excl; ++k) {
        const int p = inv[d.excl_pairs[2 * k]], q = inv[d.excl_pairs[2 * k + 1]];
        const int i = std::min(p, q), j = std::max(p, q);
        const int ib = i >> 5, jb = j >> 5;
        int2 *ent = ent_sys + (size_t)ib * kExclPerBlock;
        int slot = -1;
        for (int e = 0; e < kExclPerBlock; ++e) {
          if (ent[e].x == jb) { slot = e; break; }
          if (ent[e].x < 0) {
            ent[e] = make_int2(jb, (int)hrows.size());
            hrows.resize(hrows.size() + 32, ExclRow{0u, 0u});
            slot = e;
            break;
          }
        }
        if (slot < 0) return ib;
        ExclRow &row = hrows[ent[slot].y + (i & 31)];
        if (d.excl_kind[k] == 0) row.excl |= 1u << (j & 31);
        else row.s14 |= 1u << (j & 31);
      }
      return -1;
    };
    ord.swap(orders[s]);
    for (int l = 0; l < n; ++l) inv[ord[l]] = l;
    int over = build_excl();
    if (over >= 0 && !params->keep_atom_order) {
      for (int l = 0; l < n; ++l) ord[l] = inv[l] = l;
      over = build_excl();
    }
    if (over >= 0) {
      char buf[200];
      snprintf(buf, sizeof buf,
               "system %d: atoms %d..%d have exclusion partners in more than %d 32-atom blocks",
               s, over * 32, over * 32 + 31, kExclPerBlock);
      return fail(ctx, PB2_EINVAL, buf);
    }
    for (int l = 0; l < n; ++l) {
      const int i = ord[l];
      const int g = o + l;
      b->user_host[g] = o + i;
      b->dev_host[o + i] = g;
      hx[g] = d.positions[3 * i];
      hy[g] = d.positions[3 * i + 1];
      hz[g] = d.positions[3 * i + 2];
      hm[g] = d.masses[i];
      hsig[g] = S.c2 * std::sqrt(d.masses[i] * d.kT);
      hq[g] = d.charges[i];
      hrad[g] = d.radii[i];
      hsys[g] = s;
      hposq[g] = make_float4((float)(hx[g] - S.ox), (float)(hy[g] - S.oy), (float)(hz[g] - S.oz),
                             (float)d.charges[i]);
      double ro = d.radii[i] - kDielOffset;
      if (born_mode) ro = std::max(std::max(d.radii[i], 1e-6) - kDielOffset, 1e-4);
      hhs[g] = 0.5 * std::max(d.sigmas[i], 1e-6);
      hse[g] = std::sqrt(std::max(d.epsilons[i], 0.0));
      hro[g] = ro;
      hsr[g] = d.scaled_radii[i];
      // float copy for the pair kernels: sqrt(24 eps), so eps_ij * 24 is one product
      hpar[g] = make_float4((float)hhs[g], (float)(hse[g] * std::sqrt(24.0)), (float)ro, (float)hsr[g]);
    }
    {  // far-field tiles: every pair has r - s >= rho~ and (s/r)^2 <= u_K
      float smax = 0.f, romax = 0.f;
      for (int i = 0; i < n; ++i) {
        smax = std::max(smax, hpar[o + i].w);
        romax = std::max(romax, hpar[o + i].z);
      }
      auto bound2 = [&](double u) {
        const double r = 1.001 * std::max((double)smax / std::sqrt(u), (double)smax + (double)romax);
        return (float)(r * r);
      };
      S.far2 = bound2(kValueTierU[3]);
      for (int t = 0; t < 3; ++t) {
        S.tier2[0][t] = bound2(kValueTierU[t]);
        S.tier2[1][t] = bound2(kDerivTierU[t]);
      }
      S.ro_max = romax;
    }
    for (int bk = 0; bk < S.nblk; ++bk) {
      hblk_sys[blk_base + bk] = s;
      hblk_info[blk_base + bk] = make_int4(s, S.off + 32 * bk, std::min(32, S.n - 32 * bk), 0);
    }
    hkeys[2 * (size_t)s] = d.key[0];
    hkeys[2 * (size_t)s + 1] = d.key[1];
    blk_base += S.nblk;
  }
  {
    he64 = build_items_e64(sinfo);
    b->n_items = (int)he64.born.size();
    b->n_items_e = (int)he64.pair.size();
    b->n_tiles_e = (int)he64.tiles.size();
    const int n[2] = {b->n_items, b->n_items_e};
    for (int p = 0; p < 2; ++p)
      b->grid_e64[p] = std::max(1, std::min(energy64_occupancy(p) * ctx->sm_count, n[p]));
    b->grid_tiles_e = std::max(1, std::min(energy64_tile_occupancy() * ctx->sm_count, b->n_tiles_e));
  }
  b->sys_host = sinfo;

  // --- bonded tables (global atom indices)
  std::vector<int2> bidx, uidx;  // bonds, Urey-Bradley springs
  std::vector<double2> bpar, upar;
  std::vector<int4> aidx;
  std::vector<double2> apar;
  std::vector<int4> tidx;
  std::vector<double4> tpar;
  std::vector<int32_t> cidx;
  std::vector<double> ccoef;
  std::vector<int32_t> cgrid;
  std::vector<int64_t> cmoff;
  std::vector<int2> eidx;
  std::vector<double4> epar;
  for (int s = 0; s < n_systems; ++s) {
    const pb2_system_desc &d = systems[s];
    const int o = b->off[s];
    const std::vector<int> &inv = inv_all[s];
    auto at = [&](int32_t i) { return o + inv[i]; };  // stored batch index of input atom i
    for (int k = 0; k < d.n_bonds; ++k) {
      bidx.push_back(make_int2(at(d.bonds[2 * k]), at(d.bonds[2 * k + 1])));
      bpar.push_back(make_double2(d.bond_params[2 * k], d.bond_params[2 * k + 1]));
    }
    for (int k = 0; k < d.n_angles; ++k) {
      aidx.push_back(make_int4(at(d.angles[3 * k]), at(d.angles[3 * k + 1]), at(d.angles[3 * k + 2]), 0));
      apar.push_back(make_double2(d.angle_params[2 * k], d.angle_params[2 * k + 1]));
    }
    for (int k = 0; k < d.n_torsions; ++k)
      for (int t = 0; t < d.n_torsion_terms; ++t) {
        const double *p = d.torsion_params + ((size_t)k * d.n_torsion_terms + t) * 3;
        tidx.push_back(make_int4(at(d.torsions[4 * k]), at(d.torsions[4 * k + 1]),
                                 at(d.torsions[4 * k + 2]), at(d.torsions[4 * k + 3])));
        tpar.push_back(make_double4(p[0], p[1], p[2], kTorsProper));
      }
    for (int k = 0; k < d.n_impropers; ++k)
      for (int t = 0; t < d.n_improper_terms; ++t) {
        tidx.push_back(make_int4(at(d.impropers[4 * k]), at(d.impropers[4 * k + 1]),
                                 at(d.impropers[4 * k + 2]), at(d.impropers[4 * k + 3])));
        if (d.improper_form == 1) {
          const double *p = d.improper_params + ((size_t)k * d.n_improper_terms + t) * 2;
          tpar.push_back(make_double4(p[0], p[1], 0.0, kTorsHarmonic));
        } else {
          const double *p = d.improper_params + ((size_t)k * d.n_improper_terms + t) * 3;
          tpar.push_back(make_double4(p[0], p[1], p[2], kTorsImproper));
        }
      }
    for (int k = 0; k < d.n_urey_bradley; ++k) {
      uidx.push_back(make_int2(at(d.urey_bradley_bonds[2 * k]), at(d.urey_bradley_bonds[2 * k + 1])));
      upar.push_back(make_double2(d.urey_bradley_params[2 * k], d.urey_bradley_params[2 * k + 1]));
    }
    const int map_base = (int)cgrid.size();
    const size_t per_map = (size_t)d.cmap_grid * d.cmap_grid * 16;
    for (int m = 0; m < d.n_cmap_maps && d.n_cmap > 0; ++m) {
      cgrid.push_back(d.cmap_grid);
      cmoff.push_back((int64_t)ccoef.size());
      ccoef.insert(ccoef.end(), d.cmap_coeffs + m * per_map, d.cmap_coeffs + (m + 1) * per_map);
    }
    for (int k = 0; k < d.n_cmap; ++k) {
      for (int c = 0; c < 5; ++c) cidx.push_back(at(d.cmap_rows[5 * k + c]));
      cidx.push_back(map_base + d.cmap_map[k]);
    }
    for (int k = 0; k < d.n_exceptions; ++k) {
      const double *p = d.exception_params + 3 * (size_t)k;
      eidx.push_back(make_int2(at(d.exception_pairs[2 * k]), at(d.exception_pairs[2 * k + 1])));
      epar.push_back(make_double4(d.k_coulomb * p[0], p[1], p[2], 0.0));
    }
  }

  // terms in order of their (central) atom: with atoms in spatial order, the
  // threads of a warp then read and update nearby atoms
  auto by_atom = [N](auto &idx, auto &par, auto key) {  // stable counting sort by key in [0, N)
    std::vector<int> start(N + 1, 0);
    for (const auto &t : idx) ++start[key(t) + 1];
    for (int a = 0; a < N; ++a) start[a + 1] += start[a];
    auto idx2 = idx;
    auto par2 = par;
    for (size_t k = 0; k < idx.size(); ++k) {
      const int dst = start[key(idx[k])]++;
      idx2[dst] = idx[k];
      par2[dst] = par[k];
    }
    idx.swap(idx2);
    par.swap(par2);
  };
  by_atom(bidx, bpar, [](const int2 &t) { return std::min(t.x, t.y); });
  by_atom(uidx, upar, [](const int2 &t) { return std::min(t.x, t.y); });
  const int n_bond_plain = (int)bidx.size();  // Urey-Bradley springs follow the bonds
  bidx.insert(bidx.end(), uidx.begin(), uidx.end());
  bpar.insert(bpar.end(), upar.begin(), upar.end());
  by_atom(aidx, apar, [](const int4 &t) { return t.y; });
  by_atom(tidx, tpar, [](const int4 &t) { return std::min(t.y, t.z); });
  by_atom(eidx, epar, [](const int2 &t) { return std::min(t.x, t.y); });

  // --- device allocation
  Dev &D = b->dev;
  b->sys = D.alloc<SysInfo>(n_systems);
  b->atom_sys = D.alloc<int32_t>(N);
  b->x = D.alloc<double>(N); b->y = D.alloc<double>(N); b->z = D.alloc<double>(N);
  b->px = D.alloc<double>(N); b->py = D.alloc<double>(N); b->pz = D.alloc<double>(N);
  b->fx = D.alloc<long long>(N); b->fy = D.alloc<long long>(N); b->fz = D.alloc<long long>(N);
  b->mass = D.alloc<double>(N);
  b->sigma = D.alloc<double>(N);
  b->charge = D.alloc<double>(N);
  b->radius = D.alloc<double>(N);
  b->posq = D.alloc<float4>(N);
  b->par = D.alloc<float4>(N);
  b->born = D.alloc<float4>(N);
  b->bbox = D.alloc<float4>(2 * (size_t)blocks_total);
  b->sched = D.alloc<int32_t>(kSchedWords);
  b->blk_sys = D.alloc<int32_t>(blocks_total);
  b->blk_info = D.alloc<int4>(blocks_total);
  b->n_blocks = blocks_total;
  b->cut = cutoff_mode || gb_cut_mode || born_mode;
  {
    // bounded: every pair term in use has a finite reach, as the pair list needs
    const uint32_t t = params->terms;
    const bool direct = (t & (PB2_USE_LJ | PB2_USE_COULOMB)) != 0, gbt = (t & PB2_USE_GB) != 0;
    double reach = 0.0;
    bool bounded = b->cut && (direct || gbt);
    if (direct) {
      bounded = bounded && cutoff_mode;
      reach = std::max(reach, params->cutoff);
    }
    if (gbt) {
      bounded = bounded && gb_cut_mode;
      reach = std::max(reach, std::max(gb_cut, born_cut));
    }
    // (it saves less than its update costs where no system has many blocks:
    // us per step with and without at 1,200 atoms, 20 A: 30.7, 29.0; 2,500,
    // 9 A: 47.9, 51.2; 4,000, 12 A: 56.6, 59.7; 64 systems of 1,500 atoms,
    // 9 A: 382, 382)
    const bool many = std::any_of(sinfo.begin(), sinfo.end(), [](const SysInfo &S) { return S.nblk >= 64; });
    b->pl_on = bounded && params->skin >= 0.0 && params->pair_list >= 0 && many;
    b->pl_reach2 = (float)((reach + params->skin) * (reach + params->skin));
    if (b->params.tile_segment <= 0)
      b->params.tile_segment = b->pl_on ? listed_segment(sinfo, hposq, b->pl_reach2, ctx->sm_count)
                                        : default_segment(sinfo, bounded ? 2 : 6, ctx->sm_count);
  }
  b->hs64 = D.alloc<double>(N);
  b->se64 = D.alloc<double>(N);
  b->ro64 = D.alloc<double>(N);
  b->sr64 = D.alloc<double>(N);
  b->born64 = D.alloc<double>(N);
  b->iborn64 = D.alloc<double>(N);
  b->stage = D.alloc<double>(9 * (size_t)N);  // x, p, F rows of a host round trip
  b->user = D.alloc<int32_t>(N);
  b->devidx = D.alloc<int32_t>(N);
  b->born_acc = D.alloc<long long>(N);
  b->born_acc64 = D.alloc<long long>(N);
  b->dedb_acc = D.alloc<long long>(N);
  b->energy = D.alloc<long long>((size_t)n_systems * PB2_NTERMS);
  b->keys = D.alloc<uint32_t>(4 * (size_t)n_systems);
  b->key_splits = D.alloc<uint32_t>(8 * (size_t)n_systems);
  b->steps = D.alloc<long long>(n_systems);
  b->status = D.alloc<uint32_t>(n_systems);
  b->guard_end = D.alloc<int32_t>(1);
  b->warn_flags = D.alloc<uint32_t>(2 * (size_t)n_systems);
  b->warn_counts = D.alloc<int32_t>((size_t)n_systems * kWarnTypes);
  b->items = D.alloc<TileItem>(he64.born.size());
  b->items_e = D.alloc<TileItem>(he64.pair.size());
  b->tiles_e = D.alloc<TileItem>(he64.tiles.size());
  b->excl_ent = D.alloc<int2>(hent.size());
  b->excl_rows = D.alloc<ExclRow>(hrows.size());
  BondedArgs &B = b->bonded;
  B.n_bond = (int)bidx.size();
  B.n_bond_plain = n_bond_plain;
  B.n_angle = (int)aidx.size();
  B.n_tors = (int)tidx.size();
  B.n_cmap = (int)(cidx.size() / 6);
  B.n_exc = (int)eidx.size();
  int2 *d_eidx = D.alloc<int2>(eidx.size());
  double4 *d_epar = D.alloc<double4>(epar.size());
  int2 *d_bidx = D.alloc<int2>(bidx.size());
  double2 *d_bpar = D.alloc<double2>(bpar.size());
  int4 *d_aidx = D.alloc<int4>(aidx.size());
  double2 *d_apar = D.alloc<double2>(apar.size());
  int4 *d_tidx = D.alloc<int4>(tidx.size());
  double4 *d_tpar = D.alloc<double4>(tpar.size());
  int32_t *d_cidx = D.alloc<int32_t>(cidx.size());
  double *d_ccoef = D.alloc<double>(ccoef.size());
  int32_t *d_cgrid = D.alloc<int32_t>(cgrid.size());
  int64_t *d_cmoff = D.alloc<int64_t>(cmoff.size());
  if (D.failed) return fail(ctx, PB2_ENOMEM, "device allocation failed");

  int rc;
  if ((rc = upload(ctx, b->sys, sinfo)) || (rc = upload(ctx, b->atom_sys, hsys)) ||
      (rc = upload(ctx, b->x, hx)) || (rc = upload(ctx, b->y, hy)) || (rc = upload(ctx, b->z, hz)) ||
      (rc = upload(ctx, b->mass, hm)) || (rc = upload(ctx, b->sigma, hsig)) ||
      (rc = upload(ctx, b->charge, hq)) || (rc = upload(ctx, b->radius, hrad)) ||
      (rc = upload(ctx, b->posq, hposq)) || (rc = upload(ctx, b->par, hpar)) ||
      (rc = upload(ctx, b->hs64, hhs)) ||
      (rc = upload(ctx, b->se64, hse)) || (rc = upload(ctx, b->ro64, hro)) ||
      (rc = upload(ctx, b->sr64, hsr)) || (rc = upload(ctx, b->user, b->user_host)) ||
      (rc = upload(ctx, b->devidx, b->dev_host)) ||
      (rc = upload(ctx, b->keys, hkeys)) || (rc = upload(ctx, b->blk_sys, hblk_sys)) ||
      (rc = upload(ctx, b->blk_info, hblk_info)) || (rc = upload(ctx, b->items, he64.born)) ||
      (rc = upload(ctx, b->items_e, he64.pair)) || (rc = upload(ctx, b->tiles_e, he64.tiles)) ||
      (rc = upload(ctx, b->excl_ent, hent)) || (rc = upload(ctx, b->excl_rows, hrows)) ||
      (rc = upload(ctx, d_bidx, bidx)) || (rc = upload(ctx, d_bpar, bpar)) ||
      (rc = upload(ctx, d_aidx, aidx)) || (rc = upload(ctx, d_apar, apar)) ||
      (rc = upload(ctx, d_tidx, tidx)) || (rc = upload(ctx, d_tpar, tpar)) ||
      (rc = upload(ctx, d_cidx, cidx)) || (rc = upload(ctx, d_ccoef, ccoef)) ||
      (rc = upload(ctx, d_cgrid, cgrid)) || (rc = upload(ctx, d_cmoff, cmoff)) ||
      (rc = upload(ctx, d_eidx, eidx)) || (rc = upload(ctx, d_epar, epar)))
    return rc;
  warm_step_launch(b->n_blocks);
  CUDA_TRY(ctx, launch_key_splits(int_args(b.get(), 0, 0), nullptr));
  CUDA_TRY(ctx, cudaMemset(b->px, 0, N * sizeof(double)));
  CUDA_TRY(ctx, cudaMemset(b->py, 0, N * sizeof(double)));
  CUDA_TRY(ctx, cudaMemset(b->pz, 0, N * sizeof(double)));
  CUDA_TRY(ctx, cudaMemset(b->fx, 0, N * sizeof(long long)));
  CUDA_TRY(ctx, cudaMemset(b->fy, 0, N * sizeof(long long)));
  CUDA_TRY(ctx, cudaMemset(b->fz, 0, N * sizeof(long long)));
  CUDA_TRY(ctx, cudaMemset(b->born_acc, 0, N * sizeof(long long)));
  CUDA_TRY(ctx, cudaMemset(b->born_acc64, 0, N * sizeof(long long)));
  CUDA_TRY(ctx, cudaMemset(b->dedb_acc, 0, N * sizeof(long long)));
  CUDA_TRY(ctx, cudaMemset(b->born, 0, N * sizeof(float4)));
  CUDA_TRY(ctx, cudaMemset(b->steps, 0, n_systems * sizeof(long long)));
  CUDA_TRY(ctx, cudaMemset(b->sched, 0, kSchedWords * sizeof(int32_t)));
  CUDA_TRY(ctx, cudaMemset(b->status, 0, n_systems * sizeof(uint32_t)));
  CUDA_TRY(ctx, cudaMemset(b->guard_end, 0, sizeof(int32_t)));
  CUDA_TRY(ctx, cudaMemset(b->warn_flags, 0, 2 * (size_t)n_systems * sizeof(uint32_t)));
  CUDA_TRY(ctx, cudaMemset(b->warn_counts, 0, (size_t)n_systems * kWarnTypes * sizeof(int32_t)));
  B.atom_sys = b->atom_sys;
  B.x = b->x; B.y = b->y; B.z = b->z;
  B.fx = b->fx; B.fy = b->fy; B.fz = b->fz;
  B.energy = b->energy;
  B.terms = params->terms;
  B.bond_idx = d_bidx; B.bond_par = d_bpar;
  B.angle_idx = d_aidx; B.angle_par = d_apar;
  B.tors_idx = d_tidx; B.tors_par = d_tpar;
  B.cmap_idx = d_cidx; B.cmap_coeff = d_ccoef; B.cmap_grid = d_cgrid; B.cmap_map_off = d_cmoff;
  B.exc_idx = d_eidx; B.exc_par = d_epar;
  if (!(params->terms & PB2_USE_BONDED)) B.n_bond = B.n_angle = B.n_tors = 0;
  if (!(params->terms & PB2_USE_CMAP)) B.n_cmap = 0;
  if (!(params->terms & (PB2_USE_LJ | PB2_USE_COULOMB))) B.n_exc = 0;

  b->grid_bonded = 8 * ctx->sm_count;
  {
    // A batch of at most two waves of single tiles: thread blocks of four
    // warps spread them more evenly over the SMs than eight, and the
    // descreening pass runs faster with the registers of two resident blocks
    // than with a third (us per step with the larger batches' shapes and
    // these: 1,800 atoms 40.1, 36.1; 2,500 at 20 A 52.5, 47.4; 4,000 71.2,
    // 66.9; 6,000, 8,930 tiles 114.0, 113.7; 256 ragged systems 1313, 1341).
    long long tiles = 0;
    for (const SysInfo &S : sinfo)
      for (int ib = 0; ib < S.nblk; ib += 2) tiles += S.nblk - ib;
    if (tiles <= 2LL * 16 * ctx->sm_count)
      for (int &sh : b->shape) sh = 1;
  }
  if ((rc = setup_items2(b.get(), b->params.tile_segment))) return rc;
  if ((rc = setup_pair_list(b.get(), b->params.tile_segment))) return rc;
  {
    b->fuse = PB2_FUSE_BONDED;  // the autotuner may change this
  }
  CUDA_TRY(ctx, cudaStreamCreateWithFlags(&b->side, cudaStreamNonBlocking));
  for (auto &e : b->ev_side) CUDA_TRY(ctx, cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
  CUDA_TRY(ctx, cudaEventCreate(&b->ev[0]));
  CUDA_TRY(ctx, cudaEventCreate(&b->ev[1]));
  for (auto &e : b->ev_io) CUDA_TRY(ctx, cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
  for (auto &e : b->nl_ev) CUDA_TRY(ctx, cudaEventCreate(&e));
  CUDA_TRY(ctx, cudaDeviceSynchronize());
  *out = b.release();
  return PB2_OK;
}

extern "C" int pb2_batch_destroy(pb2_batch *b) {
  if (!b) return PB2_OK;
  cudaSetDevice(b->ctx->device);
  cudaDeviceSynchronize();
  delete b;
  return PB2_OK;
}

extern "C" int pb2_batch_info(const pb2_batch *b, int32_t *n_systems, int64_t *n_atoms_total) {
  if (!b) return PB2_EINVAL;
  if (n_systems) *n_systems = b->n_sys;
  if (n_atoms_total) *n_atoms_total = b->n_total;
  return PB2_OK;
}

// ------------------------------------------------------------ force evaluation

// In profiling mode, time one launch with CUDA events (eager runs only).
struct Timer {
  pb2_batch *b;
  cudaStream_t st;
  template <class F>
  cudaError_t operator()(int slot, F &&launch) {
    if (!b->profiling) return launch();
    cudaEventRecord(b->ev[0], st);
    const cudaError_t e = launch();
    cudaEventRecord(b->ev[1], st);
    cudaEventSynchronize(b->ev[1]);
    float ms = 0.f;
    cudaEventElapsedTime(&ms, b->ev[0], b->ev[1]);
    b->timings[slot] += ms;
    return e;
  }
};

// A pair pass: by teams where the batch has few tiles (not with the fused
// finalize, which is tail work of the one-warp kernel).
static cudaError_t enqueue_pass(pb2_batch *b, int pass, const PairArgs &a, cudaStream_t st) {
  if (b->team && !a.sys_items) return launch_team(pass, b->team, a, b->grid_team[pass], st);
  return launch_tiles(pass, a, b->grid_pair[pass], b->shape[pass], st);
}

// Force kernels on the current posq; force accumulators must be zero (or
// hold contributions to keep) and born_acc zero.  bonded_energy: also
// accumulate the (FP64) bonded energies.  The launch before (a step, a
// minimiser's move or place_kernel) wrote the block boxes and ran the pair
// list's displacement test.
static cudaError_t enqueue_forces(pb2_batch *b, cudaStream_t st, bool bonded_energy) {
  cudaError_t e;
  Timer tm{b, st};
  PairArgs pa = pair_args(b);
  const bool gb = (b->params.terms & PB2_USE_GB) != 0;
  if (b->pl_on && (e = tm(kTimBbox, [&] { return launch_pl_update(pl_args(b), b->grid_pl, st); })) != cudaSuccess)
    return e;
  if (gb) {
    FinalizeArgs fa;
    fa.sys = b->sys;
    fa.atom_sys = b->atom_sys;
    fa.radius = b->radius;
    fa.charge = b->charge;
    fa.born_acc = b->born_acc;
    fa.born = b->born;
    fa.dedb_acc = b->dedb_acc;
    fa.n_total = b->n_total;
    fa.blk_sys = b->blk_sys;
    fa.n_blocks = b->n_blocks;
    fa.sys_fin = b->sys_fin;
    fa.retired = b->retired;
    fa.status = b->status;
    // the descreening pass finalizes each block once its system's items are
    // summed (profiling keeps the separate launch, to time it)
    const bool fuse_finalize = !b->profiling && (b->fuse & PB2_FUSE_FINALIZE);
    // teams for all three passes: no finalize launch (profiling keeps it)
    if (b->team && !fuse_finalize && !b->profiling && b->force_blocks == 2) {
      pa.heads = 1;
      pa.fin = fa;
    }
    PairArgs pb = pa;
    pb.sched = b->sched + 2 * PASS_BORN;
    if (fuse_finalize) {
      pb.sys_items = b->sys_items;
      pb.fin = fa;
    }
    if ((e = tm(kTimBorn, [&] { return enqueue_pass(b, PASS_BORN, pb, st); })) != cudaSuccess) return e;
    if (!fuse_finalize && !pa.heads &&
        (e = tm(kTimFinalize, [&] { return launch_born_finalize(fa, st); })) != cudaSuccess)
      return e;
  }
  // The descreening pass lies between the positions and what follows.  A team
  // pass that is early, and a bonded launch, read positions before they wait
  // for the launch before: whatever writes positions has to be two launches
  // back or more.
  pa.early = gb;
  pa.sched = b->sched + 2 * PASS_FORCE;
  if (b->force_blocks == 4 && !b->pl_on) {
    PairArgs p4 = pa;
    p4.items = b->items4;
    p4.n_items = b->n_items4;
    p4.item_count = b->item_count4;
    if ((e = tm(kTimForce, [&] { return launch_force4(p4, b->grid4, b->shape4, st); })) != cudaSuccess) return e;
  } else if ((e = tm(kTimForce, [&] { return enqueue_pass(b, PASS_FORCE, pa, st); })) != cudaSuccess) {
    return e;
  }
  pa.sched = b->sched + 2 * PASS_CHAIN;
  BondedArgs ba = b->bonded;
  ba.energy_mode = bonded_energy ? 1 : 0;
  const int n_bonded = ba.n_bond + ba.n_angle + ba.n_tors + ba.n_cmap + ba.n_exc;
  // the bonded terms ride along as the chain pass's tail work, except when
  // their energies are wanted or there is no chain pass
  const bool fuse_bonded = gb && !bonded_energy && !b->profiling && (b->fuse & PB2_FUSE_BONDED);
  if (fuse_bonded) {
    pa.bonded = ba;
    pa.n_bonded_chunks = (n_bonded + kBondedChunk - 1) / kBondedChunk;
  }
  if (gb)
    if ((e = tm(kTimChain, [&] { return enqueue_pass(b, PASS_CHAIN, pa, st); })) != cudaSuccess) return e;
  if (fuse_bonded) return cudaSuccess;
  return tm(kTimBonded, [&] { return launch_bonded(ba, b->grid_bonded, st); });
}

// FP64 pair energies (GB polar incl. self, ACE, Coulomb, LJ) into b->energy.
static cudaError_t enqueue_energy64(pb2_batch *b, cudaStream_t st) {
  cudaError_t e;
  Energy64Args ea;
  ea.sys = b->sys;
  ea.items = b->items;
  ea.n_items = b->n_items;
  ea.terms = b->params.terms;
  ea.excl_ent = b->excl_ent;
  ea.excl_rows = b->excl_rows;
  ea.x = b->x; ea.y = b->y; ea.z = b->z;
  ea.q = b->charge; ea.hs = b->hs64; ea.se = b->se64; ea.ro = b->ro64; ea.sr = b->sr64;
  ea.radius = b->radius;
  ea.born64 = b->born64;
  ea.iborn64 = b->iborn64;
  ea.born_acc = b->born_acc64;
  ea.energy = b->energy;
  ea.bbox = b->bbox;
  ea.blk_sys = b->blk_sys;
  ea.n_blocks = b->n_blocks;
  ea.sched = b->sched + kSchedE64;
  ea.tiles = nullptr;
  ea.n_tiles = 0;
  if (b->params.terms & PB2_USE_GB) {
    if ((e = launch_energy64(0, ea, b->grid_e64[0], st)) != cudaSuccess) return e;
    if ((e = launch_finalize64(ea, st)) != cudaSuccess) return e;
  }
  ea.sched = b->sched + kSchedE64 + 2;
  ea.items = b->items_e;
  ea.n_items = b->n_items_e;
  ea.tiles = b->tiles_e;
  ea.n_tiles = b->n_tiles_e;
  if ((e = launch_energy64_tiles(ea, b->grid_tiles_e, st)) != cudaSuccess) return e;
  return launch_energy64(1, ea, b->grid_e64[1], st);
}

// Kernels of an evaluation after place_kernel.  The FP64 energies need only
// the positions, so they run beside the forces, on a stream forked from st and
// joined to it: their kernels fill the FP64 pipe and the gaps of the force
// kernels (us, one after the other and side by side: 2,500 atoms 113, 92;
// 20,000 2,070, 1,935; 32 ragged systems 448, 427).
static int enqueue_eval(pb2_batch *b, cudaStream_t st, bool energy) {
  pb2_ctx *ctx = b->ctx;
  if (energy) {
    CUDA_TRY(ctx, cudaEventRecord(b->ev_side[0], st));
    CUDA_TRY(ctx, cudaStreamWaitEvent(b->side, b->ev_side[0], 0));
    CUDA_TRY(ctx, enqueue_energy64(b, b->side));
    CUDA_TRY(ctx, cudaEventRecord(b->ev_side[1], b->side));
  }
  CUDA_TRY(ctx, enqueue_forces(b, st, energy));
  if (energy) CUDA_TRY(ctx, cudaStreamWaitEvent(st, b->ev_side[1], 0));
  return PB2_OK;
}

// A graph of chains of launches: each of `chains` enqueues one (no stream is
// captured, see GraphChain).  The thread's capture mode is relaxed meanwhile:
// a capture in progress elsewhere neither forbids this nor is ended by it.
template <class... F>
static cudaError_t build_graph(cudaGraphExec_t *out, F &&...chains) {
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  cudaError_t e = cudaThreadExchangeStreamCaptureMode(&mode);
  if (e != cudaSuccess) return e;
  cudaGraph_t g = nullptr;
  auto add = [&](auto &&enqueue) {
    if (e != cudaSuccess) return;
    GraphChain c{g};
    held_chain = &c;
    e = enqueue();
    held_chain = nullptr;
  };
  e = cudaGraphCreate(&g, 0);
  (add(chains), ...);
  if (e == cudaSuccess) e = cudaGraphInstantiate(out, g, 0);
  if (g) cudaGraphDestroy(g);
  cudaThreadExchangeStreamCaptureMode(&mode);
  if (e != cudaSuccess) *out = nullptr;
  return e;
}

// The same as a graph of two chains, for the batches that run by teams: a
// dozen launches' host time is what a small system's evaluation waits for (166
// atoms: 51 us by launches, 37 as a graph; 2,500 atoms, 1,600 tiles: 92 and
// 100, since consecutive graphs do not overlap).  Made at the third evaluation
// (a batch that is evaluated once or twice does not pay for it).  NULL: by
// launches, also where no graph could be made.
static cudaGraphExec_t eval_graph(pb2_batch *b, bool energy) {
  if (!b->team) return nullptr;
  cudaGraphExec_t &ex = b->eval_graphs[energy];
  if (ex || ++b->evals[energy] < 3) return ex;
  const auto energies = [&] { return energy ? enqueue_energy64(b, nullptr) : cudaSuccess; };
  if (build_graph(&ex, energies, [&] { return enqueue_forces(b, nullptr, energy); }) != cudaSuccess) {
    cudaGetLastError();   // the launches report their own
    b->evals[energy] = 0;  // and the third call from here tries again
  }
  return ex;
}

// Forces (and with energy set the FP64 energies) at the current positions,
// or at the caller's device rows, which then become the positions.
static int fresh_forces(pb2_batch *b, cudaStream_t st, bool energy, const double *rows = nullptr) {
  pb2_ctx *ctx = b->ctx;
  CUDA_TRY(ctx, launch_place(int_args(b, b->key_parity, 0), rows, energy ? b->energy : nullptr, st));
  // under the caller's own capture the launches become part of its graph
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  if (st) CUDA_TRY(ctx, cudaStreamIsCapturing(st, &cap));
  cudaGraphExec_t ex = nullptr;
  if (cap == cudaStreamCaptureStatusNone && !b->profiling) ex = eval_graph(b, energy);
  b->eval_replayed = ex != nullptr;
  if (ex) CUDA_TRY(ctx, cudaGraphLaunch(ex, st));
  else if (int rc = enqueue_eval(b, st, energy)) return rc;
  b->forces_valid = true;
  return PB2_OK;
}

static int copy_forces(pb2_batch *b, double *forces, cudaStream_t st) {
  pb2_ctx *ctx = b->ctx;
  const int N = b->n_total;
  CUDA_TRY(ctx, launch_fix_to_rows(b->fx, b->fy, b->fz, b->user, b->stage, N, st));
  CUDA_TRY(ctx, cudaMemcpyAsync(forces, b->stage, 3 * (size_t)N * sizeof(double), cudaMemcpyDeviceToHost, st));
  CUDA_TRY(ctx, cudaStreamSynchronize(st));
  return PB2_OK;
}

// Device-pointer variant: no host copy, no buffers of its own, no synchronisation
// (usable from an XLA custom call or under stream capture).
extern "C" int pb2_energy_forces_device(pb2_batch *b, const double *positions, double *energies,
                                        double *forces, void *stream) {
  if (!b) return PB2_EINVAL;
  pb2_ctx *ctx = b->ctx;
  cudaStream_t st = (cudaStream_t)stream;
  int rc = fresh_forces(b, st, energies != nullptr, positions);
  if (rc) return rc;
  CUDA_TRY(ctx, launch_results(b->fx, b->fy, b->fz, b->user, forces, b->n_total, b->energy, energies, b->n_sys, st));
  return PB2_OK;
}

extern "C" int pb2_energy_forces(pb2_batch *b, double *energies, double *forces, void *stream) {
  if (!b) return PB2_EINVAL;
  pb2_ctx *ctx = b->ctx;
  cudaStream_t st = (cudaStream_t)stream;
  CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  int rc = fresh_forces(b, st, energies != nullptr);
  if (rc) return rc;
  if (energies) {
    std::vector<long long> he((size_t)b->n_sys * PB2_NTERMS);
    CUDA_TRY(ctx, cudaMemcpyAsync(he.data(), b->energy, he.size() * sizeof(long long), cudaMemcpyDeviceToHost, st));
    CUDA_TRY(ctx, cudaStreamSynchronize(st));
    for (int s = 0; s < b->n_sys; ++s) {
      double tot = 0.0;
      for (int t = 0; t < PB2_TERM_TOTAL; ++t) {
        const double v = (double)he[(size_t)s * PB2_NTERMS + t] * kEnergyInv;
        energies[(size_t)s * PB2_NTERMS + t] = v;
        tot += v;
      }
      energies[(size_t)s * PB2_NTERMS + PB2_TERM_TOTAL] = tot;
    }
  }
  if (forces) return copy_forces(b, forces, st);
  CUDA_TRY(ctx, cudaStreamSynchronize(st));
  return PB2_OK;
}

extern "C" int pb2_born_radii(pb2_batch *b, double *out, void *stream) {
  if (!b || !out) return PB2_EINVAL;
  pb2_ctx *ctx = b->ctx;
  cudaStream_t st = (cudaStream_t)stream;
  if (!(b->params.terms & PB2_USE_GB)) return fail(ctx, PB2_EINVAL, "GB term disabled");
  int rc = fresh_forces(b, st, false);
  if (rc) return rc;
  std::vector<float4> hb(b->n_total);
  CUDA_TRY(ctx, cudaMemcpyAsync(hb.data(), b->born, hb.size() * sizeof(float4), cudaMemcpyDeviceToHost, st));
  CUDA_TRY(ctx, cudaStreamSynchronize(st));
  for (int g = 0; g < b->n_total; ++g) out[b->user_host[g]] = (double)hb[g].x;
  return PB2_OK;
}

// Row-major (n, 3) host arrays move through the device staging buffer in one
// copy each; the (de)interleave runs on the device.  The staging buffer is
// reused by the next transfer on the same stream, so each helper finishes
// its copy before returning.
static int upload_soa3(pb2_batch *b, const double *aos, double *dx, double *dy, double *dz, cudaStream_t st) {
  pb2_ctx *ctx = b->ctx;
  const int N = b->n_total;
  CUDA_TRY(ctx, cudaMemcpyAsync(b->stage, aos, 3 * (size_t)N * sizeof(double), cudaMemcpyHostToDevice, st));
  CUDA_TRY(ctx, launch_rows_to_soa(b->stage, b->user, dx, dy, dz, N, st));
  return PB2_OK;
}

static int download_soa3(pb2_batch *b, double *aos, const double *dx, const double *dy, const double *dz,
                         cudaStream_t st) {
  pb2_ctx *ctx = b->ctx;
  const int N = b->n_total;
  CUDA_TRY(ctx, launch_soa_to_rows(dx, dy, dz, b->user, b->stage, N, st));
  CUDA_TRY(ctx, cudaMemcpyAsync(aos, b->stage, 3 * (size_t)N * sizeof(double), cudaMemcpyDeviceToHost, st));
  CUDA_TRY(ctx, cudaStreamSynchronize(st));
  return PB2_OK;
}

extern "C" int pb2_set_positions(pb2_batch *b, const double *positions, void *stream) {
  if (!b || !positions) return PB2_EINVAL;
  b->forces_valid = false;
  int rc = upload_soa3(b, positions, b->x, b->y, b->z, (cudaStream_t)stream);
  if (rc || (rc = forces_not_from_step(b, (cudaStream_t)stream))) return rc;
  CUDA_TRY(b->ctx, cudaStreamSynchronize((cudaStream_t)stream));
  return PB2_OK;
}

// ------------------------------------------------------------ Langevin

static int run_eager(pb2_batch *b, int n_steps, cudaStream_t st) {
  pb2_ctx *ctx = b->ctx;
  Timer tm{b, st};
  for (int t = 0; t < n_steps; ++t) {
    const IntArgs ia = int_args(b, b->key_parity, t > 0);
    CUDA_TRY(ctx, tm(kTimStep, [&] { return launch_step(ia, st); }));
    CUDA_TRY(ctx, enqueue_forces(b, st, false));
    b->key_parity ^= 1;
  }
  const IntArgs fa = int_args(b, b->key_parity, 0);
  CUDA_TRY(ctx, tm(kTimStep, [&] { return launch_finish(fa, st); }));
  return PB2_OK;
}

static int get_graph(pb2_batch *b, int chunk, int parity, cudaGraphExec_t *out) {
  pb2_ctx *ctx = b->ctx;
  auto key = std::make_pair(chunk, parity);
  auto it = b->graphs.find(key);
  if (it != b->graphs.end()) {
    *out = it->second;
    return PB2_OK;
  }
  cudaGraphExec_t ex = nullptr;
  const cudaError_t e = build_graph(&ex, [&] {
    cudaError_t err = cudaSuccess;
    int p = parity;
    for (int t = 0; t < chunk && err == cudaSuccess; ++t) {
      err = launch_step(int_args(b, p, t > 0), nullptr);
      if (err == cudaSuccess) err = enqueue_forces(b, nullptr, false);
      p ^= 1;
    }
    return err == cudaSuccess ? launch_finish(int_args(b, p, 0), nullptr) : err;
  });
  if (e != cudaSuccess) return fail(ctx, PB2_ECUDA, std::string("step graph: ") + cudaGetErrorString(e));
  b->graphs[key] = ex;
  *out = ex;
  return PB2_OK;
}

extern "C" int pb2_langevin_init(pb2_batch *b, void *stream) {
  if (!b) return PB2_EINVAL;
  pb2_ctx *ctx = b->ctx;
  cudaStream_t st = (cudaStream_t)stream;
  CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  CUDA_TRY(ctx, launch_init(int_args(b, b->key_parity, 0), st));
  b->key_parity ^= 1;
  int rc = fresh_forces(b, st, false);
  if (rc || (rc = forces_not_from_step(b, st))) return rc;
  CUDA_TRY(ctx, cudaStreamSynchronize(st));
  return PB2_OK;
}

extern "C" int pb2_set_langevin_params(pb2_batch *b, const double *dt, const double *kT,
                                       const double *gamma, void *stream) {
  if (!b) return PB2_EINVAL;
  pb2_ctx *ctx = b->ctx;
  cudaStream_t st = (cudaStream_t)stream;
  const int S = b->n_sys;
  for (int s = 0; s < S; ++s)
    if ((dt && !(dt[s] > 0.0)) || (kT && !(kT[s] >= 0.0)) || (gamma && !(gamma[s] >= 0.0)))
      return fail(ctx, PB2_EINVAL, "dt > 0, kT >= 0, gamma >= 0");
  CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  // steps already queued, on any stream of the device, finish with the old
  // values: the per-system constants are overwritten in place
  CUDA_TRY(ctx, cudaDeviceSynchronize());
  for (int s = 0; s < S; ++s) {
    SysInfo &I = b->sys_host[s];
    if (dt) I.dt = dt[s];
    if (kT) I.kT = kT[s];
    if (gamma) b->gamma_host[s] = gamma[s];
    I.half_dt = 0.5 * I.dt;
    I.c1 = std::exp(-b->gamma_host[s] * I.dt);
    I.c2 = std::sqrt(1.0 - I.c1 * I.c1);
  }
  CUDA_TRY(ctx, cudaMemcpyAsync(b->sys, b->sys_host.data(), S * sizeof(SysInfo), cudaMemcpyHostToDevice, st));
  CUDA_TRY(ctx, launch_noise_scale(b->sys, b->atom_sys, b->mass, b->sigma, b->n_total, st));
  CUDA_TRY(ctx, cudaStreamSynchronize(st));
  return PB2_OK;
}

extern "C" int pb2_langevin_center_momentum(pb2_batch *b, void *stream) {
  if (!b) return PB2_EINVAL;
  pb2_ctx *ctx = b->ctx;
  cudaStream_t st = (cudaStream_t)stream;
  CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  CUDA_TRY(ctx, launch_center(int_args(b, b->key_parity, 0), st));
  CUDA_TRY(ctx, cudaStreamSynchronize(st));
  return PB2_OK;
}

extern "C" int pb2_langevin_run(pb2_batch *b, int32_t n_steps, void *stream) {
  if (!b || n_steps < 0) return PB2_EINVAL;
  pb2_ctx *ctx = b->ctx;
  cudaStream_t st = (cudaStream_t)stream;
  CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  if (n_steps == 0) return PB2_OK;
  if (!b->forces_valid) {
    int rc = fresh_forces(b, st, false);
    if (rc) return rc;
  }
  if (b->profiling) {
    for (double &t : b->timings) t = 0.0;
    cudaEvent_t a0, a1;
    cudaEventCreate(&a0);
    cudaEventCreate(&a1);
    cudaEventRecord(a0, st);
    int rc = run_eager(b, n_steps, st);
    cudaEventRecord(a1, st);
    cudaEventSynchronize(a1);
    float ms = 0.f;
    cudaEventElapsedTime(&ms, a0, a1);
    b->timings[kTimAll] = ms;
    cudaEventDestroy(a0);
    cudaEventDestroy(a1);
    if (rc) return rc;
    CUDA_TRY(ctx, cudaStreamSynchronize(st));
    return PB2_OK;
  }
  const int chunk = b->params.graph_chunk;
  int done = 0;
  while (done < n_steps) {
    const int c = std::min(chunk, n_steps - done);
    cudaGraphExec_t ex;
    int rc = get_graph(b, c, b->key_parity, &ex);
    if (rc) return rc;
    CUDA_TRY(ctx, cudaGraphLaunch(ex, st));
    b->key_parity ^= (c & 1);
    done += c;
  }
  return PB2_OK;
}

extern "C" int pb2_get_state(pb2_batch *b, double *x, double *p, double *f, uint32_t *keys,
                             int64_t *steps, void *stream) {
  if (!b) return PB2_EINVAL;
  pb2_ctx *ctx = b->ctx;
  cudaStream_t st = (cudaStream_t)stream;
  int rc;
  if (x && (rc = download_soa3(b, x, b->x, b->y, b->z, st))) return rc;
  if (p && (rc = download_soa3(b, p, b->px, b->py, b->pz, st))) return rc;
  if (f && (rc = copy_forces(b, f, st))) return rc;
  if (keys) {
    CUDA_TRY(ctx, cudaMemcpyAsync(keys, b->keys + (size_t)b->key_parity * b->n_sys * 2,
                                  (size_t)b->n_sys * 2 * sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
  }
  if (steps) {
    std::vector<long long> h(b->n_sys);
    CUDA_TRY(ctx, cudaMemcpyAsync(h.data(), b->steps, h.size() * sizeof(long long), cudaMemcpyDeviceToHost, st));
    CUDA_TRY(ctx, cudaStreamSynchronize(st));
    for (int s = 0; s < b->n_sys; ++s) steps[s] = h[s];
  }
  CUDA_TRY(ctx, cudaStreamSynchronize(st));
  return PB2_OK;
}

extern "C" int pb2_set_state(pb2_batch *b, const double *x, const double *p, const uint32_t *keys,
                             void *stream) {
  if (!b) return PB2_EINVAL;
  pb2_ctx *ctx = b->ctx;
  cudaStream_t st = (cudaStream_t)stream;
  int rc;
  if (x && (rc = upload_soa3(b, x, b->x, b->y, b->z, st))) return rc;
  if (p && (rc = upload_soa3(b, p, b->px, b->py, b->pz, st))) return rc;
  if (keys) {
    CUDA_TRY(ctx, cudaMemcpyAsync(b->keys + (size_t)b->key_parity * b->n_sys * 2, keys,
                                  (size_t)b->n_sys * 2 * sizeof(uint32_t), cudaMemcpyHostToDevice, st));
    CUDA_TRY(ctx, launch_key_splits(int_args(b, b->key_parity, 0), st));
    CUDA_TRY(ctx, cudaStreamSynchronize(st));
  }
  if (x) {  // forces must follow the positions
    rc = fresh_forces(b, st, false);
    if (rc || (rc = forces_not_from_step(b, st))) return rc;
  }
  CUDA_TRY(ctx, cudaStreamSynchronize(st));
  return PB2_OK;
}

extern "C" int pb2_set_full_state(pb2_batch *b, const double *x, const double *p, const double *f,
                                  const uint32_t *keys, void *stream) {
  if (!b || !x || !p || !f) return PB2_EINVAL;
  pb2_ctx *ctx = b->ctx;
  cudaStream_t st = (cudaStream_t)stream;
  CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  int rc;
  if ((rc = upload_soa3(b, x, b->x, b->y, b->z, st))) return rc;
  if ((rc = upload_soa3(b, p, b->px, b->py, b->pz, st))) return rc;
  CUDA_TRY(ctx, cudaMemcpyAsync(b->stage, f, 3 * (size_t)b->n_total * sizeof(double), cudaMemcpyHostToDevice, st));
  CUDA_TRY(ctx, launch_rows_to_fix(b->stage, b->user, b->fx, b->fy, b->fz, b->n_total, st));
  if (keys) {
    CUDA_TRY(ctx, cudaMemcpyAsync(b->keys + (size_t)b->key_parity * b->n_sys * 2, keys,
                                  (size_t)b->n_sys * 2 * sizeof(uint32_t), cudaMemcpyHostToDevice, st));
    CUDA_TRY(ctx, launch_key_splits(int_args(b, b->key_parity, 0), st));
  }
  CUDA_TRY(ctx, launch_posq(int_args(b, b->key_parity, 0), st));
  b->forces_valid = true;
  if ((rc = forces_not_from_step(b, st))) return rc;
  CUDA_TRY(ctx, cudaStreamSynchronize(st));
  return PB2_OK;
}


// The functional step on caller-held state: copies in on copy_in, steps on
// stream, copies out on copy_out.  kind_in / kind_out are the directions of
// the copies (host arrays, or the caller's device arrays).
static int run_caller_state(pb2_batch *b, double *x, double *p, double *f, int32_t n_steps,
                            void *stream, void *copy_in, void *copy_out, cudaMemcpyKind kind_in,
                            cudaMemcpyKind kind_out) {
  if (!b || !x || !p || !f || n_steps < 0) return PB2_EINVAL;
  pb2_ctx *ctx = b->ctx;
  cudaStream_t st = (cudaStream_t)stream, ci = (cudaStream_t)copy_in, co = (cudaStream_t)copy_out;
  const int N = b->n_total;
  const size_t rows = 3 * (size_t)N, bytes = rows * sizeof(double);
  CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  // in: the previous round trip's copies out of the staging buffer are done;
  // the three copies back to back, then one conversion
  CUDA_TRY(ctx, cudaStreamWaitEvent(ci, b->ev_io[2], 0));
  CUDA_TRY(ctx, cudaMemcpyAsync(b->stage, x, bytes, kind_in, ci));
  CUDA_TRY(ctx, cudaMemcpyAsync(b->stage + rows, p, bytes, kind_in, ci));
  CUDA_TRY(ctx, cudaMemcpyAsync(b->stage + 2 * rows, f, bytes, kind_in, ci));
  CUDA_TRY(ctx, cudaEventRecord(b->ev_io[0], ci));
  CUDA_TRY(ctx, cudaStreamWaitEvent(st, b->ev_io[0], 0));
  CUDA_TRY(ctx, launch_state_from_rows(b->stage, b->user, b->x, b->y, b->z, b->px, b->py, b->pz, b->fx, b->fy, b->fz,
                                       N, st));
  CUDA_TRY(ctx, launch_posq(int_args(b, b->key_parity, 0), st));
  b->forces_valid = true;
  int rc = pb2_langevin_run(b, n_steps, stream);
  if (rc) return rc;
  // out: one conversion, then the three copies
  CUDA_TRY(ctx, launch_state_to_rows(b->x, b->y, b->z, b->px, b->py, b->pz, b->fx, b->fy, b->fz, b->user,
                                     b->stage, N, st));
  CUDA_TRY(ctx, cudaEventRecord(b->ev_io[1], st));
  CUDA_TRY(ctx, cudaStreamWaitEvent(co, b->ev_io[1], 0));
  CUDA_TRY(ctx, cudaMemcpyAsync(x, b->stage, bytes, kind_out, co));
  CUDA_TRY(ctx, cudaMemcpyAsync(p, b->stage + rows, bytes, kind_out, co));
  CUDA_TRY(ctx, cudaMemcpyAsync(f, b->stage + 2 * rows, bytes, kind_out, co));
  CUDA_TRY(ctx, cudaEventRecord(b->ev_io[2], co));
  return PB2_OK;
}

extern "C" int pb2_langevin_run_host(pb2_batch *b, double *x, double *p, double *f, int32_t n_steps,
                                     void *stream, void *copy_in, void *copy_out) {
  return run_caller_state(b, x, p, f, n_steps, stream, copy_in, copy_out, cudaMemcpyHostToDevice,
                          cudaMemcpyDeviceToHost);
}

extern "C" int pb2_langevin_run_device(pb2_batch *b, double *x, double *p, double *f, int32_t n_steps,
                                       void *stream) {
  return run_caller_state(b, x, p, f, n_steps, stream, stream, stream, cudaMemcpyDeviceToDevice,
                          cudaMemcpyDeviceToDevice);
}

// ------------------------------------------------------------ minimisation

static MinArgs min_args(pb2_batch *b) {
  MinArgs a;
  a.sys = b->sys;
  a.atom_sys = b->atom_sys;
  a.x = b->x; a.y = b->y; a.z = b->z;
  a.px = b->px; a.py = b->py; a.pz = b->pz;
  a.fx = b->fx; a.fy = b->fy; a.fz = b->fz;
  a.mass = b->mass;
  a.charge = b->charge;
  a.posq = b->posq;
  a.x0 = b->m_x0;
  a.sel = b->m_sel;
  a.ft = b->m_ft; a.xb = b->m_xb; a.best = b->m_best;
  a.sys_dt = b->m_sys;
  a.sys_alpha = b->m_sys + b->n_sys;
  a.sys_best = b->m_sys + 2 * (size_t)b->n_sys;
  a.sys_npos = b->m_npos;
  a.status = b->status;
  a.par = b->m_par;
  a.n_total = b->n_total;
  a.n_sys = b->n_sys;
  a.blk_info = b->blk_info;
  a.n_blocks = b->n_blocks;
  a.chunks = b->m_chunks;
  a.chunk0 = b->m_chunk0;
  a.n_chunks = b->m_n_chunks;
  a.part = b->m_part;
  a.sys_done = b->m_done;
  a.mix_f = b->m_sys + 4 * (size_t)b->n_sys;
  a.mix_p = b->m_sys + 5 * (size_t)b->n_sys;
  a.sys_flags = b->m_flags;
  a.bbox = b->bbox;
  a.pl_ref = b->pl_on ? b->pl_ref : nullptr;
  a.pl_ctl = b->pl_on ? b->pl_ctl : nullptr;
  return a;
}

extern "C" int pb2_min_setup(pb2_batch *b, const uint8_t *heavy, const uint8_t *backbone) {
  if (!b) return PB2_EINVAL;
  pb2_ctx *ctx = b->ctx;
  CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  const size_t N = b->n_total;
  if (!b->min_alloc) {
    Dev &D = b->mdev;
    b->m_x0 = D.alloc<double>(3 * N);
    b->m_ft = D.alloc<double>(3 * N);
    b->m_xb = D.alloc<double>(3 * N);
    b->m_best = D.alloc<double>(3 * N);
    b->m_par = D.alloc<double>(kMinNPar);
    b->m_sys = D.alloc<double>(6 * (size_t)b->n_sys);
    b->m_npos = D.alloc<int32_t>(b->n_sys);
    b->m_sel = D.alloc<uint8_t>(N);
    std::vector<int2> chunks;
    std::vector<int32_t> first;
    for (int s = 0; s < b->n_sys; ++s) {
      first.push_back((int)chunks.size());
      for (int k = 0; k < b->sys_host[s].nblk; k += kMinChunkBlocks) chunks.push_back(make_int2(s, k));
    }
    first.push_back((int)chunks.size());
    b->m_n_chunks = (int)chunks.size();
    b->m_chunks = D.alloc<int2>(chunks.size());
    b->m_chunk0 = D.alloc<int32_t>(first.size());
    b->m_part = D.alloc<double>(3 * chunks.size());
    b->m_done = D.alloc<int32_t>(b->n_sys);
    b->m_flags = D.alloc<int32_t>(b->n_sys);
    for (const void *p : {(const void *)b->m_x0, (const void *)b->m_ft, (const void *)b->m_xb, (const void *)b->m_best,
                          (const void *)b->m_par, (const void *)b->m_sys, (const void *)b->m_npos,
                          (const void *)b->m_sel, (const void *)b->m_chunks, (const void *)b->m_chunk0,
                          (const void *)b->m_part, (const void *)b->m_done, (const void *)b->m_flags})
      if (!p) return fail(ctx, PB2_ENOMEM, "minimiser allocation failed");
    int rc;
    if ((rc = upload(ctx, b->m_chunks, chunks)) || (rc = upload(ctx, b->m_chunk0, first))) return rc;
    CUDA_TRY(ctx, cudaMemset(b->m_done, 0, b->n_sys * sizeof(int32_t)));
    b->min_alloc = true;  // a call after one that failed above starts over
  }
  // selections: heavy atoms default to mass > 1.1 amu (prolix simulate.py:596),
  // backbone to the heavy atoms
  std::vector<double> hm(N);
  CUDA_TRY(ctx, cudaMemcpy(hm.data(), b->mass, N * sizeof(double), cudaMemcpyDeviceToHost));
  std::vector<uint8_t> sel(N);
  for (size_t g = 0; g < N; ++g) {  // heavy, backbone: caller's atom order
    const int32_t u = b->user_host[g];
    const bool h = heavy ? heavy[u] != 0 : hm[g] > 1.1;
    const bool bb = backbone ? backbone[u] != 0 : h;
    sel[g] = (uint8_t)((h ? 1 : 0) | (bb ? 2 : 0));
  }
  CUDA_TRY(ctx, cudaMemcpy(b->m_sel, sel.data(), N, cudaMemcpyHostToDevice));
  CUDA_TRY(ctx, cudaMemcpy(b->m_x0, b->x, N * sizeof(double), cudaMemcpyDeviceToDevice));
  CUDA_TRY(ctx, cudaMemcpy(b->m_x0 + N, b->y, N * sizeof(double), cudaMemcpyDeviceToDevice));
  CUDA_TRY(ctx, cudaMemcpy(b->m_x0 + 2 * N, b->z, N * sizeof(double), cudaMemcpyDeviceToDevice));
  b->min_ready = true;
  return PB2_OK;
}

// mode 0: steepest descent steps; mode 1: FIRE iterations
static int min_graph(pb2_batch *b, int mode, int chunk, cudaGraphExec_t *out) {
  pb2_ctx *ctx = b->ctx;
  auto key = std::make_pair(mode, chunk);
  auto it = b->min_graphs.find(key);
  if (it != b->min_graphs.end()) {
    *out = it->second;
    return PB2_OK;
  }
  const MinArgs ma = min_args(b);
  cudaGraphExec_t ex = nullptr;
  const cudaError_t e = build_graph(&ex, [&] {
    cudaError_t err = cudaSuccess;
    for (int t = 0; t < chunk && err == cudaSuccess; ++t) {
      err = launch_min(mode == 0 ? kMinOpSd : kMinOpFireMove, ma, nullptr, nullptr);
      if (err == cudaSuccess) err = enqueue_forces(b, nullptr, false);
      if (err == cudaSuccess && mode != 0) err = launch_min(kMinOpFireClose, ma, nullptr, nullptr);
    }
    return err;
  });
  if (e != cudaSuccess) return fail(ctx, PB2_ECUDA, std::string("minimiser graph: ") + cudaGetErrorString(e));
  b->min_graphs[key] = ex;
  *out = ex;
  return PB2_OK;
}

static int min_run(pb2_batch *b, int mode, int n, cudaStream_t st) {
  pb2_ctx *ctx = b->ctx;
  int done = 0;
  while (done < n) {
    const int c = std::min(b->params.graph_chunk, n - done);
    cudaGraphExec_t ex;
    int rc = min_graph(b, mode, c, &ex);
    if (rc) return rc;
    CUDA_TRY(ctx, cudaGraphLaunch(ex, st));
    done += c;
  }
  return PB2_OK;
}

static int min_begin(pb2_batch *b, int32_t n_steps, double k, int32_t kind, cudaStream_t st) {
  pb2_ctx *ctx = b->ctx;
  if (!b->min_ready) return fail(ctx, PB2_EINVAL, "call pb2_min_setup first");
  if (n_steps < 0 || kind < 0 || kind > 2 || !(k >= 0.0)) return fail(ctx, PB2_EINVAL, "bad minimiser arguments");
  CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  b->m_par_host[kMinK] = k;
  b->m_par_host[kMinKind] = kind;
  CUDA_TRY(ctx, cudaMemcpyAsync(b->m_par, b->m_par_host, kMinNPar * sizeof(double), cudaMemcpyHostToDevice, st));
  if (!b->forces_valid) {
    int rc = fresh_forces(b, st, false);
    if (rc) return rc;
  }
  return PB2_OK;
}

extern "C" int pb2_min_sd(pb2_batch *b, int32_t n_steps, double k, int32_t kind, double dt, double max_dx,
                          void *stream) {
  if (!b) return PB2_EINVAL;
  if (!(dt > 0.0) || !(max_dx > 0.0)) return fail(b->ctx, PB2_EINVAL, "dt and max_dx must be > 0");
  b->m_par_host[kMinSdDt] = dt;
  b->m_par_host[kMinMaxDx] = max_dx;
  b->m_par_host[kMinForceCap] = 0.0;
  cudaStream_t st = (cudaStream_t)stream;
  int rc = min_begin(b, n_steps, k, kind, st);
  if (rc) return rc;
  if ((rc = min_run(b, 0, n_steps, st))) return rc;
  CUDA_TRY(b->ctx, launch_min(kMinOpRollback, min_args(b), nullptr, st));
  b->forces_valid = false;  // a rolled-back system moved
  if ((rc = forces_not_from_step(b, st))) return rc;
  CUDA_TRY(b->ctx, cudaStreamSynchronize(st));
  return PB2_OK;
}

extern "C" int pb2_min_fire(pb2_batch *b, int32_t n_steps, double k, int32_t kind, double dt_start,
                            double dt_max, double max_disp, double force_cap, int32_t flags, void *stream) {
  if (!b) return PB2_EINVAL;
  if (!(dt_start > 0.0) || !(dt_max > 0.0) || !(max_disp >= 0.0) || !(force_cap >= 0.0))
    return fail(b->ctx, PB2_EINVAL, "dt_start, dt_max must be > 0; max_disp, force_cap >= 0");
  b->m_par_host[kMinDtStart] = dt_start;
  b->m_par_host[kMinDtMax] = dt_max;
  b->m_par_host[kMinMaxDisp] = max_disp;
  b->m_par_host[kMinForceCap] = force_cap;
  cudaStream_t st = (cudaStream_t)stream;
  int rc = min_begin(b, n_steps, k, kind, st);
  if (rc) return rc;
  const MinArgs ma = min_args(b);
  CUDA_TRY(b->ctx, launch_min(kMinOpFireInit, ma, nullptr, st));
  if ((rc = min_run(b, 1, n_steps, st))) return rc;
  CUDA_TRY(b->ctx, launch_min(kMinOpFireEnd, ma, nullptr, st));
  if (flags & PB2_FIRE_KEEP_BEST) CUDA_TRY(b->ctx, launch_min(kMinOpTakeBest, ma, nullptr, st));
  CUDA_TRY(b->ctx, launch_min(kMinOpRollback, ma, nullptr, st));
  b->forces_valid = false;
  if ((rc = forces_not_from_step(b, st))) return rc;
  CUDA_TRY(b->ctx, cudaStreamSynchronize(st));
  return PB2_OK;
}


static LbfgsArgs lbfgs_args(pb2_batch *b, double tol, double max_step) {
  LbfgsArgs a;
  a.m = min_args(b);
  a.energy = b->lb_energy;
  a.g = b->lb_g; a.d = b->lb_d; a.x0 = b->lb_x0;
  a.hs = b->lb_hs; a.hy = b->lb_hy; a.rho = b->lb_rho;
  a.e0 = b->lb_sys; a.gd = b->lb_sys + b->n_sys; a.t = b->lb_sys + 2 * (size_t)b->n_sys;
  a.count = b->lb_int; a.head = b->lb_int + b->n_sys; a.flags = b->lb_int + 2 * (size_t)b->n_sys;
  a.hist = b->lb_hist;
  a.tol = tol;
  a.max_step = max_step;
  return a;
}

// Forces and FP64 energies at the current positions into lb_energy.
static int lbfgs_eval(pb2_batch *b, cudaStream_t st) {
  int rc = fresh_forces(b, st, true);
  if (rc) return rc;
  CUDA_TRY(b->ctx, launch_energies_to_double(b->energy, b->lb_energy, b->n_sys, st));
  return PB2_OK;
}

extern "C" int pb2_min_lbfgs(pb2_batch *b, int32_t n_iter, double tol, double max_step, int32_t hist,
                             int32_t max_trials, int32_t *converged, void *stream) {
  if (!b) return PB2_EINVAL;
  pb2_ctx *ctx = b->ctx;
  if (!b->min_ready) return fail(ctx, PB2_EINVAL, "call pb2_min_setup first");
  if (n_iter < 0 || hist < 1 || hist > kLbfgsMaxHist || !(max_step > 0.0) || !(tol >= 0.0) || max_trials < 1)
    return fail(ctx, PB2_EINVAL, "bad L-BFGS arguments");
  cudaStream_t st = (cudaStream_t)stream;
  CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  const size_t N3 = 3 * (size_t)b->n_total, S = b->n_sys;
  if (b->lb_hist != hist) {
    Dev &D = b->mdev;
    for (void *p : {(void *)b->lb_g, (void *)b->lb_d, (void *)b->lb_x0, (void *)b->lb_hs, (void *)b->lb_hy,
                    (void *)b->lb_rho, (void *)b->lb_sys, (void *)b->lb_energy, (void *)b->lb_int})
      if (p) D.release(p);
    b->lb_g = D.alloc<double>(N3);
    b->lb_d = D.alloc<double>(N3);
    b->lb_x0 = D.alloc<double>(N3);
    b->lb_hs = D.alloc<double>(hist * N3);
    b->lb_hy = D.alloc<double>(hist * N3);
    b->lb_rho = D.alloc<double>(hist * S);
    b->lb_sys = D.alloc<double>(3 * S);
    b->lb_energy = D.alloc<double>(S * PB2_NTERMS);
    b->lb_int = D.alloc<int32_t>(3 * S);
    if (!b->lb_g || !b->lb_d || !b->lb_x0 || !b->lb_hs || !b->lb_hy || !b->lb_rho || !b->lb_sys ||
        !b->lb_energy || !b->lb_int) {
      b->lb_hist = 0;
      return fail(ctx, PB2_ENOMEM, "L-BFGS allocation failed");
    }
    b->lb_hist = hist;
  }
  const LbfgsArgs la = lbfgs_args(b, tol, max_step);
  int rc = lbfgs_eval(b, st);
  if (rc) return rc;
  CUDA_TRY(ctx, launch_lbfgs(kLbfgsOpBegin, la, 0, st));
  std::vector<int32_t> flags(S);
  for (int it = 0; it < n_iter; ++it) {
    CUDA_TRY(ctx, launch_lbfgs(kLbfgsOpDirection, la, 0, st));
    for (int trial = 0; trial < max_trials; ++trial) {
      CUDA_TRY(ctx, launch_lbfgs(kLbfgsOpTrial, la, 0, st));
      if ((rc = lbfgs_eval(b, st))) return rc;
      CUDA_TRY(ctx, launch_lbfgs(kLbfgsOpCheck, la, trial == max_trials - 1, st));
      CUDA_TRY(ctx, cudaMemcpyAsync(flags.data(), la.flags, S * sizeof(int32_t), cudaMemcpyDeviceToHost, st));
      CUDA_TRY(ctx, cudaStreamSynchronize(st));
      bool searching = false;
      for (int32_t f : flags) searching |= !(f & (kLbfgsAccepted | kLbfgsDone));
      if (!searching) break;
    }
    bool all_done = true;
    for (int32_t f : flags) all_done &= (f & kLbfgsDone) != 0;
    if (all_done) break;
  }
  if (converged)
    for (size_t s = 0; s < S; ++s) converged[s] = (flags[s] & kLbfgsDone) ? 1 : 0;
  b->forces_valid = true;  // the last evaluation is at the final positions
  if (int rc2 = forces_not_from_step(b, st)) return rc2;
  CUDA_TRY(ctx, cudaStreamSynchronize(st));
  return PB2_OK;
}

extern "C" int pb2_min_rms(pb2_batch *b, double *rms, void *stream) {
  if (!b || !rms) return PB2_EINVAL;
  pb2_ctx *ctx = b->ctx;
  if (!b->min_ready) return fail(ctx, PB2_EINVAL, "call pb2_min_setup first");
  cudaStream_t st = (cudaStream_t)stream;
  CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  if (!b->forces_valid) {
    int rc = fresh_forces(b, st, false);
    if (rc) return rc;
  }
  double *out = b->m_sys + 3 * (size_t)b->n_sys;
  CUDA_TRY(ctx, launch_min(kMinOpRms, min_args(b), out, st));
  CUDA_TRY(ctx, cudaMemcpyAsync(rms, out, b->n_sys * sizeof(double), cudaMemcpyDeviceToHost, st));
  CUDA_TRY(ctx, cudaStreamSynchronize(st));
  return PB2_OK;
}


// Exchange the dynamical state of whole systems: slot s takes x, p and F of
// slot perm[s].  Keys, step counters and per-system constants (kT, dt)
// stay with their slots.  The systems swapped must have the same atom count.
extern "C" int pb2_permute_systems(pb2_batch *b, const int32_t *perm, void *stream) {
  if (!b || !perm) return PB2_EINVAL;
  pb2_ctx *ctx = b->ctx;
  cudaStream_t st = (cudaStream_t)stream;
  std::vector<char> seen(b->n_sys, 0);
  for (int s = 0; s < b->n_sys; ++s) {
    const int t = perm[s];
    if (t < 0 || t >= b->n_sys || seen[t]) return fail(ctx, PB2_EINVAL, "perm is not a permutation");
    seen[t] = 1;
    if (b->nat[t] != b->nat[s]) return fail(ctx, PB2_EINVAL, "permuted systems differ in atom count");
  }
  CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  if (!b->d_perm) {
    b->d_perm = b->dev.alloc<int32_t>(b->n_sys);
    if (!b->d_perm) return fail(ctx, PB2_ENOMEM, "permutation buffer allocation failed");
  }
  CUDA_TRY(ctx, cudaMemcpyAsync(b->d_perm, perm, b->n_sys * sizeof(int32_t), cudaMemcpyHostToDevice, st));
  const size_t N = b->n_total;
  void *groups[3][3] = {{b->x, b->y, b->z}, {b->px, b->py, b->pz}, {b->fx, b->fy, b->fz}};
  for (auto &g : groups) {
    for (int c = 0; c < 3; ++c)
      CUDA_TRY(ctx, launch_gather_systems(b->sys, b->atom_sys, b->d_perm, b->user, b->devidx, g[c], b->stage + c * N,
                                            b->n_total, st));
    for (int c = 0; c < 3; ++c)
      CUDA_TRY(ctx, cudaMemcpyAsync(g[c], b->stage + c * N, N * sizeof(double), cudaMemcpyDeviceToDevice, st));
  }
  CUDA_TRY(ctx, launch_posq(int_args(b, b->key_parity, 0), st));
  CUDA_TRY(ctx, cudaStreamSynchronize(st));
  return PB2_OK;
}


// ------------------------------------------------------------ trajectories

extern "C" int pb2_traj_setup(pb2_batch *b, int32_t capacity) {
  if (!b || capacity <= 0) return PB2_EINVAL;
  pb2_ctx *ctx = b->ctx;
  CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  const size_t f = 3 * (size_t)b->n_total;
  if (capacity != b->traj_cap) {
    if (b->traj_pos) {
      b->tdev.release(b->traj_pos);
      b->tdev.release(b->traj_vel);
      b->tdev.release(b->traj_steps);
    }
    b->traj_pos = b->tdev.alloc<float>((size_t)capacity * f);
    b->traj_vel = b->tdev.alloc<float>((size_t)capacity * f);
    b->traj_steps = b->tdev.alloc<long long>((size_t)capacity * b->n_sys);
    if (!b->traj_pos || !b->traj_vel || !b->traj_steps) {
      b->traj_cap = 0;
      return fail(ctx, PB2_ENOMEM, "trajectory ring allocation failed");
    }
    b->traj_cap = capacity;
  }
  return PB2_OK;
}

extern "C" int pb2_traj_snapshot(pb2_batch *b, int32_t slot, void *stream) {
  if (!b) return PB2_EINVAL;
  pb2_ctx *ctx = b->ctx;
  if (slot < 0 || slot >= b->traj_cap) return fail(ctx, PB2_EINVAL, "trajectory slot out of range");
  const size_t f = 3 * (size_t)b->n_total;
  CUDA_TRY(ctx, launch_snapshot(b->x, b->y, b->z, b->px, b->py, b->pz, b->mass, b->steps, b->user,
                                b->traj_pos + slot * f, b->traj_vel + slot * f,
                                b->traj_steps + (size_t)slot * b->n_sys, b->n_total, b->n_sys,
                                (cudaStream_t)stream));
  return PB2_OK;
}

extern "C" int pb2_traj_fetch(pb2_batch *b, int32_t first, int32_t count, float *positions, float *velocities,
                              int64_t *steps, void *stream) {
  if (!b) return PB2_EINVAL;
  pb2_ctx *ctx = b->ctx;
  if (first < 0 || count < 0 || first + count > b->traj_cap)
    return fail(ctx, PB2_EINVAL, "trajectory slots out of range");
  cudaStream_t st = (cudaStream_t)stream;
  const size_t f = 3 * (size_t)b->n_total;
  if (positions)
    CUDA_TRY(ctx, cudaMemcpyAsync(positions, b->traj_pos + first * f, count * f * sizeof(float),
                                  cudaMemcpyDeviceToHost, st));
  if (velocities)
    CUDA_TRY(ctx, cudaMemcpyAsync(velocities, b->traj_vel + first * f, count * f * sizeof(float),
                                  cudaMemcpyDeviceToHost, st));
  if (steps)
    CUDA_TRY(ctx, cudaMemcpyAsync(steps, b->traj_steps + (size_t)first * b->n_sys,
                                  (size_t)count * b->n_sys * sizeof(long long), cudaMemcpyDeviceToHost, st));
  CUDA_TRY(ctx, cudaStreamSynchronize(st));
  return PB2_OK;
}

extern "C" int pb2_get_status(pb2_batch *b, uint32_t *status, int clear, void *stream) {
  if (!b || !status) return PB2_EINVAL;
  pb2_ctx *ctx = b->ctx;
  cudaStream_t st = (cudaStream_t)stream;
  CUDA_TRY(ctx, cudaMemcpyAsync(status, b->status, b->n_sys * sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
  if (clear) CUDA_TRY(ctx, cudaMemsetAsync(b->status, 0, b->n_sys * sizeof(uint32_t), st));
  CUDA_TRY(ctx, cudaStreamSynchronize(st));
  return PB2_OK;
}

extern "C" int pb2_set_safeguards(pb2_batch *b, double vlimit, double max_dx, double force_cap) {
  if (!b) return PB2_EINVAL;
  pb2_ctx *ctx = b->ctx;
  if (!std::isfinite(vlimit) || !std::isfinite(max_dx) || !std::isfinite(force_cap))
    return fail(ctx, PB2_EINVAL, "safeguard limits must be finite");
  const double g[3] = {vlimit > 0.0 ? vlimit : 0.0, max_dx > 0.0 ? max_dx : 0.0,
                       force_cap > 0.0 ? force_cap : 0.0};
  if (g[0] == b->guard[0] && g[1] == b->guard[1] && g[2] == b->guard[2]) return PB2_OK;
  CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  CUDA_TRY(ctx, cudaDeviceSynchronize());
  for (int k = 0; k < 3; ++k) b->guard[k] = g[k];
  for (auto &kv : b->graphs) cudaGraphExecDestroy(kv.second);  // they hold the old limits
  b->graphs.clear();
  return PB2_OK;
}

extern "C" int pb2_get_safeguards(const pb2_batch *b, double *vlimit, double *max_dx, double *force_cap) {
  if (!b) return PB2_EINVAL;
  if (vlimit) *vlimit = b->guard[0];
  if (max_dx) *max_dx = b->guard[1];
  if (force_cap) *force_cap = b->guard[2];
  return PB2_OK;
}

extern "C" int pb2_get_warn_counts(pb2_batch *b, int32_t *counts, int reset, void *stream) {
  if (!b || !counts) return PB2_EINVAL;
  pb2_ctx *ctx = b->ctx;
  cudaStream_t st = (cudaStream_t)stream;
  const size_t S = (size_t)b->n_sys;
  std::vector<uint32_t> flags(2 * S);
  CUDA_TRY(ctx, cudaMemcpyAsync(counts, b->warn_counts, S * kWarnTypes * sizeof(int32_t), cudaMemcpyDeviceToHost, st));
  CUDA_TRY(ctx, cudaMemcpyAsync(flags.data(), b->warn_flags, 2 * S * sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
  if (reset) {
    CUDA_TRY(ctx, cudaMemsetAsync(b->warn_counts, 0, S * kWarnTypes * sizeof(int32_t), st));
    CUDA_TRY(ctx, cudaMemsetAsync(b->warn_flags, 0, 2 * S * sizeof(uint32_t), st));
  }
  CUDA_TRY(ctx, cudaStreamSynchronize(st));
  // caps recorded by the last launch and not yet folded into the counts
  for (size_t h = 0; h < 2; ++h)
    for (size_t s = 0; s < S; ++s)
      for (int k = 0; k < kWarnTypes; ++k)
        if (flags[h * S + s] & (1u << k)) counts[s * kWarnTypes + k] += 1;
  return PB2_OK;
}

extern "C" int pb2_set_tile_segment(pb2_batch *b, int32_t segment) {
  if (!b || segment <= 0) return PB2_EINVAL;
  pb2_ctx *ctx = b->ctx;
  CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  if (segment == b->params.tile_segment) return PB2_OK;
  CUDA_TRY(ctx, cudaDeviceSynchronize());
  b->params.tile_segment = segment;
  if (int rc = setup_items2(b, segment)) return rc;
  if (int rc = setup_pair_list(b, segment)) return rc;
  b->drop_graphs();  // they hold the old list
  return PB2_OK;
}

extern "C" int pb2_retire_system(pb2_batch *b, int32_t sys, void *stream) {
  if (!b) return PB2_EINVAL;
  pb2_ctx *ctx = b->ctx;
  if (sys < 0 || sys >= b->n_sys) return fail(ctx, PB2_EINVAL, "system index out of range");
  CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  if (b->retired_host[sys]) return PB2_OK;
  b->retired_host[sys] = 1;
  CUDA_TRY(ctx, launch_retire(sys, b->retired, b->items2_all, b->n_items2, b->items2, b->item_count,
                              b->pl_on ? b->pl_ctl : nullptr, (cudaStream_t)stream));
  CUDA_TRY(ctx, launch_retire(-1, b->retired, b->items4_all, b->n_items4, b->items4, b->item_count4, nullptr,
                              (cudaStream_t)stream));
  return PB2_OK;
}

extern "C" int pb2_test_hold_system(pb2_batch *b, int32_t sys, int32_t hold) {
  if (!b) return PB2_EINVAL;
  pb2_ctx *ctx = b->ctx;
  if (sys < 0 || sys >= b->n_sys || hold < 0) return fail(ctx, PB2_EINVAL, "bad system or hold");
  if (b->pl_on) return fail(ctx, PB2_EINVAL, "the pair list writes its own item counts");
  CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  CUDA_TRY(ctx, cudaDeviceSynchronize());
  const int32_t v = b->sys_items_host[sys] + hold;
  CUDA_TRY(ctx, cudaMemcpy(b->sys_items + sys, &v, sizeof v, cudaMemcpyHostToDevice));
  return PB2_OK;
}

extern "C" int pb2_test_schedule(const pb2_batch *b, int32_t *pair_list, int32_t *team, int32_t *replayed) {
  if (!b) return PB2_EINVAL;
  if (pair_list) *pair_list = b->pl_on;
  if (team) *team = b->team;
  if (replayed) *replayed = b->eval_replayed;
  return PB2_OK;
}

extern "C" int pb2_get_tile_segment(const pb2_batch *b, int32_t *segment) {
  if (!b || !segment) return PB2_EINVAL;
  *segment = b->params.tile_segment;
  return PB2_OK;
}

static void any_shape(int pass, int k, int *t, int *m) {
  if (pass == 3) force4_shape(k, t, m);
  else tile_shape(pass, k, t, m);
}

extern "C" int pb2_block_shapes(int32_t pass, int32_t *threads, int32_t *min_blocks, int32_t capacity) {
  if (pass < 0 || pass > 3) return PB2_EINVAL;
  for (int k = 0; k < kShapesPerPass && k < capacity; ++k) {
    int t = 0, m = 0;
    any_shape(pass, k, &t, &m);
    if (threads) threads[k] = t;
    if (min_blocks) min_blocks[k] = m;
  }
  return kShapesPerPass;
}

extern "C" int pb2_set_block_shape(pb2_batch *b, int32_t pass, int32_t threads, int32_t min_blocks) {
  if (!b || pass < 0 || pass > 3) return PB2_EINVAL;
  pb2_ctx *ctx = b->ctx;
  int found = -1;
  for (int k = 0; k < kShapesPerPass; ++k) {
    int t = 0, m = 0;
    any_shape(pass, k, &t, &m);
    if (t == threads && m == min_blocks) found = k;
  }
  if (found < 0) return fail(ctx, PB2_EINVAL, "block shape not compiled for this pass (see pb2_block_shapes)");
  if (found == (pass == 3 ? b->shape4 : b->shape[pass])) return PB2_OK;
  CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  CUDA_TRY(ctx, cudaDeviceSynchronize());
  if (pass == 3) {
    b->shape4 = found;
    set_force4_grid(b);
  } else {
    b->shape[pass] = found;
    set_pair_grid(b, pass);
  }
  b->drop_graphs();  // they hold the old kernel
  return PB2_OK;
}

extern "C" int pb2_get_block_shape(const pb2_batch *b, int32_t pass, int32_t *threads, int32_t *min_blocks) {
  if (!b || pass < 0 || pass > 3 || !threads || !min_blocks) return PB2_EINVAL;
  int t = 0, m = 0;
  any_shape(pass, pass == 3 ? b->shape4 : b->shape[pass], &t, &m);
  *threads = t;
  *min_blocks = m;
  return PB2_OK;
}

extern "C" int pb2_set_force_blocks(pb2_batch *b, int32_t blocks) {
  if (!b || (blocks != 2 && blocks != 4)) return PB2_EINVAL;
  if (blocks == b->force_blocks) return PB2_OK;
  CUDA_TRY(b->ctx, cudaSetDevice(b->ctx->device));
  CUDA_TRY(b->ctx, cudaDeviceSynchronize());
  b->force_blocks = blocks;
  b->drop_graphs();  // they hold the other kernel
  return PB2_OK;
}

extern "C" int pb2_get_force_blocks(const pb2_batch *b, int32_t *blocks) {
  if (!b || !blocks) return PB2_EINVAL;
  *blocks = b->force_blocks;
  return PB2_OK;
}

extern "C" int pb2_set_fusion(pb2_batch *b, int32_t flags) {
  if (!b || (flags & ~(PB2_FUSE_BONDED | PB2_FUSE_FINALIZE))) return PB2_EINVAL;
  if (flags == b->fuse) return PB2_OK;
  CUDA_TRY(b->ctx, cudaSetDevice(b->ctx->device));
  CUDA_TRY(b->ctx, cudaDeviceSynchronize());
  b->fuse = flags;
  b->drop_graphs();  // they hold the old schedule
  return PB2_OK;
}

extern "C" int pb2_get_fusion(const pb2_batch *b, int32_t *flags) {
  if (!b || !flags) return PB2_EINVAL;
  *flags = b->fuse;
  return PB2_OK;
}

extern "C" int pb2_set_profiling(pb2_batch *b, int enable) {
  if (!b) return PB2_EINVAL;
  b->profiling = enable != 0;
  return PB2_OK;
}

extern "C" int pb2_last_timings(pb2_batch *b, double *out_ms) {
  if (!b || !out_ms) return PB2_EINVAL;
  for (int k = 0; k < kTimSlots; ++k) out_ms[k] = b->timings[k];
  return PB2_OK;
}

// Neighbour-list entry points: the list is built in pb2_nlist.cu.
