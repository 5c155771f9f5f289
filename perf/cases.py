"""The work a user has this framework do, as cases to time and to compare.

Three paths through the public entry points, over the sizes of the
repository's own configurations (one chain of 166 atoms, a 2,500-atom globule
with CMAP and a 20 A cutoff, 20,000 atoms, ragged batches of 150-4,000 and
100-10,000 atoms):

* ``energy``: ``make_energy_fn(...)`` called on a CUDA tensor, as a program
  that holds float32 coordinates calls it (line searches, reporting,
  reweighting, force matching): total energy in float64 and the forces,
  handed on in the precision of the coordinates;
* ``batch_energy`` / ``batch_forces``: the same for many systems at once on
  device arrays (``Batch.energy_forces_device``), with the energies per term
  or for the forces alone (an integrator that lives elsewhere);
* ``md``: ``Batch.langevin_run`` and the frame a trajectory keeps of its end
  (float32 positions and velocities, the step counters);
* ``minimize``: restrained steepest descent and FIRE from given positions,
  and the structure it ends at as a float32 frame.

``exact`` restates the formulas in plain torch, in 64 bits.
"""

import math

import numpy as np
import torch

from prolix_b200 import engine, synth
from prolix_b200.system import make_energy_fn

DENSITY = 0.075   # atoms / A^3 of a globule
MAX_CHAIN = 4000  # larger systems are assemblies of chains


def listed():
  return [
      # one small peptide: every launch and every wait counts
      dict(name="energy_166", kind="energy", systems=1, lo=166, hi=166, cutoff=0.0, cmap=False),
      # an ordinary protein with CMAP; direct terms cut off at 20 A, GB over all pairs
      dict(name="energy_2500_cut20", kind="energy", systems=1, lo=2500, hi=2500, cutoff=20.0, cmap=True),
      # a large assembly, all pairs
      dict(name="energy_20000", kind="energy", systems=1, lo=20000, hi=20000, cutoff=0.0, cmap=True),
      # decomposed energies of an ensemble (reweighting, exchange)
      dict(name="batch_energy_32", kind="batch_energy", systems=32, lo=150, hi=4000, mix=2024, cutoff=0.0, cmap=False),
      # forces of an ensemble, for an integrator outside the library
      dict(name="batch_forces_64", kind="batch_forces", systems=64, lo=150, hi=4000, mix=2024, cutoff=0.0, cmap=False),
      # dynamics of one peptide, a chunk of 50 steps
      dict(name="md_166", kind="md", systems=1, lo=166, hi=166, cutoff=0.0, cmap=False, steps=50, guards=False),
      # dynamics of one protein, every term cut off at 20 A with the skin list
      dict(name="md_2500_cut20", kind="md", systems=1, lo=2500, hi=2500, cutoff=20.0, cmap=True, steps=25,
           guards=False),
      # dynamics of a large assembly, with the list and over all pairs
      dict(name="md_20000_cut20", kind="md", systems=1, lo=20000, hi=20000, cutoff=20.0, cmap=True, steps=10,
           guards=False),
      dict(name="md_20000", kind="md", systems=1, lo=20000, hi=20000, cutoff=0.0, cmap=True, steps=5,
           guards=False),
      # the ragged ensemble the framework is built for
      dict(name="md_ragged_256", kind="md", systems=256, lo=150, hi=4000, mix=2024, cutoff=0.0, cmap=False, steps=5,
           guards=False),
      # a served cohort of uneven systems, with the batched step's safeguards
      dict(name="md_served_16", kind="md", systems=16, lo=100, hi=10000, mix=2024, cutoff=0.0, cmap=False, steps=25,
           guards=True),
      # preparing an ensemble for dynamics
      dict(name="minimize_16", kind="minimize", systems=16, lo=150, hi=4000, mix=2024, cutoff=0.0, cmap=False, sd=20,
           fire=30),
  ]


def _log_uniform(rng, lo, hi):
  return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
  kind = rng.choice(["energy", "energy", "batch_energy", "batch_forces", "md", "md", "md", "minimize"])
  cutoff = rng.choice([0.0, 0.0, 20.0, round(rng.uniform(9.0, 22.0), 2)])
  cmap = rng.random() < 0.4
  if kind == "energy" or (kind == "md" and rng.random() < 0.6):
    n = _log_uniform(rng, 100, 20000)
    case = dict(kind=kind, systems=1, lo=n, hi=n, cutoff=cutoff, cmap=cmap)
  else:
    systems = _log_uniform(rng, 2, 64 if kind != "md" else 128)
    lo = _log_uniform(rng, 100, 400)
    case = dict(kind=kind, systems=systems, lo=lo, hi=_log_uniform(rng, 500, 4000), mix=rng.randint(0, 9999),
                cutoff=cutoff, cmap=cmap)
  if kind == "md":
    most = 50 if case["hi"] <= 4000 and case["systems"] <= 4 else 10 if case["hi"] <= 10000 else 5
    case.update(steps=rng.randint(1, most), guards=rng.random() < 0.3)
  if kind == "minimize":
    case.update(sd=rng.randint(5, 20), fire=rng.randint(5, 30))
  return case


# ------------------------------------------------------------------- inputs


def _sizes(case):
  if case["lo"] == case["hi"]:
    return [case["lo"]] * case["systems"]
  return [int(n) for n in synth.batch_sizes(case["systems"], case["mix"], case["lo"], case["hi"])]


def _globules(n, seed, cmap):
  """``n`` atoms: one compact chain, or an assembly of equal chains on a
  cubic grid (an oligomer) where one chain would be larger than MAX_CHAIN."""
  chains = max(1, math.ceil(n / 2500)) if n > MAX_CHAIN else 1
  cuts = np.linspace(0, n, chains + 1).astype(int)
  parts = [synth.make_chain(int(b - a), seed + 7919 * k, compact=True, cmap=cmap, **synth.PHYSICAL_RANGES)
           for k, (a, b) in enumerate(zip(cuts[:-1], cuts[1:]))]
  if chains == 1:
    return parts[0]
  gap = 2.0 * max(float(np.abs(p["positions"]).max()) for p in parts) + 2.5
  side = math.ceil(chains ** (1.0 / 3.0))
  out = {"seed": seed}
  for k, p in enumerate(parts):
    cell = np.array([k % side, (k // side) % side, k // (side * side)], dtype=np.float64)
    p["positions"] = p["positions"] + gap * (cell - 0.5 * (side - 1))
    for key in ("bonds", "angles", "dihedrals", "cmap_torsions"):
      if key in p:
        p[key] = p[key] + np.int32(cuts[k])
    if cmap:
      p["cmap_indices"] = p["cmap_indices"] + np.int32(k)
  for key in parts[0]:
    if key != "seed":
      out[key] = np.concatenate([p[key] for p in parts])
  return out


def _systems(case, seed):
  out = []
  for k, n in enumerate(_sizes(case)):
    s = _globules(n, (seed * 1000003 + 17 * k) % (1 << 31), case["cmap"])
    # chain neighbours: one and two bonds apart excluded, three scaled
    b = s["bonds"]
    bonded = np.zeros(n, dtype=bool)
    bonded[b[:, 0]] = True  # atom i is bonded to i + 1
    i = np.arange(n)
    pairs, kind = [], []
    ok = np.ones(n, dtype=bool)
    for d in (1, 2, 3):
      ok = ok & np.concatenate([bonded[d - 1:], np.zeros(d - 1, dtype=bool)])
      pairs.append(np.stack([i[ok], i[ok] + d], axis=1))
      kind.append(np.full(int(ok.sum()), 1 if d == 3 else 0))
    s["excl_pairs"] = np.concatenate(pairs).astype(np.int32)
    s["excl_kind"] = np.concatenate(kind).astype(np.int32)
    s["key"] = (seed & 0xFFFFFFFF, k)
    out.append(s)
  return out


def _coordinates(systems, seed):
  """Coordinates to evaluate at: the structures after small thermal
  displacements, in float32."""
  rng = np.random.default_rng(seed + 1)
  x = np.concatenate([s["positions"] for s in systems])
  return (x + 0.02 * rng.standard_normal(x.shape)).astype(np.float32)


def prepare(case, seed):
  systems = _systems(case, seed)
  kind = case["kind"]
  if kind == "energy":
    fn = make_energy_fn(None, systems[0], cutoff=case["cutoff"], implicit_solvent=True)
    return {"kind": kind, "fn": fn, "r": torch.from_numpy(_coordinates(systems, seed)).cuda()}
  b = engine.Batch(systems, cutoff=case["cutoff"], skin=2.0)
  state = {"kind": kind, "batch": b}
  if kind in ("batch_energy", "batch_forces"):
    state["r"] = torch.from_numpy(_coordinates(systems, seed)).cuda()
    state["f"] = torch.empty((b.n_atoms, 3), dtype=torch.float64, device="cuda")
    if kind == "batch_energy":
      state["e"] = torch.empty((b.n_systems, 12), dtype=torch.float64, device="cuda")
  elif kind == "md":
    if case["guards"]:
      b.set_safeguards(**engine.BATCHED_SAFEGUARDS)
    b.traj_setup(1)
    b.langevin_init()
    state["steps"] = case["steps"]
  else:
    state["x0"] = np.concatenate([s["positions"] for s in systems])
    state["sd"], state["fire"] = case["sd"], case["fire"]
  return state


def run(state):
  kind = state["kind"]
  if kind == "energy":
    e, f = state["fn"].energy_and_forces(state["r"])
    return {"energy": e, "forces": f.to(state["r"].dtype)}
  b = state["batch"]
  stream = torch.cuda.current_stream().cuda_stream
  if kind in ("batch_energy", "batch_forces"):
    x = state["r"].to(torch.float64)
    e = state.get("e")
    b.energy_forces_device(x.data_ptr(), e.data_ptr() if e is not None else 0, state["f"].data_ptr(), stream)
    out = {"forces": state["f"].to(state["r"].dtype)}
    if e is not None:
      out["energies"] = e
    return out
  if kind == "md":
    b.langevin_run(state["steps"], stream)
    b.traj_snapshot(0, stream)
    pos, vel, steps = b.traj_fetch(0, 1, stream)
    return {"positions": pos, "velocities": vel, "steps": steps}
  b.set_positions(state["x0"], stream)
  b.min_setup()
  b.min_sd(state["sd"], k=500.0, kind="heavy", dt=0.002, max_dx=0.01, stream=stream)
  b.min_fire(state["fire"], k=0.0, kind="all", dt_start=1e-4, dt_max=1e-3, max_disp=0.1, stream=stream)
  return {"positions": b.get_state(stream, fields=("position",))["position"].astype(np.float32)}


# -------------------------------------------------------------- minimal work

# Floating-point operations per unique pair within reach (fused multiply-add
# = 2): descreening 33, pair forces 55, chain rule 49; an energy adds the
# descreening integrals and the three pair terms once more.
PAIR_FORCE = 33 + 55 + 49
PAIR_ENERGY = 33 + 45


def _pairs(n, cutoff):
  full = 0.5 * n * (n - 1)
  return full if cutoff <= 0 else min(full, 0.5 * n * DENSITY * 4.18879 * cutoff ** 3)


def work(case):
  sizes = _sizes(case)
  atoms = sum(sizes)
  all_pairs = sum(_pairs(n, 0.0) for n in sizes)
  cut_pairs = sum(_pairs(n, case["cutoff"]) for n in sizes)
  kind = case["kind"]
  if kind == "energy":  # GB over all pairs, direct terms within the cutoff
    return {"bytes": atoms * (24 + 24 + 64), "flops": all_pairs * (PAIR_FORCE - 20 + 33 + 25) + cut_pairs * 40}
  if kind == "batch_energy":
    return {"bytes": atoms * (24 + 24 + 64), "flops": cut_pairs * (PAIR_FORCE + PAIR_ENERGY)}
  if kind == "batch_forces":
    return {"bytes": atoms * (24 + 24 + 64), "flops": cut_pairs * PAIR_FORCE}
  if kind == "md":  # state, parameters and noise of a step: 184 B per atom
    return {"bytes": atoms * (184 * case["steps"] + 24), "flops": cut_pairs * PAIR_FORCE * case["steps"]}
  evals = case["sd"] + case["fire"] + 1
  return {"bytes": atoms * 184 * evals, "flops": cut_pairs * PAIR_FORCE * evals}


# ------------------------------------------------------------------ 64 bits

K_COULOMB = 332.0637
LJ14, COUL14 = float(np.float32(0.5)), float(np.float32(0.83333333))
OFFSET = 0.09
ROWS = 1 << 23  # pairs held at once


def _dihedral(x, idx):
  ri, rj, rk, rl = (x[idx[:, c]] for c in range(4))
  b0, b1, b2 = ri - rj, rk - rj, rl - rk
  u = b1 / (b1.norm(dim=1, keepdim=True) + 1e-8)
  v = b0 - (b0 * u).sum(1, keepdim=True) * u
  w = b2 - (b2 * u).sum(1, keepdim=True) * u
  return torch.atan2((torch.linalg.cross(u, v) * w).sum(1), (v * w).sum(1))


def _spline_slope(g):
  """Matrix of the knot derivatives of a periodic cubic spline through g
  values at spacing 2 pi / g."""
  h = 2.0 * math.pi / g
  eye = torch.eye(g, dtype=torch.float64)
  nxt, prv = eye.roll(1, dims=1), eye.roll(-1, dims=1)
  second = torch.linalg.solve(4.0 * h * eye + h * nxt + h * prv, 6.0 / h * (nxt - 2.0 * eye + prv))
  return (nxt - eye) / h - h / 6.0 * (2.0 * second + nxt @ second)


class _System:
  """Energy terms and forces of one system, in 64 bits on the GPU."""

  def __init__(self, s, cutoff, gb_cutoff):
    t = lambda k: torch.as_tensor(np.asarray(s[k]), dtype=torch.float64).cuda()  # noqa: E731
    i = lambda k: torch.as_tensor(np.asarray(s[k]), dtype=torch.int64).cuda()  # noqa: E731
    self.n = len(s["charges"])
    self.q, self.sig, self.eps = t("charges"), t("sigmas"), t("epsilons")
    self.rad, self.sr, self.m = t("radii"), t("scaled_radii"), t("masses")
    self.cut2, self.gcut2 = cutoff * cutoff, gb_cutoff * gb_cutoff
    self.bonds, self.bp = i("bonds"), t("bond_params")
    self.angles, self.ap = i("angles"), t("angle_params")
    self.dih, self.dp = i("dihedrals"), t("dihedral_params").reshape(-1, 3)
    self.excl, self.kind = i("excl_pairs"), i("excl_kind")
    self.cmap = None
    if "cmap_torsions" in s and len(s["cmap_torsions"]):
      e = torch.as_tensor(np.asarray(s["cmap_energy_grids"]), dtype=torch.float64).transpose(1, 2)  # (phi, psi)
      d = _spline_slope(e.shape[1])
      dv = e @ d.T
      self.cmap = [m.cuda() for m in (e, d @ e, dv, d @ dv)]
      self.crow, self.cmapi = i("cmap_torsions"), i("cmap_indices")

  def bonded(self, x):
    """(bond, angle, dihedral, cmap) energies."""
    b = (x[self.bonds[:, 0]] - x[self.bonds[:, 1]]).norm(dim=1)
    e_b = (0.5 * self.bp[:, 1] * (b - self.bp[:, 0]) ** 2).sum()
    va, vb = x[self.angles[:, 0]] - x[self.angles[:, 1]], x[self.angles[:, 2]] - x[self.angles[:, 1]]
    c = (va * vb).sum(1) / (va.norm(dim=1) * vb.norm(dim=1) + 1e-8)
    e_a = (0.5 * self.ap[:, 1] * (torch.arccos(c.clamp(-0.999999, 0.999999)) - self.ap[:, 0]) ** 2).sum()
    e_d = (self.dp[:, 2] * (1.0 + torch.cos(self.dp[:, 0] * _dihedral(x, self.dih) - self.dp[:, 1]))).sum()
    e_c = torch.zeros((), dtype=torch.float64, device=x.device)
    if self.cmap is not None:
      g = self.cmap[0].shape[1]
      delta = 2.0 * math.pi / g
      p = torch.remainder(_dihedral(x, self.crow[:, :4]), 2.0 * math.pi) / delta
      s = torch.remainder(_dihedral(x, self.crow[:, 1:]), 2.0 * math.pi) / delta
      ia, ib = p.detach().floor().long() % g, s.detach().floor().long() % g
      hermite = lambda u: ((1 + 2 * u) * (1 - u) ** 2, u * u * (3 - 2 * u), u * (1 - u) ** 2, u * u * (u - 1))  # noqa: E731
      hu, hv = hermite(p - ia), hermite(s - ib)
      for a in (0, 1):
        for b_ in (0, 1):
          e, du, dv, duv = (t[self.cmapi, (ia + a) % g, (ib + b_) % g] for t in self.cmap)
          e_c = e_c + (e * hu[a] * hv[b_] + delta * (du * hu[2 + a] * hv[b_] + dv * hu[a] * hv[2 + b_])
                       + delta * delta * duv * hu[2 + a] * hv[2 + b_]).sum()
    return e_b, e_a, e_d, e_c

  def _rows(self):
    step = max(1, ROWS // self.n)
    for a in range(0, self.n, step):
      yield a, min(self.n, a + step)

  def _geometry(self, x, a, b):
    """r^2 of rows a..b against all atoms (1 where i = j) and the i != j mask."""
    r2 = torch.zeros((b - a, self.n), dtype=torch.float64, device=x.device)
    for c in range(3):
      r2 = r2 + (x[a:b, c, None] - x[None, :, c]) ** 2
    other = torch.ones(r2.shape, dtype=torch.bool, device=x.device)
    other[torch.arange(b - a), torch.arange(a, b)] = False
    return torch.where(other, r2, 1.0), other

  def _integral(self, r2, other, a, b):
    """The OBC integral of the rows' atoms by all others' scaled radii."""
    r, rho, s = torch.sqrt(r2 + 1e-12), (self.rad - OFFSET)[a:b, None], self.sr[None, :]
    L = torch.maximum(rho.expand_as(r), (r - s).abs())
    U = r + s
    v = 0.5 * (1 / L - 1 / U) + 0.25 * torch.log(L / U) / r + 0.125 * (r - s * s / r) * (1 / U ** 2 - 1 / L ** 2)
    keep = other & (U > rho)
    if self.gcut2 > 0:
      keep = keep & (r2 < self.gcut2)
    return torch.where(keep, v, 0.0)

  def _born(self, sums):
    rho = self.rad - OFFSET
    psi = rho * sums
    inv = 1 / rho - torch.tanh(psi - 0.8 * psi ** 2 + 4.85 * psi ** 3) / self.rad
    return 1 / (inv.clamp_min(1e-4) if self.gcut2 > 0 else inv)

  def _scales(self, a, b, device):
    """Exclusion factors (lj, coulomb) of rows a..b."""
    lj = torch.ones((b - a, self.n), dtype=torch.float64, device=device)
    co = torch.ones_like(lj)
    p = torch.cat([self.excl, self.excl.flip(1)])
    k = torch.cat([self.kind, self.kind])
    on = (p[:, 0] >= a) & (p[:, 0] < b)
    p, k = p[on], k[on]
    lj[p[:, 0] - a, p[:, 1]] = torch.where(k == 1, LJ14, 0.0).to(torch.float64)
    co[p[:, 0] - a, p[:, 1]] = torch.where(k == 1, COUL14, 0.0).to(torch.float64)
    return lj, co

  def evaluate(self, x):
    """(energies of bond, angle, dihedral, cmap, lj, coulomb, gb, nonpolar; forces)."""
    x = x.detach().requires_grad_(True)
    with torch.no_grad():
      sums = torch.cat([self._integral(*self._geometry(x, a, b), a, b).sum(1) for a, b in self._rows()])
    sums.requires_grad_(True)
    radii = self._born(sums)
    born = radii.detach().requires_grad_(True)
    pref = -0.5 * K_COULOMB * (1.0 - 1.0 / 78.5)
    r_nm = (self.rad - OFFSET) / 10.0 + 0.009
    ace = (28.3919551 * (r_nm + 0.14) ** 2 * (r_nm / (born / 10.0)) ** 6 * 0.239006).sum()
    self_gb = pref * (self.q ** 2 / born).sum()
    bonded = self.bonded(x)
    (sum(bonded) + ace + self_gb).backward()
    e_gb, e_lj, e_co = self_gb.detach(), 0.0, 0.0
    for a, b in self._rows():
      r2, other = self._geometry(x, a, b)
      qq = self.q[a:b, None] * self.q[None, :]
      bb = born[a:b, None] * born[None, :]
      g_on = other & (r2 < self.gcut2) if self.gcut2 > 0 else other
      d_on = other & (r2 < self.cut2) if self.cut2 > 0 else other
      gb = torch.where(g_on, pref * qq / torch.sqrt(r2 + bb * torch.exp(-r2 / (4 * bb))), 0.0).sum()
      lj, co = self._scales(a, b, x.device)
      inv = torch.rsqrt(r2)
      coul = torch.where(d_on, 0.5 * K_COULOMB * qq * co * inv, 0.0).sum()
      s6 = ((0.5 * (self.sig[a:b, None] + self.sig[None, :])) * inv) ** 6
      el = torch.where(d_on, 2.0 * torch.sqrt(self.eps[a:b, None] * self.eps[None, :]) * lj * (s6 * s6 - s6), 0.0).sum()
      (gb + coul + el).backward()
      e_gb, e_lj, e_co = e_gb + gb.detach(), e_lj + el.detach(), e_co + coul.detach()
    radii.backward(born.grad)
    for a, b in self._rows():
      r2, other = self._geometry(x, a, b)
      (self._integral(r2, other, a, b) * sums.grad[a:b, None]).sum().backward()
    return [*(e.detach() for e in bonded), e_lj, e_co, e_gb, ace.detach()], -x.grad


def _threefry(k0, k1, x0, x1):
  """Threefry-2x32 with 20 rounds on uint32 arrays (Salmon et al., SC'11)."""
  ks = (np.uint32(k0), np.uint32(k1), np.uint32(k0) ^ np.uint32(k1) ^ np.uint32(0x1BD11BDA))
  rot = (13, 15, 26, 6, 17, 29, 16, 24)
  with np.errstate(over="ignore"):
    x0, x1 = x0 + ks[0], x1 + ks[1]
    for r in range(20):
      x0 = x0 + x1
      x1 = ((x1 << np.uint32(rot[r % 8])) | (x1 >> np.uint32(32 - rot[r % 8]))) ^ x0
      if r % 4 == 3:
        j = r // 4 + 1
        x0, x1 = x0 + ks[j % 3], x1 + ks[(j + 1) % 3] + np.uint32(j)
  return x0, x1


def _split(key):
  a, b = _threefry(key[0], key[1], np.zeros(2, np.uint32), np.arange(2, dtype=np.uint32))
  return (a[0], b[0]), (a[1], b[1])


def _normal(key, n):
  """(n, 3) standard normals of a key: float32 uniforms, as they are drawn,
  through the inverse error function in 64 bits."""
  a, b = _threefry(key[0], key[1], np.zeros(3 * n, np.uint32), np.arange(3 * n, dtype=np.uint32))
  f = (((a ^ b) >> np.uint32(9)) | np.uint32(0x3F800000)).view(np.float32) - np.float32(1.0)
  lo = np.nextafter(np.float32(-1.0), np.float32(0.0))
  u = torch.from_numpy(np.maximum(lo, f * np.float32(2.0) + lo)).double()
  return (math.sqrt(2.0) * torch.erfinv(u)).reshape(n, 3).cuda()


def _limit(v, most, eps):
  """min(1, most / |v|) per row, and where |v| is above ``most``."""
  m = torch.sqrt((v * v).sum(1, keepdim=True) + eps)
  return (most / m).clamp(max=1.0), m > most


def _dynamics(y, s, case):
  dt, kT = 1.0 / 48.88821291839, 300.0 * 0.0019872041
  c1 = math.exp(-48.88821291839e-3 * dt)
  m = y.m[:, None]
  noise = math.sqrt(1.0 - c1 * c1) * torch.sqrt(m * kT)
  key, sub = _split(s["key"])
  x = torch.as_tensor(s["positions"], dtype=torch.float64).cuda()
  p = torch.sqrt(m * kT) * _normal(sub, y.n)
  f = y.evaluate(x)[1]
  for _ in range(case["steps"]):
    p = p + 0.5 * dt * f
    if case["guards"]:
      scale, over = _limit(p / m, 20.0, 1e-30)
      p = torch.where(over, p * scale, p)
    old = x
    x = x + 0.5 * dt * p / m
    key, sub = _split(key)
    p = c1 * p + noise * _normal(sub, y.n)
    x = x + 0.5 * dt * p / m
    if case["guards"]:
      scale, over = _limit(x - old, 0.5, 1e-30)
      x, p = old + (x - old) * scale, torch.where(over, p * scale, p)
    f = y.evaluate(x)[1]
    if case["guards"]:
      f = f * _limit(f, 1e4, 1e-12)[0]
    p = p + 0.5 * dt * f
  return x, p / m


def _minimum(y, s, case):
  x = torch.as_tensor(s["positions"], dtype=torch.float64).cuda()
  x0, heavy, m = x, (y.m > 1.1)[:, None], y.m[:, None]
  f = y.evaluate(x)[1]
  for _ in range(case["sd"]):
    d = 0.002 * (f - torch.where(heavy, 500.0 * (x - x0), 0.0))
    x = x + d * (0.01 / torch.sqrt((d * d).sum(1, keepdim=True) + 1e-30)).clamp(max=1.0)
    f = y.evaluate(x)[1]
  p, dt, alpha, ahead, best, least = torch.zeros_like(x), 1e-4, 0.1, 0, x, 1e10
  for _ in range(case["fire"]):
    rms = float(torch.sqrt((f * f).sum() / y.n))
    if rms < least:
      least, best = rms, x
    p = p + 0.5 * dt * f
    old = x
    x = x + dt * p / m
    f = y.evaluate(x)[1]
    p = p + 0.5 * dt * f
    power = float((f * p).sum())
    mix = alpha * float(torch.sqrt((p * p).sum())) / math.sqrt(float((f * f).sum()) + 1e-6)
    p = p + (mix * f - alpha * p)
    ahead = ahead + 1 if power >= 0 else 0
    if power > 0 and ahead > 5:
      dt, alpha = min(1.1 * dt, 1e-3), alpha * 0.99
    if power < 0:
      dt, alpha, p = 0.5 * dt, 0.1, torch.zeros_like(p)
    d = x - old
    scale = (0.1 / torch.sqrt((d * d).sum(1, keepdim=True) + 1e-30)).clamp(max=1.0)
    x, p = old + d * scale, p * scale
  return best


def exact(case, seed):
  kind, cutoff = case["kind"], case["cutoff"]
  if case["systems"] * (case.get("steps", 0) + case.get("sd", 0) + case.get("fire", 0)) > 2500:
    return None  # one system at a time: too long
  systems = _systems(case, seed)
  ys = [_System(s, cutoff, 0.0 if kind == "energy" else cutoff) for s in systems]
  if kind in ("energy", "batch_energy", "batch_forces"):
    r = torch.from_numpy(_coordinates(systems, seed)).cuda().double()
    parts = torch.split(r, [y.n for y in ys])
    got = [y.evaluate(p) for y, p in zip(ys, parts)]
    out = {"forces": torch.cat([f for _, f in got])}
    if kind == "energy":
      out["energy"] = sum(got[0][0])
    if kind == "batch_energy":  # exception pairs, impropers and Urey-Bradley springs: none here
      rows = torch.zeros((len(ys), 12), dtype=torch.float64, device="cuda")
      for k, (e, _) in enumerate(got):
        rows[k, :8] = torch.stack([torch.as_tensor(v, dtype=torch.float64, device="cuda") for v in e])
        rows[k, 11] = rows[k, :8].sum()
      out["energies"] = rows
    return out
  if kind == "md":
    ends = [_dynamics(y, s, case) for y, s in zip(ys, systems)]
    return {"positions": torch.cat([x for x, _ in ends])[None], "velocities": torch.cat([v for _, v in ends])[None],
            "steps": None}
  return {"positions": torch.cat([_minimum(y, s, case) for y, s in zip(ys, systems)])}
