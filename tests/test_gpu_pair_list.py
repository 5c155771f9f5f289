"""Runs with the pair list, which needs a system of 64 blocks (2,017 atoms)
or more, against the same runs without: steps, minimisation, states set from
outside and retirements, with a skin so small that the list is rebuilt during
the run (a list that missed a rebuild would drop pairs)."""

import numpy as np
import pytest

from gpu_schedule import schedule
from prolix_b200 import engine, synth

pytestmark = pytest.mark.gpu

SKIN = 0.2
FIELDS = ("position", "momentum", "force")
CUTOFFS = [dict(cutoff=9.0), dict(cutoff=8.0, gb_cutoff=12.0), dict(cutoff=10.0, born_cutoff=7.0)]


def _systems(sizes):
  return [dict(synth.make_chain(n, 700 + n, compact=True, cmap=n % 2 == 0, **synth.PHYSICAL_RANGES), key=(0, n))
          for n in sizes]


def _batch(systems, listed, **kw):
  b = engine.Batch(systems, skin=SKIN, pair_list=listed, dt=engine.akma_dt(2.0), kT=600 * engine.KB_KCAL, **kw)
  assert schedule(b)["pair_list"] == int(listed)
  return b


def _both(systems, run, **kw):
  out = []
  for listed in (True, False):
    with _batch(systems, listed, **kw) as b:
      out.append(run(b))
  for a, c in zip(*out):
    np.testing.assert_array_equal(a, c)
  return out[0]


def _state(b):
  st = b.get_state(fields=FIELDS)
  return [st[f] for f in FIELDS]


def _moved(systems, x):
  return np.linalg.norm(x - np.concatenate([s["positions"] for s in systems]), axis=1).max()


@pytest.mark.parametrize("cutoffs", CUTOFFS)
@pytest.mark.parametrize("sizes", [(2017,), (300, 2500, 2049, 33)])
def test_steps(sizes, cutoffs):
  systems = _systems(sizes)

  def run(b):
    e, f = b.energy_forces()
    b.langevin_init()
    b.langevin_run(70)
    b.langevin_run(50)
    return [e, f, *_state(b)]

  out = _both(systems, run, **cutoffs)
  assert np.isfinite(out[2]).all() and _moved(systems, out[2]) > 5 * SKIN


@pytest.mark.parametrize("segment", [2, 5])
def test_steps_at_other_item_lengths(segment):
  systems = _systems((2200, 40))

  def run(b):
    b.set_tile_segment(segment)
    b.langevin_init()
    b.langevin_run(60)
    return _state(b)

  _both(systems, run, cutoff=9.0)


def test_minimisation():
  systems = _systems((2100, 500))

  def run(b):
    b.min_setup()
    b.min_sd(40, k=10.0, kind="heavy", dt=0.002, max_dx=0.05)
    x1 = b.get_state(fields=("position",))["position"]
    b.min_fire(40, k=5.0, kind="heavy", dt_start=1e-3, dt_max=1e-2, max_disp=0.1)
    return [x1, *_state(b), b.min_rms()]

  out = _both(systems, run, cutoff=9.0)
  assert _moved(systems, out[1]) > 2 * SKIN


def test_states_set_from_outside():
  # positions far from those the list was built for, by every entry that
  # sets them, each followed by steps or an evaluation
  import torch
  systems = _systems((2300, 90))
  x0 = np.concatenate([s["positions"] for s in systems])
  far = x0[:, ::-1] * 1.02  # another orientation and scale

  def run(b):
    out = [b.forces()]
    b.set_positions(far)
    out.append(b.forces())
    b.langevin_init()
    b.langevin_run(5)
    st = b.get_state()
    b.set_state(position=x0)
    b.langevin_run(5)
    out += _state(b)
    b.set_full_state(st["position"], st["momentum"], st["force"])
    b.langevin_run(5)
    out += _state(b)
    x, p, f = (v.copy() for v in (x0, st["momentum"], out[0]))  # overwritten
    b.langevin_run_host(x, p, f, 5)
    torch.cuda.synchronize()
    out += [x, p, f]
    t = torch.from_numpy(np.ascontiguousarray(far)).cuda()
    e = torch.zeros((2, 12), dtype=torch.float64, device="cuda")
    g = torch.zeros_like(t)
    for _ in range(4):
      b.energy_forces_device(t.data_ptr(), e.data_ptr(), g.data_ptr(), torch.cuda.current_stream().cuda_stream)
    return out + [e.cpu().numpy(), g.cpu().numpy()]

  _both(systems, run, cutoff=9.0)


@pytest.mark.parametrize("retire", [0, 1])
def test_a_retired_system_leaves_the_list(retire):
  # the rest end bit for bit as in a batch that never held it, with the list
  # and (the small systems alone) without one
  systems = _systems((2100, 2400, 500))
  rest = [k for k in range(3) if k != retire]
  with _batch(systems, True, cutoff=9.0) as b:
    b.langevin_init()
    b.langevin_run(30)
    gone = b.split(b.get_state(fields=("position",))["position"])[retire]
    b.retire(retire)
    b.langevin_run(25)
    b.langevin_run(40)
    mixed = [b.split(v) for v in _state(b)]
  np.testing.assert_array_equal(mixed[0][retire], gone)
  for group, listed in ((rest, True), (rest, False)):
    with _batch([systems[k] for k in group], listed, cutoff=9.0) as b:
      b.langevin_init()
      b.langevin_run(95)
      alone = [b.split(v) for v in _state(b)]
    for m, a in zip(mixed, alone):
      for k, s in enumerate(group):
        np.testing.assert_array_equal(m[s], a[k])
