"""Evaluations of batches that run by teams, replayed as graphs: the forces
and energies of the first launches bit for bit, after every setter that drops
the graphs, after a retirement and after steps in between."""

import numpy as np
import pytest

from gpu_schedule import schedule
from prolix_b200 import _lib, autotune, engine, synth

pytestmark = pytest.mark.gpu

BATCHES = [((166,), 0.0, 8), ((40, 300, 700), 0.0, 8), ((40, 300, 700), 12.0, 8), ((900, 60, 700), 0.0, 4),
           ((900, 60, 700), 9.0, 4)]


@pytest.mark.parametrize("sizes,cutoff,team", BATCHES)
def test_replays_after_every_change(sizes, cutoff, team):
  import torch
  systems = [synth.make_chain(n, 620 + n, compact=True, cmap=n > 64, **synth.PHYSICAL_RANGES) for n in sizes]
  x0 = np.concatenate([s["positions"] for s in systems])
  rng = np.random.default_rng(5)
  xs = [torch.from_numpy(x0 + 0.03 * rng.standard_normal(x0.shape)).cuda() for _ in range(2)]
  stream = torch.cuda.current_stream().cuda_stream
  ref = []
  for x in xs:
    with engine.Batch(systems, cutoff=cutoff) as b:
      b.set_positions(x.cpu().numpy())
      ref.append(b.energy_forces())
      assert not schedule(b)["replayed"]

  def check(b, k, energies, first_atom=0, first=0):
    e = torch.zeros((len(sizes), 12), dtype=torch.float64, device="cuda")
    f = torch.zeros(x0.shape, dtype=torch.float64, device="cuda")
    b.energy_forces_device(xs[k].data_ptr(), e.data_ptr() if energies else 0, f.data_ptr(), stream)
    np.testing.assert_array_equal(f.cpu().numpy()[first_atom:], ref[k][1][first_atom:])
    if energies:
      np.testing.assert_array_equal(e.cpu().numpy()[first:], ref[k][0][first:])
    return schedule(b)["replayed"]

  with engine.Batch(systems, cutoff=cutoff) as b:
    assert schedule(b)["team"] == team == autotune.team_warps(sizes)
    # the third evaluation of each kind is the first replay
    assert [check(b, n % 2, True) for n in range(5)] == [0, 0, 1, 1, 1]
    assert [check(b, n % 2, False) for n in range(5)] == [0, 0, 1, 1, 1]
    changes = [lambda: b.set_fusion(0), lambda: b.set_fusion(_lib.FUSE_BONDED | _lib.FUSE_FINALIZE),
               lambda: b.set_force_blocks(4), lambda: b.set_fusion(_lib.FUSE_BONDED), lambda: b.set_force_blocks(2),
               lambda: b.set_block_shape(1, *b.block_shapes(1)[-1]),
               lambda: b.set_langevin_params(kT=0.5), lambda: b.set_safeguards(vlimit=20.0)]
    for change in changes:
      change()
      for n in range(3):
        assert check(b, n % 2, True) == 1
        assert check(b, n % 2, False) == 1
    b.set_tile_segment(3)  # no teams, no graphs
    assert [check(b, n % 2, n > 1) for n in range(4)] == [0, 0, 0, 0]
    b.set_tile_segment(1)
    assert [check(b, n % 2, n % 2 == 0) for n in range(4)] == [1, 1, 1, 1]
    b.set_profiling(True)
    assert check(b, 0, True) == 0
    b.set_profiling(False)
    b.langevin_init()
    b.langevin_run(7)
    assert check(b, 1, True) == 1
    b.langevin_run(3)
    assert check(b, 0, True) == 1
    b.retire(0)  # the graphs stay: they read the list of live items
    if len(sizes) > 1:
      for n in range(4):
        assert check(b, n % 2, n < 2, sizes[0], 1) == 1
