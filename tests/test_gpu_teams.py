"""The team kernels (a thread block per tile, for batches of few tiles) give
the one-warp kernel's forces and trajectories bit for bit: at block edges, at
the tile counts where the team's size changes (296 and 640) and ends, with
cutoffs, term subsets and retired systems.  The default work list is a team's
where the batch has few tiles; a work item of two tiles is never one."""

import numpy as np
import pytest

from prolix_b200 import _lib, engine, synth

pytestmark = pytest.mark.gpu

SIZES = (1, 2, 31, 32, 33, 65, 300, 1056, 1057, 1120, 1568, 1600)
FIELDS = ("position", "momentum", "force")


def _run(systems, segment, **kw):
  with engine.Batch(systems, **kw) as b:
    if segment:
      b.set_tile_segment(segment)
    else:
      assert b.tile_segment() == 1
    f = b.forces()
    b.langevin_init()
    b.langevin_run(3)
    b.langevin_run(2)
    return f, b.get_state(fields=FIELDS)


def _same(systems, **kw):
  f1, s1 = _run(systems, 0, **kw)
  f2, s2 = _run(systems, 2, **kw)
  np.testing.assert_array_equal(f1, f2)
  for k in FIELDS:
    np.testing.assert_array_equal(s1[k], s2[k])


@pytest.mark.parametrize("cutoff", [0.0, 9.0])
@pytest.mark.parametrize("n", SIZES)
def test_team_sums_equal_the_one_warp_sums(n, cutoff):
  _same([synth.make_chain(n, 60 + n, compact=True, cmap=n > 64, **synth.PHYSICAL_RANGES)], cutoff=cutoff)


@pytest.mark.parametrize("terms", [_lib.USE_GB, _lib.USE_LJ | _lib.USE_BONDED, _lib.USE_COULOMB | _lib.USE_GB])
def test_team_sums_with_term_subsets(terms):
  _same([synth.make_chain(n, 70 + n, compact=True, **synth.PHYSICAL_RANGES) for n in (40, 200, 333)], terms=terms)


def test_retired_systems_leave_a_team_batch():
  systems = [synth.make_chain(n, 80 + n, compact=True, **synth.PHYSICAL_RANGES) for n in (50, 170, 300)]
  with engine.Batch(systems) as b, engine.Batch([systems[0], systems[2]]) as c:
    for x in (b, c):
      x.langevin_init()
    b.retire(1)
    b.langevin_run(6)
    c.langevin_run(6)
    xb, xc = (v.get_state(fields=("position",))["position"] for v in (b, c))
  np.testing.assert_array_equal(np.concatenate([xb[:50], xb[220:]]), xc)


def test_single_tile_items_of_long_rows_leave_the_forces_equal():
  s = synth.make_chain(4000, 91, compact=True, **synth.PHYSICAL_RANGES)
  with engine.Batch([s]) as b:
    ref = b.forces()
    for seg in (2, 6, 7):
      b.set_tile_segment(seg)
      np.testing.assert_array_equal(b.forces(), ref)
