"""Default work-item lengths: single tiles go with the pair list, not with
every cutoff."""

import numpy as np
import pytest

from prolix_b200 import engine, serving, synth

pytestmark = pytest.mark.gpu


def _segment(systems, **kw):
  with engine.Batch(systems, **kw) as b:
    return b.tile_segment(), b.forces()


def test_a_cutoff_without_a_pair_list_does_not_force_single_tiles():
  # 40 systems of 47 blocks: 23,040 tiles, enough for items of two and more
  systems = [synth.make_chain(1500, 300 + k, compact=True, **synth.PHYSICAL_RANGES) for k in range(40)]
  whole, _ = _segment(systems)
  assert whole > 1
  # GB over all pairs beside a direct cutoff: every tile is evaluated
  seg, f = _segment(systems, cutoff=9.0, gb_cutoff=0.0)
  assert seg == whole
  np.testing.assert_array_equal(f, _segment(systems, cutoff=9.0, gb_cutoff=0.0, tile_segment=1)[1])
  # every term cut off, no list (no system of 64 blocks)
  seg, f = _segment(systems, cutoff=9.0)
  assert seg == 2
  np.testing.assert_array_equal(f, _segment(systems, cutoff=9.0, tile_segment=1)[1])


def test_single_tiles_with_a_pair_list():
  systems = [synth.make_chain(2500, 340 + k, compact=True, **synth.PHYSICAL_RANGES) for k in range(16)]
  seg, f = _segment(systems, cutoff=9.0)
  seg_off, f_off = _segment(systems, cutoff=9.0, pair_list=False)
  assert (seg, seg_off) == (1, 2)
  np.testing.assert_array_equal(f, f_off)


def _device_bytes(systems, **kw):
  """What the batch holds of the device's memory pool."""
  from cuda.bindings import runtime as rt
  attr = rt.cudaMemPoolAttr.cudaMemPoolAttrUsedMemCurrent
  engine.Context.get(0)
  pool = rt.cudaDeviceGetDefaultMemPool(0)[1]
  before = int(rt.cudaMemPoolGetAttribute(pool, attr)[1])
  with engine.Batch(systems, **kw):
    return int(rt.cudaMemPoolGetAttribute(pool, attr)[1]) - before


def test_the_pair_list_replaces_the_other_work_lists():
  # 36 B per tile with it (two buffers of items and the j-blocks) against 48
  # without at the same item length (two- and four-block items, all and live)
  systems = [synth.make_chain(4000, 350, compact=True, **synth.PHYSICAL_RANGES)]
  tiles = sum(125 - ib for ib in range(0, 125, 2))
  listed = _device_bytes(systems, cutoff=12.0)
  plain = _device_bytes(systems, cutoff=12.0, pair_list=False, tile_segment=1)
  # the displacement reference and the rows: 16 B per atom and per pair of blocks
  assert listed <= plain + 16 * 4000 + 16 * 63 + 8192, (listed, plain, tiles)


@pytest.mark.parametrize("cutoff", [0.0, 12.0])
def test_the_server_counts_what_a_cohort_holds(cutoff):
  # at most the server's figure, and no less than four fifths of it (a cohort
  # of several systems has longer items than the figure takes for each alone)
  for sizes in ((100,) * 40, (300, 900, 1900), (2500, 150), (10000,), (20000,)):
    systems = []
    for k, n in enumerate(sizes):
      parts = [synth.make_chain(min(n, 2500), 360 + k, compact=True, **synth.PHYSICAL_RANGES) for _ in range(max(1, n // 2500))]
      s = {f: np.concatenate([p[f] for p in parts]) for f in
           ("charges", "sigmas", "epsilons", "radii", "scaled_radii", "masses", "bond_params", "angle_params",
            "dihedral_params")}
      for f in ("bonds", "angles", "dihedrals"):
        s[f] = np.concatenate([p[f] + 2500 * j for j, p in enumerate(parts)])
      s["positions"] = np.concatenate([p["positions"] + np.array([50.0 * j, 0.0, 0.0]) for j, p in enumerate(parts)])
      systems.append(s)
    held = _device_bytes(systems, cutoff=cutoff)
    counted = sum(serving.system_bytes(n, cutoff) for n in sizes)
    assert 0.8 * counted <= held <= counted, (sizes, held, counted)


def test_item_length_with_a_pair_list_follows_the_tiles_within_reach():
  # 24 systems of 2,500 atoms at 40 A list nearly all of their 38,400 tiles:
  # two per item; at 6 A a third of them: one
  systems = [synth.make_chain(2500, 340, compact=True, **synth.PHYSICAL_RANGES)] * 24
  wide, f = _segment(systems, cutoff=40.0)
  narrow, _ = _segment(systems, cutoff=6.0)
  assert (wide, narrow) == (2, 1)
  np.testing.assert_array_equal(f, _segment(systems, cutoff=40.0, pair_list=False)[1])
