"""Default work-item lengths: single tiles go with the pair list, not with
every cutoff."""

import numpy as np
import pytest

from prolix_b200 import engine, synth

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
