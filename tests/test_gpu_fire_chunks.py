"""FIRE at the edges of its 256-atom chunks, in one run and across the graph
chunk's end, against the FP64 restatement, and the same in a batch."""

import numpy as np
import pytest

from oracle import minimize as om
from prolix_b200 import engine, synth

pytestmark = pytest.mark.gpu

ARGS = dict(k=125.0, kind="backbone", dt_start=1e-3, dt_max=1e-2, max_disp=0.1)


def _sys(n):
  s = synth.make_chain(n, 500 + n, compact=True, **synth.PHYSICAL_RANGES)
  return dict(s, origin=engine.default_origin(s["positions"]))


def _fire(systems, **kw):
  with engine.Batch(systems, **kw) as b:
    b.min_setup()
    b.min_fire(12, **ARGS)
    return b.split(b.get_state(fields=("position",))["position"])


@pytest.mark.parametrize("n", [1, 32, 255, 256, 257, 513, 800])
def test_fire_at_chunk_edges(n):
  s = _sys(n)
  got = _fire([s])[0]
  heavy = (np.asarray(s["masses"]) > 1.1).astype(float)
  best, _ = om.fire(s, s["positions"], s["positions"], heavy, s["masses"], 12, 125.0, 1e-3, 1e-2, 0.1)
  # twelve steps of float32-accurate forces (1e-5 relative at most) move an
  # atom by at most 0.1 A each: 12 * 0.1 * 1e-5
  assert np.max(np.abs(got - best)) < 1.2e-5
  np.testing.assert_array_equal(_fire([s], graph_chunk=5)[0], got)
  np.testing.assert_array_equal(_fire([_sys(300), s])[1], got)
