"""Bonded terms give the same forces bit for bit in the chain pass's tail, in
a team's units and in a kernel of their own: where they run is a matter of
schedule (forces alone against forces with energies, fusion on and off)."""

import numpy as np
import pytest

from prolix_b200 import _lib, engine, synth

pytestmark = pytest.mark.gpu


def _with_every_term(n, seed):
  s = synth.make_chain(n, seed, compact=True, cmap=True, **synth.PHYSICAL_RANGES)
  i = np.arange(n // 4)
  m = len(i)
  s["urey_bradley_bonds"] = np.stack([i, i + 2], 1).astype(np.int32)
  s["urey_bradley_params"] = np.stack([2.5 + 0 * i, 5.0 + 0 * i], 1)
  s["impropers"] = np.stack([i + k for k in range(4)], 1).astype(np.int32)
  s["improper_params"] = np.stack([np.full((m, 1), 2.0), np.full((m, 1), 0.3), np.full((m, 1), 1.0)], -1)
  s["exception_pairs"] = np.stack([i, i + 4], 1).astype(np.int32)
  s["exception_chargeprods"] = np.full(m, 0.05)
  s["exception_sigmas"] = np.full(m, 2.5)
  s["exception_epsilons"] = np.full(m, 0.05)
  return s


@pytest.mark.parametrize("terms", [_lib.USE_GB | _lib.USE_CMAP, _lib.USE_ALL])
@pytest.mark.parametrize("sizes,evaluations", [((3500, 4200, 2600), 60), ((900,), 400)])
def test_forces_with_and_without_energies(sizes, evaluations, terms):
  # a last bit of an FP64 force shows in the 2^-32 fixed point about once in
  # 1e5 terms: some 2e5 CMAP terms in each case
  systems = [_with_every_term(n, 700 + n) for n in sizes]
  x0 = np.concatenate([s["positions"] for s in systems])
  rng = np.random.default_rng(11)
  with engine.Batch(systems, terms=terms) as b:
    assert b.fusion() == _lib.FUSE_BONDED
    for _ in range(evaluations):
      b.set_positions(x0 + 0.02 * rng.standard_normal(x0.shape))
      np.testing.assert_array_equal(b.forces(), b.energy_forces()[1])


def test_steps_with_and_without_the_fusion():
  systems = [dict(_with_every_term(n, 900 + n), key=(0, n)) for n in (3500, 4200, 2600)]
  out = []
  for fusion in (0, _lib.FUSE_BONDED):
    with engine.Batch(systems) as b:
      b.set_fusion(fusion)
      b.langevin_init()
      b.langevin_run(300)
      out.append(b.get_state(fields=("position", "momentum", "force")))
  for k in out[0]:
    np.testing.assert_array_equal(out[0][k], out[1][k])
