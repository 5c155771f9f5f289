"""FP64 pair energies at the sizes where their work items change: the edges
of 32-atom blocks, of the splits of a tile's steps over 8, 4, 2 and 1 items
(28, 40, 57 blocks) and of the longer items of large systems (160, 256 and
400 blocks), with and without a cutoff."""

import numpy as np
import pytest

from oracle import cforces
from prolix_b200 import engine, synth

pytestmark = pytest.mark.gpu

SIZES = [(n, 0.0) for n in (1, 2, 31, 33, 65, 896, 897, 1280, 1281, 1824, 1825, 5088, 5121)]
SIZES += [(33, 9.0), (897, 9.0), (1825, 20.0), (5121, 12.0)]


def _bound(s, n, cutoff):
  """What the arithmetic may differ from exact by, kcal/mol.  Each item's
  three sums and each atom's two energies are rounded to 2^-24; a Born sum
  is rounded to 2^-40 once per item that touches the atom, which moves an
  energy by at most P q^2 per unit of the sum (dE/dB dB/dI <= P q^2 / B^2 *
  B^2, and the neighbours' terms as much again); and the double arithmetic
  by 1e-12 of the pair terms' absolute sum, which 332 q^2 n^2 / 2 per 1 A
  bounds."""
  nblk = (n + 31) // 32
  items = nblk * nblk // 4 * 8 + 8 * nblk + 8
  q2 = float(np.max(np.abs(s["charges"])) ** 2)
  per_atom = 8 * (nblk + 2) * 2.0 ** -41 * 2 * 164.0 * max(q2, 1e-3)
  reach = n if cutoff <= 0 else min(n, int(0.1 * 4.19 * cutoff ** 3) + 32)
  return (items + 2 * n) * 2.0 ** -25 + n * per_atom + 1e-12 * 332.0 * q2 * n * reach / 2


@pytest.mark.parametrize("n,cutoff", SIZES)
def test_pair_energies_at_item_edges(n, cutoff):
  s = synth.make_chain(n, 900 + n, compact=True, **synth.PHYSICAL_RANGES)
  with engine.Batch([s], cutoff=cutoff, pair_list=False) as b:
    e, _ = b.energy_forces()
    e2, _ = b.energy_forces()
  np.testing.assert_array_equal(e, e2)
  ref, _ = cforces.energy_forces(s, s["positions"], cutoff=cutoff)
  got = dict(zip(("lj", "coulomb", "gb", "nonpolar"), (e[0][4], e[0][5], e[0][6], e[0][7])))
  tol = _bound(s, n, cutoff)
  for name, v in got.items():
    assert abs(v - ref[name]) <= tol, (name, v, ref[name], tol)


def test_energies_do_not_depend_on_the_batch_or_the_segment():
  systems = [synth.make_chain(n, 40 + n, compact=True, **synth.PHYSICAL_RANGES) for n in (40, 700, 1500, 3000)]
  with engine.Batch(systems) as b:
    e, _ = b.energy_forces()
    b.set_tile_segment(4)
    e4, _ = b.energy_forces()
  np.testing.assert_array_equal(e, e4)
  for k, s in enumerate(systems):
    with engine.Batch([s]) as b1:
      np.testing.assert_array_equal(b1.energy_forces()[0][0], e[k])
