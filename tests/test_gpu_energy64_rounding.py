"""FP64 energies to the rounding of their fixed-point sums: the errors of
2^-24 per added sum and 2^-40 per part of a descreening sum add like
independent ones, and six standard deviations of their total (5e-7 to 8e-6
kcal/mol) leave no room for an unrefined reciprocal or root (1e-6 relative)
or a lost pair.  A series tier off by one is not among what they show: it
moves these energies by 4e-7 at most, below the rounding itself."""

import numpy as np
import pytest

from oracle import gbsa
from prolix_b200 import _lib, engine, synth

pytestmark = pytest.mark.gpu


def _tolerances(s, n, extras, energies):
  nblk = -(-n // 32)
  tiles = sum(range(nblk, 0, -2))
  parts = 8 if nblk <= 28 else 4 if nblk <= 40 else 2 if nblk <= 57 else 1
  # sums added per term: two i-blocks of each item (a tile at most); the GB
  # self terms and ACE are rounded per atom
  e_var, i_var = (2.0 ** -25) ** 2 / 3, (2.0 ** -41) ** 2 / 3
  ace6 = 6.0 * gbsa.ace_energy(s["radii"], extras["born_radii"]) / extras["born_radii"]
  # parts of an atom's descreening sum: its row's and column's items, and the
  # pairs near enough for the closed form, each rounded by itself
  per_atom = parts * (nblk + 2) + 64
  d_ace = ace6 * extras["dbdi"]
  d_gb = extras["dedb"] * extras["dbdi"] + d_ace
  x, q = s["positions"], np.abs(s["charges"])
  scale = 0.0  # absolute sum of the pair terms, for the double arithmetic
  for a in range(0, n, 512):
    r = np.sqrt(((x[a:a + 512, None] - x[None]) ** 2).sum(-1) + 1.0)
    scale += 332.0 * (q[a:a + 512, None] * q[None] / r).sum()
  arithmetic = 1e-14 * (scale + sum(abs(v) for v in energies.values()))
  sd = {"lj": np.sqrt(2 * tiles * e_var), "coulomb": np.sqrt(2 * tiles * e_var),
        "gb": np.sqrt((2 * tiles + n) * e_var + per_atom * i_var * (d_gb ** 2).sum()),
        "nonpolar": np.sqrt(n * e_var + per_atom * i_var * (d_ace ** 2).sum())}
  return {k: 6.0 * v + arithmetic for k, v in sd.items()}


@pytest.mark.parametrize("cutoff", [0.0, 14.0])
@pytest.mark.parametrize("n,compact", [(166, True), (700, False), (1290, False), (1900, False), (2600, True)])
def test_energies_to_the_rounding(n, compact, cutoff):
  s = synth.make_chain(n, 800 + n, compact=compact, **synth.PHYSICAL_RANGES)
  ref, _, extras = gbsa.nonbonded(s, s["positions"], cutoff=cutoff)
  with engine.Batch([s], cutoff=cutoff) as b:
    got = dict(zip(_lib.TERM_NAMES, b.energy_forces()[0][0]))
  tol = _tolerances(s, n, extras, ref)
  for k, t in tol.items():
    assert abs(got[k] - ref[k]) <= t, (k, got[k], ref[k], t)
