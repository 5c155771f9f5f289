"""FP64 pair energies at inputs that have no ordinary value: what the
formulas give in double, and nothing that only looks like it."""

import numpy as np
import pytest

from oracle import gbsa
from prolix_b200 import _lib, engine, synth

pytestmark = pytest.mark.gpu


def _two_atoms(r, radius):
  return dict(positions=np.array([[0.0, 0.0, 0.0], [r, 0.0, 0.0]]), charges=np.array([0.3, -0.3]),
              sigmas=np.ones(2), epsilons=np.zeros(2), radii=np.array([radius, 1.7]),
              scaled_radii=np.array([0.0, 0.72 * 1.61]), masses=np.ones(2), bonds=np.zeros((0, 2), np.int32))


def _terms(system, **kw):
  with engine.Batch([system], **kw) as b:
    return dict(zip(_lib.TERM_NAMES, b.energy_forces()[0][0]))


@pytest.mark.parametrize("r,radius", [(1.1, 0.05), (1.0, 0.03), (1.3, 0.01), (0.9, 0.02)])
def test_a_negative_born_radius_keeps_the_exponential(r, radius):
  # a radius below the dielectric offset gives one atom B < 0: the pair's
  # exponential has a positive argument, and f^2 is well below r^2.  Three
  # roundings to 2^-24, and 1e-9 relative for the descreening sums' 2^-40.
  s = _two_atoms(r, radius)
  born, _, _ = gbsa.born_radii(s["positions"], s["radii"], s["scaled_radii"])
  assert born[0] * born[1] < 0.0
  ref = gbsa.nonbonded(s, s["positions"])[0]["gb"]
  assert np.isfinite(ref)
  got = _terms(s, terms=_lib.USE_GB)["gb"]
  assert abs(got - ref) <= 4 * 2.0 ** -25 + 1e-9 * abs(ref), (got, ref)


@pytest.mark.parametrize("r,radius", [(0.9, 0.05), (3.0, 0.05), (30.0, 0.05)])
def test_a_pair_without_a_value_shows_in_the_energy(r, radius):
  # f^2 < 0: no finite energy.  A NaN is the lowest fixed-point number
  # (-2^63 of 2^-24), far from any energy.
  s = _two_atoms(r, radius)
  with np.errstate(all="ignore"):
    assert not np.isfinite(gbsa.nonbonded(s, s["positions"])[0]["gb"])
  assert abs(_terms(s, terms=_lib.USE_GB)["gb"]) > 1e11


def test_a_lost_atom_leaves_the_other_atoms_descreening_sums():
  # one atom of an extended chain without a position (NaN): its pairs count
  # as nothing in the descreening sums, near and far, so the nonpolar energy
  # is that of the chain without the atom plus the atom's own, alone.  Each
  # atom's energy is rounded to 2^-24; a Born sum to 2^-40 in each of at most
  # 8 parts of each tile that touches the atom, and dACE/dI is below 20.
  s = synth.make_chain(600, 5, compact=False, **synth.PHYSICAL_RANGES)
  n, k = 600, 301
  x = s["positions"].copy()
  keep = np.arange(n) != k
  born, _, _ = gbsa.born_radii(x[keep], s["radii"][keep], s["scaled_radii"][keep])
  ref = gbsa.ace_energy(s["radii"][keep], born).sum()
  ref += gbsa.ace_energy(s["radii"][k:k + 1], s["radii"][k:k + 1] - gbsa.DIELECTRIC_OFFSET)[0]
  x[k, 1] = np.nan
  with engine.Batch([s], terms=_lib.USE_GB) as b:
    b.set_positions(x)
    got = dict(zip(_lib.TERM_NAMES, b.energy_forces()[0][0]))["nonpolar"]
  assert abs(got - ref) <= n * (2.0 ** -25 + 20.0 * 8 * 20 * 2.0 ** -41), (got, ref)


@pytest.mark.parametrize("cutoff", [4.0, 8.0, 9.0, 16.0])
def test_a_pair_at_the_cutoff_is_outside_it(cutoff):
  # r < cutoff counts: at the cutoff itself the energies are those of two
  # atoms far apart, to the last bit
  s = _two_atoms(cutoff, 1.5)
  s["scaled_radii"][:] = 1.1
  at = _terms(s, cutoff=cutoff)
  assert at == _terms(dict(s, positions=s["positions"] * 3.0), cutoff=cutoff)
  assert at != _terms(dict(s, positions=s["positions"] * 0.999), cutoff=cutoff)
