"""FP64 pair energies at inputs that have no ordinary value: what the
formulas give in double, and nothing that only looks like it."""

import numpy as np
import pytest

from oracle import gbsa
from prolix_b200 import _lib, engine

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
