"""The generated FP64 polynomials of the energy path."""

import importlib.util
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "prolix_b200" / "csrc"


def test_series64_header_is_what_the_generator_writes():
  spec = importlib.util.spec_from_file_location("gen_obc_series", CSRC / "gen_obc_series.py")
  gen = importlib.util.module_from_spec(spec)
  spec.loader.exec_module(gen)
  assert (CSRC / "pb2_series64.cuh").read_text() == gen.header64()  # raises where a bound is missed
