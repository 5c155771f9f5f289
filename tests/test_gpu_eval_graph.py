"""Evaluations replayed as a graph give what the first, launched one by one,
gave: forces and energies bit for bit, at new positions, after the work items
or kernels changed, after a retirement, and inside a caller's capture."""

import numpy as np
import pytest

from prolix_b200 import engine, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes,cutoff", [((166,), 0.0), ((40, 700, 2300), 0.0), ((2300, 90), 12.0)])
def test_replayed_evaluations_equal_the_first(sizes, cutoff):
  import torch
  systems = [synth.make_chain(n, 600 + n, compact=True, cmap=n > 64, **synth.PHYSICAL_RANGES) for n in sizes]
  x0 = np.concatenate([s["positions"] for s in systems])
  rng = np.random.default_rng(3)
  xs = [torch.from_numpy(x0 + 0.03 * rng.standard_normal(x0.shape)).cuda() for _ in range(2)]
  ref = []
  for x in xs:
    with engine.Batch(systems, cutoff=cutoff) as b:
      b.set_positions(x.cpu().numpy())
      ref.append(b.energy_forces())
  stream = torch.cuda.current_stream().cuda_stream

  def check(b, k, energies=True):
    e = torch.zeros((len(sizes), 12), dtype=torch.float64, device="cuda")
    f = torch.zeros(x0.shape, dtype=torch.float64, device="cuda")
    b.energy_forces_device(xs[k].data_ptr(), e.data_ptr() if energies else 0, f.data_ptr(), stream)
    np.testing.assert_array_equal(f.cpu().numpy(), ref[k][1])
    if energies:
      np.testing.assert_array_equal(e.cpu().numpy(), ref[k][0])

  with engine.Batch(systems, cutoff=cutoff) as b:
    for call in range(8):
      check(b, call % 2, energies=call % 3 != 1)
    b.set_tile_segment(3)
    check(b, 0)
    b.set_block_shape(1, *b.block_shapes(1)[-1])
    b.set_fusion(0)
    check(b, 1)
    check(b, 0, energies=False)
    g = torch.cuda.CUDAGraph()
    f = torch.zeros(x0.shape, dtype=torch.float64, device="cuda")
    e = torch.zeros((len(sizes), 12), dtype=torch.float64, device="cuda")
    with torch.cuda.graph(g):
      b.energy_forces_device(xs[1].data_ptr(), e.data_ptr(), f.data_ptr(),
                             torch.cuda.current_stream().cuda_stream)
    g.replay()
    torch.cuda.synchronize()
    np.testing.assert_array_equal(f.cpu().numpy(), ref[1][1])
    np.testing.assert_array_equal(e.cpu().numpy(), ref[1][0])
    b.retire(0)
    if len(sizes) > 1:
      n0 = sizes[0]
      b.energy_forces_device(xs[0].data_ptr(), e.data_ptr(), f.data_ptr(), stream)
      np.testing.assert_array_equal(f.cpu().numpy()[n0:], ref[0][1][n0:])
      np.testing.assert_array_equal(e.cpu().numpy()[1:], ref[0][0][1:])
