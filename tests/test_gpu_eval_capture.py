"""Evaluations while something else is being captured: the call that makes an
evaluation's graph is as free of side effects as the ones before it."""

import threading

import numpy as np
import pytest

from prolix_b200 import engine, synth

pytestmark = pytest.mark.gpu

MODES = ("global", "thread_local", "relaxed")


def _calls(b, x, n, stream):
  import torch
  out = []
  for _ in range(n):
    e = torch.zeros((1, 12), dtype=torch.float64, device="cuda")
    f = torch.zeros_like(x)
    out.append((e, f))
  torch.cuda.synchronize()

  def go():
    for e, f in out:
      b.energy_forces_device(x.data_ptr(), e.data_ptr(), f.data_ptr(), stream.cuda_stream)
  return out, go


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("other_thread", [False, True])
def test_evaluations_beside_a_capture_of_another_stream(mode, other_thread):
  # the third call of a small batch instantiates its graph; a capture in
  # progress on another stream, of this thread or another one, neither stops
  # it nor is broken by it
  import torch
  s = synth.make_chain(166, 11, compact=True, **synth.PHYSICAL_RANGES)
  x = torch.from_numpy(s["positions"]).cuda()
  y = torch.zeros(1024, device="cuda")
  st = torch.cuda.Stream()
  with engine.Batch([s]) as b:
    out, go = _calls(b, x, 6, st)
    with engine.Batch([s]) as ref_batch:  # loads every kernel
      ref = ref_batch.energy_forces()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    errors = []

    def run():
      try:
        go()
      except Exception as err:  # noqa: BLE001
        errors.append(err)

    with torch.cuda.graph(g, capture_error_mode=mode):
      y.add_(1.0)
      if other_thread:
        t = threading.Thread(target=run)
        t.start()
        t.join()
      else:
        run()
      y.mul_(2.0)
    assert not errors
    g.replay()
    torch.cuda.synchronize()
    assert float(y[0]) == 2.0
    for e, f in out:
      np.testing.assert_array_equal(e.cpu().numpy(), ref[0])
      np.testing.assert_array_equal(f.cpu().numpy(), ref[1])
