"""Evaluations in several threads, beside others that use the default stream
and wait for the device: an evaluation puts no stream into capture, which
would make those calls fail in every thread of the process."""

import threading
import time

import numpy as np
import pytest

from prolix_b200 import engine, synth

pytestmark = pytest.mark.gpu


def test_evaluations_leave_other_threads_calls_alone():
  # two threads take batch after batch to their replayed evaluations (the
  # third of each kind makes the graph); two others launch on the default
  # stream, allocate, and wait for streams and for the device
  import torch
  s = synth.make_chain(60, 3, compact=True, **synth.PHYSICAL_RANGES)
  x = torch.from_numpy(s["positions"]).cuda()
  with engine.Batch([s]) as b:
    e0, f0 = b.energy_forces()
  warm = torch.ones(256, device="cuda")
  (warm * 2.0).sum().item()
  stop = threading.Event()
  errors, results = [], []

  def evaluate():
    try:
      torch.cuda.set_device(0)
      st = torch.cuda.Stream()
      for _ in range(60):
        with engine.Batch([s]) as b:
          e = torch.zeros((1, 12), dtype=torch.float64, device="cuda")
          f = torch.zeros_like(x)
          torch.cuda.current_stream().synchronize()
          for _ in range(5):
            b.energy_forces_device(x.data_ptr(), e.data_ptr(), f.data_ptr(), st.cuda_stream)
            b.energy_forces_device(x.data_ptr(), 0, f.data_ptr(), st.cuda_stream)
          st.synchronize()
          results.append((e.cpu().numpy(), f.cpu().numpy()))
    except Exception as err:  # noqa: BLE001
      errors.append(err)

  def others(wait):
    try:
      torch.cuda.set_device(0)
      while not stop.is_set():
        y = torch.ones(4096, device="cuda") * 2.0
        assert float(y.sum()) == 8192.0
        if wait:
          torch.cuda.synchronize()
        time.sleep(0)
    except Exception as err:  # noqa: BLE001
      errors.append(err)

  busy = [threading.Thread(target=others, args=(w,)) for w in (False, True)]
  work = [threading.Thread(target=evaluate) for _ in range(2)]
  for t in busy + work:
    t.start()
  for t in work:
    t.join()
  stop.set()
  for t in busy:
    t.join()
  assert not errors, errors
  assert len(results) == 120
  for e, f in results:
    np.testing.assert_array_equal(e, e0)
    np.testing.assert_array_equal(f, f0)
