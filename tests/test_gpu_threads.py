"""Batches worked by several threads at once, each on a stream of its own,
from creation through evaluations, steps and minimisation: what each gives
alone, bit for bit.  No graph of a batch is made by capturing a stream, which
would make the other threads' creation, transfers and waits fail."""

import threading

import numpy as np
import pytest

from prolix_b200 import engine, synth

pytestmark = pytest.mark.gpu

SIZES = (22, 100, 166, 400, 900, 1500, 2200)


def _work(seed, out):
  import torch
  torch.cuda.set_device(0)
  stream = torch.cuda.Stream()
  st = stream.cuda_stream
  rng = np.random.default_rng(seed)
  for _ in range(4):
    systems = [dict(synth.make_chain(int(rng.choice(SIZES)), int(rng.integers(1 << 30)), compact=True,
                                     **synth.PHYSICAL_RANGES), key=(0, int(rng.integers(1 << 30))))
               for _ in range(int(rng.integers(1, 4)))]
    x0 = np.concatenate([s["positions"] for s in systems])
    with engine.Batch(systems, cutoff=float(rng.choice([0.0, 9.0])), graph_chunk=int(rng.choice([3, 50]))) as b:
      out.extend(b.energy_forces(st))
      with torch.cuda.stream(stream):
        for k in range(5):
          x = torch.tensor(x0 + 0.01 * rng.standard_normal(x0.shape), device="cuda")
          e = torch.zeros((len(systems), 12), dtype=torch.float64, device="cuda")
          f = torch.zeros_like(x)
          b.energy_forces_device(x.data_ptr(), e.data_ptr() if k % 3 else 0, f.data_ptr(), st)
          del x
          out += [e.cpu().numpy(), f.cpu().numpy()]
      b.langevin_init(st)
      b.langevin_run(int(rng.integers(1, 30)), st)
      b.min_setup()
      b.min_sd(4, stream=st)
      b.min_fire(4, dt_start=1e-3, dt_max=1e-2, stream=st)
      b.langevin_run(int(rng.integers(1, 30)), st)
      s = b.get_state(stream=st)
      out += [s["position"], s["momentum"], s["force"]]


def test_threads_give_what_they_give_alone():
  n = 5
  for trial in range(2):
    alone = [[] for _ in range(n)]
    beside = [[] for _ in range(n)]
    for k in range(n):
      _work(100 * trial + k, alone[k])
    threads = [threading.Thread(target=_work, args=(100 * trial + k, beside[k])) for k in range(n)]
    for t in threads:
      t.start()
    for t in threads:
      t.join()
    for a, b in zip(alone, beside):
      assert len(a) == len(b) > 0
      for u, v in zip(a, b):
        np.testing.assert_array_equal(u, v)
