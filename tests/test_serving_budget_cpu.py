"""The server's memory budget counts what a cohort holds on the device: the
atoms and the work lists, which grow with the system's tiles."""

import numpy as np

from prolix_b200 import serving
from test_serving_cpu import FakeBatch


def _request(n, rid, **extra):
  system = dict(positions=np.zeros((n, 3)), charges=np.zeros(n), excl_pairs=np.zeros((0, 2), np.int32),
                excl_kind=np.zeros(0, np.int32), **extra)
  return serving.Request(system=system, n_steps=10, key=(0, rid), rid=rid)


def _serve(requests, **kw):
  srv = serving.Server(batch_factory=FakeBatch, chunk=10, **kw)
  srv.run(requests)
  return srv


def test_large_listed_systems_wait_for_each_other():
  # 40,000 atoms at 12 A hold 34.6 MB (measured): two do not fit 60 MB at once
  srv = _serve([_request(40_000, k) for k in range(2)], cutoff=12.0, hbm_budget_bytes=60e6)
  assert srv.cohorts_created == 2
  assert all(r.error is None for r in srv.results.values())
  srv = _serve([_request(40_000, k) for k in range(2)], cutoff=12.0, hbm_budget_bytes=75e6)
  assert srv.cohorts_created == 1


def test_cmap_tables_count():
  grids = dict(cmap_energy_grids=np.zeros((4, 24, 24)))
  assert serving._request_bytes(_request(100, 0, **grids), 0.0) \
      == serving._request_bytes(_request(100, 0), 0.0) + 4 * 24 * 24 * 128
  srv = _serve([_request(100, 0, **grids)], hbm_budget_bytes=200e3)
  assert srv.results[0].error is not None


def test_the_work_lists_count_at_every_size():
  sizes = (1, 32, 33, 896, 897, 1281, 1825, 2016, 2017, 5120, 8192, 12_800, 100_000)
  for cutoff in (0.0, 12.0):
    assert all(serving.BYTES_PER_ATOM * n < serving.system_bytes(n, cutoff) for n in sizes)
