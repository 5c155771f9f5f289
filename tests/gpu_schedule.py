"""How a batch runs (pb2_test_schedule), for tests that are about one way of
running."""

import ctypes


def schedule(batch) -> dict:
  v = [ctypes.c_int32(-1) for _ in range(3)]
  batch._check(batch.lib.pb2_test_schedule(batch.handle, *[ctypes.byref(x) for x in v]))
  return dict(zip(("pair_list", "team", "replayed"), (x.value for x in v)))
