"""Which stored autotuner choices a batch takes up."""

import json

from prolix_b200 import autotune
from test_autotune_cpu import FakeBatch


def test_a_choice_stored_for_other_schedules_is_not_applied(tmp_path, monkeypatch):
  # an entry as stored before one tile per item was among the candidates
  path = tmp_path / "t.json"
  monkeypatch.setenv("PROLIX_B200_TUNE_CACHE", str(path))
  old = "FAKE|sys1|atoms256|nmax256|all"
  path.write_text(json.dumps({old: {"segment": 2, "shapes": [[256, 3]] * 4, "force_blocks": 2, "fusion": 1,
                                    "ms": 1.0, "timings": {}}}))
  monkeypatch.setattr(autotune, "_gpu_name", lambda: "FAKE")
  monkeypatch.setattr(autotune, "_time", lambda b, steps=4: float(b.seg))
  fb = FakeBatch([166])
  r = autotune.tune(fb)
  assert not r["cached"] and r["segment"] == 1 and fb.seg == 1
  assert old in json.loads(path.read_text())  # another package's entries stay


def test_a_bucket_does_not_straddle_the_team_sizes():
  # both round to 2,048 atoms; 1,100 run by teams at one tile per item (315
  # tiles), 2,000 do not (1,024)
  a, b, c = (autotune.bucket_key(FakeBatch([n]), "GPU") for n in (1100, 2000, 1900))
  assert a != b and b == c


def test_team_tiles():
  # 1,056 atoms: 33 blocks, 289 tiles; 1,088: 34, 306; 1,568: 49, 625; 1,569: 50, 650
  assert [autotune.team_warps([n]) for n in (166, 1056, 1088, 1568, 1569)] == [8, 8, 4, 4, 1]
  assert autotune.team_warps([900, 900]) == 4
