"""Autotuner host logic on CPU: cache keys, the JSON cache and candidate
selection with a fake timer (the GPU test times real launches)."""
import json

from diffren_gb300 import _lib, autotune, kernels


def batch_and_config():
  b = kernels.ImageBatch([256, 512], [256, 512], [100, 200], [1000, 3000])
  c = kernels.raster_config(3, 1, 0)
  return b, c


def test_signature_groups_similar_batches():
  b, c = batch_and_config()
  k1 = autotune.signature("GB300", b, c, 4)
  b2 = kernels.ImageBatch([256, 512], [256, 512], [100, 210], [1000, 3100])
  assert autotune.signature("GB300", b2, c, 4) == k1
  assert autotune.signature("GB300", b, c, 3) != k1
  assert autotune.signature("B200", b, c, 4) != k1
  c5 = kernels.raster_config(5, 1, 0)
  assert autotune.signature("GB300", b, c5, 4) != k1


def test_cache_round_trip(tmp_path):
  path = str(tmp_path / "tune.json")
  autotune.clear_memory()
  assert autotune.lookup("k", path) is None
  autotune.store("k", (32, 16, 8), path)
  autotune.clear_memory()
  assert autotune.lookup("k", path) == (32, 16, 8)
  with open(path) as f:
    assert json.load(f) == {"k": [32, 16, 8]}
  autotune.store("k2", (16, 16, 16), path)
  with open(path) as f:
    assert set(json.load(f)) == {"k", "k2"}
  autotune.clear_memory()


def test_corrupt_cache_is_ignored(tmp_path):
  path = tmp_path / "tune.json"
  path.write_text("not json")
  autotune.clear_memory()
  assert autotune.lookup("k", str(path)) is None
  autotune.store("k", (8, 8, 16), str(path))
  assert json.loads(path.read_text()) == {"k": [8, 8, 16]}
  autotune.clear_memory()


def test_time_candidates_picks_fastest_and_skips_rejected():
  cost = {(16, 16, 16): 3.0, (32, 16, 16): 1.5, (8, 8, 16): 2.0, (32, 32, 16): None}
  current = {}

  def run(cand):
    if cost[cand] is None:
      raise _lib.DiffrenError("rejected")
    current["c"] = cand

  def timer(fn):
    fn()
    return cost[current["c"]]

  times = autotune.time_candidates(run, list(cost), repeats=2, timer=timer)
  assert set(times) == {(16, 16, 16), (32, 16, 16), (8, 8, 16)}
  assert min(times, key=times.get) == (32, 16, 16)


def test_candidates_fit_the_rasterizer_limits():
  for w, h, large in autotune.CANDIDATES:
    assert 0 < w <= 128 and 0 < h <= 128 and w * h <= 1024 and large > 0


def test_choices_of_other_kernels_are_not_found(tmp_path, monkeypatch):
  b, c = batch_and_config()
  path = str(tmp_path / "tune.json")
  keys = []
  for k in range(2):
    lib = tmp_path / ("lib%d.so" % k)
    lib.write_bytes(b"kernels %d" % k)
    monkeypatch.setenv("DIFFREN_GB300_LIBRARY", str(lib))
    autotune.kernels_digest.cache_clear()
    keys.append(autotune.signature("GB300", b, c, 4))
  autotune.kernels_digest.cache_clear()
  autotune.clear_memory()
  autotune.store(keys[0], (8, 8, 16), path)
  autotune.clear_memory()
  assert autotune.lookup(keys[0], path) == (8, 8, 16)
  assert autotune.lookup(keys[1], path) is None
  autotune.clear_memory()


def test_default_tiles_are_candidates():
  """The tile that no configuration gives shows in the workspace it needs
  (which also covers 16x16): it is that of a candidate with 16 tiles as the
  large threshold, as in the default."""
  chosen = set()
  for w, h, images, tris, layers in (
      (64, 64, 1, 5000, 3), (256, 256, 1, 300, 3), (256, 256, 1, 20000, 1), (352, 340, 1, 20000, 3),
      (640, 480, 1, 20000, 4), (1024, 1024, 8, 100000, 3), (1000, 1000, 64, 20000, 3),
      (1000, 1000, 64, 20000, 8), (2047, 2047, 4, 1000000, 3)):
    batch = kernels.ImageBatch([w] * images, [h] * images, [3] * images, [tris] * images)

    def need(tile, large):
      return kernels.raster_workspace_bytes(batch, kernels.raster_config(layers, 1, 0, tile, large))
    base = need((16, 16), 16)
    fits = {c for c in autotune.CANDIDATES
            if c[2] == 16 and max(base, need(c[:2], 16)) == need((0, 0), 0)}
    assert fits
    chosen |= fits
  assert {(16, 16, 16), (8, 8, 16), (16, 8, 16)} <= chosen
