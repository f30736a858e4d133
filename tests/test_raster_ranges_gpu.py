"""GPU rasterizer against the oracle over the ranges its dispatch rules split:
edge-function magnitudes, row alignments and channel counts of the background
rows, layer counts, the default tile."""
import ctypes

import numpy as np
import pytest
import torch

from diffren_gb300 import _lib, kernels
from oracle import raster
from test_raster_gpu import _scene, assert_same, run_abi

pytestmark = pytest.mark.gpu


# Scaling a scene's clip coordinates by 2^k leaves its image alone and scales
# the edge coefficients by 2^2k: they cross 2^43 (from where edge functions may
# wrap) at k of about 4 to 8, the fixed-point coordinates 2^31 at k = 14, and
# the products wrap and the conversions saturate above that.
@pytest.mark.parametrize("kind,n", [("soup", 1500), ("big", 30), ("near", 600)])
@pytest.mark.parametrize("k", [-9, -4, -1, 0, 1, 2, 3, 4, 6, 9, 13, 14, 15, 18, 23, 31, 48, 60])
def test_clip_scale_matches_oracle(kind, n, k, device):
  verts, tris = _scene(kind, n, 96, 71, 3)
  verts = (np.asarray(verts, np.float64) * 2.0**k).astype(np.float32)
  for cull, mode, oracle_mode in ((0, _lib.DR_DEPTH_DISCRETIZED, raster.DEPTH_DISCRETIZED),
                                  (1, _lib.DR_DEPTH_DISCRETIZED, raster.DEPTH_DISCRETIZED),
                                  (2, _lib.DR_DEPTH_FLOAT, raster.DEPTH_FLOAT)):
    ref = raster.rasterize(verts, tris, 96, 71, 3, cull, oracle_mode)
    assert_same(run_abi(verts, tris, 96, 71, 3, cull, mode, device), ref)


# Background rows are written as float4s where every row starts and ends on
# 16 bytes (all of W, tile width and channels decide) and as floats elsewhere;
# empty tiles go eight at a time; layers are listed up to any L.
@pytest.mark.parametrize("w,h", [(64, 48), (96, 71), (97, 61), (16, 16), (15, 3), (130, 5), (260, 16)])
@pytest.mark.parametrize("layers,channels", [(1, 4), (2, 3), (3, 9), (3, 2), (4, 1), (5, 16)])
def test_background_and_layers_match_oracle(w, h, layers, channels, device):
  verts, tris = _scene("soup", 60, w, h, 5)
  clip = torch.tensor(np.asarray(verts, np.float32), device=device)
  tri = torch.tensor(np.asarray(tris, np.int32), device=device)
  attr = torch.rand(clip.shape[0], channels, device=device) + 0.5
  batch = kernels.ImageBatch.single(w, h, clip.shape[0], tri.shape[0])
  for tile in ((0, 0), (8, 8), (5, 7), (32, 8)):
    cfg = kernels.raster_config(layers, 1, _lib.DR_DEPTH_DISCRETIZED, tile)
    ref = raster.rasterize(verts, tris, w, h, layers, 1, raster.DEPTH_DISCRETIZED)
    n = layers * w * h
    out = (torch.full((n,), -7, dtype=torch.int32, device=device),
           torch.full((n,), float("nan"), device=device),
           torch.full((n, 3), float("nan"), device=device))
    ids, z, bary = kernels.rasterize_packed(clip, tri, batch, cfg, out=out)
    assert_same((ids.view(layers, h, w).cpu().numpy(), z.view(layers, h, w).cpu().numpy(),
                 bary.view(layers, h, w, 3).cpu().numpy()), ref)
    a, pos, ids2, z2, bary2 = kernels.rasterize_interpolate_packed(
        attr, clip, tri, batch, cfg, kernels.Workspace(device))
    assert torch.equal(ids, ids2) and torch.equal(z, z2) and torch.equal(bary, bary2)
    want, want_pos = kernels.interpolate_with_positions_packed(attr, clip, bary, tri, ids, z,
                                                               batch, layers)
    assert torch.equal(a, want)  # 0 on background
    fg = z != 1.0
    assert torch.equal(pos[fg][:, :3], want_pos[fg][:, :3])


# The default tile follows the batch's 16x16 tiles (512, 1536, 6144, 16384),
# triangles per tile (16, 24) and widths off 32 bytes: both sides of each line
# give the bits of an explicit tile, and a workspace for 16x16 tiles is enough.
@pytest.mark.parametrize("images,w,h,tris,layers", [
    (1, 352, 360, 300, 3), (1, 352, 376, 300, 3), (1, 352, 376, 9000, 2), (6, 256, 256, 5000, 3),
    (6, 256, 272, 5000, 3), (10, 256, 256, 200, 1), (11, 256, 256, 200, 4), (11, 256, 256, 4500, 3),
    (24, 256, 256, 5000, 3), (64, 256, 256, 300, 3), (64, 250, 256, 300, 4), (64, 256, 256, 300, 5),
    (64, 256, 256, 6200, 3), (64, 255, 256, 6200, 3), (64, 253, 256, 300, 6), (130, 64, 48, 40, 3)])
def test_default_tile_rule(images, w, h, tris, layers, device):
  clips = []
  for i in range(min(images, 3)):
    verts, tri = _scene("soup", tris, w, h, i)
    clips.append(torch.tensor(np.asarray(verts, np.float32), device=device))
  v, t = len(clips[0]), len(tri)
  clip = torch.cat([clips[i % len(clips)] for i in range(images)])
  tri = torch.tensor(np.asarray(tri, np.int32), device=device).repeat(images, 1)
  batch = kernels.ImageBatch([w] * images, [h] * images, [v] * images, [t] * images)
  config = lambda tile: kernels.raster_config(layers, 1, _lib.DR_DEPTH_DISCRETIZED, tile)
  want = kernels.rasterize_packed(clip, tri, batch, config((16, 16)))
  got = kernels.rasterize_packed(clip, tri, batch, config((0, 0)))
  for a, b in zip(got, want):
    assert torch.equal(a, b)
  need = kernels.raster_workspace_bytes(batch, config((16, 16)))
  assert kernels.raster_workspace_bytes(batch, config((0, 0))) >= need
  lib, P = _lib.load(), kernels._p
  ws = torch.empty(need, dtype=torch.uint8, device=device)
  for size, ok in ((need, True), (need - 256, False)):
    out = [torch.full_like(x, -7) for x in want]
    cfg = config((0, 0))
    rc = lib.dr_rasterize_batch(P(clip), P(tri), batch.ptr, batch.n, ctypes.byref(cfg), P(out[0]),
                                P(out[1]), P(out[2]), P(ws), size, kernels._stream(device))
    assert (rc == 0) == ok
    if ok:
      for a, b in zip(out, want):
        assert torch.equal(a, b)


# Tiles with more than 768 keys take triangles 64 at a time, the others 128: the
# same bits with one triangle less and more than whole chunks in a tile.
@pytest.mark.parametrize("count", [1, 63, 64, 65, 127, 128, 129, 257])
@pytest.mark.parametrize("layers", [1, 3, 4, 16])
def test_chunk_of_large_tiles(count, layers, device):
  g = torch.Generator(device=device).manual_seed(count)
  w, h = 37, 29
  clip = torch.rand(3 * count, 4, generator=g, device=device) * 2 - 1
  clip[:, 3] = 1.0
  tri = torch.arange(3 * count, dtype=torch.int32, device=device).view(-1, 3)
  batch = kernels.ImageBatch([w], [h], [3 * count], [count])
  out = [kernels.rasterize_packed(clip, tri, batch, kernels.raster_config(
      layers, culling, _lib.DR_DEPTH_DISCRETIZED, tile, large))
         for culling in (0, 1) for large in (1, 16)
         for tile in ((16, 16), (32, 16), (32, 32), (17, 16), (64, 5))]
  for k in range(0, len(out), 5):
    for got in out[k + 1:k + 5]:
      for a, b in zip(got, out[k]):
        assert torch.equal(a, b)


# An image with more large triangles than a chunk holds (128, or 64 above 768 keys
# a tile) has its chunks gathered from the list 128 boxes at a time, after the
# bins' last ones: a threshold of 1 tile (nearly all are large), one in between,
# and one that leaves the list empty give the same bits, as does the oracle.
@pytest.mark.parametrize("wide,small", [(63, 5), (65, 0), (127, 1), (128, 200), (129, 0), (255, 130),
                                        (257, 7), (512, 64), (513, 0), (900, 900)])
@pytest.mark.parametrize("layers,tile", [(3, (16, 16)), (1, (8, 8)), (5, (16, 16)), (3, (32, 16))])
def test_large_list_is_gathered(wide, small, layers, tile, device):
  w, h = 150, 90
  rng = np.random.default_rng(wide)
  center = rng.uniform(-1, 1, (wide + small, 1, 3))
  reach = np.where(np.arange(wide + small) < wide, 0.7, 0.02)[:, None, None]
  verts = (center + reach * rng.uniform(-1, 1, (wide + small, 3, 3))).reshape(-1, 3)
  order = rng.permutation(wide + small)
  clip = np.concatenate([verts, np.ones((len(verts), 1))], 1).astype(np.float32)
  tri = np.arange(len(verts), dtype=np.int32).reshape(-1, 3)[order]
  dclip, dtri = torch.tensor(clip, device=device), torch.tensor(tri, device=device)
  # a second image with an empty list, and a third like the first
  tiny = dclip[:3] * torch.tensor([0.05, 0.05, 1.0, 1.0], device=device)
  batch = kernels.ImageBatch([w, 40, w], [h, 30, h], [len(clip), 3, len(clip)],
                             [len(tri), 1, len(tri)])
  clips = torch.cat([dclip, tiny, dclip])
  tris = torch.cat([dtri, torch.arange(3, dtype=torch.int32, device=device)[None], dtri])
  out = [kernels.rasterize_packed(clips, tris, batch, kernels.raster_config(
      layers, 0, _lib.DR_DEPTH_DISCRETIZED, tile, large)) for large in (100000, 1, 6)]
  for got in out[1:]:
    for a, b in zip(got, out[0]):
      assert torch.equal(a, b)
  n = layers * w * h
  ref = raster.rasterize(clip, tri, w, h, layers, 0, raster.DEPTH_DISCRETIZED)
  for part in (slice(0, n), slice(out[1][0].numel() - n, None)):
    ids, z, bary = (x[part].cpu().numpy() for x in out[1])
    assert_same((ids.reshape(layers, h, w), z.reshape(layers, h, w),
                 bary.reshape(layers, h, w, 3)), ref)


# Empty tiles come in runs of one to eight, by their number: the depths of nearly
# empty images from hundreds to a hundred thousand tiles, and of one with none.
@pytest.mark.parametrize("w,h", [(260, 250), (1111, 700), (2304, 2200)])
@pytest.mark.parametrize("tile", [(8, 8), (16, 16), (128, 8)])
@pytest.mark.parametrize("empty", [False, True])
def test_empty_runs(w, h, tile, empty, device):
  clip = torch.tensor([[0.5, 0.5, 0.1, 1.0], [0.9, 0.5, 0.1, 1.0], [0.5, 0.95, 0.1, 1.0]],
                      device=device)
  tri = torch.arange(0 if empty else 3, dtype=torch.int32, device=device).view(-1, 3)
  batch = kernels.ImageBatch.single(w, h, 3, len(tri))
  out = (torch.full((2 * w * h,), -7, dtype=torch.int32, device=device),
         torch.full((2 * w * h,), float("nan"), device=device),
         torch.full((2 * w * h, 3), float("nan"), device=device))
  ids, z, bary = kernels.rasterize_packed(
      clip, tri, batch, kernels.raster_config(2, 0, _lib.DR_DEPTH_FLOAT, tile), out=out)
  z = z.view(2, h, w)
  covered = z[0] != 1.0
  assert not torch.isnan(z).any() and not torch.isnan(bary).any() and (z[1] == 1.0).all()
  assert torch.equal(ids.view(2, h, w)[0], torch.where(covered, 0, -1).int())
  assert (ids.view(2, h, w)[1] == -1).all() and not bary.view(2, h, w, 3)[1].any()
  # half of a 0.2 x 0.225 box of the image, within its outline's pixels
  want = 0 if empty else 0.5 * 0.2 * 0.225 * w * h
  assert abs(int(covered.sum()) - want) <= (0 if empty else 0.3 * (w + h))


# A row's keys are permuted within the power of two in the tile's width (up to 16).
@pytest.mark.parametrize("tile", [(1, 16), (2, 3), (6, 10), (12, 20), (4, 40), (8, 33), (24, 16),
                                  (20, 9), (48, 16), (128, 8), (3, 128)])
@pytest.mark.parametrize("layers", [1, 3, 6])
def test_tile_widths_match_oracle(tile, layers, device):
  for kind, n in (("big", 40), ("soup", 300)):
    verts, tris = _scene(kind, n, 131, 77, 5)
    ref = raster.rasterize(verts, tris, 131, 77, layers, 1, raster.DEPTH_DISCRETIZED)
    clip = torch.tensor(np.asarray(verts, np.float32), device=device)
    tri = torch.tensor(np.asarray(tris, np.int32), device=device)
    batch = kernels.ImageBatch.single(131, 77, len(clip), len(tri))
    got = kernels.rasterize_packed(clip, tri, batch, kernels.raster_config(
        layers, 1, _lib.DR_DEPTH_DISCRETIZED, tile))
    shape = (layers, 77, 131)
    assert_same((got[0].view(shape).cpu().numpy(), got[1].view(shape).cpu().numpy(),
                 got[2].view(*shape, 3).cpu().numpy()), ref)
