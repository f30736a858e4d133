"""The splat forward's and the samples VJP's dispatch edges: pixels whose
surroundings hold foreground in layer 0 only, sample counts and image sizes on
both sides of the VJP's block rule."""
import numpy as np
import pytest
import torch

from diffren_gb300 import _lib, kernels, workloads

pytestmark = pytest.mark.gpu


# Both calls see the same samples; without a depth buffer the foreground
# weight travels in the positions and every pixel takes the general surface
# test, so the images agree bit for bit (also for equal, infinite and NaN
# depths, whose comparisons are all false).
@pytest.mark.parametrize("layers", [1, 2, 3, 5, 9])
@pytest.mark.parametrize("channels", [1, 3, 4, 7])
def test_single_layer_surroundings_match_general_test(layers, channels, device):
  w, h = 75, 50
  g = torch.Generator(device=device).manual_seed(layers * 16 + channels)
  rand = lambda *s: torch.rand(*s, generator=g, device=device)
  count = torch.zeros(h, w, dtype=torch.long, device=device)  # foreground layers per pixel
  count[4:46, 3:70] = 1
  count[20:30, 40:60] = min(2, layers)
  count[33:, 10:20] = layers
  count[rand(h, w) < 0.2] = 0
  z = torch.full((layers, h, w), 1.0, device=device)
  depth = 0.5 + 0.49 * rand(layers, h, w)
  depth = torch.where(rand(layers, h, w) < 0.3, torch.round(depth * 8) / 8 - 0.01, depth)
  depth[:, 10, 10:14] = float("nan")
  depth[:, 12, 10:14] = float("inf")
  fg = torch.arange(layers, device=device)[:, None, None] < count
  z[fg] = 0.5
  pos = torch.zeros(layers, h, w, 4, device=device)
  pos[..., 0] = torch.arange(w, device=device) + 0.5 + 0.2 * (rand(layers, h, w) - 0.5)
  pos[..., 1] = torch.arange(h, device=device)[:, None] + 0.5 + 0.2 * (rand(layers, h, w) - 0.5)
  pos[..., 2] = torch.where(fg, depth, torch.ones_like(depth))
  pos[..., 3] = fg.float()
  colors = rand(layers, h, w, channels)
  batch = kernels.ImageBatch.single(w, h, 0, 0)
  flat = pos.view(-1, 4)
  general = kernels.splat_packed(flat, colors.view(-1, channels), batch, layers)
  for grad in (False, True):  # one block per tile, and the listed tiles
    c = colors.view(-1, channels).clone().requires_grad_(grad)
    out = kernels.splat_packed(flat, c, batch, layers, z=z.view(-1)).detach()
    assert torch.equal(out, general) and not torch.isnan(out).any()


def _reference(attr, clip, bary, vid, sizes, g_attr, g_pos):
  """64-bit gradients of the interpolation and the splat positions of
  foreground samples."""
  attr = attr.double().requires_grad_()
  clip = clip.double().requires_grad_()
  b = bary.double()[:, :, None]
  a = (attr[vid] * b).sum(1)
  c = (clip[vid] * b).sum(1)
  xy = (c[:, :2] / c[:, 3:] + 1.0) * sizes * 0.5
  loss = (a * g_attr.double()).sum() + (xy * g_pos.double()[:, :2]).sum()
  return torch.autograd.grad(loss, [attr, clip])


# One sample a thread below 3.7 M samples, eight above; a block that spans
# images looks each sample up.
@pytest.mark.parametrize("sizes,layers,channels", [
    ([(9, 7)] * 40, 3, 4), ([(1, 1), (33, 5), (64, 64), (3, 100)], 2, 3), ([(300, 211)], 1, 5),
    ([(1201, 1050)], 3, 4), ([(640, 480)] * 5 + [(31, 17)] * 30 + [(900, 800)], 2, 2)])
@pytest.mark.parametrize("deterministic", [False, True])
def test_samples_vjp_block_rule(sizes, layers, channels, deterministic, device):
  n = len(sizes)
  m = workloads.soup_workload(400, seed=3, mu=-2.0, sigma=0.5)
  eyes = workloads.sphere_eyes(n, seed=4)
  cams = torch.tensor(np.stack([workloads.camera_matrix(e, w, h)
                                for e, (w, h) in zip(eyes, sizes)]), device=device)
  V, T = len(m.vertices), len(m.triangles)
  batch = kernels.ImageBatch([s[0] for s in sizes], [s[1] for s in sizes], [V] * n, [T] * n)
  verts = torch.tensor(m.vertices, device=device).repeat(n, 1)
  tri = torch.tensor(m.triangles, device=device).repeat(n, 1)
  clip = kernels.transform(verts, cams, batch).requires_grad_()
  g = torch.Generator(device=device).manual_seed(1)
  attr = torch.rand(n * V, channels, generator=g, device=device).requires_grad_()
  cfg = kernels.raster_config(layers, 1, _lib.DR_DEPTH_DISCRETIZED)
  a, pos, ids, z, bary = kernels.rasterize_interpolate_packed(
      attr, clip, tri, batch, cfg, kernels.Workspace(device), deterministic=deterministic)
  g_attr = torch.randn(a.shape, generator=g, device=device)
  g_pos = torch.randn(pos.shape, generator=g, device=device)
  got = torch.autograd.grad([a, pos], [attr, clip], [g_attr, g_pos])
  per = torch.tensor([layers * w * h for w, h in sizes], device=device)
  img = torch.repeat_interleave(torch.arange(n, device=device), per)
  fg = z != 1.0
  vid = tri[img[fg] * T + ids[fg].long()].long() + V * img[fg][:, None]
  wh = torch.tensor(sizes, dtype=torch.float64, device=device)[img[fg]]
  want = _reference(attr.detach(), clip.detach(), bary[fg], vid, wh, g_attr[fg], g_pos[fg])
  for x, y in zip(got, want):
    assert (x.double() - y).abs().max() <= 1e-4 * y.abs().max()


# Four samples a thread from 467k samples on, to 1.4 M, or 3.7 M in fixed point;
# the first two sizes lie on both sides of the lower line.
@pytest.mark.parametrize("sizes,layers,channels", [
    ([(683, 683)], 1, 4), ([(684, 684)], 1, 4), ([(97, 131)] * 40 + [(3, 1)] * 9, 2, 3),
    ([(1183, 1184)], 1, 2), ([(1184, 1184)], 1, 2), ([(640, 480), (901, 703)], 3, 9)])
@pytest.mark.parametrize("deterministic", [False, True])
def test_samples_vjp_four_a_thread(sizes, layers, channels, deterministic, device):
  test_samples_vjp_block_rule(sizes, layers, channels, deterministic, device)


# Four channels in a 16-byte aligned buffer save float4 planes, anything else
# one plane per value; both hold the same numbers.
@pytest.mark.parametrize("layers", [1, 2, 3])
@pytest.mark.parametrize("listed", [True, False])
def test_saved_planes_aligned_and_not(layers, listed, device):
  w, h, C = 83, 37, 4
  g = torch.Generator(device=device).manual_seed(layers)
  rand = lambda *s: torch.rand(*s, generator=g, device=device)
  fg = torch.arange(layers, device=device)[:, None, None] < (rand(h, w) * (layers + 1)).long()
  z = torch.where(fg, 0.5, 1.0).contiguous()
  pos = torch.zeros(layers, h, w, 4, device=device)
  pos[..., 0] = torch.arange(w, device=device) + rand(layers, h, w)
  pos[..., 1] = torch.arange(h, device=device)[:, None] + rand(layers, h, w)
  pos[..., 2] = torch.where(fg, rand(layers, h, w), 1.0)
  pos[..., 3] = fg.float()
  colors = rand(layers, h, w, C)
  d_out = torch.randn(h, w, C, generator=g, device=device)
  batch = kernels.ImageBatch.single(w, h, 0, 0)
  lib, P, st = _lib.load(), kernels._p, kernels._stream(device)
  zb = z if listed else None
  results = []
  for offset in (0, 1):
    saved = torch.empty((3 * (C + 1) + 2) * w * h + 1, device=device)[offset:]
    out = torch.empty(h, w, C, device=device)
    d_c, d_p = torch.zeros_like(colors), torch.zeros_like(pos)
    assert lib.dr_splat_fwd(P(pos), P(zb), P(colors), C, batch.ptr, 1, layers, P(out), P(saved),
                            None, None, st) == 0
    assert lib.dr_splat_bwd(P(d_out), P(pos), P(zb), P(colors), P(saved), C, batch.ptr, 1, layers,
                            P(d_c), P(d_p), st) == 0
    results.append((out, d_c, d_p))
  for a, b in zip(*results):
    assert torch.equal(a, b) and torch.count_nonzero(a) > 0


# The layout follows the buffer's alignment in the forward: a saved-tensor hook
# (or a caller of the registered op) that hands the backward a copy elsewhere
# gets the same gradients.
@pytest.mark.parametrize("layers", [1, 2, 3, 4])
@pytest.mark.parametrize("offset", [1, 2, 3])
def test_saved_buffer_moved_off_its_alignment(layers, offset, device):
  from diffren_gb300 import ops
  w, h, C = 70, 33, 4
  g = torch.Generator(device=device).manual_seed(layers)
  rand = lambda *s: torch.rand(*s, generator=g, device=device)
  fg = torch.arange(layers, device=device)[:, None, None] < (rand(h, w) * (layers + 1)).long()
  z = torch.where(fg, 0.5, 1.0).contiguous()
  pos = torch.zeros(layers, h, w, 4, device=device)
  pos[..., 0] = torch.arange(w, device=device) + rand(layers, h, w)
  pos[..., 1] = torch.arange(h, device=device)[:, None] + rand(layers, h, w)
  pos[..., 2] = torch.where(fg, rand(layers, h, w), 1.0)
  pos[..., 3] = fg.float()
  colors = rand(layers, h, w, C)
  d_out = torch.randn(h, w, C, generator=g, device=device)
  batch = kernels.ImageBatch.single(w, h, 0, 0)
  rows = 3 * (C + 1) + 2

  def moved(t):
    if t.shape[0] != rows:
      return t
    buf = torch.empty(t.numel() + offset, device=device)
    return buf[offset:].view_as(t).copy_(t)

  def grads(unpack):
    p, c = pos.view(-1, 4).clone().requires_grad_(), colors.view(-1, C).clone().requires_grad_()
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t, unpack):
      out = kernels.splat_packed(p, c, batch, layers, z=z.view(-1))
      d_p, d_c = torch.autograd.grad(out, [p, c], d_out.view(-1, C))
    return torch.where(fg.view(-1, 1), d_p, 0.0), d_c
  want = grads(lambda t: t)
  for a, b in zip(grads(moved), want):
    assert torch.equal(a, b) and torch.count_nonzero(a) > 0
  image, saved = ops.splat_fwd(pos, colors, z)
  d_p, d_c = ops.splat_bwd(d_out, pos, colors, z, moved(saved))
  assert torch.equal(d_c.view(-1, C), want[1]) and torch.equal(d_p.view(-1, 4), want[0])
