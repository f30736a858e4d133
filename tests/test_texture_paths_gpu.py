"""The texture kernels at the edges of their dispatch: one to five channels,
point counts around a block's, buffers off the wide loads' alignment."""
import numpy as np
import pytest
import torch

from diffren_gb300 import shaders
from oracle import texture

pytestmark = pytest.mark.gpu


def _at_offset(a, floats, device):
  """A contiguous CUDA copy of `a` that starts `floats` floats into its storage."""
  buf = torch.empty(a.size + floats, dtype=torch.float32, device=device)
  out = buf[floats:].view(a.shape)
  out.copy_(torch.tensor(a))
  return out


@pytest.mark.parametrize("channels", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("points", [1, 255, 257, 511, 512, 513, 1025])
@pytest.mark.parametrize("offset", [0, 1, 2])
def test_texture_dispatch(channels, points, offset, device):
  rng = np.random.default_rng(points + channels)
  tex = rng.uniform(-1, 1, (6, 9, channels)).astype(np.float32)
  uv = rng.uniform(-0.2, 1.2, (points, 2)).astype(np.float32)
  g = rng.standard_normal((points, channels)).astype(np.float32)
  g[::5] = 0.0  # points without gradient
  g[1::7, 0] = 0.0  # and channels
  du = _at_offset(uv, offset, device).requires_grad_()
  dt = _at_offset(tex, offset, device).requires_grad_()
  out = shaders.texture_map(du, dt)
  np.testing.assert_array_equal(out.detach().cpu().numpy(), texture.texture_map(uv, tex))
  got = torch.autograd.grad(out, (du, dt), _at_offset(g, offset, device))
  tu = torch.tensor(uv, dtype=torch.float64, requires_grad=True)
  tt = torch.tensor(tex, dtype=torch.float64, requires_grad=True)
  want = torch.autograd.grad(texture.texture_map_t(tu, tt), (tu, tt),
                             torch.tensor(g, dtype=torch.float64))
  # A texel sums up to 4 points / 54 texels of products of three rounded
  # factors, a coordinate channels x 2 of them times 9: below 1e-4 of the
  # largest magnitude.
  for x, y in zip(got, want):
    assert (x.cpu().double() - y).abs().max() <= 1e-4 * y.abs().max()


# One point a thread up to 466,944 points, two above: both sides of the line, and
# counts that leave a block one point.
@pytest.mark.parametrize("points", [466_943, 466_944, 466_945, 467_457, 467_458])
@pytest.mark.parametrize("channels", [1, 2, 3, 4])
def test_points_a_thread(points, channels, device):
  rng = np.random.default_rng(points)
  tex = rng.uniform(-1, 1, (6, 9, channels)).astype(np.float32)
  uv = rng.uniform(-0.2, 1.2, (points, 2)).astype(np.float32)
  g = rng.standard_normal((points, channels)).astype(np.float32)
  du, dt = _at_offset(uv, 0, device).requires_grad_(), _at_offset(tex, 0, device).requires_grad_()
  out = shaders.texture_map(du, dt)
  np.testing.assert_array_equal(out.detach().cpu().numpy(), texture.texture_map(uv, tex))
  got = torch.autograd.grad(out, (du, dt), _at_offset(g, 0, device))
  tu = torch.tensor(uv, dtype=torch.float64, requires_grad=True)
  tt = torch.tensor(tex, dtype=torch.float64, requires_grad=True)
  want = torch.autograd.grad(texture.texture_map_t(tu, tt), (tu, tt),
                             torch.tensor(g, dtype=torch.float64))
  # A coordinate's gradient sums channels x 2 rounded products, as above, but for
  # the points whose float32 location falls on the other side of a texel's center
  # (2^-21 of a texel on either axis: some 1e-6 of them). A texel sums up to 4 x
  # 467k / 54 products of either sign, each within 2^-24 of its magnitude: below
  # 1e-3 of the largest sum.
  far = (got[0].cpu().double() - want[0]).abs().max(1).values > 1e-4 * want[0].abs().max()
  assert far.double().mean() <= 3e-5
  assert (got[1].cpu().double() - want[1]).abs().max() <= 1e-3 * want[1].abs().max()


# float32 rounds sides above 2^24 to even numbers: 2^24 + 3 becomes 2^24 + 4, one
# past the last padded texel. Coordinates at and beyond the far edge are the last
# texel and its gradient, those at the near edge the first.
@pytest.mark.parametrize("side", [2**24 - 1, 2**24, 2**24 + 3])
@pytest.mark.parametrize("channels,rows", [(1, True), (1, False), (2, True), (3, False), (4, True)])
def test_far_edge_of_long_sides(side, channels, rows, device):
  far = [1.0, 1.25, 2.0, 1e9, float("inf")]
  at = torch.tensor([0.0, -1.0] + far, device=device)
  mid = torch.full_like(at, 0.5)
  uv = torch.stack((mid, at) if rows else (at, mid), -1).requires_grad_()
  tex = torch.zeros(side, channels, device=device)
  tex[0] = torch.arange(1, channels + 1, device=device)
  tex[-1] = -torch.arange(3, channels + 3, device=device)
  tex = (tex[:, None] if rows else tex[None]).requires_grad_()
  ends = tex.detach().view(side, channels)[[0, 0] + [-1] * len(far)]
  out = shaders.texture_map(uv, tex)
  assert torch.equal(out, ends)
  g = torch.arange(1, out.numel() + 1, device=device).float().view_as(out)
  d_tex = torch.autograd.grad(out, tex, g)[0].view(side, channels)
  assert torch.equal(d_tex[0], g[:2].sum(0)) and torch.equal(d_tex[-1], g[2:].sum(0))
  assert int((d_tex != 0).sum()) == 2 * channels
