"""Packing attribute columns and splitting them again: values, gradients (also
where the parts' gradients already share one buffer, or are missing) and
forward mode, against torch.cat and torch.split."""
import ctypes

import pytest
import torch

from diffren_gb300 import _lib, kernels


def test_pack_columns_rejects_bad_arguments():
  lib = _lib.load()
  one = (ctypes.c_int32 * 1)(3)
  stride = (ctypes.c_int64 * 1)(3)
  ptr = (ctypes.c_void_p * 1)(None)
  for args in ((None, one, stride, 1, 4), (ptr, one, stride, 0, 4), (ptr, one, stride, 1, -1),
               (ptr, (ctypes.c_int32 * 1)(17), stride, 1, 4), (ptr, one, stride, 1, 4)):
    assert lib.dr_pack_columns(*args, None, None) == 1
  two = (ctypes.c_int32 * 2)(9, 8)
  assert lib.dr_pack_columns((ctypes.c_void_p * 2)(), two, (ctypes.c_int64 * 2)(9, 8), 2, 4, None,
                             None) == 1
  assert lib.dr_pack_columns(ptr, one, stride, 1, 0, None, None) == 0


@pytest.mark.gpu
@pytest.mark.parametrize("rows", [0, 1, 127, 128, 129, 5000])
@pytest.mark.parametrize("widths", [(3, 3, 3), (1, 1), (4, 12), (16,), (2, 5, 1, 7), (1,) * 16])
def test_pack_and_split(rows, widths, device):
  g = torch.Generator(device=device).manual_seed(rows)
  wide = torch.randn(rows, 20, generator=g, device=device)
  parts = [torch.randn(rows, w, generator=g, device=device).requires_grad_() for w in widths]
  strided = [wide[:, i:i + w] for i, w in enumerate(widths) if i + w <= 20]
  packed = kernels.pack_columns(parts)
  assert torch.equal(packed, torch.cat(parts, 1))
  if len(strided) == len(widths):
    assert torch.equal(kernels._pack(strided, list(widths), rows, device), torch.cat(strided, 1))
  split = kernels.split_channels(packed, list(widths))
  for a, b in zip(split, torch.split(packed, list(widths), 1)):
    assert torch.equal(a, b)
  seeds = [torch.randn(rows, w, generator=g, device=device) for w in widths]
  whole = torch.randn(rows, sum(widths), generator=g, device=device)
  for grads in (seeds, torch.split(whole, list(widths), 1)):
    used = list(range(0, len(widths), 2))  # every other part unused: no gradient
    for which in (list(range(len(widths))), used):
      got = torch.autograd.grad([split[i] for i in which], parts, [grads[i] for i in which],
                                retain_graph=True, allow_unused=True)
      for i, x in enumerate(got):
        assert torch.equal(x, grads[i] if i in which else torch.zeros_like(grads[i]))


# Gradients that share a buffer are that buffer where it starts on 16 bytes, and
# are packed into one that does elsewhere (float offsets 1 to 3).
@pytest.mark.parametrize("offset", [0, 1, 2, 3, 4])
def test_one_buffer_is_aligned(offset):
  whole = torch.arange(40.0 + offset)[offset:].view(10, 4)
  got = kernels._one_buffer(torch.split(whole, [3, 1], 1), (10, 4), (4, 1), [0, 3])
  assert got is None if offset % 4 else torch.equal(got, whole)


@pytest.mark.gpu
@pytest.mark.parametrize("offset", [0, 1, 2, 4])
def test_split_gradients_off_alignment_reach_the_rasterizer(offset, device):
  w, h, layers = 24, 20, 2
  clip = torch.tensor([[-0.9, -0.9, 0.1, 1.0], [0.9, -0.8, 0.2, 1.0], [0.0, 0.9, 0.3, 1.0]],
                      device=device)
  tri = torch.tensor([[0, 1, 2]], dtype=torch.int32, device=device)
  attr = torch.rand(3, 4, device=device).requires_grad_()
  cfg = kernels.raster_config(layers, 0, _lib.DR_DEPTH_DISCRETIZED)
  batch = kernels.ImageBatch.single(w, h, 3, 1)
  out, _, _, z, bary = kernels.rasterize_interpolate_packed(attr, clip, tri, batch, cfg,
                                                            kernels.Workspace(device))
  n = out.shape[0]
  d = torch.ones(4 * n + offset, device=device)[offset:].view(n, 4)
  got = torch.autograd.grad(kernels.split_channels(out, [3, 1]), attr, torch.split(d, [3, 1], 1))[0]
  want = bary[z != 1.0].double().sum(0)  # the same for every channel
  # sums of some hundred products in [0, 1]
  assert (got.double() - want[:, None]).abs().max() <= 1e-5 * want.max() and want.min() > 10


@pytest.mark.gpu
def test_pack_and_split_forward_mode(device):
  import torch.autograd.forward_ad as fwAD
  a, b = torch.randn(50, 3, device=device), torch.randn(50, 4, device=device)
  da = torch.randn_like(a)
  with fwAD.dual_level():
    packed = kernels.pack_columns([fwAD.make_dual(a, da), b])
    x, y = kernels.split_channels(packed, [3, 4])
    assert torch.equal(fwAD.unpack_dual(x).tangent, da)
    assert not fwAD.unpack_dual(y).tangent.any()


# The columns of one [n, 9] buffer, in any order, get their gradients as the
# columns of one buffer; the values are those of separate inputs.
@pytest.mark.gpu
@pytest.mark.parametrize("rows", [1, 3, 255, 256, 257, 1000])
@pytest.mark.parametrize("order", [(0, 1, 2), (2, 0, 1)])
@pytest.mark.parametrize("alpha", [False, True])
def test_point_light_packed_gradients(rows, order, alpha, device):
  from diffren_gb300 import shaders
  g = torch.Generator(device=device).manual_seed(rows)
  packed = torch.randn(rows, 9, generator=g, device=device)
  seed = torch.randn(rows, 4 if alpha else 3, generator=g, device=device)
  results = []
  for split in (True, False):
    p = packed.clone().requires_grad_()
    cols = kernels.split_channels(p, [3, 3, 3])
    if not split:
      cols = [c.contiguous() for c in cols]
    c = [cols[i] for i in order]
    out = shaders.point_light(c[0], c[1], c[2], (2.0, 2.0, 2.0), ks=0.4, ns=3.0, alpha=alpha)
    results.append((out.detach(), *torch.autograd.grad(out, [p], seed)))
  for a, b in zip(*results):
    assert torch.equal(a, b)


# Saved-tensor hooks hand back tensors with strides of their own: the gradients
# of packed columns are those without hooks.
@pytest.mark.gpu
@pytest.mark.parametrize("rows", [2, 300])
@pytest.mark.parametrize("unpack", [lambda t: t.contiguous(), lambda t: t.t().contiguous().t(),
                                    lambda t: torch.cat([t, t], 1)[:, 3:]])
def test_point_light_under_saved_tensor_hooks(rows, unpack, device):
  from diffren_gb300 import shaders
  g = torch.Generator(device=device).manual_seed(rows)
  packed = torch.randn(rows, 9, generator=g, device=device)
  seed = torch.randn(rows, 3, generator=g, device=device)

  def grad(hooks):
    p = packed.clone().requires_grad_()
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t, hooks):
      out = shaders.point_light(*kernels.split_channels(p, [3, 3, 3]), (2.0, 2.0, 2.0), ks=0.4,
                                ns=3.0)
      return torch.autograd.grad(out, p, seed)[0]
  assert torch.equal(grad(unpack), grad(lambda t: t))


# A gradient that is differentiated again (create_graph) goes through the
# split and through the layer slices as through torch's own operations.
@pytest.mark.gpu
@pytest.mark.parametrize("rows", [1, 130])
def test_second_derivatives(rows, device):
  from diffren_gb300 import render
  g = torch.Generator(device=device).manual_seed(rows)
  t = torch.randn(2, rows, 1, 7, generator=g, device=device)

  def columns(split):
    def f(x):
      a, b = split(x, [3, 4])
      return (a ** 3).sum() + (a * a).sum() * (b ** 2).sum()
    return f

  def layers(shade):
    def f(x):
      y = shade(x)
      return (y[0] * y[1]).pow(2).sum()
    return f
  pairs = [(columns(kernels.split_channels), columns(lambda x, w: torch.split(x, w, -1))),
           (layers(lambda x: render._shade_layers(lambda a: a["c"] ** 2, {"c": x}, 2, False)),
            layers(lambda x: x ** 2)),
           (layers(lambda x: render._shade_layers(lambda a: a["c"], {"c": x}, 2, False)),
            layers(lambda x: x))]
  for pair in pairs:
    second = []
    for f in pair:
      x = t.clone().requires_grad_()
      first, = torch.autograd.grad(f(x), x, create_graph=True)
      second.append(torch.autograd.grad(first.pow(2).sum(), x)[0])
    assert (second[0] - second[1]).abs().max() <= 1e-5 * second[1].abs().max()
