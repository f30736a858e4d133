"""Shading layer by layer and compositing: every way a shader may treat its
slices gives the gradients of a plain expression, and the OVER kernels for
aligned RGBA agree with the general ones at every layer bound."""
import pytest
import torch

from diffren_gb300 import constants, kernels, render, workloads

pytestmark = pytest.mark.gpu


def _inplace(a):
  c = a["rgba"]
  c.mul_(0.5)
  return c


def _unused_layer():
  calls = []

  def shade(a):
    calls.append(0)
    return a["rgba"] if len(calls) % 2 else torch.zeros_like(a["rgba"])
  return shade


@pytest.mark.parametrize("mode", [constants.CompositingMode.SPLAT_OVER,
                                  constants.CompositingMode.OVER])
@pytest.mark.parametrize("batched", [False, True])
@pytest.mark.parametrize("layers", [1, 2, 3])
def test_shader_slices(mode, batched, layers, device):
  m = workloads.icosphere_workload(5, seed=1)
  eyes = workloads.sphere_eyes(2, seed=2)
  w, h = 45, 38
  cams = torch.stack([torch.tensor(workloads.camera_matrix(e, w, h)) for e in eyes]).to(device)
  cam = cams if batched else cams[0]
  tri = torch.tensor(m.triangles, device=device)
  seed = torch.rand((2, h, w, 4) if batched else (h, w, 4), device=device)

  def run(shade, extra=False):
    v = torch.tensor(m.vertices, device=device, requires_grad=True)
    c = torch.cat([torch.tensor(m.colors), torch.ones(len(m.colors), 1)], 1).to(
        device).requires_grad_()
    attrs = {"rgba": c, "pos": v} if extra else {"rgba": c}
    options = dict(compositing_mode=mode,
                   compute_diff_barys=mode == constants.CompositingMode.OVER)
    out = render.render_triangles(v, attrs, tri, cam, w, h, shade, layers, **options)
    with torch.no_grad():
      still = render.render_triangles(v, attrs, tri, cam, w, h, shade, layers, **options)
    assert torch.equal(out, still)
    return (out.detach(), *torch.autograd.grad(out, [v, c], seed))

  pairs = [(lambda a: a["rgba"], lambda a: a["rgba"] * 1.0, False),
           (_inplace, lambda a: a["rgba"] * 0.5, False),
           (lambda a: a["rgba"], lambda a: a["rgba"] + 0.0 * a["pos"].sum(-1, keepdim=True), True)]
  for shade, plain, extra in pairs:
    got, want = run(shade, extra), run(plain, extra)
    assert torch.equal(got[0], want[0])
    for x, y in zip(got[1:], want[1:]):  # float atomics: 1e-5 of the largest magnitude
      assert (x - y).abs().max() <= 1e-5 * y.abs().max()
  if layers == 2 and not batched:
    out = run(_unused_layer())
    assert all(torch.isfinite(x).all() for x in out)
  kept = []

  def keep(a):
    kept.append(a["rgba"])
    return a["rgba"]
  v = torch.tensor(m.vertices, device=device, requires_grad=True)
  c = torch.rand(len(m.vertices), 4, device=device, requires_grad=True)
  out = render.render_triangles(v, {"rgba": c}, tri, cam, w, h, keep, layers,
                                compositing_mode=mode)
  grads = torch.autograd.grad(out, kept, seed)  # the shader's input is part of the graph
  assert all(g.shape == k.shape for g, k in zip(grads, kept)) and grads[0].abs().sum() > 0


@pytest.mark.parametrize("layers", [1, 2, 3, 4, 5, 8, 9, 16])
def test_over_aligned_rgba_matches_general(layers, device):
  sizes = [(37, 21), (5, 1), (64, 8)]
  batch = kernels.ImageBatch([s[0] for s in sizes], [s[1] for s in sizes], [0] * 3, [0] * 3)
  g = torch.Generator(device=device).manual_seed(layers)
  n = layers * batch.total_pixels
  z = (torch.rand(n, generator=g, device=device) > 0.4).float()
  results = []
  for offset in (0, 1):
    buf = torch.empty(4 * n + 4, device=device)
    shaded = buf[offset:offset + 4 * n].view(n, 4)
    shaded.copy_(torch.rand(n, 4, generator=torch.Generator(device=device).manual_seed(5),
                            device=device))
    shaded.requires_grad_()
    out = kernels.over_packed(shaded, z, batch, layers)
    d = torch.randn(out.shape, generator=torch.Generator(device=device).manual_seed(6),
                    device=device)
    results.append((out.detach(), *torch.autograd.grad(out, [shaded], d)))
  for a, b in zip(*results):
    assert torch.equal(a, b)
