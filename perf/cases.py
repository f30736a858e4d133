"""The work that users of this framework have it do, as measurable cases.

A case is a dict of plain values. ``prepare`` makes its seeded inputs and what
a program keeps between calls (a ``BatchRenderer``, a captured step), ``run``
makes one pass through the public entry points, and ``exact`` restates the
same outputs in 64-bit torch. The meshes, cameras and sizes follow the
framework's own workloads (diffren_gb300/workloads.py); a case's seed moves
vertices, colors, cameras and targets, never its sizes.
"""
import math

import numpy as np
import torch

from diffren_gb300 import batch as batch_lib
from diffren_gb300 import constants
from diffren_gb300 import losses
from diffren_gb300 import mesh as mesh_lib
from diffren_gb300 import rasterize
from diffren_gb300 import render
from diffren_gb300 import shaders
from diffren_gb300 import workloads

LIGHT = (2.0, 2.0, 2.0)


def listed():
  return [
      # Fitting one small mesh with render_triangles, as the first script of a
      # user and most tests do: call latency.
      dict(name="fit_small", kind="single", mesh="sphere", size=8, width=64, height=64,
           layers=3),
      # A lit mesh-fitting step captured once and replayed (vertex normals and
      # a point light recomputed every step): launch-bound.
      dict(name="lit_256", kind="fit", mesh="sphere", size=16, images=1, width=256, height=256,
           layers=3, shade="lit", graph=True, deterministic=False),
      # One mesh seen by eight cameras: many tiny triangles on few pixels.
      dict(name="soup_512", kind="fit", mesh="soup", size=200000, images=8, width=512,
           height=512, layers=3, shade="rgba", graph=False, deterministic=False),
      # The same with a closed surface: few triangles per pixel, one layer deep.
      dict(name="sphere_1024", kind="fit", mesh="sphere", size=71, images=8, width=1024,
           height=1024, layers=3, shade="rgba", graph=False, deterministic=False),
      # Textured terrain at high resolution, gradients to vertices and texture.
      dict(name="terrain_2048", kind="fit", mesh="terrain", size=708, images=4, width=2048,
           height=2048, layers=3, shade="texture", graph=False, deterministic=False),
      # The largest: a ragged batch of 64 meshes, each with its own camera and
      # resolution.
      dict(name="ragged_64", kind="ragged", images=64, median=20000, most=500000, sizes=1024,
           odd=False, layout=0, layers=3, deterministic=False),
      # A small ragged batch of odd sizes, two layers, reproducible gradients.
      dict(name="ragged_odd", kind="ragged", images=11, median=3000, most=40000, sizes=420,
           odd=True, layout=5, layers=2, deterministic=True),
      # Forward only: a preview image of a detailed mesh, no gradients kept.
      dict(name="preview", kind="preview", mesh="sphere", size=71, width=1283, height=717,
           layers=1),
      # The rasterizer by itself: ids, depths and barycentrics of four layers,
      # both faces, for a shader or an analysis outside of the framework.
      dict(name="raster_layers", kind="raster", mesh="soup", size=20000, width=640, height=479,
           layers=4),
      # Interior gradients without splatting: differentiable barycentrics,
      # interpolation and OVER compositing.
      dict(name="over_diff", kind="over", mesh="sphere", size=40, width=517, height=389,
           layers=2),
      # The texture shader by itself, RGB, forward and backward.
      dict(name="texture_rgb", kind="texture", points=1500001, width=1023, height=767,
           channels=3),
      # Vertex normals of a large mesh, forward and backward.
      dict(name="normals", kind="normals", size=708),
  ]


def _log(rng, lo, hi):
  return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
  """One more case of the listed ranges."""
  kind = rng.choice(["single", "fit", "fit", "fit", "ragged", "ragged", "preview", "raster",
                     "over", "texture", "normals"])
  if kind == "texture":
    return dict(kind=kind, points=_log(rng, 20000, 6000000), width=_log(rng, 40, 2048),
                height=_log(rng, 40, 2048), channels=rng.choice([1, 3, 4, 4]))
  if kind == "normals":
    return dict(kind=kind, size=_log(rng, 20, 900))
  if kind == "ragged":
    return dict(kind=kind, images=rng.randint(2, 64), median=_log(rng, 800, 20000), most=300000,
                sizes=_log(rng, 100, 900), odd=rng.random() < 0.7, layout=rng.randint(0, 9999),
                layers=rng.choice([1, 2, 3, 3, 3]), deterministic=rng.random() < 0.25)
  if kind == "fit":
    mesh = rng.choice(["soup", "sphere", "terrain"])
    images = rng.choice([1, 2, 3, 4, 8])
    side = _log(rng, 100, {1: 2000, 2: 1600, 3: 1300, 4: 1100, 8: 900}[images])
    size = {"soup": _log(rng, 500, 200000), "sphere": _log(rng, 5, 80),
            "terrain": _log(rng, 20, 500)}[mesh]
    shade = "texture" if mesh == "terrain" else rng.choice(["rgba", "lit"])
    return dict(kind=kind, mesh=mesh, size=size, images=images, width=side,
                height=max(60, int(side * rng.uniform(0.6, 1.1))), layers=rng.choice([1, 2, 3, 3, 3]),
                shade=shade, graph=rng.random() < 0.3, deterministic=rng.random() < 0.2)
  mesh = rng.choice(["soup", "sphere"])
  size = _log(rng, 200, 100000) if mesh == "soup" else _log(rng, 3, 71)
  width = _log(rng, 64, 1400)
  return dict(kind=kind, mesh=mesh, size=size, width=width,
              height=max(48, int(width * rng.uniform(0.5, 1.2))),
              layers=1 if kind == "preview" else rng.choice([1, 2, 3, 4]))


# ----------------------------------------------------------------- inputs
def _generator(seed):
  return torch.Generator(device="cuda").manual_seed(int(seed))


def _mesh(kind, size, gen, seed):
  """(vertices [V, 3], triangles [T, 3], uv or None) of one mesh on the GPU."""
  dev = gen.device
  if kind == "sphere":
    v, f = workloads.icosphere(size)
    v = torch.tensor(v, dtype=torch.float32, device=dev)
    v = v * (1.0 + 0.02 * torch.randn(len(v), 1, generator=gen, device=dev))
    return v, torch.tensor(f, device=dev), None
  if kind == "soup":
    c = torch.rand(size, 1, 3, generator=gen, device=dev) * 2.0 - 1.0
    d = torch.randn(size, 3, 3, generator=gen, device=dev)
    d = d / d.norm(dim=-1, keepdim=True)
    r = torch.exp(-4.0 + 0.7 * torch.randn(size, 3, 1, generator=gen, device=dev))
    return ((c + d * r).reshape(-1, 3),
            torch.arange(3 * size, dtype=torch.int32, device=dev).view(-1, 3), None)
  h = torch.tensor(workloads.value_noise(size, seed), dtype=torch.float32, device=dev)
  g = torch.linspace(-1.0, 1.0, size, device=dev)
  v = torch.stack([g[None, :].expand(size, size), h, -g[:, None].expand(size, size)], -1)
  w = torch.linspace(0.0, 1.0, size, device=dev)
  uv = torch.stack([w[None, :].expand(size, size), w[:, None].expand(size, size)], -1)
  return (v.reshape(-1, 3), torch.tensor(workloads.grid_triangles(size), device=dev),
          uv.reshape(-1, 2).contiguous())


def _cameras(sizes, seed, mesh="sphere"):
  terrain = mesh == "terrain"
  eyes = workloads.sphere_eyes(len(sizes), seed=seed + 1, radius=2.2 if terrain else 3.0,
                               upper_only=terrain)
  cams = [workloads.camera_matrix(e, w, h) for e, (w, h) in zip(eyes, sizes)]
  return torch.tensor(np.stack(cams), device="cuda")


def _layout(case):
  """[(mesh kind, size), ...] and [(width, height), ...] of a case's images."""
  if case["kind"] != "ragged":
    n = case.get("images", 1)
    return [(case["mesh"], case["size"])] * n, [(case["width"], case["height"])] * n
  rng = np.random.default_rng(case["layout"])
  n = case["images"]
  counts = np.clip(rng.lognormal(math.log(case["median"]), 1.2, n), 500, case["most"]).astype(int)
  meshes = [("soup", int(c)) if k else ("sphere", workloads.frequency_for_triangles(c))
            for k, c in zip(rng.integers(0, 2, n), counts)]
  top = case["sizes"]
  if not case["odd"]:
    return meshes, [(int(s), int(s)) for s in rng.choice([top // 4, top // 2, top], n)]
  return meshes, [(int(w), int(h)) for w, h in rng.integers(max(top // 6, 16), top + 1, (n, 2))]


def _scene(case, seed):
  """Packed inputs of a case's images, as a program holds them on the GPU."""
  gen = _generator(seed)
  meshes, sizes = _layout(case)
  if case["kind"] == "ragged":
    parts = [_mesh(k, s, gen, seed) for k, s in meshes]
  else:  # one mesh, every image its own copy with its own camera
    parts = [_mesh(*meshes[0], gen, seed)] * len(meshes)
  v = torch.cat([p[0] for p in parts])
  pixels = sum(w * h for w, h in sizes)
  s = dict(vertices=v, triangles=[p[1] for p in parts], counts=[len(p[0]) for p in parts],
           sizes=sizes, cameras=_cameras(sizes, seed, case.get("mesh", "sphere")))
  shade = case.get("shade", "rgba")
  if shade == "texture":
    s["uv"] = torch.cat([p[2] for p in parts])
    s["texture"] = torch.randint(0, 256, (1024, 1024, 4), generator=gen,
                                 device=gen.device).float() / 255.0
  else:
    s["colors"] = torch.rand(len(v), 3 if shade == "lit" else 4, generator=gen,
                             device=gen.device)
    if shade == "rgba":
      s["colors"][:, 3] = 1.0
  if case["kind"] in ("fit", "ragged", "single", "over"):
    s["target"] = torch.rand(pixels, 4, generator=gen, device=gen.device)
    s["target"][:, 3] = 1.0
  return s


def _texture_inputs(case, seed):
  """Texture coordinates as a render gives them: rows of neighbouring
  pixels, a tenth of them background (all zero, with a zero gradient)."""
  gen = _generator(seed)
  n = case["points"]
  cols = max(1, int(math.sqrt(n)))
  i = torch.arange(n, device=gen.device)
  uv = torch.stack([(i % cols).float() / cols, (i // cols).float() / (n // cols + 1)], -1)
  uv = uv + 0.002 * torch.randn(n, 2, generator=gen, device=gen.device)
  hidden = torch.rand(n // 64 + 1, generator=gen, device=gen.device)[i // 64] < 0.1
  uv = torch.where(hidden[:, None], torch.zeros_like(uv), uv)
  tex = torch.rand(case["height"], case["width"], case["channels"], generator=gen,
                   device=gen.device)
  g = torch.randn(n, case["channels"], generator=gen, device=gen.device)
  return uv, tex, torch.where(hidden[:, None], torch.zeros_like(g), g)


def _normal_inputs(case, seed):
  gen = _generator(seed)
  v, f, _ = _mesh("terrain", case["size"], gen, seed)
  v = v + (0.2 / case["size"]) * torch.randn(v.shape, generator=gen, device=gen.device)
  return v, f, torch.randn(v.shape, generator=gen, device=gen.device)


def _lit(a):
  return shaders.point_light(a["rgb"], a["normals"], a["pos"], LIGHT, alpha=True)


def _batch_step(case, s):
  """A fitting step of a BatchRenderer: loss, image and gradients."""
  r = s["renderer"]
  v = s["vertices"]
  shade = case.get("shade", "rgba")
  if shade == "texture":
    params = [v, s["texture"]]
    out = r.render(v, {"uv": s["uv"]}, s["cameras"],
                   lambda a: shaders.texture_map(a["uv"], s["texture"],
                                                 deterministic=case["deterministic"]))
  elif shade == "lit":
    params = [v, s["colors"]]
    out = r.render(v, {"rgb": s["colors"], "normals": r.vertex_normals(v), "pos": v},
                   s["cameras"], _lit)
  else:
    params = [v, s["colors"]]
    out = r.render(v, {"rgba": s["colors"]}, s["cameras"], lambda a: a["rgba"])
  loss, g = losses.squared_error_seed(out, s["target"])
  d_v, d_c = torch.autograd.grad(out, params, grad_outputs=g)
  return [out.detach(), loss, d_v, d_c]


def prepare(case, seed):
  kind = case["kind"]
  if kind == "texture":
    uv, tex, g = _texture_inputs(case, seed)
    return dict(case=case, uv=uv.requires_grad_(), texture=tex.requires_grad_(), g=g)
  if kind == "normals":
    v, f, g = _normal_inputs(case, seed)
    return dict(case=case, vertices=v.requires_grad_(), triangles=f, g=g)
  s = _scene(case, seed)
  s["case"] = case
  if kind in ("fit", "ragged", "single", "over"):
    s["vertices"].requires_grad_()
    s["texture" if "texture" in s else "colors"].requires_grad_()
  if kind in ("fit", "ragged"):
    s["renderer"] = batch_lib.BatchRenderer(s["triangles"], s["counts"], s["sizes"],
                                            case["layers"],
                                            deterministic_gradients=case["deterministic"])
    if case.get("graph"):
      stream = torch.cuda.Stream()
      stream.wait_stream(torch.cuda.current_stream())
      with torch.cuda.stream(stream):
        for _ in range(2):
          _batch_step(case, s)
      torch.cuda.current_stream().wait_stream(stream)
      s["graph"] = torch.cuda.CUDAGraph()
      with torch.cuda.graph(s["graph"]):
        s["outputs"] = _batch_step(case, s)
  return s


def run(s):
  case = s["case"]
  kind = case["kind"]
  if kind == "texture":
    out = shaders.texture_map(s["uv"], s["texture"])
    return [out.detach(), *torch.autograd.grad(out, [s["uv"], s["texture"]], grad_outputs=s["g"])]
  if kind == "normals":
    out = mesh_lib.compute_vertex_normals(s["vertices"], s["triangles"])
    return [out.detach(), *torch.autograd.grad(out, [s["vertices"]], grad_outputs=s["g"])]
  if kind in ("fit", "ragged"):
    if "graph" in s:
      s["graph"].replay()
      return s["outputs"]
    return _batch_step(case, s)
  v, tri, cam = s["vertices"], s["triangles"][0], s["cameras"][0]
  w, h = s["sizes"][0]
  if kind == "raster":
    f = rasterize.rasterize_triangles(v, tri, cam, w, h, case["layers"],
                                      constants.FaceCullingMode.NONE)
    return [f.triangle_id, f.z_buffer, f.barycentrics]
  attrs = {"rgba": s["colors"]}
  if kind == "preview":
    with torch.no_grad():
      return [render.render_triangles(v, attrs, tri, cam, w, h, lambda a: a["rgba"],
                                      case["layers"])]
  over = kind == "over"
  out = render.render_triangles(
      v, attrs, tri, cam, w, h, lambda a: a["rgba"], case["layers"],
      compositing_mode=(constants.CompositingMode.OVER if over
                        else constants.CompositingMode.SPLAT_OVER),
      compute_diff_barys=over)
  loss = losses.squared_error(out.view(-1, 4), s["target"], 1.0 / out.numel())
  d_v, d_c = torch.autograd.grad(loss, [v, s["colors"]])
  return [out.detach(), loss.detach(), d_v, d_c]


def work(case):
  """Each input read once and each output written once; the operations of the
  transform, the triangle setup and, per covered sample (a third of the
  pixels), the depth test and the splat's nine taps."""
  kind = case["kind"]
  if kind == "texture":
    n, c = case["points"], case["channels"]
    texels = case["width"] * case["height"]
    return dict(bytes=4 * (n * (2 + c + c + 2) + 2 * texels * c), flops=n * (24 + 28 * c))
  if kind == "normals":
    v, t = case["size"]**2, 2 * (case["size"] - 1)**2
    return dict(bytes=12 * (4 * v + t), flops=40 * t + 60 * v)
  meshes, sizes = _layout(case)
  counts = [(10 * s * s + 2, 20 * s * s) if k == "sphere" else
            (3 * s, s) if k == "soup" else (s * s, 2 * (s - 1)**2) for k, s in meshes]
  v, t = sum(c[0] for c in counts), sum(c[1] for c in counts)
  p = sum(w * h for w, h in sizes)
  covered = p // 3
  back = kind not in ("preview", "raster")
  if kind == "raster":
    return dict(bytes=12 * v + 12 * t + 20 * case["layers"] * p, flops=28 * v + 60 * t +
                40 * covered)
  extra = 2 * 4 * 1024 * 1024 * 4 if case.get("shade") == "texture" else 0
  attr = {"texture": 2, "lit": 3}.get(case.get("shade"), 4)
  per_vertex = (12 + 4 * attr) * (2 if back else 1)
  return dict(bytes=per_vertex * v + 12 * t + 16 * p * (2 if back else 1) + extra,
              flops=(28 * v + 60 * t + 40 * covered + 9 * 10 * covered) * (3 if back else 1))


# ------------------------------------------------------- 64-bit restatement
def _fma(a, b, c):
  return (a.double() * b.double() + c.double()).float()


def _exact_raster(clip, tri, w, h, layers, both_faces):
  """The samples of one image: (layer, pixel, triangle) indices, float32 and
  64-bit barycentrics and the float32 depth, in the rasterizer's fixed-point
  and float32 arithmetic, which defines which triangle a sample shows."""
  p = clip[tri.long()]  # [T, 3, 4]
  fx = (p * 65536.0).double().trunc().long()
  x, y, q = fx[..., 0].unbind(1), fx[..., 1].unbind(1), fx[..., 3].unbind(1)
  m = []
  for i, j in ((1, 2), (2, 0), (0, 1)):
    m.append((y[i] * q[j] - q[i] * y[j], x[j] * q[i] - q[j] * x[i], x[i] * y[j] - y[i] * x[j]))
  if both_faces:
    det = (x[0] * m[0][0] + x[1] * m[1][0] + x[2] * m[2][0]).float()
    sign = torch.copysign(torch.ones_like(det), det)
    m = [tuple((c.float() * sign).double().trunc().long() for c in r) for r in m]
  px = 0.5 * (p[..., 0] / p[..., 3] + 1.0) * w
  py = 0.5 * (p[..., 1] / p[..., 3] + 1.0) * h
  lo = torch.stack([px.amin(1).floor(), py.amin(1).floor()], 1).clamp(min=0).long()
  hi = torch.stack([px.amax(1).ceil().clamp(max=w), py.amax(1).ceil().clamp(max=h)], 1).long()
  span = (hi - lo).clamp(min=0)
  n = span[:, 0] * span[:, 1]

  def center(i, size):
    s = torch.tensor(2.0, device=i.device) / float(size)
    c = _fma(s, i.float() + 0.5, torch.tensor(-1.0, device=i.device))
    return (c * 65536.0).double().trunc().long()

  keep = []
  first, most = 0, 1 << 25
  ends = torch.cumsum(n, 0).cpu()
  while first < len(n):  # chunks of triangles with a bounded candidate count
    base = int(ends[first - 1]) if first else 0
    last = max(first + 1, int(torch.searchsorted(ends, base + most, right=True)))
    part = torch.arange(first, last, device=clip.device)
    t = torch.repeat_interleave(part, n[first:last])
    r = torch.arange(len(t), device=clip.device) - (torch.cumsum(n, 0) - n)[t] + base
    cx, cy = lo[t, 0] + r % span[t, 0], lo[t, 1] + r // span[t, 0]
    gx, gy = center(cx, w), center(cy, h)
    e = [m[i][0][t] * gx + m[i][1][t] * gy + m[i][2][t] * 65536 for i in range(3)]
    inside = (e[0] >= 0) & (e[1] >= 0) & (e[2] >= 0) & ((e[0] + e[1] + e[2]) > 0)
    keep.append([a[inside] for a in (t, cy * w + cx, *e)])
    first = last
  t, pix, e0, e1, e2 = (torch.cat(a) for a in zip(*keep))
  total = (e0 + e1 + e2).float()
  b = torch.stack([e0.float() / total, e1.float() / total, e2.float() / total], 1)
  c = p[t]

  def dot(k):
    return _fma(b[:, 2], c[:, 2, k], _fma(b[:, 0], c[:, 0, k], b[:, 1] * c[:, 1, k]))

  z = dot(2) / dot(3)
  d = ((z.double() + 1.0) * 2147483647.0).trunc().long()
  ok = (z >= -1.0) & (z <= 1.0) & (d < 4294967294)
  t, pix, b, d = t[ok], pix[ok], b[ok], d[ok]
  e = torch.stack([e0, e1, e2], 1)[ok].double()
  order = torch.argsort(t, stable=True)
  order = order[torch.argsort(d[order], stable=True)]
  order = order[torch.argsort(pix[order], stable=True)]
  ps = pix[order]
  start = torch.searchsorted(ps, ps)
  layer = torch.arange(len(ps), device=ps.device) - start
  order, layer = order[layer < layers], layer[layer < layers]
  depth = (d[order].double() / 2147483647.0 - 1.0)
  e = e[order]
  return layer, pix[order], t[order], b[order], e / e.sum(1, keepdim=True), depth


def _exact_clip32(v, cam):
  m, x = cam, v
  rows = [((m[i, 0] * x[:, 0] + m[i, 1] * x[:, 1]) + m[i, 2] * x[:, 2]) + m[i, 3]
          for i in range(4)]
  return torch.stack(rows, 1)


def _unit(x):
  return x * torch.rsqrt((x * x).sum(-1, keepdim=True) + 1e-12)


def _exact_normals(v, tri):
  a, b, c = (v[tri[:, i].long()] for i in range(3))
  n = torch.linalg.cross(b - a, c - a)
  s = torch.zeros_like(v)
  for i in range(3):
    s = s.index_add(0, tri[:, i].long(), n)
  return _unit(s)


def _exact_texture(uv, tex):
  h, w, c = tex.shape
  size = torch.tensor([w, h], device=uv.device)
  loc = uv * size - 0.5
  # The texel and its clamping follow the float32 location.
  loc32 = (uv.detach().float() * size.float() - 0.5) + 1.0
  f = torch.minimum(loc32.floor().clamp(min=0.0), size.float())
  t = (loc + 1.0) - f.double()
  t = torch.minimum(torch.maximum(t, torch.zeros_like(t)), torch.ones_like(t))
  i0 = (f - 1.0).clamp(min=0.0).long()
  i1 = torch.minimum(f, size.float() - 1.0).long()
  flat = tex.reshape(-1, c)
  out = 0.0
  for ix, wx in ((i0[:, 0], 1.0 - t[:, 0]), (i1[:, 0], t[:, 0])):
    for iy, wy in ((i0[:, 1], 1.0 - t[:, 1]), (i1[:, 1], t[:, 1])):
      out = out + flat[iy * w + ix] * (wx * wy)[:, None]
  return out


def _exact_light(rgb, n, pos):
  to = torch.tensor(LIGHT, dtype=torch.float64, device=pos.device) - pos
  nol = (n * _unit(to)).sum(-1, keepdim=True).clamp(0.0, 1.0)
  dist = torch.linalg.vector_norm(to, dim=-1, keepdim=True)
  out = rgb * (0.3 + 1.4 * nol) / (1.0 + 0.7 * dist + 1.8 * dist * dist)
  return torch.cat([out, torch.ones_like(out[:, :1])], 1)


def _exact_splat(clip, clip32, vid, b, b32, layer, pix, color, w, h, layers):
  """Splats one image's shaded samples, normalizes and composites."""
  lerp = lambda a, k: (a[:, 0] * k[:, :1] + a[:, 1] * k[:, 1:2]) + a[:, 2] * k[:, 2:]
  c = lerp(clip[vid], b)
  size = torch.tensor([w, h], dtype=torch.float64, device=clip.device)
  xy = (c[:, :2] / c[:, 3:] + 1.0) * size * 0.5
  c32 = lerp(clip32[vid], b32)
  z = torch.ones(layers, h * w, device=clip.device)
  z[layer, pix] = (c32[:, 2] / c32[:, 3] + 1.0) * 0.5
  px, py = pix % w, pix // w
  g = torch.tensor([-1.0, 0.0, 1.0], dtype=torch.float64)
  coef = float(1.05 / torch.exp(-2.0 * g * g).sum()**2)
  acc = torch.zeros(3 * h * w, color.shape[1] + 1, dtype=torch.float64, device=clip.device)
  splat = torch.cat([color, torch.ones_like(color[:, :1])], 1)
  for u in (-1, 0, 1):
    for v in (-1, 0, 1):
      x, y = px + u, py + v
      on = (x >= 0) & (y >= 0) & (x < w) & (y < h)
      dst = (y * w + x)[on]
      src, l = pix[on], layer[on]
      near = (z[:, src] - z[0, dst]).abs()
      far = (z[:, dst] - z[0, src]).abs()
      cm, ci = near.min(0)
      tm, ti = far.min(0)
      ci = (near == cm).int().argmax(0)
      ti = (far == tm).int().argmax(0)
      s = torch.where(tm < cm, -ti, ci)
      k = torch.where(s > l, 0, torch.where(s == l, 1, 2))
      off = (xy[on].detach().floor() + 0.5) - xy[on] + torch.tensor(
          [u, v], dtype=torch.float64, device=clip.device)
      wgt = coef * torch.exp(-2.0 * (off * off).sum(1, keepdim=True))
      acc = acc.index_add(0, k * (h * w) + dst, wgt * splat[on])
  acc = acc.view(3, h * w, -1)
  total = acc[..., -1:] - 1.0
  n = acc[..., :-1] / (torch.maximum(total, torch.zeros_like(total)) + 1.0)
  a = n[..., -1:]
  return n[0] + (1.0 - a[0]) * (n[1] + (1.0 - a[1]) * n[2])


def _exact_diff_barys(clip, vid, pix, w, h):
  p = clip[vid]
  mat = torch.stack([p[..., 0], p[..., 1], p[..., 3]], 1)  # rows x, y, w
  at = torch.stack([(2.0 * (pix % w) + 1.0) / w - 1.0, (2.0 * (pix // w) + 1.0) / h - 1.0,
                    torch.ones_like(pix)], 1).double()
  cols = mat.unbind(2)
  u = torch.stack([(torch.linalg.cross(cols[(i + 1) % 3], cols[(i + 2) % 3]) * at).sum(1)
                   for i in range(3)], 1)
  return u / u.sum(1, keepdim=True)


def _exact_image(case, s, first, i, v, attr, tex):
  """One image's [H W, C] in 64 bits from the packed 64-bit parameters."""
  w, h = s["sizes"][i]
  rows = slice(first, first + s["counts"][i])
  tri = s["triangles"][i]
  cam = s["cameras"][i]
  clip32 = _exact_clip32(s["vertices"][rows], cam)
  clip = torch.cat([v, torch.ones_like(v[:, :1])], 1) @ cam.double().t()
  layer, pix, t, b32, b, _ = _exact_raster(clip32, tri, w, h, case["layers"], False)
  vid = tri[t].long()
  if case["kind"] == "over":
    b = _exact_diff_barys(clip, vid, pix, w, h)
  lerp = lambda a: (a[vid] * b[:, :, None]).sum(1)
  shade = case.get("shade", "rgba")
  if shade == "texture":
    color = _exact_texture(lerp(attr), tex)
  elif shade == "lit":
    color = _exact_light(lerp(attr), lerp(_exact_normals(v, tri)), lerp(v))
  else:
    color = lerp(attr)
  if case["kind"] == "over":
    out = torch.zeros(h * w, color.shape[1], dtype=torch.float64, device=v.device)
    for l in reversed(range(case["layers"])):
      on = layer == l
      full = torch.zeros_like(out).index_add(0, pix[on], color[on])
      out = full + (1.0 - full[:, -1:]) * out if l < case["layers"] - 1 else full
    return out
  return _exact_splat(clip, clip32, vid, b, b32, layer, pix, color, w, h, case["layers"])


def exact(case, seed):
  kind = case["kind"]
  if kind == "texture":
    uv, tex, g = _texture_inputs(case, seed)
    uv, tex = uv.double().requires_grad_(), tex.double().requires_grad_()
    out = _exact_texture(uv, tex)
    return [out.detach(), *torch.autograd.grad(out, [uv, tex], grad_outputs=g.double())]
  if kind == "normals":
    v, f, g = _normal_inputs(case, seed)
    v = v.double().requires_grad_()
    out = _exact_normals(v, f)
    return [out.detach(), *torch.autograd.grad(out, [v], grad_outputs=g.double())]
  s = _scene(case, seed)
  if kind == "raster":
    w, h = s["sizes"][0]
    tri = s["triangles"][0]
    clip = _exact_clip32(s["vertices"], s["cameras"][0])
    layer, pix, t, _, b, depth = _exact_raster(clip, tri, w, h, case["layers"], True)
    z = torch.ones(case["layers"], h * w, dtype=torch.float64, device=clip.device)
    z[layer, pix] = depth
    bary = torch.zeros(case["layers"], h * w, 3, dtype=torch.float64, device=clip.device)
    bary[layer, pix] = b
    return [None, z.view(-1, h, w), bary.view(-1, h, w, 3)]
  # Image by image, each with its own gradients: the images are independent.
  grad = kind != "preview"
  tex = s["texture"].double().requires_grad_(grad) if "texture" in s else None
  images, d_v, d_c, loss = [], [], [], 0.0
  d_tex = torch.zeros_like(tex) if tex is not None else None
  row = pixel = 0
  for i, (w, h) in enumerate(s["sizes"]):
    rows = slice(row, row + s["counts"][i])
    v = s["vertices"][rows].double().requires_grad_(grad)
    attr = (s["uv"] if tex is not None else s["colors"])[rows].double().requires_grad_(
        grad and tex is None)
    with torch.set_grad_enabled(grad):
      out = _exact_image(case, s, row, i, v, attr, tex)
    images.append(out.detach())
    if grad:
      diff = out.detach() - s["target"][pixel:pixel + h * w].double()
      scale = 1.0 if kind in ("fit", "ragged") else 1.0 / out.numel()
      loss = loss + scale * (diff * diff).sum()
      gv, gc = torch.autograd.grad(out, [v, tex if tex is not None else attr],
                                   grad_outputs=2.0 * scale * diff)
      d_v.append(gv)
      if tex is not None:
        d_tex = d_tex + gc
      else:
        d_c.append(gc)
    row += s["counts"][i]
    pixel += h * w
  if kind in ("single", "preview", "over"):
    images = [images[0].view(h, w, -1)]
  if not grad:
    return images
  return [torch.cat(images) if kind in ("fit", "ragged") else images[0], loss, torch.cat(d_v),
          d_tex if tex is not None else torch.cat(d_c)]
