"""Main entry point (diffren/jax/render.py:28-140).

``render_triangles`` keeps the reference's signature and behaviour:
rasterize, interpolate the attribute dict, run the user's deferred shader
(any differentiable torch function of a dict of [H, W, K] buffers) on each
layer, then splat+composite (SPLAT_OVER), composite (OVER) or return the
layers (NONE). Gradients reach vertices, attributes and camera through the
CUDA VJP kernels; the shader's own VJP is torch autograd.

A leading batch dimension on vertices / camera (/ attributes / triangles)
renders all images in one launch per kernel, the batched counterpart of
jax.vmap(render_triangles).
"""
from typing import Callable, Dict

import torch

from . import constants
from . import interpolate
from . import kernels
from . import rasterize
from . import splat


class _Slices(torch.autograd.Function):
  """The slices of a tensor along its first dimension, as tensors over the
  same memory. Their gradients come back as the buffer they share (what
  stacking the shaded slices gives, when the shader returns its input) or
  stacked in one pass, where a select per slice fills and adds a whole tensor
  each. Plain tensors rather than views, so that a shader may still write to
  its input; with several attributes (`views`) it may not, as with the views
  of torch.split."""

  @staticmethod
  def forward(ctx, t, views):
    ctx.shape, ctx.stride = t.shape, t.stride()
    ctx.set_materialize_grads(False)
    if views:
      return t.unbind(0)
    step = t.stride(0)
    return tuple(
        torch.empty(0, dtype=t.dtype, device=t.device).set_(
            t.untyped_storage(), t.storage_offset() + i * step, t.shape[1:], t.stride()[1:])
        for i in range(t.shape[0]))

  @staticmethod
  def jvp(ctx, d, _):
    return tuple(d.unbind(0))

  @staticmethod
  def backward(ctx, *grads):
    like = next((g for g in grads if g is not None), None)
    if like is None:
      return None, None
    # (a gradient that is itself differentiated keeps its graph: stacked)
    if not torch.is_grad_enabled() and all(g is not None and g.is_contiguous() for g in grads):
      n = like.numel()
      whole = kernels._one_buffer(grads, ctx.shape, (n, *like.stride()),
                                  [i * n for i in range(len(grads))])
      if whole is not None:
        return whole, None
    return torch.stack([torch.zeros_like(like) if g is None else g for g in grads]), None


def _shade_layers(shading_function, interpolated, num_layers, batched):
  """vmap(shading_function) over layers (and images), as render.py:128."""
  first = next(iter(interpolated.values()))
  lead = first.shape[:2] if batched else first.shape[:1]
  n = lead.numel()
  slices = {}
  for k, v in interpolated.items():
    flat = v.flatten(0, 1) if batched else v
    if torch.is_grad_enabled() and v.requires_grad:
      slices[k] = _Slices.apply(flat, len(interpolated) > 1)
    else:
      slices[k] = [flat[i] for i in range(n)]
  outs = [shading_function({k: v[i] for k, v in slices.items()}) for i in range(n)]
  if outs and not torch.is_grad_enabled():
    for k, v in slices.items():
      if all(o is s for o, s in zip(outs, v)):
        return interpolated[k]  # the shader returned its input: nothing to stack
  shaded = torch.stack(outs)
  return shaded.view(*lead, *shaded.shape[1:]) if batched else shaded


def _render_fused(geom, attributes, shading_function, num_layers, face_culling_mode,
                  depth_semantics, return_accum_buffers, recompute_raster=False,
                  deterministic_gradients=False):
  """SPLAT_OVER through the rasterizer that interpolates the attributes and
  the splat positions in its epilogue; None when the attributes exceed its
  channel limit."""
  keys = list(attributes.keys())
  parts = []
  for k in keys:
    a = torch.as_tensor(attributes[k], device=geom.clip.device)
    a = a.float() if not a.is_floating_point() or a.dtype != torch.float32 else a
    if geom.batched:
      a = (a.expand(geom.B, *a.shape) if a.dim() == 2 else a).reshape(-1, a.shape[-1])
    parts.append(a)
  widths = [p.shape[1] for p in parts]
  if sum(widths) > kernels._lib.DR_MAX_CHANNELS:
    return None
  cat = kernels.pack_columns(parts).contiguous()
  # Background samples are told by the depth buffer downstream, so their
  # ids and barycentrics need not be written; with a pass-through shader
  # (None) the splat is the only reader of the attributes, so neither are
  # their attributes nor their color gradients.
  passthrough = shading_function is None
  cfg = kernels.raster_config(num_layers, face_culling_mode, int(depth_semantics),
                              flags=kernels._lib.DR_RASTER_FOREGROUND_ONLY |
                              (kernels._lib.DR_RASTER_FOREGROUND_ATTRIBUTES if passthrough
                               else 0))
  interp, vp, ids, z, bary = kernels.rasterize_interpolate_packed(
      cat, geom.clip, geom.triangles_packed, geom.batch, cfg,
      kernels.default_workspace(geom.clip.device), recompute_raster, deterministic_gradients)
  lead = (geom.B,) if geom.batched else ()
  H, W = geom.batch.heights[0], geom.batch.widths[0]
  interp = interp.view(*lead, num_layers, H, W, -1)
  if passthrough:
    shaded = interp
  else:
    interpolated = dict(zip(keys, kernels.split_channels(interp, widths)))
    shaded = _shade_layers(shading_function, interpolated, num_layers, geom.batched)
  colors = splat._shaded_flat(shaded)
  res = kernels.splat_packed(vp, colors, geom.batch, num_layers, return_accum_buffers, z=z,
                             foreground_gradients=passthrough)
  return splat._shape_outputs(res, lead, H, W, colors.shape[1], return_accum_buffers)


def render_triangles(vertices, attributes: Dict[str, torch.Tensor], triangles,
                     camera_matrices, image_width: int, image_height: int,
                     shading_function: Callable[[Dict[str, torch.Tensor]],
                                                torch.Tensor],
                     num_layers: int = 1,
                     face_culling_mode=constants.FaceCullingMode.BACK,
                     compositing_mode=constants.CompositingMode.SPLAT_OVER,
                     return_accum_buffers=False, compute_diff_barys=False,
                     depth_semantics=constants.DepthSemantics.CUDA,
                     recompute_raster=False, deterministic_gradients=False):
  """Rendering with differentiable occlusion using rasterize-then-splat.

  Returns [H, W, C] ([num_layers, H, W, C] for CompositingMode.NONE), with a
  leading batch dimension when the inputs are batched. ``recompute_raster``
  (SPLAT_OVER, beyond the reference's arguments): the backward reruns the
  rasterizer instead of keeping its per-sample triangle ids, barycentrics
  and vertex ids, for memory-tight renders. ``shading_function`` None (also
  beyond the reference's arguments): the single attribute is the color, as
  ``lambda a: a[key]`` gives, and background samples' attributes and color
  gradients, which nothing then reads, are not written.
  ``deterministic_gradients`` (SPLAT_OVER; also beyond the reference): the
  vertex and attribute gradients of the fused pass are summed in fixed
  point, the same bits on every run.

  Raises:
    ValueError: if face_culling_mode is not BACK and compositing_mode is
      SPLAT_OVER (back faces would count as occluding layers).
  """
  if (compositing_mode == constants.CompositingMode.SPLAT_OVER and
      face_culling_mode != constants.FaceCullingMode.BACK):
    raise ValueError("Backface culling must be enabled when using splatting.")
  if shading_function is None and len(attributes) != 1:
    raise ValueError("shading_function=None needs exactly one attribute")
  vertices = torch.as_tensor(vertices)
  triangles = torch.as_tensor(triangles)
  camera = None if camera_matrices is None else torch.as_tensor(camera_matrices)
  rasterize._validate(vertices, triangles, camera, image_width, image_height,
                      num_layers)
  geom = rasterize.Geometry(vertices, triangles, camera, image_width, image_height)
  if (compositing_mode == constants.CompositingMode.SPLAT_OVER and not compute_diff_barys
      and attributes):
    fused = _render_fused(geom, attributes, shading_function, num_layers,
                          face_culling_mode, depth_semantics, return_accum_buffers,
                          recompute_raster, deterministic_gradients)
    if fused is not None:
      return fused
  frame, _ = rasterize.rasterize_geometry(geom, num_layers, face_culling_mode,
                                          depth_semantics, compute_diff_barys)
  interpolated = interpolate.interpolate_vertex_attributes(attributes, frame)
  if shading_function is None:
    shaded = next(iter(interpolated.values()))
  else:
    shaded = _shade_layers(shading_function, interpolated, num_layers, geom.batched)

  if compositing_mode == constants.CompositingMode.SPLAT_OVER:
    return splat.splat_clip(geom.clip, frame, shaded, return_accum_buffers)

  if compositing_mode == constants.CompositingMode.OVER:
    # Foreground mask and composite.over in one kernel.
    C = shaded.shape[-1]
    out = kernels.over_packed(shaded.reshape(-1, C), frame.z_buffer.reshape(-1), geom.batch,
                              num_layers)
    lead = (geom.B,) if geom.batched else ()
    return out.view(*lead, image_height, image_width, C)
  return shaded * frame.foreground_mask
