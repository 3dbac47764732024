"""The work that performance is measured on: what a user's program has this package do each step,
through its public entry points, from the smallest calls to the largest.

frame   real-time tier: refit_bvh, render and the image views of every camera, the loop of a
        vision policy or a sensor simulation (poses already on the device)
path    path-traced tier: refit_bvh, render and one of the two denoisers, HDR and display images out
train   one training step of the learned denoiser (forward, loss, backward, Adam)
conv    one 3 x 3 convolution layer of that network: forward, input gradient or weight gradient

Sizes are those of the package's own scenes (16 x 64 x 64 primitives, 4096 x 128 x 128 meshes with
image-based lighting, 2048 worlds with three uneven cameras, 1024 x 128 x 128 path-traced, two
256 x 256 cameras with four environments, batches of 16 training crops) and odd ones in between.
"""

from __future__ import annotations

import ctypes
from typing import Any

import torch

import mujoco_warp_pbr_gb300 as mjpbr
from mujoco_warp_pbr_gb300 import _lib
from mujoco_warp_pbr_gb300 import kpcn
from mujoco_warp_pbr_gb300 import synthetic
from mujoco_warp_pbr_gb300 import train_kpcn

DEPTH_SCALE = 8.0  # metres that get_depth maps to 1
WEIGHTS = "mujoco_warp_pbr_gb300/weights/kpcn_path.npz"


def listed() -> list[dict[str, Any]]:
  return [
    # the package's smallest configuration: a handful of environments, latency is what counts
    {"name": "frame_primitives_16x64", "kind": "frame", "scene": "primitives", "worlds": 16, "width": 64, "height": 64, "samples": 1},
    # a reinforcement-learning batch with a small camera that no tile divides
    {"name": "frame_primitives_500x84", "kind": "frame", "scene": "primitives", "worlds": 500, "width": 84, "height": 84, "samples": 1},
    # a few environments with a larger, ragged camera: meshes, textures, environment light, mirror floor
    {"name": "frame_meshes_24x200x150", "kind": "frame", "scene": "meshes", "worlds": 24, "width": 200, "height": 150, "samples": 2},
    # the package's headline workload
    {"name": "frame_meshes_4096x128", "kind": "frame", "scene": "meshes", "worlds": 4096, "width": 128, "height": 128, "samples": 2},
    # three cameras of uneven size per world with per-pixel rays (two pinholes and a fisheye)
    {"name": "frame_batched_2048", "kind": "frame", "scene": "batched", "worlds": 2048, "width": 256, "height": 256, "samples": 1},
    # terrain from a height field under primitives
    {"name": "frame_terrain_300x96", "kind": "frame", "scene": "terrain", "worlds": 300, "width": 96, "height": 96, "samples": 1},
    # path-traced preview of a few worlds at an odd size and sample count, a-trous filtered
    {"name": "path_atrous_20x90x61", "kind": "path", "scene": "path", "worlds": 20, "width": 90, "height": 61, "spp": 3, "filter": "atrous"},
    # the path-traced configuration: data generation at two samples per pixel, a-trous filtered
    {"name": "path_atrous_1024x128", "kind": "path", "scene": "path", "worlds": 1024, "width": 128, "height": 128, "spp": 2, "filter": "atrous"},
    # two large cameras and four environments per world, filtered by the network
    {"name": "path_learned_128x2x256", "kind": "path", "scene": "large", "worlds": 128, "width": 256, "height": 256, "spp": 2, "filter": "learned"},
    # a training step at the training script's batch size
    {"name": "train_16x128", "kind": "train", "crops": 16, "res": 128},
    # the decoder's first full-resolution layer, on a chunk of images as inference meets it
    {"name": "conv_forward_256x128", "kind": "conv", "direction": "forward", "images": 256, "height": 128, "width": 128, "c_in": 32, "c_skip": 48, "c_out": 32},
    # the same level's second layer in training, large batch
    {"name": "conv_weight_grad_64x128", "kind": "conv", "direction": "weight_grad", "images": 64, "height": 128, "width": 128, "c_in": 32, "c_skip": 0, "c_out": 32},
  ]


def _between(rng, low: int, high: int) -> int:
  """A whole number between low and high, spread over the logarithm."""
  return int(round(low * (high / low) ** rng.random()))


def draw(rng) -> dict[str, Any]:
  kind = rng.choice(["frame", "frame", "path", "path", "train", "conv"])
  if kind == "frame":
    scene = rng.choice(["primitives", "meshes", "batched", "terrain"])
    if scene == "batched":
      r = _between(rng, 32, 256)
      return {"kind": kind, "scene": scene, "worlds": _between(rng, 4, 2048), "width": r, "height": r, "samples": 1}
    samples = rng.choice([1, 2]) if scene != "meshes" else rng.choice([1, 2, 2])
    width, height = _between(rng, 24, 256), _between(rng, 24, 256)
    most = min(4096, max(8, 4096 * 128 * 128 * 4 // (width * height * samples**2)))
    return {"kind": kind, "scene": scene, "worlds": _between(rng, 4, most), "width": width, "height": height, "samples": samples}
  if kind == "path":
    scene = rng.choice(["path", "large"])
    filt = rng.choice(["atrous", "atrous", "learned"])
    spp = rng.choice([1, 2, 3, 4])
    if filt == "learned":  # sizes the network's tiles cover
      width, height = rng.choice([128, 256]), 64 * _between(rng, 1, 4)
    else:
      width, height = _between(rng, 24, 256), _between(rng, 24, 256)
    cams = 2 if scene == "large" else 1
    most = min(1024, max(4, 1024 * 128 * 128 * 2 // (width * height * spp * cams)))
    return {"kind": kind, "scene": scene, "worlds": _between(rng, 2, most), "width": width, "height": height, "spp": spp, "filter": filt}
  if kind == "train":
    res = rng.choice([128, 128, 256])
    return {"kind": kind, "crops": _between(rng, 4, 64 * 128 * 128 // res**2), "res": res}
  widths = (32, 48, 64, 96)
  level = rng.randrange(4)
  c_in, c_out = widths[level], widths[level]
  c_skip = widths[level + 1] if level < 3 and rng.random() < 0.4 else 0
  width = 128 >> level
  height = (128 // width) * _between(rng, 8, 128 >> level if level < 2 else 32)
  images = _between(rng, 4, 256 << level)
  return {
    "kind": kind, "direction": rng.choice(["forward", "input_grad", "weight_grad"]), "images": images, "height": height, "width": width,
    "c_in": c_in, "c_skip": c_skip, "c_out": c_out,
  }


# ---------------------------------------------------------------- rendering
def _scene(case: dict[str, Any], seed: int) -> synthetic.SyntheticScene:
  n, w, h = case["worlds"], case["width"], case["height"]
  kind = case["scene"]
  if kind == "primitives":
    sc = synthetic.primitive_scene(seed=seed, nworld=n, res=w)
  elif kind == "meshes":
    sc = synthetic.mesh_ibl_scene(seed=seed, nworld=n, res=w)
  elif kind == "batched":
    return synthetic.batched_scene(seed=seed, nworld=n, res=(max(8, w // 4), max(8, w // 2), w))
  elif kind == "terrain":
    sc = synthetic.hfield_scene(seed=seed, nworld=n, res=w)
  elif kind == "path":
    sc = synthetic.path_scene(seed=seed, nworld=n, res=w, spp=case["spp"])
  else:
    sc = synthetic.large_path_scene(seed=seed, nworld=n, res=w)
    sc.options["path_samples"] = case["spp"]
  sc.options["cam_res"] = [(w, h)] * sc.mjm.ncam
  return sc


def _prepare_render(case: dict[str, Any], seed: int) -> dict[str, Any]:
  sc = _scene(case, seed)
  opts = dict(sc.options)
  if case["kind"] == "path":
    opts.update({"denoise": True, "render_hdr": True})
  else:
    opts["samples_per_pixel"] = case["samples"]
  m = mjpbr.put_model(sc.mjm)
  d = mjpbr.put_data(sc.mjm, sc.mjd, nworld=sc.nworld)
  rc = mjpbr.create_render_context(sc.mjm, sc.nworld, data=sc.mjd, **opts)
  synthetic.apply_per_world(sc, m, rc)
  images = []
  for w, h in rc.base.cam_res:
    shape = (sc.nworld, h, w)
    views = {"rgb": torch.zeros((*shape, 3), device=rc.device)}
    if case["kind"] == "path":
      views["hdr"] = torch.zeros((*shape, 3), device=rc.device)
    else:
      views["depth"] = torch.zeros(shape, device=rc.device)
      views["seg"] = torch.zeros((*shape, 2), dtype=torch.int32, device=rc.device)
    images.append(views)
  net = kpcn.KPCN.load(WEIGHTS) if case.get("filter") == "learned" else None
  return {"m": m, "d": d, "rc": rc, "images": images, "net": net, "seed": seed & 0xFFFF}


def _run_render(s: dict[str, Any]) -> list[dict[str, torch.Tensor]]:
  m, d, rc = s["m"], s["d"], s["rc"]
  mjpbr.refit_bvh(m, d, rc)
  if s["net"] is not None:
    mjpbr.render(m, d, rc, seed=s["seed"], denoise=False)
    s["net"].denoise(m, d, rc)
  else:
    mjpbr.render(m, d, rc, seed=s["seed"])
  for cam, views in enumerate(s["images"]):
    mjpbr.get_rgb(rc, cam, views["rgb"])
    if "hdr" in views:
      mjpbr.get_hdr(rc, cam, views["hdr"])
    if "depth" in views:
      mjpbr.get_depth(rc, cam, DEPTH_SCALE, views["depth"])
      mjpbr.get_segmentation(rc, cam, views["seg"])
  return s["images"]


def _pixels(case: dict[str, Any]) -> int:
  w, h, n = case["width"], case["height"], case["worlds"]
  if case["scene"] == "batched":
    return n * sum(r * r for r in (max(8, w // 4), max(8, w // 2), w))
  return n * w * h * (2 if case["scene"] == "large" else 1)


# ---------------------------------------------------------------- training
def _prepare_train(case: dict[str, Any], seed: int) -> dict[str, Any]:
  x0, radiance, target, _, _ = train_kpcn.make_dataset(case["crops"], case["crops"], case["res"], target_spp=64, seed0=seed)
  return {"net": kpcn.KPCN.load(WEIGHTS), "x0": x0, "radiance": radiance, "target": target}


def _run_train(s: dict[str, Any]) -> dict[str, Any]:
  sums = s["net"].train_step(s["x0"], s["radiance"], s["target"], 3.0e-4)
  layers = s["net"].layers
  return {
    "loss": sums, "w": [l.w for l in layers.values()], "b": [l.b for l in layers.values()],
    "grad_w": [l.mw for l in layers.values()], "grad_b": [l.mb for l in layers.values()],
  }


# ---------------------------------------------------------------- convolution layers
def _conv_inputs(case: dict[str, Any], seed: int) -> dict[str, torch.Tensor | None]:
  """Activations after a ReLU, He-scaled weights, small biases; gradients centred on zero."""
  n, h, w, c1, c2, co = (case[k] for k in ("images", "height", "width", "c_in", "c_skip", "c_out"))
  g = torch.Generator(device="cuda").manual_seed(seed)

  def normal(*shape, scale=1.0):
    return (torch.randn(shape, generator=g, device="cuda") * scale).to(torch.bfloat16)

  x = normal(n, h, w, c1).relu_()
  skip = normal(n, h, w, c2).relu_() if c2 else None
  weight = normal(co, 9, c1 + c2, scale=(2.0 / (9 * (c1 + c2))) ** 0.5)
  bias = torch.randn(co, generator=g, device="cuda") * 0.1
  grad = normal(n, h, w, co, scale=1.0e-2) if case["direction"] != "forward" else None
  return {"x": x, "skip": skip, "weight": weight, "bias": bias, "grad": grad}


def _ptr(t: torch.Tensor | None) -> int | None:
  return t.data_ptr() if t is not None else None


def _prepare_conv(case: dict[str, Any], seed: int) -> dict[str, Any]:
  n, h, w, c1, c2, co = (case[k] for k in ("images", "height", "width", "c_in", "c_skip", "c_out"))
  s: dict[str, Any] = {"direction": case["direction"], **_conv_inputs(case, seed)}
  s["error"] = torch.zeros(1, dtype=torch.int32, device="cuda")
  if case["direction"] == "forward":
    s["out"] = torch.zeros((n, h, w, co), dtype=torch.bfloat16, device="cuda")
    s["call"] = _lib.Conv(
      in_=_ptr(s["x"]), in2=_ptr(s["skip"]), weight=_ptr(s["weight"]), bias=_ptr(s["bias"]), out=_ptr(s["out"]), out_f32=None, mask=None,
      error_word=_ptr(s["error"]), nimg=n, height=h, width=w, c_in=c1, c_in2=c2, c_out=co, relu=1, in2_full=1,
    )
  elif case["direction"] == "input_grad":
    # a layer fed by one tensor masks with that tensor's ReLU; a concatenated one leaves FP32 for the split
    s["flipped"] = s["weight"].flip(1).permute(2, 1, 0).contiguous()
    s["out"] = torch.zeros((n, h, w, c1 + c2), dtype=torch.float32 if c2 else torch.bfloat16, device="cuda")
    s["call"] = _lib.Conv(
      in_=_ptr(s["grad"]), in2=None, weight=_ptr(s["flipped"]), bias=None, out=None if c2 else _ptr(s["out"]),
      out_f32=_ptr(s["out"]) if c2 else None, mask=None if c2 else _ptr(s["x"]), error_word=_ptr(s["error"]), nimg=n, height=h, width=w,
      c_in=co, c_in2=0, c_out=c1 + c2, relu=0,
    )
  else:
    s["out"] = {"weight": torch.zeros((co, 9, c1 + c2), device="cuda"), "bias": torch.zeros(co, device="cuda")}
    s["call"] = _lib.ConvGrad(
      in_=_ptr(s["x"]), in2=_ptr(s["skip"]), grad_out=_ptr(s["grad"]), grad_weight=_ptr(s["out"]["weight"]), grad_bias=_ptr(s["out"]["bias"]),
      error_word=_ptr(s["error"]), nimg=n, height=h, width=w, c_in=c1, c_in2=c2, c_out=co,
      tiles_per_cta=max(8, (n * h * w // 128 + 2047) // 2048), in2_full=1,
    )
  return s


def _run_conv(s: dict[str, Any]) -> Any:
  stream = torch.cuda.current_stream().cuda_stream
  if s["direction"] == "weight_grad":  # the gradients accumulate: a step starts from zero
    s["out"]["weight"].zero_()
    s["out"]["bias"].zero_()
    _lib.call("mjpbr_conv3x3_wgrad_bf16", ctypes.byref(s["call"]), stream)
  else:
    _lib.call("mjpbr_conv3x3_bf16", ctypes.byref(s["call"]), stream)
  return s["out"]


def _shifted(x: torch.Tensor, tap: int) -> torch.Tensor:
  """x (n, h, w, c) as the 3 x 3 tap `tap` reads it: shifted, zero outside the image."""
  h, w = x.shape[1:3]
  padded = torch.nn.functional.pad(x, (0, 0, 1, 1, 1, 1))
  dy, dx = divmod(tap, 3)
  return padded[:, dy : dy + h, dx : dx + w]


def _conv64(x: torch.Tensor, weight: torch.Tensor) -> torch.Tensor:
  return sum(_shifted(x, tap) @ weight[:, tap].T for tap in range(9))


def exact(case: dict[str, Any], seed: int) -> Any:
  """The convolution layers in 64 bits; images and training steps have no independent 64-bit form
  that is quick enough."""
  if case["kind"] != "conv":
    return None
  s = _conv_inputs(case, seed)
  weight, n, c1, c2, co = s["weight"].double(), case["images"], case["c_in"], case["c_skip"], case["c_out"]
  step = max(1, (1 << 21) // (case["height"] * case["width"]))
  if case["direction"] == "weight_grad":
    gw, gb = torch.zeros((co, 9, c1 + c2), dtype=torch.float64, device="cuda"), torch.zeros(co, dtype=torch.float64, device="cuda")
  parts = []
  for k in range(0, n, step):
    x = s["x"][k : k + step].double()
    if s["skip"] is not None:
      x = torch.cat([x, s["skip"][k : k + step].double()], -1)
    if case["direction"] == "forward":
      parts.append((_conv64(x, weight) + s["bias"].double()).relu_())
      continue
    grad = s["grad"][k : k + step].double()
    if case["direction"] == "input_grad":
      out = _conv64(grad, weight.flip(1).permute(2, 1, 0))
      parts.append(out if c2 else torch.where(x > 0, out, 0.0))
      continue
    flat = grad.reshape(-1, co)
    for tap in range(9):
      gw[:, tap] += flat.T @ _shifted(x, tap).reshape(-1, c1 + c2)
    gb += flat.sum(0)
  if case["direction"] == "weight_grad":
    return {"weight": gw, "bias": gb}
  return torch.cat(parts)


# ---------------------------------------------------------------- the measured calls
def prepare(case: dict[str, Any], seed: int) -> dict[str, Any]:
  make = {"frame": _prepare_render, "path": _prepare_render, "train": _prepare_train, "conv": _prepare_conv}[case["kind"]]
  return {"kind": case["kind"], **make(case, seed)}


def run(state: dict[str, Any]) -> Any:
  return {"frame": _run_render, "path": _run_render, "train": _run_train, "conv": _run_conv}[state["kind"]](state)


def work(case: dict[str, Any]) -> dict[str, float]:
  """Bytes: inputs once, outputs once. FLOPs of a frame: one ray per camera sample (per path
  vertex) and one shadow ray at it, 250 each; of a convolution: its multiply-adds."""
  if case["kind"] in ("frame", "path"):
    px = _pixels(case)
    per_world = 2700.0  # poses, tables and the packed block of a world
    if case["kind"] == "frame":
      # packed colour, depth, segmentation and their views
      return {"bytes": px * (16 + 24.0) + case["worlds"] * per_world, "flops": px * case["samples"] ** 2 * 2 * 250.0}
    flops = px * case["spp"] * 2 * 2 * 250.0
    if case["filter"] == "learned":
      flops += float(kpcn.forward_flops(1, 128, 128)) / (128 * 128) * px
    return {"bytes": px * (16 + 24.0) + case["worlds"] * per_world, "flops": flops}
  if case["kind"] == "train":
    px = case["crops"] * case["res"] ** 2
    params = sum(9 * (s.c_in + s.c_in2) * s.c_out for s in kpcn.layer_specs())
    return {"bytes": px * 64.0 + params * 28.0, "flops": 3.0 * kpcn.forward_flops(case["crops"], case["res"], case["res"])}
  px = case["images"] * case["height"] * case["width"]
  c, co = case["c_in"] + case["c_skip"], case["c_out"]
  size = 4.0 if case["direction"] == "input_grad" and case["c_skip"] else 2.0
  moved = {"forward": c * 2.0 + co * 2.0, "input_grad": co * 2.0 + c * size + (0.0 if case["c_skip"] else c * 2.0), "weight_grad": c * 2.0 + co * 2.0}
  weights = 9 * c * co * (4.0 if case["direction"] == "weight_grad" else 2.0)
  return {"bytes": px * moved[case["direction"]] + weights, "flops": 2.0 * 9 * c * co * px}
