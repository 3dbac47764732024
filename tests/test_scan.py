"""Scenes of up to 32 geoms are traced by a warp-wide scan of the geoms (csrc/scan.cuh) where larger
ones walk the scene BVH: the same hits, bit for bit. The queue schedule (real-time tier) and the
persistent path kernel (grid schedule) always walk the BVH, so their images are the reference, at
the edges of the rule: 1, 2, 31, 32 and 33 geoms, with meshes and without, hidden geoms, coincident
ones (whose hits the order of the tests decides), mirrors, more lights than the fused kernel
counts, and several samples per pixel."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from mujoco_warp_pbr_gb300 import synthetic  # noqa: E402
from tests import helpers  # noqa: E402


def scene(ngeom, nlight=2, mesh=False, coincident=False, mirror=False, nworld=3, seed=0):
  """A floor and ngeom - 1 geoms, per-world poses; every fifth geom hidden in one of the worlds."""
  rng = np.random.default_rng(seed + 100 * ngeom)
  b = synthetic.Builder()
  floor = b.material(rgba=(0.6, 0.6, 0.6, 1), metallic=0.0, roughness=0.4, reflectance=0.4 if mirror else 0.0)
  b.geom(synthetic.GEOM_PLANE, (3.0, 3.0, 0.1), matid=floor)
  kinds = [synthetic.GEOM_SPHERE, synthetic.GEOM_BOX, synthetic.GEOM_CAPSULE, synthetic.GEOM_ELLIPSOID, synthetic.GEOM_CYLINDER]
  mid = -1
  if mesh:
    v, f = synthetic.icosphere(2)
    mid = b.mesh(v * 0.25, f)
  for k in range(ngeom - 1):
    if mesh and k % 3 == 0:
      b.geom(synthetic.GEOM_MESH, (0.25, 0.25, 0.25), dataid=mid)
    else:
      b.geom(kinds[k % len(kinds)], tuple(rng.uniform(0.08, 0.25, 3)))
  for k in range(nlight):
    kind = (synthetic.LIGHT_DIRECTIONAL, synthetic.LIGHT_POINT)[k % 2]
    b.light(kind, pos=tuple(rng.uniform(-1, 1, 2)) + (2.0,), dir=(0.2, 0.1, -1.0), diffuse=(0.3, 0.3, 0.3), bulbradius=0.05 * (k + 1))
  b.camera((0.0, -3.0, 2.0), (0.0, 0.0, 0.25), fovy=45.0, resolution=(37, 29))
  mjm, mjd0 = b.build()
  n = mjm.ngeom
  xpos = np.broadcast_to(mjd0.geom_xpos, (nworld, n, 3)).copy()
  xmat = np.broadcast_to(mjd0.geom_xmat, (nworld, n, 9)).copy()
  xpos[:, 1:, :2] = rng.uniform(-1.0, 1.0, (nworld, n - 1, 2))
  xpos[:, 1:, 2] = rng.uniform(0.1, 0.8, (nworld, n - 1))
  xmat[:, 1:] = synthetic.quat_to_mat(synthetic.random_quats(rng, (nworld, n - 1)))
  if coincident and n > 6:  # pairs and a triple of one pose: equal and nearly equal distances
    for a, c in ((1, 6), (2, 7), (3, 8), (3, 13)):
      if c < n:
        xpos[:, c], xmat[:, c] = xpos[:, a], xmat[:, a]
        mjm.geom_size[c] = mjm.geom_size[a]
  rgba = np.concatenate([rng.uniform(0.1, 0.9, (nworld, n, 3)), np.ones((nworld, n, 1))], -1).astype(np.float32)
  rgba[1, 1::5, 3] = 0.0
  mjd = synthetic.HostData(
    geom_xpos=xpos.astype(np.float32), geom_xmat=xmat.astype(np.float32),
    cam_xpos=np.broadcast_to(mjd0.cam_xpos, (nworld, 1, 3)).astype(np.float32),
    cam_xmat=np.broadcast_to(mjd0.cam_xmat, (nworld, 1, 9)).astype(np.float32),
    light_xpos=np.broadcast_to(mjd0.light_xpos, (nworld, mjm.nlight, 3)).astype(np.float32),
    light_xdir=np.broadcast_to(mjd0.light_xdir, (nworld, mjm.nlight, 3)).astype(np.float32),
  )
  options = {"cam_res": (37, 29), "render_rgb": True, "render_depth": True, "render_seg": True, "render_hdr": True, "shadow_samples": 3}
  return synthetic.SyntheticScene(name="scan", mjm=mjm, mjd=mjd, nworld=nworld, options=options, per_world={"geom_rgba": rgba}, seed=seed)


def images(sc, **options):
  m, d, rc = helpers.gpu_scene(sc, **options)
  return helpers.render_gpu(m, d, rc, seed=11)


@pytest.mark.gpu
@pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a CUDA GPU")
@pytest.mark.parametrize("coincident", [False, True])
@pytest.mark.parametrize("mesh", [False, True])
@pytest.mark.parametrize("ngeom", [1, 2, 17, 31, 32, 33])
def test_real_time_scan_matches_the_bvh(ngeom, mesh, coincident):
  sc = scene(ngeom, mesh=mesh and ngeom > 1, coincident=coincident, mirror=ngeom % 2 == 0)
  samples = 2 if ngeom % 2 else 1
  ref = images(sc, schedule="queue", samples_per_pixel=samples)
  got = images(sc, schedule="wavefront", samples_per_pixel=samples)
  for key in ("rgb", "depth", "seg", "hdr"):
    np.testing.assert_array_equal(got[key], ref[key], err_msg=key)


@pytest.mark.gpu
@pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a CUDA GPU")
@pytest.mark.parametrize("nlight,samples", [(0, 1), (16, 1), (17, 2), (3, 4), (2, 16)])
def test_fused_kernel_edges_match_the_bvh(nlight, samples):
  """No light, as many as the fused kernel counts and one more; as many samples per pixel as a CTA has
  threads."""
  sc = scene(9, nlight=nlight, mirror=True, nworld=2)
  ref = images(sc, schedule="queue", samples_per_pixel=samples)
  got = images(sc, schedule="wavefront", samples_per_pixel=samples)
  for key in ("rgb", "depth", "seg", "hdr"):
    np.testing.assert_array_equal(got[key], ref[key], err_msg=key)


@pytest.mark.gpu
@pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a CUDA GPU")
@pytest.mark.parametrize("mesh", [False, True])
@pytest.mark.parametrize("ngeom", [2, 17, 32, 33])
def test_path_scan_matches_the_bvh(ngeom, mesh):
  sc = scene(ngeom, mesh=mesh, coincident=True, mirror=ngeom == 17)
  options = {"tier": 1, "path_samples": 2, "max_depth": 3}
  ref = images(sc, schedule="grid", **options)
  got = images(sc, schedule="wavefront", **options)
  for key in ("rgb", "depth", "seg", "hdr"):
    np.testing.assert_array_equal(got[key], ref[key], err_msg=key)


@pytest.mark.gpu
@pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a CUDA GPU")
@pytest.mark.parametrize("nworld,samples", [(210, 1), (60, 2), (25, 3), (3, 16)])
def test_large_frames_match_the_bvh(nworld, samples):
  """Frames of at least four 512-thread CTAs per SM are rendered by them: the same images, at sample counts that
  divide 512 and 256 and one that divides neither."""
  sc = scene(9, mirror=True, nworld=nworld)
  ref = images(sc, schedule="queue", samples_per_pixel=samples)
  got = images(sc, schedule="wavefront", samples_per_pixel=samples)
  for key in ("rgb", "depth", "seg", "hdr"):
    np.testing.assert_array_equal(got[key], ref[key], err_msg=key)


def far_scene(distance, mesh, nworld=8, res=160):
  """Axis-aligned boxes around the origin (every third geom a mesh of one) seen, and lit, from `distance` metres
  away. Their silhouettes are their leaf boxes': rays pass them by less than the rounding of the distance, and a
  box test that rounds otherwise loses hits."""
  sc = scene(17, mesh=mesh, nworld=nworld)
  boxes = sc.mjm.geom_type != synthetic.GEOM_MESH
  boxes[0] = False
  sc.mjm.geom_type[boxes] = synthetic.GEOM_BOX
  sc.mjd.geom_xmat[:, boxes] = np.eye(3, dtype=np.float32).reshape(9)
  eye = np.array([0.3, -0.8, 0.5]) * distance
  sc.mjm.cam_fovy[:] = np.degrees(2.0 * np.arctan(1.3 / np.linalg.norm(eye)))
  sc.mjd.cam_xpos[:] = eye
  sc.mjd.cam_xmat[:] = synthetic.look_at(eye, np.array([0.0, 0.0, 0.4])).reshape(9)
  sc.mjd.light_xpos[:, 1] = (0.2 * distance, 0.3 * distance, 0.9 * distance)
  sc.options["cam_res"] = (res, res)
  return sc


@pytest.mark.gpu
@pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a CUDA GPU")
@pytest.mark.parametrize("mesh", [False, True])
@pytest.mark.parametrize("distance", [50.0, 400.0, 4000.0])
def test_far_cameras_match_the_bvh(distance, mesh):
  sc = far_scene(distance, mesh)
  for options, schedule in (({}, "queue"), ({"tier": 1, "path_samples": 1, "max_depth": 1}, "grid")):
    ref = images(sc, schedule=schedule, **options)
    got = images(sc, schedule="wavefront", **options)
    assert (ref["seg"][..., 0] > 0).mean() > 0.1
    for key in ("rgb", "depth", "seg", "hdr"):
      np.testing.assert_array_equal(got[key], ref[key], err_msg=key)


@pytest.mark.gpu
@pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a CUDA GPU")
@pytest.mark.parametrize("mesh", [False, True])
def test_large_coordinates_match_the_bvh(mesh):
  """The scene kilometres from the origin, where a coordinate's rounding is as large as the boxes' padding is
  elsewhere."""
  sc = scene(17, mesh=mesh, mirror=True, nworld=4)
  for field in ("geom_xpos", "cam_xpos", "light_xpos"):
    getattr(sc.mjd, field)[...] += np.array([3000.0, -2000.0, 500.0], np.float32)
  for options, schedule in (({}, "queue"), ({"tier": 1, "path_samples": 2, "max_depth": 2}, "grid")):
    ref = images(sc, schedule=schedule, **options)
    got = images(sc, schedule="wavefront", **options)
    assert (ref["seg"][..., 0] > 0).mean() > 0.1
    for key in ("rgb", "depth", "seg", "hdr"):
      np.testing.assert_array_equal(got[key], ref[key], err_msg=key)


@pytest.mark.gpu
@pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a CUDA GPU")
@pytest.mark.parametrize("name", ["hfield", "translucent", "translucent_mesh"])
def test_path_scan_of_height_fields_and_translucent_geoms(name):
  if name == "hfield":
    sc = synthetic.hfield_scene(seed=2, nworld=3, res=36)
    sc.options.pop("shadow_samples")
  else:
    sc = scene(17, mesh=name.endswith("mesh"), nworld=3)
    sc.per_world["geom_rgba"][:, 2::4, 3] = 0.5
  got = []
  for schedule in ("grid", "wavefront"):
    m, d, rc = helpers.gpu_scene(sc, schedule=schedule, tier=1, path_samples=2, max_depth=3, render_hdr=True)
    rc.has_transparency = name != "hfield"
    got.append(helpers.render_gpu(m, d, rc, seed=11))
  for key in ("rgb", "depth", "seg", "hdr"):
    np.testing.assert_array_equal(got[1][key], got[0][key], err_msg=key)
