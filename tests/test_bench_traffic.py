"""The bench's DRAM traffic is of the kernels that rendered the frame: the lines of profiles/ncu_traffic.txt are
chosen by workload and kernels, and kernels that were not measured have none."""

import types

from mujoco_warp_pbr_gb300 import _lib


def _context(**changes):
  base = types.SimpleNamespace(render_rgb=[True])
  rc = types.SimpleNamespace(tier=0, schedule=2, has_transparency=False, has_reflection=True, use_shadows=True, mesh_nface=[12], nhfield=0, base=base)
  s = _lib.Scene()
  s.nbvh_geom, s.nlight, s.nmesh, s.blas_root = 17, 1, 1, 0x1000
  s.settings.schedule, s.settings.samples_per_axis, s.settings.stack_depth = 2, 2, 8
  for name, value in changes.items():
    setattr(rc if hasattr(rc, name) else s, name, value)
  return rc, s


def test_traffic_is_chosen_by_the_kernels_that_ran():
  import bench

  rc, s = _context()
  scanned = bench.render_kernels(rc, s)
  assert "wave_mirror_mesh" in scanned and bench.render_launches(rc, s, 4) == 28
  now = bench._traffic("mesh_ibl_4096x128", scanned)
  assert now is not None and now != bench._traffic("mesh_ibl_4096x128")
  rc, s = _context(nbvh_geom=33)
  assert bench._traffic("mesh_ibl_4096x128", bench.render_kernels(rc, s)) == bench._traffic("mesh_ibl_4096x128")
  assert bench._traffic("mesh_ibl_4096x128", ["rt"]) is None and bench._traffic("mesh_ibl_1024x128", scanned) is None
  rc, s = _context(tier=1)
  assert bench._traffic("path_1024x128_spp2", bench.render_kernels(rc, s)) < bench._traffic("path_1024x128_spp2")
  rc, s = _context(mesh_nface=[], nmesh=0, blas_root=None)
  assert bench.render_kernels(rc, s) == ["rt_fused"] and bench.render_launches(rc, s, 1) == 1
  rc, s = _context(mesh_nface=[], nmesh=0, blas_root=None, nlight=17)  # staged, without triangle BVHs: one mirror kernel
  assert bench.render_launches(rc, s, 1) == 6
  rc, s = _context(has_transparency=True)
  assert bench.render_kernels(rc, s) == ["rt"]
