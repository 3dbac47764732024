"""The persistent trace stages refill their lanes from the queues (csrc/refill.cuh): frames whose queues hold
several times the lanes that are resident, so that lanes take second and third rays while others of their
warp are at other steps, against the schedules without queues, bit for bit. Scanned mesh scenes (voted_loop
for mirror rays, refill_loop for the rest) with coincident geoms, whose hits the order of the tests decides, and
scenes past 32 geoms (refill_loop over the BVH)."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from tests import helpers  # noqa: E402
from tests.test_scan import scene  # noqa: E402

RES = 64


def _resident_lanes() -> int:
  return torch.cuda.get_device_properties(0).multi_processor_count * 2048


def _frame(sc, **options):
  m, d, rc = helpers.gpu_scene(sc, cam_res=(RES, RES), **options)
  return rc, helpers.render_gpu(m, d, rc, seed=11)


@pytest.mark.gpu
@pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a CUDA GPU")
@pytest.mark.parametrize("ngeom,mesh", [(17, True), (32, True), (33, True), (33, False)])
def test_long_queues_of_the_real_time_tier(ngeom, mesh):
  sc = scene(ngeom, mesh=mesh, coincident=True, mirror=True, nworld=400)
  _, ref = _frame(sc, schedule="queue", samples_per_pixel=2)
  rc, got = _frame(sc, schedule="wavefront", samples_per_pixel=2)
  # the queues' lengths stand at the start of the scratch: mirror rays, shadow entries, mirror rays with meshes
  lengths = rc.wave_scratch[:32].view(torch.int32).cpu().numpy()
  assert lengths[0] > 3 * _resident_lanes() and lengths[1] > 3 * _resident_lanes()
  assert ngeom > 32 or lengths[6] > 2 * _resident_lanes()
  for key in ("rgb", "depth", "seg", "hdr"):
    np.testing.assert_array_equal(got[key], ref[key], err_msg=key)


@pytest.mark.gpu
@pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a CUDA GPU")
@pytest.mark.parametrize("ngeom,mesh", [(17, True), (32, True), (33, True), (33, False)])
def test_long_queues_of_the_path_tier(ngeom, mesh):
  sc = scene(ngeom, mesh=mesh, coincident=True, mirror=True, nworld=100)
  assert 100 * RES * RES * 3 > 3 * _resident_lanes()
  options = {"tier": 1, "path_samples": 3, "max_depth": 3}
  _, ref = _frame(sc, schedule="grid", **options)
  _, got = _frame(sc, schedule="wavefront", **options)
  for key in ("rgb", "depth", "seg", "hdr"):
    np.testing.assert_array_equal(got[key], ref[key], err_msg=key)
