"""Refit: a world's block does not depend on how many worlds are refitted with it, although the number decides
where the sweep keeps its nodes (csrc/refit.cu, refit_launch): in shared memory for the few worlds, in global
memory for the many, at sizes on both sides of the rule and where it never changes."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")

import mujoco_warp_pbr_gb300 as mjpbr  # noqa: E402
from tests import helpers  # noqa: E402
from tests.test_scan import scene  # noqa: E402


@pytest.mark.gpu
@pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a CUDA GPU")
@pytest.mark.parametrize("ngeom", [40, 221, 300, 580])
def test_blocks_do_not_depend_on_the_number_of_worlds(ngeom):
  few = scene(ngeom, nworld=7, nlight=5)
  m, d, rc = helpers.gpu_scene(few, cam_res=(4, 4))
  mjpbr.refit_bvh(m, d, rc)
  ref = rc.world_blocks.cpu().numpy().view(np.uint32)
  many = 3003
  period = np.arange(many) % 7
  sc = scene(ngeom, nworld=7, nlight=5)
  for field in ("geom_xpos", "geom_xmat", "cam_xpos", "cam_xmat", "light_xpos", "light_xdir"):
    setattr(sc.mjd, field, getattr(sc.mjd, field)[period])
  sc.nworld = many
  sc.per_world = {k: v[period] for k, v in sc.per_world.items()}
  m, d, rc = helpers.gpu_scene(sc, cam_res=(4, 4))
  mjpbr.refit_bvh(m, d, rc)
  got = rc.world_blocks.cpu().numpy().view(np.uint32)
  np.testing.assert_array_equal(got, ref[period])
