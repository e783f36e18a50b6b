"""The full-size step with the launch shapes that the library gives the grid, bit for bit the step with the shapes
that test_gpu_wide.py pins against the oracle (a shape changes no value)."""
import numpy as np
import pytest

from helpers import SKY, make_env, small_case
from skewtcloudsim_gb300 import SolverConfig

pytestmark = pytest.mark.gpu


def test_full_size_step_with_the_default_shapes(gpu_lib):
    init, dt, speed = small_case((512, 512, 256), name="precision-512x512x256")
    got = []
    for pinned in (False, True):
        env = make_env(init, SolverConfig(use_graph=1))
        if pinned:
            env.set_tuning(diffuse_depth=2, diffuse_rows=14, diffuse2_bps=4, ppm_x_bps=8, ppm_y_bps=32, ppm_z_bps=8)
        else:
            assert env.get_tuning()["diffuse2_bps"] == 8 and env.get_tuning()["ppm_x_bps"] == 16
        env.update_gpu(dt, speed)
        got.append({k: env.read(k) for k in SKY})
        env.close()
    for k in SKY:
        assert np.array_equal(got[0][k].view(np.uint32), got[1][k].view(np.uint32)), k
