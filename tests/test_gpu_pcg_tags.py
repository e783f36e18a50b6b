"""The one-launch PCG over more reductions than its tags have numbers (2^20, some 2600 solves of 200 iterations in one
environment): a solve after the tags have come round gives the bits of the same solve in a new environment."""
import numpy as np
import pytest

from helpers import make_env, small_case
from skewtcloudsim_gb300 import SolverConfig

pytestmark = pytest.mark.gpu


def test_solve_after_the_tags_came_round(gpu_lib):
    init, dt, speed = small_case((24, 20, 12))
    env = make_env(init, SolverConfig(pcg_tol=0.0))
    sky = env.sky_mask()
    rng = np.random.default_rng(1)
    wind = {k: np.where(sky, rng.uniform(-1.0, 1.0, sky.shape), 0.0).astype(np.float32) for k in ("u", "v", "w")}
    state = {k: env.read(k) for k in ("p", "rho")}
    reductions = 0
    while reductions < 2 ** 20 + 5000:
        for k, v in {**state, **wind}.items():
            env.write(k, v)
        st = env.run_stage(3, 0, dt * speed)
        assert st["pcg_iters"] == 200
        reductions += 2 * st["pcg_iters"]
    fresh = make_env(init, SolverConfig(pcg_tol=0.0))
    for k, v in {**state, **wind}.items():
        fresh.write(k, v)
    fresh.run_stage(3, 0, dt * speed)
    for k in ("u", "v", "w", "p", "debug3"):
        np.testing.assert_array_equal(env.read(k).view(np.uint32), fresh.read(k).view(np.uint32), err_msg=k)
    env.close()
    fresh.close()
