"""The V-cycle's coarsest level (k_mg_coarse_run, k_mg_coarse), where it can go wrong: a grid that has no coarser level, at
the largest size the kernel takes, with one of its planes in two and so the largest zero planes around the
iterate (more shared memory than a launch has by default), coarsest levels whose cells end inside a warp,
terrain. The mixed projection against the FP64 oracle solved to 1e-13: relative L2 1e-6 on u, w, p and rho
as in the mixed tests, the solver's own residual below 1e-8. Sizes are x, y (vertical), z."""
import numpy as np
import pytest

import oracle
from helpers import make_env, push_oracle_to_env, rel_l2, small_case
from skewtcloudsim_gb300 import SolverConfig
from test_gpu_mixed import FP64_CFG, _to64

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("x,y,z,hills", [
    (16, 8, 16, 0), (32, 16, 8, 0),   # the coarsest level alone, 2048 and 4096 cells
    (64, 32, 2, 0),                   # two planes of 2048
    (32, 16, 16, 0), (40, 24, 56, 0), (72, 40, 72, 0),
    (24, 16, 30, 1),                  # an odd number of planes, half a run at the end
    (128, 64, 64, 1),
])
def test_coarsest_level_matches_fp64(gpu_lib, x, y, z, hills):
    init, dt, speed = small_case((x, z, y))
    if hills:
        xx, zz = np.meshgrid(np.arange(init.nx), np.arange(init.nz))
        h = np.round(5.0 * np.exp(-((xx - 0.4 * x) ** 2 + (zz - 0.6 * z) ** 2) / (0.04 * x * z)))
        init.ground_height = np.clip(h, 0, init.ny - 2).astype(np.int32).reshape(-1)
    st32 = oracle.OracleState(init, np.float32)
    rng = np.random.default_rng(x * y + z)
    sky = st32.sky_mask()
    for k in ("u", "v", "w"):
        st32.a[k] += np.where(sky, rng.uniform(-1.0, 1.0, sky.shape), 0.0).astype(np.float32)
    ref = _to64(st32, init)
    env = make_env(init, SolverConfig(precision=1))
    push_oracle_to_env(st32, env)
    env.run_stage(3, 0, dt * speed)
    st = env.stats()
    assert st["converged"] and st["pcg_residual"] <= 1e-8, st
    assert ref.stage(oracle.Config(**FP64_CFG), 3, 0, dt * speed)["pcg_iters"] < 20000
    for k in ("u", "w", "p", "rho"):
        assert rel_l2(env.read(k), ref.a[k], sky) <= 1e-6, k
    env.close()
