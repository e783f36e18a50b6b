"""The PCG's three streaming launches on grids of any x (k_matvec, k_update, k_search) where they can go
wrong: cells that leave one, two and three over from the float4 streams, fewer cells than one float4 per
thread, x at and around a warp, rows that leave one to three of a lane's four, one plane, runs that end
below a tile's planes, more tiles than blocks, terrain; against the oracle's projection, with the bound
of the other projection tests (relative L2 1e-5: the rounding differences of the same FP32 iteration).
Sizes are x, y (vertical), z."""
import numpy as np
import pytest

import oracle
from helpers import gpu_cfg, make_env, oracle_cfg, push_oracle_to_env, rel_l2, small_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("x,y,z,hills,sem", [
    (5, 3, 1, 0, 0), (33, 9, 5, 1, 0), (31, 18, 7, 0, 1), (29, 35, 11, 1, 0), (61, 16, 3, 0, 1),
    (95, 33, 26, 1, 0),
    (1, 4, 9001, 0, 0),   # a column of planes one cell wide
])
def test_three_launch_pcg_matches_oracle(gpu_lib, x, y, z, hills, sem):
    init, dt, speed = small_case((x, z, y))
    if hills:
        xx, zz = np.meshgrid(np.arange(init.nx), np.arange(init.nz))
        h = np.round(4.0 * np.exp(-((xx - 0.4 * x) ** 2 + (zz - 0.6 * z) ** 2) / (0.04 * x * z)))
        init.ground_height = np.clip(h, 0, init.ny - 2).astype(np.int32).reshape(-1)
    st = oracle.OracleState(init, np.float32)
    rng = np.random.default_rng(x * y * z)
    sky = st.sky_mask()
    for k in ("u", "v", "w"):
        st.a[k] += np.where(sky, rng.uniform(-1.0, 1.0, sky.shape), 0.0).astype(np.float32)
    env = make_env(init, gpu_cfg(sem, pcg_fused=0))
    push_oracle_to_env(st, env)
    o = st.stage(oracle_cfg(sem), 3, 0, dt * speed)
    g = env.run_stage(3, 0, dt * speed)
    assert abs(g["pcg_iters"] - o["pcg_iters"]) <= 1, (g, o)
    for k in ("u", "v", "w", "p"):
        assert rel_l2(env.read(k), st.a[k], sky) <= 1e-5, k
    env.close()
