"""The PCG in one cooperative launch (grids up to about a million cells) at the sizes where it can go
wrong: one block that is not full, a block boundary inside a row, rows that are no multiple of a
warp, each count of cells per thread, a halo row longer than a block's share, terrain; against the
oracle's projection, with the bound of the other projection tests (relative L2 1e-5: the rounding
differences of the same FP32 iteration). Sizes are x, y (vertical), z."""
import numpy as np
import pytest

import oracle
from helpers import gpu_cfg, make_env, oracle_cfg, push_oracle_to_env, rel_l2, small_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("x,y,z,hills,sem", [
    (5, 4, 3, 0, 0),        # 60 cells: one block, mostly empty
    (32, 16, 2, 0, 1),      # 1024 cells: one full block
    (33, 31, 2, 0, 0),      # two blocks, the second with 1022 cells
    (1031, 5, 4, 0, 0),     # a row longer than a block's 1024 cells
    (47, 43, 49, 1, 0),     # 97 blocks of two cells a thread: four cells a thread instead
    (90, 51, 75, 0, 1),     # eight cells a thread
    (101, 83, 97, 1, 0),    # fourteen cells a thread, odd in every direction
])
def test_one_launch_pcg_matches_oracle(gpu_lib, x, y, z, hills, sem):
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
    env = make_env(init, gpu_cfg(sem))
    push_oracle_to_env(st, env)
    o = st.stage(oracle_cfg(sem), 3, 0, dt * speed)
    g = env.run_stage(3, 0, dt * speed)
    assert abs(g["pcg_iters"] - o["pcg_iters"]) <= 1, (g, o)
    for k in ("u", "v", "w", "p"):
        assert rel_l2(env.read(k), st.a[k], sky) <= 1e-5, k
    env.close()
