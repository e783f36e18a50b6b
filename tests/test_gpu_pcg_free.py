"""The matrix-free PCG operator fed by TMA (grids above the one-launch solver's size, x a multiple of
four) where it can go wrong: a last block of one lane, rows of blocks with a remainder of one row, runs of
planes with a remainder, terrain, both forms of the lower coefficients, densities whose coefficients cross
whole numbers (Q3's truncation), and stops after one to nine iterations (the pressure updates go four at a
time); against the oracle's projection, with the bound of the other projection tests (relative L2 1e-5).
Sizes are x, y (vertical), z."""
import numpy as np
import pytest

import oracle
from helpers import gpu_cfg, make_env, oracle_cfg, push_oracle_to_env, rel_l2, small_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("x,y,z,hills,sem,cap", [
    (132, 65, 131, 0, 0, 40),   # a second block with one lane, 9 rows of blocks, the last of one row
    (1028, 9, 123, 0, 1, 40),   # nine blocks along x, two along y
    (260, 41, 107, 1, 0, 40),   # terrain
    (128, 100, 89, 1, 1, 40),
    (64, 136, 128, 0, 0, 1), (64, 136, 128, 0, 0, 4), (64, 136, 128, 0, 0, 5), (64, 136, 128, 0, 0, 9),
])
def test_matrix_free_pcg_matches_oracle(gpu_lib, x, y, z, hills, sem, cap):
    init, dt, speed = small_case((x, z, y))
    if hills:
        xx, zz = np.meshgrid(np.arange(init.nx), np.arange(init.nz))
        h = np.round(6.0 * np.exp(-((xx - 0.4 * x) ** 2 + (zz - 0.6 * z) ** 2) / (0.04 * x * z)))
        init.ground_height = np.clip(h, 0, init.ny - 2).astype(np.int32).reshape(-1)
    st = oracle.OracleState(init, np.float32)
    rng = np.random.default_rng(x + y + z)
    sky = st.sky_mask()
    for k in ("u", "v", "w"):
        st.a[k] += np.where(sky, rng.uniform(-1.0, 1.0, sky.shape), 0.0).astype(np.float32)
    env = make_env(init, gpu_cfg(sem, pcg_max_iter=cap))
    push_oracle_to_env(st, env)
    o = st.stage(oracle_cfg(sem, pcg_max_iter=cap), 3, 0, dt * speed)
    g = env.run_stage(3, 0, dt * speed)
    assert g["pcg_iters"] == o["pcg_iters"] == cap
    for k in ("u", "v", "w", "p"):
        assert rel_l2(env.read(k), st.a[k], sky) <= 1e-5, k
    env.close()
