"""Grids of short rows above the one-launch solver's size: rows below 24 cells run the three launches, from 24 on the
matrix-free form, flat and over hills, both against the oracle's projection (relative L2 1e-5 as in the other
projection tests), and the captured step against the stream-ordered one. Sizes are x, y (vertical), z."""
import numpy as np
import pytest

import oracle
from helpers import SKY, gpu_cfg, make_env, oracle_cfg, push_oracle_to_env, rel_l2, small_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("x,y,z,hills,form", [
    (4, 128, 2400, 0, "three launches"), (20, 100, 601, 1, "three launches"), (20, 100, 601, 0, "three launches"),
    (24, 100, 501, 0, "matrix-free"), (24, 100, 501, 1, "matrix-free"),
])
def test_short_rows(gpu_lib, x, y, z, hills, form):
    init, dt, speed = small_case((x, z, y))
    if hills:
        xx, zz = np.meshgrid(np.arange(init.nx), np.arange(init.nz))
        init.ground_height = np.clip(np.round(4.0 * np.sin(0.4 * xx) ** 2 * np.cos(0.05 * zz) ** 2), 0, 4).astype(np.int32).reshape(-1)
    st = oracle.OracleState(init, np.float32)
    rng = np.random.default_rng(x + z)
    sky = st.sky_mask()
    for k in ("u", "v", "w"):
        st.a[k] += np.where(sky, rng.uniform(-1.0, 1.0, sky.shape), 0.0).astype(np.float32)
    env = make_env(init, gpu_cfg(0, pcg_max_iter=20))
    push_oracle_to_env(st, env)
    env.profile(True)
    g = env.run_stage(3, 0, dt * speed)
    assert ("pcg_search" in env.profile_read()) == (form == "three launches")
    env.profile(False)
    o = st.stage(oracle_cfg(0, pcg_max_iter=20), 3, 0, dt * speed)
    assert g["pcg_iters"] == o["pcg_iters"]
    for k in ("u", "v", "w", "p"):
        assert rel_l2(env.read(k), st.a[k], sky) <= 1e-5, k
    env.close()
    a, b = make_env(init, gpu_cfg(0, pcg_max_iter=11)), make_env(init, gpu_cfg(0, pcg_max_iter=11, use_graph=1))
    a.update_gpu(dt, speed)
    b.update_gpu(dt, speed)
    for k in SKY:
        np.testing.assert_array_equal(a.read(k).view(np.uint32), b.read(k).view(np.uint32), err_msg=k)
    a.close()
    b.close()
