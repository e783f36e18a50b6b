"""Diffusion and advection away from the flat x-multiple-of-four grids (k_diffuse, k_ppm_x, k_ppm_march),
stage by stage against the oracle where they can go wrong: x at and around a warp's 28 and 32 cells, fewer
cells than a window, rows that fill a lane's four exactly or leave one, one plane and fewer planes than the
loads ahead, flat ground, single steep towers that end below the top, and rough ground where every
neighbour may be a ground cell. Bound: 2e-5 of the field's largest value, as in the stage tests (a stage
makes 20 sweeps, or two substeps of 5 passes of some ten roundings, over a companion of 0.4 or more:
10 * 10 * 6e-8 / 0.4 = 1.5e-5). Sizes are x, y
(vertical), z."""
import numpy as np
import pytest

import oracle
from helpers import gpu_cfg, make_env, oracle_cfg, push_oracle_to_env, rel_max, small_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("x,y,z,ground", [
    (28, 17, 9, "towers"), (29, 18, 5, "flat"), (57, 33, 3, "rough"), (33, 6, 35, "rough"),
    (31, 21, 12, "flat"), (2, 9, 7, "towers"), (64, 20, 2, "rough"), (90, 5, 1, "flat"),
])
def test_stages_on_any_grid(gpu_lib, x, y, z, ground):
    init, dt, speed = small_case((x, z, y))
    rng = np.random.default_rng(100 * x + z)
    h = np.zeros((z, x), np.int32)
    if ground == "towers":
        h[rng.uniform(size=h.shape) < 0.1] = y - 2
    elif ground == "rough":
        h = rng.integers(0, y - 1, h.shape).astype(np.int32)
    init.ground_height = h.reshape(-1)
    st = oracle.OracleState(init, np.float32)
    sky = st.sky_mask()
    # winds that do not change along their own axis: no cell's companion falls below 1 - 0.6, at a ground face
    yy, zz, xx = np.meshgrid(np.arange(y), np.arange(z), np.arange(x), indexing="ij")
    yy, zz, xx = (a.transpose(1, 0, 2).reshape(-1) for a in (yy, zz, xx))  # the fields' order: x fastest, then y, z
    wind = {"u": 6.0 * np.sin(0.3 * yy + 0.2 * zz), "v": 4.0 * np.cos(0.25 * xx + 0.4 * zz), "w": 5.0 * np.sin(0.35 * xx - 0.2 * yy)}
    for k, a in wind.items():
        st.a[k] = np.where(sky, a.reshape(sky.shape), 0.0).astype(np.float32)
    for k in ("qw", "qr"):
        st.a[k] = np.where(sky, rng.uniform(5e-4, 1e-3, sky.shape), 0.0).astype(np.float32)
    before = {k: v.copy() for k, v in st.a.items()}
    env = make_env(init, gpu_cfg())
    for stage, names in ((0, ("th", "qv", "u", "v", "w", "qw")), (1, ("th", "u", "v", "w", "qv", "qw"))):
        for arg, name in enumerate(names):
            for k, v in before.items():
                st.a[k][...] = v
            push_oracle_to_env(st, env)
            g = env.run_stage(stage, arg, 20.0)
            o = st.stage(oracle_cfg(), stage, arg, 20.0)
            if stage == 1:
                assert g["nsub"] == o["nsub"]
            assert rel_max(env.read(name), st.a[name], sky) <= 2e-5, (stage, name)
    env.close()
