"""The moisture fields swept and carried together (a launch per pass for all of them): whole steps
against the oracle where the number of passes is odd (a third buffer per field, or a copy for one
pass) or two sweeps share a pass, on flat terrain with x a multiple of four, on an odd size and over
hills, with two wind substeps. Bound: the whole-step tolerance of the parity tests (relative L2 1e-5)."""
import numpy as np
import pytest

import oracle
from helpers import SKY, gpu_cfg, make_env, oracle_cfg, push_oracle_to_env, rel_l2, small_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(32, 32, 16), (30, 25, 17)], ids=["vec", "odd"])  # x, y, z (z vertical)
@pytest.mark.parametrize("sweeps,depth,hills", [(1, 1, 0), (3, 1, 0), (6, 2, 0), (7, 2, 0), (3, 1, 1)])
def test_step_with_fields_together(gpu_lib, shape, sweeps, depth, hills):
    init, dt, speed = small_case(shape)
    if hills:
        xx, zz = np.meshgrid(np.arange(init.nx), np.arange(init.nz))
        init.ground_height = np.clip(np.round(3.0 * np.exp(-((xx - 12) ** 2 + (zz - 14) ** 2) / 40.0)), 0, 3).astype(np.int32).reshape(-1)
    st = oracle.OracleState(init, np.float32)
    rng = np.random.default_rng(sweeps * 10 + depth)
    sky = st.sky_mask()
    for k, size in (("qw", 1e-3), ("qc", 5e-4), ("qr", 1e-3), ("qs", 5e-4), ("qi", 5e-4)):
        st.a[k] = np.where(sky, rng.uniform(0.0, size, sky.shape), 0.0).astype(np.float32)
    env = make_env(init, gpu_cfg(diffuse_sweeps=sweeps))
    env.set_tuning(diffuse_depth=depth, diffuse_rows=14)
    push_oracle_to_env(st, env)
    o = st.step(oracle_cfg(diffuse_sweeps=sweeps), dt, speed)
    env.update_gpu(dt, speed)
    assert env.stats()["nsub"] == o["nsub"]
    for k in SKY:
        assert rel_l2(env.read(k), st.a[k], sky) <= 1e-5, (k, rel_l2(env.read(k), st.a[k], sky))
    env.close()
