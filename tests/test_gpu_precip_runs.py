"""The falling species in runs of rows (eight warps share 32 columns): heights with no row for some
warps, one row each, a remainder in the last run, ground inside a run and at a run's first row, and
columns that do not fill a block. The launch of the three species together is reached by a whole step:
one without wind, sweeps and pressure iterations, whose rain, snow and ice are compared with the oracle's
step within the stage tolerance (max-norm 2e-5). Sizes are x, y (vertical), z."""
import numpy as np
import pytest

import oracle
from helpers import gpu_cfg, make_env, oracle_cfg, push_oracle_to_env, rel_max, small_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("x,y,z,hills", [(4, 3, 4, 0), (7, 9, 5, 0), (32, 10, 3, 1), (33, 40, 7, 1), (16, 129, 4, 0)])
def test_fall_in_runs(gpu_lib, x, y, z, hills):
    init, dt, speed = small_case((x, z, y))
    if hills:
        h = np.arange(init.nx * init.nz) % max(1, min(8, init.ny - 2))
        init.ground_height = h.astype(np.int32)
    st = oracle.OracleState(init, np.float32)
    rng = np.random.default_rng(x * y + z)
    sky = st.sky_mask()
    for k, size in (("qr", 1e-3), ("qs", 5e-4), ("qi", 5e-4)):
        q = rng.uniform(0.0, size, sky.shape) * (rng.random(sky.shape) < 0.7)  # some cells hold none
        st.a[k] = np.where(sky, q, 0.0).astype(np.float32)
    cfg = dict(diffuse_sweeps=0, pcg_max_iter=0)
    for k in ("u", "v", "w"):
        st.a[k][:] = 0.0
    env = make_env(init, gpu_cfg(**cfg))
    push_oracle_to_env(st, env)
    st.step(oracle_cfg(**cfg), dt, speed)
    env.update_gpu(dt, speed)
    for k in ("qr", "qs", "qi"):
        assert rel_max(env.read(k), st.a[k], sky) <= 2e-5, k
    env.close()
