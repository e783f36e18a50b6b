"""skt_autotune on grids that the two-sweep diffusion does not take (terrain, x no multiple of four): it measures no
depth there, so the size's own depth stays, in the environment and in the cache that a flat terrain of the same
grid reads."""
import json

import numpy as np
import pytest

from helpers import make_env, small_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("x,hills", [(64, True), (62, False)])
def test_depth_stays_where_it_is_not_measured(gpu_lib, tmp_path, x, hills):
    cache = str(tmp_path / "tuning.json")
    init, dt, speed = small_case((x, 48, 32))
    flat = init.ground_height.copy()
    if hills:
        h = np.zeros((init.nz, init.nx), np.int32)
        h[10:20, 20:30] = 3
        init.ground_height = h.reshape(-1)
    env = make_env(init)
    own = env.get_tuning()
    assert own["diffuse_depth"] == 2
    t = env.autotune(cache)
    assert t["diffuse_depth"] == own["diffuse_depth"] and env.get_tuning()["diffuse_depth"] == own["diffuse_depth"]
    env.close()
    assert len(json.load(open(cache))) == 1
    init.ground_height = flat
    b = make_env(init)
    assert b.autotune(cache)["from_cache"] and b.get_tuning()["diffuse_depth"] == own["diffuse_depth"]
    b.close()
