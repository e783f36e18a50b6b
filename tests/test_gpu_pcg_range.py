"""The plain projection of winds far smaller and far larger than FP32's squares: it is linear in the wind, so a
wind scaled by a power of two must give the correction scaled by the same power. At 2^-70 the residual's and
the direction's products lie below FP32's smallest number, at 2^70 above its largest; the sums hold them. Grids
of x no multiple of four, whose dot products take exact terms: one block, the one-launch solver's 4 and 14
cells a thread, the three streaming launches, terrain, both semantics. The boundary columns are 0, the
tolerance 0, ten iterations each. Bound: relative L2 1e-5 as in the projection tests (scaling by a power of
two keeps every rounding but those of numbers below 2^-126). Sizes are x, y (vertical), z."""
import numpy as np
import pytest

from helpers import gpu_cfg, make_env, rel_l2, small_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("x,y,z,hills,sem,fused", [
    (13, 9, 7, 0, 0, 1), (45, 43, 51, 1, 0, 1), (101, 83, 97, 0, 1, 1),
    (13, 9, 7, 0, 0, 0), (61, 33, 26, 1, 1, 0),
])
def test_projection_scales_with_the_wind(gpu_lib, x, y, z, hills, sem, fused):
    init, dt, speed = small_case((x, z, y))
    if hills:
        xx, zz = np.meshgrid(np.arange(init.nx), np.arange(init.nz))
        h = np.round(4.0 * np.exp(-((xx - 0.4 * x) ** 2 + (zz - 0.6 * z) ** 2) / (0.04 * x * z)))
        init.ground_height = np.clip(h, 0, init.ny - 2).astype(np.int32).reshape(-1)
    env = make_env(init, gpu_cfg(sem, pcg_tol=0.0, pcg_max_iter=10, pcg_fused=fused))
    state = {k: env.read(k) for k in ("th", "qv", "p", "rho")}
    sky = env.sky_mask()
    rng = np.random.default_rng(x * y * z)
    wind = {k: np.where(sky, rng.uniform(-1.0, 1.0, sky.shape), 0.0).astype(np.float32) for k in ("u", "v", "w")}
    for k in ("defU", "defW"):
        env.write(k, np.zeros(init.ny, np.float32))
    got = {}
    for power in (0, -70, 70):
        for k, v in state.items():
            env.write(k, v)
        for k, v in wind.items():
            env.write(k, v * np.float32(2.0 ** power))
        st = env.run_stage(3, 0, dt * speed)
        assert st["pcg_iters"] == 10, st
        got[power] = env.read("debug3").astype(np.float64) * 2.0 ** -power
    assert np.linalg.norm(got[0][sky]) > 0
    for power in (-70, 70):
        assert rel_l2(got[power], got[0], sky) <= 1e-5, power
    env.close()
