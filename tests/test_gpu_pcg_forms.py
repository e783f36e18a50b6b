"""Every form of the plain PCG where a small grid's default does not reach it: the form is told by the stages that
the library profiles (one launch: pcg_grid; matrix-free: pcg_matvec and pcg_update; three launches: pcg_search
too). For each: a NaN and a zero density end the step with SKT_NAN_DETECTED and leave the environment usable;
the iteration cap after odd and even numbers; and the captured step's loop against the stream-ordered one, bit
for bit, with caps before, at and inside a replayed chunk of eight iterations, one to four directions pending,
and a stop by the tolerance. The matrix-free grids have 1.6M cells, well above the one-launch solver's 1.1M.
Sizes are x, y (vertical), z."""
import numpy as np
import pytest

from helpers import SKY, make_env, rel_l2, small_case
from skewtcloudsim_gb300 import SktError, SolverConfig
from skewtcloudsim_gb300.environment import Status

pytestmark = pytest.mark.gpu

FORMS = {  # name: (size, configuration, stages)
    "one launch": ((32, 32, 32), {}, {"pcg_grid"}),
    "one launch, x odd": ((33, 18, 21), {}, {"pcg_grid"}),
    "matrix-free": ((128, 100, 128), {}, {"pcg_matvec", "pcg_update"}),
    "three launches": ((64, 24, 40), {"pcg_fused": 0}, {"pcg_matvec", "pcg_update", "pcg_search"}),
    "three launches, x odd": ((61, 24, 40), {"pcg_fused": 0}, {"pcg_matvec", "pcg_update", "pcg_search"}),
    "three launches by size": ((127, 101, 127), {}, {"pcg_matvec", "pcg_update", "pcg_search"}),
}


def _env(form, **kw):
    (x, y, z), cfg, stages = FORMS[form]
    init, dt, speed = small_case((x, z, y))
    return make_env(init, SolverConfig(**cfg, **kw)), dt, speed, stages


@pytest.mark.parametrize("form", list(FORMS))
def test_form_of_the_grid(gpu_lib, form):
    env, dt, speed, stages = _env(form)
    env.profile(True)
    env.update_gpu(dt, speed)
    ran = {k for k in env.profile_read() if k.startswith("pcg_")}
    env.close()
    assert ran == stages


@pytest.mark.parametrize("form", list(FORMS))
@pytest.mark.parametrize("field,value", [("th", np.nan), ("p", 0.0)])
@pytest.mark.parametrize("graph", [0, 1])
def test_nan_is_reported(gpu_lib, form, field, value, graph):
    env, dt, speed, _ = _env(form, use_graph=graph)
    env.update_gpu(dt, speed)
    good = {k: env.read(k) for k in SKY}
    (x, y, z), _, _ = FORMS[form]
    a = good[field].copy()
    a[x // 2 + x * (y // 2 + y * (z // 2))] = value
    env.write(field, a)
    # theta's NaN reaches the projection through the density, without a step's wind maximum before it
    with pytest.raises(SktError) as ei:
        env.run_stage(3, 0, dt * speed)
    assert ei.value.status == Status.NAN_DETECTED
    for k, v in good.items():
        env.write(k, v)
    env.write(field, a)
    with pytest.raises(SktError) as ei:
        env.update_gpu(dt, speed)
    assert ei.value.status == Status.NAN_DETECTED
    for k, v in good.items():
        env.write(k, v)
    assert env.update_gpu(dt, speed) in (Status.OK, Status.NOT_CONVERGED)
    for k in SKY:
        assert np.isfinite(env.read(k)[env.sky_mask()]).all(), k
    env.close()


@pytest.mark.parametrize("form", ["one launch", "matrix-free", "three launches", "three launches, x odd"])
def test_cap_after_any_number_of_iterations(gpu_lib, form):
    """The same pressure as the three-launch iteration's (a vertical neighbour's sum order apart: 1e-6)."""
    (x, y, z), cfg, _ = FORMS[form]
    init, dt, speed = small_case((x, z, y))
    start = None
    for cap in (1, 2, 3, 6, 7, 8):
        got = {}
        for fused in (cfg.get("pcg_fused", 1), 0):
            env = make_env(init, SolverConfig(pcg_fused=fused, pcg_max_iter=cap))
            if start is None:
                rng = np.random.default_rng(7)
                sky = env.sky_mask()
                start = {k: env.read(k) + np.where(sky, rng.uniform(-1, 1, sky.shape), 0.0).astype(np.float32) for k in ("u", "v", "w")}
            for k, v in start.items():
                env.write(k, v)
            st = env.run_stage(3, 0, dt * speed)
            assert st["pcg_iters"] == cap and not st["converged"]
            got[fused] = {k: env.read(k) for k in ("u", "v", "w", "p")}
            env.close()
        for k, v in got[0].items():
            assert rel_l2(got[cfg.get("pcg_fused", 1)][k], v, sky) <= 1e-6, (cap, k)


@pytest.mark.parametrize("form,sem,stops", [
    ("matrix-free", 0, (1, 5, 9, 10, 11, 12)), ("matrix-free", 1, (2, 3, 4, 8, 17)),
    ("three launches", 0, (1, 9, 10)), ("three launches by size", 1, (1, 9, 12)), ("one launch, x odd", 0, (1, 5)),
])
def test_captured_loop_equals_stream_ordered(gpu_lib, form, sem, stops):
    for cap in stops + ("tolerance",):
        kw = dict(semantics=sem, pcg_max_iter=cap) if cap != "tolerance" else dict(semantics=1, pcg_max_iter=500, pcg_tol=3e-4)
        a, dt, speed, _ = _env(form, **kw)
        b, _, _, _ = _env(form, use_graph=1, **kw)
        for _ in range(2):
            a.update_gpu(dt, speed)
            b.update_gpu(dt, speed)
        sa, sb = a.stats(), b.stats()
        assert sa["pcg_iters"] == sb["pcg_iters"] and sa["converged"] == sb["converged"] and sa["nsub"] == sb["nsub"], (cap, sa, sb)
        assert sa["converged"] if cap == "tolerance" else sa["pcg_iters"] <= cap
        for k in SKY:
            np.testing.assert_array_equal(a.read(k).view(np.uint32), b.read(k).view(np.uint32), err_msg=f"{cap} {k}")
        a.close()
        b.close()
