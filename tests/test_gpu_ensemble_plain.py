"""Ensembles of plain members whose one-launch solves do not fit the chip side by side (each wants most SMs to
itself), one of them of a size with exact products and one above the one-launch size: stepped by one graph and by
host threads, with the bits of the members stepped alone."""
import numpy as np
import pytest

from helpers import SKY, make_env, small_case
from skewtcloudsim_gb300 import Ensemble, SolverConfig, step_ensemble

pytestmark = pytest.mark.gpu

SHAPES = [(128, 64, 100), (120, 70, 110), (127, 64, 99), (96, 64, 96), (128, 100, 96)]  # x, y (vertical), z


def _members():
    out = []
    for i, (x, y, z) in enumerate(SHAPES):
        init, dt, speed = small_case((x, z, y), seed=i + 1)
        out.append((make_env(init, SolverConfig()), dt, speed))
    return out


@pytest.mark.parametrize("runner", ["graph", "threads"])
def test_members_whose_solves_do_not_fit_together(gpu_lib, runner):
    a, b = _members(), _members()
    dts = [m[1] for m in a]
    if runner == "graph":
        ens = Ensemble([m[0] for m in a])
        ens.step(dts, 1.0, nsteps=2)
        ens.close()
    else:
        step_ensemble([m[0] for m in a], dts, 1.0, nsteps=2, threads=len(a))
    for env, dt, _ in b:
        env.update_gpu(dt, 1.0, nsteps=2)
    for (ea, *_), (eb, *_) in zip(a, b):
        m = ea.sky_mask()
        for k in SKY:
            assert np.isfinite(ea.read(k)[m]).all(), k
            np.testing.assert_array_equal(ea.read(k).view(np.uint32), eb.read(k).view(np.uint32), err_msg=k)
        assert ea.stats()["pcg_iters"] == eb.stats()["pcg_iters"] > 0
    for m in a + b:
        m[0].close()
