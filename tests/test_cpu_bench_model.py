"""bench.py's byte models are those of the PCG form that ran, which the profiled stages name: the launches of an
iteration add up to its bytes, no stage has a model of another form, and the one-launch form has none."""
import os
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)

import bench  # noqa: E402


def test_forms_by_stage_names():
    assert bench.plain_form({"pcg_grid": 1, "diffuse": 1}) == "one launch"
    assert bench.plain_form({"pcg_matvec": 1, "pcg_update": 1, "pcg_search": 1}) == "three launches"
    assert bench.plain_form({"pcg_matvec": 1, "pcg_update": 1}) == "matrix-free"


def test_bytes_of_an_iteration():
    launches = {"matrix-free": {"pcg_matvec": 1, "pcg_update": 5 / 4}, "three launches": {"pcg_matvec": 1, "pcg_update": 1, "pcg_search": 1}}
    for form, n in launches.items():
        stages, total = bench.PLAIN_FORMS[form]
        assert set(stages) == set(n) and sum(stages[k] * v for k, v in n.items()) == total
    # the arrays of 4 B a cell: matvec 5 read, 1 written; update 5 read, 2 written; search 3 read, 1 written
    assert bench.PLAIN_FORMS["three launches"] == ({"pcg_matvec": 6 * 4.0, "pcg_update": 7 * 4.0, "pcg_search": 4 * 4.0}, 68.0)
    assert bench.PLAIN_FORMS["one launch"] == ({}, 0.0)


def test_step_bytes_by_form():
    assert bench.plain_step_bytes("matrix-free", 200, 2) == 1734.0 + 50.0 * 200
    assert bench.plain_step_bytes("three launches", 200, 1) == 2534.0 + 68.0 * 200
    assert bench.plain_step_bytes("one launch", 200, 2) == 1734.0


def test_sweeps_per_pass_where_the_two_sweep_kernel_runs():
    import numpy as np
    flat, hill = np.zeros(12, np.int32), np.array([0] * 11 + [1], np.int32)
    assert bench.sweeps_per_pass({"diffuse_depth": 2}, 64, flat) == 2
    assert bench.sweeps_per_pass({"diffuse_depth": 1}, 64, flat) == 1
    assert bench.sweeps_per_pass({"diffuse_depth": 2}, 62, flat) == 1
    assert bench.sweeps_per_pass({"diffuse_depth": 2}, 64, hill) == 1
