"""The counts that size launches (skt_rules.hpp, compiled for the host) on the largest grids that skt_create
accepts, nx*ny*nz < 2^31: the blocks of a grid, and the far sides' faces, of which there are more than 2^31 where
two dimensions are 1 and 2."""
import ctypes
import subprocess

import pytest

from skewtcloudsim_gb300 import build


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    d = tmp_path_factory.mktemp("rules")
    (d / "rules.cpp").write_text('#include "skt_rules.hpp"\nextern "C" int blocks(int n, int p) { return skt::blocks_for(n, p); }\n'
                                 'extern "C" unsigned faces(int x, int y, int z) { return skt::far_faces(x, y, z); }\n')
    so = str(d / "rules.so")
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-I", build.CSRC, str(d / "rules.cpp"), "-o", so], check=True)
    lib = ctypes.CDLL(so)
    lib.faces.restype = ctypes.c_uint
    return lib


@pytest.mark.parametrize("per", [1024, 2048, 4096, 7168])
def test_blocks(rules, per):
    for n in (1, per - 1, per, per + 1, 10 ** 6, 2 ** 31 - per, 2 ** 31 - per + 1, 2 ** 31 - 1):
        assert rules.blocks(n, per) == -(-n // per), n


@pytest.mark.parametrize("x,y,z", [(1, 2, 1), (32, 32, 32), (512, 256, 512), (2 ** 30 - 1, 2, 1), (1, 2, 2 ** 30 - 1), (46340, 2, 23170), (1, 2 ** 30, 1),
                                   (2, 32768, 32767)])
def test_far_faces(rules, x, y, z):
    assert x * y * z < 2 ** 31
    assert rules.faces(x, y, z) == x * y + x * z + y * z < 2 ** 32
