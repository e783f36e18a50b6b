"""The launch shapes that skt_create gives a grid lie on the side of each rule where that grid measured faster:
6 rows a tile and the x pass's longer runs at 256x128x256 and 320x128x320, 14 rows at 320x160x320 (nx, ny, nz), and
the larger count of blocks above."""
import pytest

from skewtcloudsim_gb300 import Environment

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,rows,x_bps", [
    ((64, 32, 64), 6, 8), ((256, 128, 256), 6, 8), ((320, 128, 320), 6, 8), ((320, 160, 320), 14, 8), ((512, 128, 512), 14, 16),
])
def test_default_shapes(gpu_lib, shape, rows, x_bps):
    env = Environment(*shape, 100.0)
    t = env.get_tuning()
    env.close()
    assert (t["diffuse_depth"], t["diffuse_rows"], t["ppm_x_bps"]) == (2, rows, x_bps)
