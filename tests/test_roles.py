"""The role-specialised step kernel where its tiles, rings and segments have edges: the smallest height
(a tile of 512/NX rows and its halo), heights that the tile's rows do not divide (the last tile overlaps
the one before), the smallest column, one and two segments, both ways of copying a plane.

Against the gather kernel with the tolerances of the tiled kernels (FP32 2e-6 on rho, 50 times that on
the velocity). The two copy paths deliver the same bytes, and the step's sums are added in a fixed order:
runs agree bit for bit."""
import numpy as np
import pytest

from conftest import rel_l2
from test_chunk import params, solve

pytestmark = pytest.mark.gpu

# the last number: steps compared. The reference scheme itself diverges (oracle, hill and channel: max |u|
# above 1e3) within two steps on 128x10x8 and 256x8x16 and within ten on 256x11x24, whose spanwise
# spacing is far below the time step's reach; no two summation orders agree past that.
GRIDS = [(32, 22, 8, 20), (32, 23, 17, 20), (32, 49, 24, 20), (64, 14, 9, 20), (64, 17, 33, 20), (128, 10, 8, 1), (128, 13, 40, 20),
         (256, 8, 16, 1), (256, 11, 24, 3)]


@pytest.mark.parametrize("les", [0.0, 0.1])
@pytest.mark.parametrize("channel", [False, True])
@pytest.mark.parametrize("nx,ny,nz,steps", GRIDS)
def test_edges_match_gather(islbm_lib, monkeypatch, nx, ny, nz, steps, channel, les):
    kw = params(nx, ny, nz, precision="fp32", les_cs=les, mass_interval=7, geometry=int(channel))
    a = solve(islbm_lib, steps, kernel=islbm_lib.KERNEL_GATHER, **kw)
    b = solve(islbm_lib, steps, **kw)
    assert rel_l2(b[0], a[0]) <= 2e-6
    assert rel_l2(b[1], a[1]) <= 50 * 2e-6
    assert abs(b[3] - a[3]) <= 1e-3 * abs(a[3])
    monkeypatch.setenv("ISLBM_PAIR_COPIES", "bulk")
    c = solve(islbm_lib, steps, **kw)
    np.testing.assert_array_equal(c[2], b[2])
    if nz >= 16:
        monkeypatch.setenv("ISLBM_TILED_ZSEGS", "2")
        d = solve(islbm_lib, steps, **kw)
        assert rel_l2(d[2], b[2]) <= 2e-6
