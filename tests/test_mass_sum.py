"""The mass sum of the role-specialised kernel on a column marched as one segment: FP32 partial sums of at most 16
densities per lane, then FP64. The bound is the worst case of such sums: adding the k-th density of about 1
rounds by at most half a unit of the last place of k, in all 6e-6 over 16 terms of a lane; the two lanes of
a pair and their sum make 1.3e-5 for 32 densities, 4.1e-7 of each. The state is uniform, so that every
thread rounds alike (sums of 96 terms lose 8e-7 of each)."""
import numpy as np
import pytest

from test_chunk import params
from test_chunk_order import ROLES, step_kernel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ulps", [0, 3, 5, 12, 21])
def test_mass_of_a_uniform_state(islbm_lib, monkeypatch, ulps):
    monkeypatch.setenv("ISLBM_TILED_ZSEGS", "1")
    nx, ny, nz = 32, 64, 96
    w = np.array([1/3] + [1/18]*6 + [1/36]*12)
    f = np.broadcast_to(w[:, None, None, None]*(1.0 + ulps*2.0**-23), (19, nz, ny, nx)).copy()
    p = islbm_lib.default_params(**dict(params(nx, ny, nz, precision="fp32", geometry=1, mass_interval=1), NDTFRC=1000))
    with islbm_lib.Solver(p) as s:
        assert step_kernel(islbm_lib, s) == ROLES
        s.set_populations(f)
        s.force = 0.0
        s.step(1)
        rho = s.fields()["rho"]
        got = s.scalars()["rho_modify"]
    n = rho.size
    assert abs(got - (n - rho.sum())/n) <= 4.1e-7
