"""Batches of different kernels in one server, with the same storage format, width and number of work items: each is
stepped with a block count of its own kernel, and gives the solve's results bit for bit."""
import numpy as np
import pytest

from test_chunk import params

pytestmark = pytest.mark.gpu


def test_kinds_in_turn(islbm_lib):
    # NX 32: 16 rows step with the paired kernel, 64 with the role-specialised one, 20 with the tiled one
    grids = [(32, 16, 16), (32, 64, 48), (32, 20, 24), (32, 16, 16), (32, 64, 48)]
    ps = [islbm_lib.default_params(**params(*g, precision="fp16", init_mode=1, seed=i)) for i, g in enumerate(grids)]
    with islbm_lib.Server(steps_per_chunk=20) as srv:
        for p in ps:   # one after the other, then together
            i = srv.submit(p, max_steps=30, tol=0.0, keep_fields=True)
            srv.drain()
            check(islbm_lib, p, srv.fields(i))
        ids = [srv.submit(p, max_steps=30, tol=0.0, keep_fields=True) for p in ps]
        srv.drain()
        for p, i in zip(ps, ids):
            check(islbm_lib, p, srv.fields(i))


def check(islbm, p, got):
    with islbm.Solver(p) as s:
        s.step(30)
        f = s.fields()
    for c in ("rho", "u", "v", "w"):
        assert np.isfinite(f[c]).all()
        np.testing.assert_array_equal(got[c], f[c])
