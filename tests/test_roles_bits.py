"""The role-specialised kernel gives the paired kernel's bits in every storage format: tile edges (heights that its
tiles do not divide, so that the last one overlaps the one before; the smallest heights), two segments,
both ways of copying a plane, the steep hill, whose first wall rows are nearer than half a cell, both BFL
table modes, the channel, LES; the same in a batch of the serving loop."""
import numpy as np
import pytest

from conftest import rel_l2
from test_chunk import params
from test_chunk_order import PAIRED, ROLES, step_kernel

pytestmark = pytest.mark.gpu

GRIDS = [(32, 24, 16), (32, 40, 33), (64, 16, 25), (64, 20, 32), (128, 10, 57), (128, 14, 64), (256, 8, 104), (256, 11, 112)]
OPTS = [dict(les_cs=0.1), dict(alpha=0.73), dict(alpha=0.73, bfl_mode=1, les_cs=0.1), dict(geometry=1)]


def steps(islbm, paired, **kw):
    with islbm.Solver(islbm.default_params(**kw)) as s:
        if paired:
            islbm.check(s._L.islbm_use_paired(s._h))
        assert step_kernel(islbm, s) == (PAIRED if paired else ROLES)
        s.step(2)
        s.step(7)
        f = s.fields()
        return s.populations(), np.stack([f[c] for c in ("rho", "u", "v", "w")])


@pytest.mark.parametrize("prec", ["fp32", "fp16", "bf16"])
@pytest.mark.parametrize("opts", OPTS)
@pytest.mark.parametrize("nx,ny,nz", GRIDS)
def test_same_bits_as_paired(islbm_lib, monkeypatch, nx, ny, nz, opts, prec):
    kw = params(nx, ny, nz, precision=prec, init_mode=1, seed=7, **opts)
    a, b = steps(islbm_lib, True, **kw), steps(islbm_lib, False, **kw)
    assert np.isfinite(a[0]).all()
    np.testing.assert_array_equal(b[0], a[0])
    np.testing.assert_array_equal(b[1], a[1])
    monkeypatch.setenv("ISLBM_PAIR_COPIES", "bulk")
    np.testing.assert_array_equal(steps(islbm_lib, False, **kw)[0], a[0])
    if nz >= 16:
        monkeypatch.setenv("ISLBM_TILED_ZSEGS", "2")
        np.testing.assert_array_equal(steps(islbm_lib, False, **kw)[0], a[0])


@pytest.mark.parametrize("prec,tol", [("fp16", 2e-3), ("bf16", 1e-2)])
def test_near_rows_against_fp64(islbm_lib, prec, tol):
    """The steep hill of the request stream over 300 steps, with the tolerances of the formats."""
    out = {}
    for p in (prec, "fp64"):
        with islbm_lib.Solver(islbm_lib.default_params(**params(32, 64, 48, tau=0.64, precision=p, alpha=0.73))) as s:
            s.step(300)
            f = s.fields()
            out[p] = f["rho"], np.stack([f[c] for c in "uvw"])
    assert rel_l2(out[prec][0], out["fp64"][0]) <= tol
    assert rel_l2(out[prec][1], out["fp64"][1]) <= 50*tol


@pytest.mark.parametrize("prec", ["fp32", "fp16"])
def test_batch_same_bits_as_alone(islbm_lib, prec):
    ps = [islbm_lib.default_params(**params(32, 64, 48, tau=0.64 + 0.002*i, precision=prec, alpha=0.73, init_mode=1, seed=i))
          for i in range(5)]
    with islbm_lib.Server(steps_per_chunk=50) as srv:
        ids = [srv.submit(p, max_steps=120, tol=0.0, keep_fields=True) for p in ps]
        srv.drain()
        got = [srv.fields(i) for i in ids]
    for p, g in zip(ps, got):
        with islbm_lib.Solver(p) as s:
            s.step(120)
            f = s.fields()
        for c in ("rho", "u", "v", "w"):
            np.testing.assert_array_equal(g[c], f[c])
