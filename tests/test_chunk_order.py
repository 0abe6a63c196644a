"""The chunk-marching kernel in FP32 adds its terms in the gather kernel's order: the same populations and
fields, bit for bit, on grids without a tiled layout. Widths below, at and above a tile's lanes, odd
counts in every direction, partial tiles, the hill's steep form (wall rows nearer than half a cell),
both BFL table modes, the channel, with and without LES, the controller on."""
import ctypes

import numpy as np
import pytest

from test_chunk import params

pytestmark = pytest.mark.gpu

GATHER, CHUNK, TILED, PAIRED, ROLES = range(5)
GRIDS = [(1, 14, 16), (2, 15, 16), (5, 17, 17), (7, 14, 16), (9, 16, 9), (16, 24, 24), (21, 35, 23), (31, 16, 20), (33, 21, 24),
         (45, 31, 33), (91, 30, 41), (97, 25, 40), (130, 24, 50), (260, 19, 104)]
OPTS = [dict(), dict(les_cs=0.1, alpha=0.9), dict(alpha=0.73), dict(alpha=0.73, bfl_mode=1, les_cs=0.1), dict(geometry=1, les_cs=0.1)]


def step_kernel(islbm, solver):
    k = ctypes.c_int()
    islbm.check(solver._L.islbm_step_kernel(solver._h, ctypes.byref(k)))
    return k.value


def run(islbm, expected, calls, **kw):
    with islbm.Solver(islbm.default_params(**kw)) as s:
        assert step_kernel(islbm, s) == expected
        for n in calls:
            s.step(n)
        f = s.fields()
        return s.populations(), np.stack([f[c] for c in ("rho", "u", "v", "w")]), s.force


@pytest.mark.parametrize("opts", OPTS)
@pytest.mark.parametrize("nx,ny,nz", GRIDS)
def test_fp32_same_bits_as_gather(islbm_lib, nx, ny, nz, opts):
    kw = params(nx, ny, nz, precision="fp32", init_mode=1, seed=5, **opts)
    a = run(islbm_lib, GATHER, [1, 1, 21], kernel=islbm_lib.KERNEL_GATHER, **kw)
    b = run(islbm_lib, CHUNK, [1, 1, 21], **kw)
    assert np.isfinite(a[0]).all()
    np.testing.assert_array_equal(b[0], a[0])
    np.testing.assert_array_equal(b[1], a[1])
    assert abs(b[2] - a[2]) <= 1e-12*abs(a[2])
