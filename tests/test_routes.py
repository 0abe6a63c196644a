"""Which kernel steps a grid, and that the choice does not change its results: the role-specialised kernel takes
the grids of the paired one; grids that the paired kernel does not divide keep the results of the
one-node-per-thread tiled kernel or of the gather kernel, bit for bit."""
import numpy as np
import pytest

from conftest import rel_l2
from test_chunk import params
from test_chunk_order import CHUNK, GATHER, PAIRED, ROLES, TILED, run, step_kernel

pytestmark = pytest.mark.gpu

# NX, NY, NZ and the automatic choice in FP32, 16-bit storage
CHOICES = [(32, 24, 16, ROLES, ROLES), (32, 16, 16, PAIRED, PAIRED), (64, 20, 24, ROLES, ROLES), (64, 12, 24, PAIRED, PAIRED),
           (128, 14, 40, ROLES, ROLES), (128, 8, 16, PAIRED, PAIRED), (256, 11, 24, ROLES, ROLES), (384, 8, 16, PAIRED, PAIRED),
           (32, 20, 24, TILED, TILED), (64, 14, 24, TILED, TILED), (128, 13, 56, TILED, TILED),
           (32, 23, 17, CHUNK, GATHER), (64, 17, 33, CHUNK, GATHER), (33, 24, 16, CHUNK, GATHER)]


@pytest.mark.parametrize("nx,ny,nz,fp32,half", CHOICES)
def test_choice(islbm_lib, nx, ny, nz, fp32, half):
    for prec, want in (("fp32", fp32), ("fp16", half), ("bf16", half), ("fp64", CHUNK)):
        with islbm_lib.Solver(islbm_lib.default_params(**params(nx, ny, nz, precision=prec))) as s:
            assert step_kernel(islbm_lib, s) == want, prec


@pytest.mark.parametrize("prec,tol", [("fp32", 2e-6), ("fp16", 2e-3)])
@pytest.mark.parametrize("nx,ny,nz", [(32, 16, 16), (64, 12, 32), (128, 8, 56), (384, 8, 160)])
def test_paired_grids_match_gather(islbm_lib, prec, tol, nx, ny, nz):
    """The grids that the paired kernel still steps, with the tolerances of the formats."""
    kw = params(nx, ny, nz, precision=prec, init_mode=1, seed=4, les_cs=0.1)
    a = run(islbm_lib, GATHER, [20], kernel=islbm_lib.KERNEL_GATHER, **kw)
    b = run(islbm_lib, PAIRED, [20], **kw)
    assert np.isfinite(a[0]).all()
    assert rel_l2(b[1][0], a[1][0]) <= tol
    assert rel_l2(b[1][1:], a[1][1:]) <= 50*tol


@pytest.mark.parametrize("prec", ["fp32", "fp16"])
@pytest.mark.parametrize("nx,ny,nz", [c[:3] for c in CHOICES if c[3] in (TILED, CHUNK) and c[0] != 33])
def test_undivided_grids_keep_their_results(islbm_lib, prec, nx, ny, nz):
    kw = params(nx, ny, nz, precision=prec, init_mode=1, seed=9, les_cs=0.1)
    fp32, half = [c[3:] for c in CHOICES if c[:3] == (nx, ny, nz)][0]
    auto = fp32 if prec == "fp32" else half
    named = (islbm_lib.KERNEL_TILED_SINGLE, TILED) if auto == TILED else (islbm_lib.KERNEL_GATHER, GATHER)
    a = run(islbm_lib, named[1], [3, 12], kernel=named[0], **kw)
    b = run(islbm_lib, auto, [3, 12], **kw)
    assert np.isfinite(a[0]).all()
    np.testing.assert_array_equal(b[0], a[0])
    np.testing.assert_array_equal(b[1], a[1])
    if auto == TILED:
        np.testing.assert_array_equal(run(islbm_lib, TILED, [3, 12], kernel=islbm_lib.KERNEL_TILED, **kw)[0], a[0])
    else:
        with pytest.raises(islbm_lib.IslbmError):
            islbm_lib.Solver(islbm_lib.default_params(kernel=islbm_lib.KERNEL_TILED, **kw))
