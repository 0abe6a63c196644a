"""Step kernels that start before the previous step has ended (dependent launches): many steps in one call
give the same bytes as the same steps one by one with a synchronisation after each, where no two steps
are resident at the same time. Grids of a few blocks, so that several steps would fit on the GPU at
once, read the buffer that the step before last read through the same L1 caches."""
import numpy as np
import pytest

from test_chunk import params

pytestmark = pytest.mark.gpu

# chunk-marching kernel (FP64; FP32 without a tiled layout) and role-specialised kernel
CASES = [("fp64", 8, 16, 16, 0.0), ("fp64", 16, 24, 24, 0.1), ("fp64", 33, 21, 24, 0.0), ("fp32", 9, 16, 16, 0.0),
         ("fp32", 33, 21, 24, 0.1), ("fp32", 32, 24, 16, 0.0), ("fp16", 64, 16, 24, 0.1)]


@pytest.mark.parametrize("prec,nx,ny,nz,les", CASES)
def test_chains_of_steps_match_single_steps(islbm_lib, prec, nx, ny, nz, les):
    kw = params(nx, ny, nz, precision=prec, les_cs=les, init_mode=1, seed=3)
    with islbm_lib.Solver(islbm_lib.default_params(**kw)) as a, islbm_lib.Solver(islbm_lib.default_params(**kw)) as b:
        for _ in range(60):
            a.step(1)
            a.sync()
        b.step(60)
        b.sync()
        fa, fb = a.populations(), b.populations()
        assert np.isfinite(fa).all()
        np.testing.assert_array_equal(fa, fb)
        for _ in range(5):
            b.step(200)
            for _ in range(200):
                a.step(1)
                a.sync()
            np.testing.assert_array_equal(a.populations(), b.populations())
