"""Reads into pinned host buffers (written by the conversion kernels directly) give the same bytes as reads
into pageable ones (converted on the device, then copied): fields, populations and time means, every
storage format, an odd node count, a buffer inside a larger pinned allocation."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["fp64", "fp32", "fp16", "bf16"])
@pytest.mark.parametrize("nx,ny,nz", [(7, 15, 17), (32, 32, 24)])
def test_pinned_and_pageable_reads_agree(islbm_lib, prec, nx, ny, nz):
    torch = pytest.importorskip("torch")
    min_size = (3.036 - 1.0) / nz * 0.6
    p = islbm_lib.default_params(NX=nx, NY=ny, NZ=nz, Re=3 * 0.05 / (0.5 * min_size), precision=prec)
    n = nx * ny * nz
    vp = ctypes.c_void_p
    with islbm_lib.Solver(p) as s:
        s.stats_reset()
        s.step(3)
        s.stats_accumulate()
        f, pop, mean = s.fields(), s.population(7), s.stats_mean("VV")
        pin = torch.zeros(n + 3, dtype=torch.float64).pin_memory()
        out = pin[1:n + 1]
        read = lambda: out.numpy().reshape(nz, ny, nx).copy()
        for i, c in enumerate(("rho", "u", "v", "w")):
            args = [vp(out.data_ptr()) if i == j else None for j in range(4)]
            islbm_lib.check(s._L.islbm_fields(s._h, *args, islbm_lib.LAYOUT_UNIQUE))
            np.testing.assert_array_equal(read(), f[c])
        islbm_lib.check(s._L.islbm_get_population(s._h, 7, vp(out.data_ptr()), islbm_lib.LAYOUT_UNIQUE))
        np.testing.assert_array_equal(read(), pop)
        islbm_lib.check(s._L.islbm_stats_mean(s._h, islbm_lib.STATS.index("VV"), vp(out.data_ptr()), islbm_lib.LAYOUT_UNIQUE))
        np.testing.assert_array_equal(read(), mean)
        assert pin[0] == 0 and (pin[n + 1:] == 0).all()   # nothing beside the buffer
