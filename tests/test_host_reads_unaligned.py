"""Reads into pinned host buffers that do not start at a double's boundary take the copy (a conversion kernel's
stores would be misaligned) and give the same bytes: fields, populations and time means in every format."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["fp64", "fp32", "fp16", "bf16"])
@pytest.mark.parametrize("offset", [1, 4, 12])
def test_unaligned_pinned_reads(islbm_lib, prec, offset):
    torch = pytest.importorskip("torch")
    nx, ny, nz = 7, 15, 17
    n = nx*ny*nz
    vp = ctypes.c_void_p
    with islbm_lib.Solver(islbm_lib.default_params(NX=nx, NY=ny, NZ=nz, Re=60.0, precision=prec)) as s:
        s.stats_reset()
        s.step(3)
        s.stats_accumulate()
        f, pop, mean = s.fields(), s.population(7), s.stats_mean("VV")
        pin = torch.zeros(8*n + 64, dtype=torch.uint8).pin_memory()
        at = vp(pin.data_ptr() + offset)

        def taken():
            raw = pin.numpy()
            assert not raw[:offset].any() and not raw[offset + 8*n:].any()
            return np.frombuffer(raw[offset:offset + 8*n].tobytes()).reshape(nz, ny, nx)

        for i, c in enumerate(("rho", "u", "v", "w")):
            islbm_lib.check(s._L.islbm_fields(s._h, *[at if i == j else None for j in range(4)], islbm_lib.LAYOUT_UNIQUE))
            np.testing.assert_array_equal(taken(), f[c])
        islbm_lib.check(s._L.islbm_get_population(s._h, 7, at, islbm_lib.LAYOUT_UNIQUE))
        np.testing.assert_array_equal(taken(), pop)
        islbm_lib.check(s._L.islbm_stats_mean(s._h, islbm_lib.STATS.index("VV"), at, islbm_lib.LAYOUT_UNIQUE))
        np.testing.assert_array_equal(taken(), mean)
