"""FP64 fields and time means go to any host buffer, also to one that is pinned in part or in several pieces (which
a plain copy refuses)."""
import ctypes

import numpy as np
import pytest

from test_chunk import params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pieces", ["front", "back", "both"])
@pytest.mark.parametrize("prec", ["fp64", "fp32"])
def test_partly_pinned_buffers(islbm_lib, prec, pieces):
    cu = ctypes.CDLL("libcuda.so.1")
    nx, ny, nz = 32, 64, 48
    n, vp = nx*ny*nz, ctypes.c_void_p
    with islbm_lib.Solver(islbm_lib.default_params(**params(nx, ny, nz, precision=prec))) as s:
        s.stats_reset()
        s.step(2)
        s.stats_accumulate()
        v, mean = s.fields()["v"], s.stats_mean("VV")
        buf = np.zeros(n + 1024)
        at = (buf.ctypes.data + 4095)//4096*4096
        half = 8*n//2//4096*4096
        out = np.ctypeslib.as_array(ctypes.cast(at, ctypes.POINTER(ctypes.c_double)), (nz, ny, nx))
        parts = ([(at, half)] if pieces != "back" else []) + ([(at + half, 8*n - half)] if pieces != "front" else [])
        for a, size in parts:
            assert cu.cuMemHostRegister_v2(vp(a), ctypes.c_size_t(size), 2) == 0
        try:
            if prec == "fp64":
                islbm_lib.check(s._L.islbm_fields(s._h, None, None, vp(at), None, islbm_lib.LAYOUT_UNIQUE))
                np.testing.assert_array_equal(out, v)
                out[:] = 0
            islbm_lib.check(s._L.islbm_stats_mean(s._h, islbm_lib.STATS.index("VV"), vp(at), islbm_lib.LAYOUT_UNIQUE))
            np.testing.assert_array_equal(out, mean)
        finally:
            for a, _ in parts:
                cu.cuMemHostUnregister(vp(a))
