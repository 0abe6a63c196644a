"""Reading time means takes no device memory, whatever kind of host buffer it goes to; pageable, pinned and
unaligned buffers get the same bytes."""
import ctypes

import numpy as np
import pytest

from test_chunk import params

pytestmark = pytest.mark.gpu


def test_means_take_no_device_memory(islbm_lib):
    torch = pytest.importorskip("torch")
    nx, ny, nz = 64, 128, 96   # 6.3 MB a quantity
    n = nx*ny*nz
    with islbm_lib.Solver(islbm_lib.default_params(**params(nx, ny, nz, precision="fp32"))) as s:
        s.stats_reset()
        for _ in range(3):
            s.step(2)
            s.stats_accumulate()
        s.sync()
        free = torch.cuda.mem_get_info()[0]
        mean = s.stats_mean("UV")
        s.stats_mean("UV", islbm_lib.LAYOUT_REFERENCE)
        raw = np.zeros(8*n + 8, np.uint8)
        q = islbm_lib.STATS.index("UV")
        islbm_lib.check(s._L.islbm_stats_mean(s._h, q, ctypes.c_void_p(raw.ctypes.data + 4), islbm_lib.LAYOUT_UNIQUE))
        assert torch.cuda.mem_get_info()[0] == free
        np.testing.assert_array_equal(np.frombuffer(raw[4:4 + 8*n].tobytes()), mean.ravel())
        pin = torch.zeros(n, dtype=torch.float64).pin_memory()
        islbm_lib.check(s._L.islbm_stats_mean(s._h, q, ctypes.c_void_p(pin.data_ptr()), islbm_lib.LAYOUT_UNIQUE))
        np.testing.assert_array_equal(pin.numpy(), mean.ravel())
