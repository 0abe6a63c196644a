"""Steps captured from a solve's stream into a CUDA graph and replayed: the same bytes as the steps launched one
after the other. The captured number of steps is even (the two population buffers change places) and a
multiple of the controller's interval. Grids whose launches fill the GPU with one block per SM, and small ones."""
import numpy as np
import pytest

from test_chunk import params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,nx,ny,nz", [("fp32", 128, 64, 96), ("fp16", 256, 64, 104), ("fp32", 32, 64, 48), ("fp32", 384, 32, 160),
                                           ("fp64", 16, 24, 24), ("fp32", 33, 40, 24)])
def test_replayed_steps(islbm_lib, prec, nx, ny, nz):
    torch = pytest.importorskip("torch")
    kw = params(nx, ny, nz, precision=prec, init_mode=1, seed=2, les_cs=0.1)
    with islbm_lib.Solver(islbm_lib.default_params(**kw)) as a, islbm_lib.Solver(islbm_lib.default_params(**kw)) as b:
        a.step(60)
        b.step(10)
        b.sync()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=torch.cuda.ExternalStream(b.stream_handle())):
            b.step(10)
        with torch.cuda.stream(torch.cuda.ExternalStream(b.stream_handle())):
            for _ in range(5):
                g.replay()
        b.sync()
        f = a.populations()
        assert np.isfinite(f).all()
        np.testing.assert_array_equal(b.populations(), f)
        assert abs(b.force - a.force) <= 1e-12*abs(a.force)
