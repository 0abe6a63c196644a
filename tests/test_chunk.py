"""The chunk-marching step kernel (FP64 on every grid, FP32 on grids without a tiled layout; the 16-bit
formats keep the gather kernel there) where its tiles, chunks and segments have edges: widths below, at
and above the 32 lanes of a tile, odd counts in every direction, the smallest column, partial tiles, both
BFL table modes.

FP64 against the oracle: both evaluate the same sums in another order; a step's relative rounding
difference is a few 1e-16 and grows at most in proportion to the steps here, so 1e-12 holds. The
other formats against the gather kernel, as the tiled kernels are (FP32 2e-6 on rho, 50 times that on
the velocity; FP16 and BF16 2e-3 and 1e-2)."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


def params(nx, ny, nz, tau=1.0, **kw):
    min_size = (3.036 - 1.0) / nz * 0.6
    return dict(NX=nx, NY=ny, NZ=nz, Re=3.0 * 0.05 / ((tau - 0.5) * min_size), Uref=0.05, NDTFRC=10, **kw)


def solve(islbm, steps, **kw):
    with islbm.Solver(islbm.default_params(**kw)) as s:
        s.step(steps)
        f = s.fields()
        return f["rho"], np.stack([f[c] for c in "uvw"]), s.populations(), s.force


GRIDS = [(1, 14, 16), (2, 15, 16), (5, 17, 17), (9, 16, 8), (16, 24, 24), (21, 35, 23), (31, 16, 20), (32, 20, 31), (33, 21, 24),
         (45, 31, 33), (64, 33, 29), (97, 25, 40)]


@pytest.mark.parametrize("nx,ny,nz", GRIDS)
def test_fp64_vs_oracle(islbm_lib, oracle_mod, nx, ny, nz):
    opts = {0: dict(les_cs=0.1, mass_interval=7), 1: dict(bfl_mode=1), 2: dict(alpha=0.9)}[nx % 3]
    kw = params(nx, ny, nz, precision="fp64", **opts)
    steps = 23
    rho, vel, f, force = solve(islbm_lib, steps, **kw)
    if nx < 3:
        # the oracle keeps the reference's ghost columns, whose copies are periodic only for three
        # unique columns or more: the gather kernel wraps by index on any width
        want = solve(islbm_lib, steps, kernel=islbm_lib.KERNEL_GATHER, **kw)
        assert rel_l2(rho, want[0]) <= 1e-12 and rel_l2(vel, want[1]) <= 1e-12 and rel_l2(f, want[2]) <= 1e-12
        return
    o = oracle_mod.Oracle(nx, ny, nz, re=kw["Re"], ndtfrc=10, **opts)
    o.step(steps)
    assert rel_l2(rho, o.unique(o.get("rho"))) <= 1e-12
    assert rel_l2(vel, np.stack([o.unique(o.get(c)) for c in "uvw"])) <= 1e-12
    assert rel_l2(f, np.stack([o.unique(o.get("f", q)) for q in range(19)])) <= 1e-12
    assert abs(force - o.force) <= 1e-12 * abs(o.force)


@pytest.mark.parametrize("prec,tol", [("fp32", 2e-6), ("fp16", 2e-3), ("bf16", 1e-2)])
@pytest.mark.parametrize("nx,ny,nz", [(7, 14, 16), (33, 21, 24), (91, 30, 41), (128, 37, 40), (130, 24, 50)])
def test_formats_match_gather(islbm_lib, prec, tol, nx, ny, nz):
    kw = params(nx, ny, nz, precision=prec, les_cs=0.1, mass_interval=7)
    a = solve(islbm_lib, 20, kernel=islbm_lib.KERNEL_GATHER, **kw)
    b = solve(islbm_lib, 20, **kw)
    assert rel_l2(b[0], a[0]) <= tol
    assert rel_l2(b[1], a[1]) <= 50 * tol
    assert abs(b[3] - a[3]) <= 1e-3 * abs(a[3])
