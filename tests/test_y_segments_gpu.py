"""Y sweeps whose row segments are sized for the device: grids from two rows up, across the widths of a block and rows that
the segments do not divide, bit for bit against the oracle."""
import numpy as np
import pytest

import oracle as O
from vanguard_b200 import workloads as wl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx", [3, 64, 131])
@pytest.mark.parametrize("ny", [2, 3, 5, 17, 63, 260])
def test_euler_rows(gpu, oracle_lib, nx, ny):
    W = wl.euler_quadrants_2d(nx, ny, seed=ny)
    prm = wl.euler_params(1.4)
    ref = W.copy()
    O.run(O.EULER, ref, 1.0 / nx, 0.8, steps=3, limiter=0, params=prm)
    with gpu.Solver(gpu.EULER, nx, ny, prm) as s:
        s.upload(W)
        s.run(1.0 / nx, 0.8, steps=3, limiter=0)
        assert np.array_equal(s.download(), ref)


@pytest.mark.parametrize("ny", [2, 7, 130])
def test_mhd_rows_periodic(gpu, oracle_lib, ny):
    nx = 70
    W = wl.mhd_vortex_2d(nx, ny, seed=ny)
    prm = wl.mhd_params(5.0 / 3.0)
    ref = W.copy()
    O.run(O.MHD, ref, 1.0 / nx, 0.8, steps=3, limiter=1, params=prm, bc=1)
    with gpu.Solver(gpu.MHD, nx, ny, prm, boundary=gpu.PERIODIC) as s:
        s.upload(W)
        s.run(1.0 / nx, 0.8, steps=3, limiter=1)
        assert np.array_equal(s.download(), ref)
