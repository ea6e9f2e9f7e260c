"""The CFL maximum folded into the last X sweep, whose bound skips most cells, for MHD with all nine planes: transverse velocity
and field components, one cell whose speed is in them, and unphysical cells beside it."""
import numpy as np
import pytest

from vanguard_b200 import workloads as wl

pytestmark = pytest.mark.gpu

NX, NY = 1500, 901


@pytest.mark.parametrize("p_inf", [0.0, 0.2])
@pytest.mark.parametrize("mixed", [False, True])
def test_folded_maximum_equals_the_separate_one(gpu, mixed, p_inf):
    W = wl.mhd_vortex_2d(NX, NY, seed=4)
    rng = np.random.default_rng(4)
    W[3] = 0.3 * rng.standard_normal((NY, NX))
    W[7] = 0.4 * rng.standard_normal((NY, NX))
    W[7, 400, 700] = 9.0  # the fastest cell, by its transverse field
    W[4, 300, 200:203] = -1e-3  # negative pressures among the cells that the bound looks at
    out = []
    for separate in (0, 1):
        with gpu.Solver(gpu.MHD, NX, NY, wl.mhd_params(5.0 / 3.0, p_inf), precision=gpu.MIXED if mixed else gpu.FP64,
                        boundary=gpu.PERIODIC) as s:
            s.upload(W)
            s.set_schedule(separate)
            t, it = s.run(1.0 / NX, 0.8, steps=6, limiter=1, allow_nan=True)
            out.append((t, it, s.download()))
    assert out[0][:2] == out[1][:2]
    assert np.array_equal(out[0][2], out[1][2], equal_nan=True)
