"""The CFL maximum folded into the last X sweep skips cells that are certainly below what earlier blocks found: on grids of
more blocks than the device holds at once, the run equals the one whose maximum is a pass of its own over every cell."""
import numpy as np
import pytest

import oracle as O
from vanguard_b200 import workloads as wl

pytestmark = pytest.mark.gpu

NX, NY = 1500, 901
CASES = {
    "euler": (O.EULER, lambda: wl.euler_quadrants_2d(NX, NY, seed=1), wl.euler_params(1.4)),
    "euler_pinf": (O.EULER, lambda: wl.euler_quadrants_2d(NX, NY, seed=2), wl.euler_params(1.4, 0.3)),
    "mhd": (O.MHD, lambda: wl.mhd_vortex_2d(NX, NY, seed=1), wl.mhd_params(5.0 / 3.0)),
    "reduced": (O.EULER_REDUCED, lambda: wl.reduced_bubble_2d(NX, NY), wl.reduced_params(1.4, 0.0, 1.67, 0.0)),
}


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("name", list(CASES))
def test_folded_maximum_equals_the_separate_one(gpu, name, mixed):
    model, make, prm = CASES[name]
    W = make()
    if name == "mhd":
        W[2, 400, 700] = 3.0  # one fast cell among slow ones
    out = []
    for separate in (0, 1):
        with gpu.Solver(model, NX, NY, prm, precision=gpu.MIXED if mixed else gpu.FP64) as s:
            s.upload(W)
            s.set_schedule(separate)
            t, it = s.run(1.0 / NX, 0.8, steps=7)
            out.append((t, it, s.download()))
    assert out[0][:2] == out[1][:2]
    assert np.array_equal(out[0][2], out[1][2])
