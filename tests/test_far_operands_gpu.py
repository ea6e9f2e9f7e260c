"""Stages with one operand outside the proven range of the shared reciprocals: a transverse velocity or heat flux that is far
below 2^-764 enters the other components nowhere and itself linearly, so that a run with it scaled by 2^-300 or 2^-600 (all
operands in range) and one with it scaled by 2^-900 differ in nothing but its own exponent."""
import numpy as np
import pytest

from vanguard_b200 import workloads as wl

pytestmark = pytest.mark.gpu

FIELDS = {"euler": [2], "mhd": [3, 7], "hpr": [16]}  # MHD: w, and the Bz that it makes


def _start(name, shape):
    ny, nx = shape
    field = 1.0 + 0.5 * np.random.default_rng(5).random(shape)
    if name == "euler":  # v of a run along x alone
        W = wl.sod_1d(nx)
        return W, wl.euler_params(1.4), field[0]
    if name == "mhd":
        W = wl.mhd_vortex_2d(nx, ny, seed=2)
        return W, wl.mhd_params(5.0 / 3.0), field
    W = wl.hpr_smooth_2d(nx, ny, seed=2)
    return W, wl.hpr_params(tau1=5e-3, tau2=5e-3), field


@pytest.mark.parametrize("limiter", [0, 1, 2])
@pytest.mark.parametrize("subcycles", [0, 3])
@pytest.mark.parametrize("name", list(FIELDS))
def test_small_field_scales(gpu, name, subcycles, limiter):
    if name != "hpr" and subcycles:
        pytest.skip("no forcing with this field")
    ny, nx = (1, 2500) if name == "euler" else (37, 53)
    out = []
    for power in (-300, -600, -900):
        W, prm, field = _start(name, (ny, nx))
        W[FIELDS[name][0]] = np.ldexp(field, power)
        with gpu.Solver({"euler": gpu.EULER, "mhd": gpu.MHD, "hpr": gpu.HPR}[name], nx, ny, prm) as s:
            s.upload(W)
            s.run(1.0 / nx, 0.8, steps=4, limiter=limiter, subcycles=subcycles)
            W = s.download()
        f = W[FIELDS[name]].copy()
        W[FIELDS[name]] = 0.0
        out.append((W, np.ldexp(f, -power)))
    assert np.isfinite(out[0][1]).all() and np.abs(out[0][1][0]).max() > 0.05
    for other in out[1:]:
        assert np.array_equal(out[0][0], other[0])
        assert np.array_equal(out[0][1], other[1])
