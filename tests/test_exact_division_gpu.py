"""Sweeps of the exact form where the shared-reciprocal division is at its edges: divisors whose upper significand bits
are all ones, operands that are zero, subnormal or far from 1 (the stages that go through the compiler's division
again), beside ordinary cells, bit for bit against the oracle."""
import numpy as np
import pytest

import oracle as O
from vanguard_b200 import workloads as wl

pytestmark = pytest.mark.gpu

DENSITIES = [2.0 - 2.0 ** -52, 2.0 - 2.0 ** -20, 2.0 - 2.0 ** -19, 1.0, 1.0 + 2.0 ** -52, 2.0 ** -250, 2.0 ** -260, 2.0 ** 250,
             2.0 ** 258, 0.7]
VELOCITIES = [0.0, -0.0, 5e-324, 1e-310, -1e-200, 1e-153, 3e-17, 0.3, -1.5]


def _edges(W, density, velocities, rng):
    """Every combination of the edge densities and velocities scattered over the grid among ordinary cells."""
    flat = [W[k].reshape(-1) for k in range(W.shape[0])]
    cells = rng.permutation(flat[0].size)
    for n, c in enumerate(cells[:flat[0].size // 2]):
        for k in density:
            flat[k][c] = DENSITIES[n % len(DENSITIES)]
        for i, k in enumerate(velocities):
            flat[k][c] = VELOCITIES[(n // len(DENSITIES) + 3 * i) % len(VELOCITIES)]
    return W


CASES = {
    "euler": (O.EULER, lambda nx, ny: wl.euler_quadrants_2d(nx, ny, seed=1), wl.euler_params(1.4), [0], [1, 2]),
    "mhd": (O.MHD, lambda nx, ny: wl.mhd_vortex_2d(nx, ny, seed=1), wl.mhd_params(5.0 / 3.0), [0], [1, 2]),
    "hpr": (O.HPR, lambda nx, ny: wl.hpr_smooth_2d(nx, ny, seed=1), wl.hpr_params(), [0], [11, 12, 14]),
}


@pytest.mark.parametrize("limiter", [0, 1, 2])
@pytest.mark.parametrize("axis", [0, 1])
@pytest.mark.parametrize("name", list(CASES))
def test_sweep_at_the_edges_of_the_range(gpu, oracle_lib, name, axis, limiter):
    model, make, prm, density, velocities = CASES[name]
    nx, ny = 150, 70
    W = _edges(make(nx, ny), density, velocities, np.random.default_rng(3 + limiter))
    ref = W.copy()
    with np.errstate(all="ignore"):
        O.sweep(model, ref, axis, 1.0 / nx, 1e-4, limiter=limiter, params=prm)
    with gpu.Solver(model, nx, ny, prm) as s:
        s.upload(W)
        s.sweep(axis, 1.0 / nx, 1e-4, limiter=limiter)
        out = s.download()
    finite = np.isfinite(ref).all(0)
    assert finite.sum() > nx * ny // 4
    assert np.array_equal(np.isfinite(out).all(0), finite)
    assert np.array_equal(out[:, finite], ref[:, finite])


@pytest.mark.parametrize("nx", [40, 3000])  # the one-launch loop and the graph-driven one
def test_run_1d_at_the_edges_of_the_range(gpu, oracle_lib, nx):
    W = wl.sod_1d(nx)
    W[0, ::7] = 2.0 - 2.0 ** -52
    W[1, ::3] = 1e-310
    W[1, 1::5] = -1e-170
    prm = wl.euler_params(1.4)
    ref = W.copy()
    O.run(O.EULER, ref, 1.0 / nx, 0.8, steps=8, limiter=0, params=prm)
    with gpu.Solver(gpu.EULER, nx, 1, prm) as s:
        s.upload(W)
        s.run(1.0 / nx, 0.8, steps=8, limiter=0)
        assert np.array_equal(s.download(), ref)


@pytest.mark.parametrize("name", ["reduced", "mhd_reduced"])
def test_two_materials_at_the_edges_of_the_range(gpu, oracle_lib, name):
    nx, ny = 70, 45
    if name == "reduced":
        model, W, prm, vel = O.EULER_REDUCED, wl.reduced_bubble_2d(nx, ny), wl.reduced_params(1.4, 0.0, 1.67, 0.0), (1, 2)
        rho = (4, 5)
    else:
        model, W, prm, vel = O.MHD_REDUCED, wl.mhd_reduced_dumbser_2d(nx, ny), wl.mhd_reduced_params(1.4, 0.0, 1.67, 0.0), (1, 2, 3)
        rho = (4, 5)
    flat = [W[k].reshape(-1) for k in range(W.shape[0])]
    for k in rho:
        flat[k][::11] = 2.0 - 2.0 ** -52
    for k in vel:
        flat[k][k::7] = 1e-310
        flat[k][k::13] = -1e-170
    ref = W.copy()
    sub = 1 if name == "mhd_reduced" else 0
    O.run_two_material(model, ref, 1.0 / nx, 0.8, steps=4, limiter=1, params=prm, reinit=0, subcycles=sub)
    with gpu.Solver(model, nx, ny, prm) as s:
        s.upload(W)
        s.run(1.0 / nx, 0.8, steps=4, limiter=1, subcycles=sub)
        assert np.array_equal(s.download(), ref)
