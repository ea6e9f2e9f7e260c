"""Runs of tiles per block in the batch's step and reverse kernels: batches of fewer tiles than the device holds blocks, a few
more, and several rounds, whose runs begin and end inside instances."""
import numpy as np
import pytest

import oracle as O
from vanguard_b200 import workloads as wl

pytestmark = pytest.mark.gpu

CFL = 0.8


def _steps(gpu, ncell, gamma, W, target, steps):
    with gpu.Batch(ncell, 1.0 / ncell, gamma) as b:
        b.upload(W)
        dts = b.run(CFL, steps)
        out = b.download()
        b.upload(W)
        _, g, gg, _, _ = b.gradient(target, CFL, steps, checkpoints=2)
    return out, dts, g, gg


# tiles of 124 cells (forward) and 118 (reverse); a B200 holds 592 reverse and 740 forward blocks
@pytest.mark.parametrize("k", [3, 197, 198, 247, 249, 600])
def test_instances_do_not_depend_on_the_runs(gpu, oracle_lib, k):
    rng = np.random.default_rng(k)
    ncell = rng.integers(250, 355, k)  # three tiles each, forward and reverse
    theta = np.stack([rng.uniform(lo, hi, k) for lo, hi in ((0.1, 2.0), (-1.0, 1.0), (0.1, 10.0)) * 2], 1)
    W = wl.batch_planes(ncell, theta)
    W[[0, 4]] *= 1.0 + 0.01 * rng.standard_normal((2, W.shape[1]))
    gamma, target = rng.uniform(1.2, 1.67, k), rng.uniform(0.1, 2.0, W.shape[1])
    steps = 7
    out, dts, g, gg = _steps(gpu, ncell, gamma, W, target, steps)
    first = np.concatenate([[0], np.cumsum(ncell)])
    for i in sorted({0, 1, k // 2, k - 2, k - 1}):
        c = slice(first[i], first[i + 1])
        alone = _steps(gpu, ncell[i:i + 1], gamma[i:i + 1], np.ascontiguousarray(W[:, c]), target[c].copy(), steps)
        for a, b in zip((out[:, c], dts[i:i + 1], g[:, c], gg[i:i + 1]), alone):
            assert np.array_equal(a, b)
    # every cell of every instance against the oracle
    for i in range(k) if k <= 3 else rng.integers(0, k, 20):
        c = slice(first[i], first[i + 1])
        ref = np.ascontiguousarray(W[:, c])
        O.run(O.EULER, ref, 1.0 / ncell[i], CFL, steps=steps, limiter=0, params=wl.euler_params(gamma[i]))
        assert np.array_equal(out[:, c], ref)
