"""The two forms of the batch's step kernel and the shared-reciprocal division of its adjoint, at the edges of their ranges."""
import numpy as np
import pytest

from oracle import tangent
from vanguard_b200 import workloads as wl

pytestmark = pytest.mark.gpu

CFL = 0.8


def _batch(ncell, seed):
    rng = np.random.default_rng(seed)
    k = len(ncell)
    theta = np.stack([rng.uniform(lo, hi, k) for lo, hi in ((0.1, 2.0), (-1.0, 1.0), (0.1, 10.0)) * 2], 1)
    W = wl.batch_planes(ncell, theta)
    W[[0, 4]] *= 1.0 + 0.01 * rng.standard_normal((2, W.shape[1]))  # no ties, not all slopes floored
    W[1] += 0.01 * rng.standard_normal(W.shape[1])
    return rng.uniform(1.2, 1.67, k), W, rng.uniform(0.1, 2.0, W.shape[1])


@pytest.mark.parametrize("limiter", [0, 1, 2])
def test_batch_without_p_inf_equals_the_general_form(gpu, limiter):
    """One more instance with p_inf > 0 sends the batch to the general kernel: the others keep every bit."""
    ncell = np.array([2, 3, 126, 127, 128, 400, 50])
    gamma, W, _ = _batch(ncell, limiter)
    W[1, ::9] = 0.0
    W[1, 4::31] = 1e-310
    W[0, 5::17] = 2.0 - 2.0 ** -52
    n = int(ncell[:-1].sum())
    out = []
    for last in (0.0, 0.3):
        p_inf = np.zeros(len(ncell))
        p_inf[-1] = last
        with gpu.Batch(ncell, 1.0 / ncell, gamma, p_inf) as b:
            b.upload(W)
            dts = b.run(CFL, 25, limiter=limiter)
            out.append((b.download()[:, :n], dts[:-1]))
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])


# ordinary states; a bias that the shared form covers, and one that it leaves to the compiler's division; divisors next to a
# power of two beside subnormal and zero velocities; pressures whose energies are past the proven range (2^513)
@pytest.mark.parametrize("limiter", [0, 1, 2])
@pytest.mark.parametrize("edge", ["bias", "wide_bias", "operands", "range"])
def test_adjoint_at_the_edges_of_the_range(gpu, edge, limiter):
    ncell = np.array([2, 19, 33])
    gamma, W, target = _batch(ncell, 20 + limiter)
    bias = {"bias": 0.4, "wide_bias": 1.2}.get(edge, 0.0)
    if edge == "operands":
        W[0, ::5] = 2.0 - 2.0 ** -52
        W[1, ::4] = 0.0
        W[1, 1::7] = -1e-310
    elif edge == "range":
        W[4] *= 1e160  # a gas of sound speeds about 1e80: velocities of that order keep it in the same regime
        W[1] *= 1e80
    steps = 8
    with gpu.Batch(ncell, 1.0 / ncell, gamma) as b:
        b.upload(W)
        L, G, gg, _, _ = b.gradient(target, CFL, steps, bias=bias, limiter=limiter, checkpoints=3)
    Lt, Gt, ggt = tangent.gradient(ncell, 1.0 / ncell, gamma, W, target, CFL, steps, bias, limiter)
    assert abs(L - Lt) <= 1e-12 * Lt
    # round-off of a few hundred operations a step: 1e-9 of each plane's largest component, as for ordinary states
    for v in (0, 1, 4):
        assert np.abs(G[v] - Gt[v]).max() <= 1e-9 * np.abs(Gt[v]).max()
    assert np.allclose(gg, ggt, rtol=1e-9, atol=1e-9 * np.abs(ggt).max())
