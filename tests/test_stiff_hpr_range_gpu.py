"""Stiff relaxation where the Newton step's operands leave the shared reciprocals' range: rates so small that its residuals
are below 2^-511 go through the compiler's division; beside them rates on either side of that."""
import numpy as np
import pytest

import oracle as O
from vanguard_b200 import workloads as wl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tau1", [1e-3, 1e150, 1e157, 1e200, 1e290])
def test_relaxation_at_the_edge_of_the_range(gpu, oracle_lib, tau1):
    n = 24
    W = wl.hpr_smooth_2d(n, n, seed=4)
    rng = np.random.default_rng(4)
    W[2:11] += 0.05 * rng.standard_normal((9, n, n))
    W[14:17] = 0.1 * rng.standard_normal((3, n, n))
    prm = wl.hpr_params(tau1=tau1, tau2=1e-3)
    ref = W.copy()
    O.run(O.HPR, ref, 1.0 / n, 0.8, steps=2, limiter=0, params=prm, subcycles=-1)
    assert np.isfinite(ref).all()
    with gpu.Solver(gpu.HPR, n, n, prm) as s:
        s.upload(W)
        s.run(1.0 / n, 0.8, steps=2, limiter=0, stiff=True)
        out = s.download()
    # exp, log and pow of CUDA and glibc may differ in the last place
    assert (np.abs(out - ref) / np.maximum(np.abs(ref), 1e-3)).max() <= 1e-10
