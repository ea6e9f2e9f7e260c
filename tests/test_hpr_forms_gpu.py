"""The HPR model's form without p_inf against its general form at p_inf = 0: fluxes and source, every bit but the signs of zeros
(a product in one operation with the 0.0 that it is added to keeps the sign of what underflows), on states whose products underflow
and whose sums vanish."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from vanguard_b200 import workloads as wl

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")


@pytest.fixture(scope="module")
def probe(gpu, tmp_path_factory):
    so = tmp_path_factory.mktemp("probe") / "hpr_forms_probe.so"
    env = {k: v for k, v in os.environ.items() if k not in ("CXX", "CC")}
    # the flags of the exact form's units (vanguard_b200/build.py)
    subprocess.run([NVCC, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-fmad=false", "-shared",
                    "-Xcompiler", "-fPIC", "-ccbin", "g++", "-o", str(so), os.path.join(HERE, "device", "hpr_forms_probe.cu")],
                   check=True, env=env)
    return ctypes.CDLL(str(so))


def test_forms_agree_but_for_the_sign_of_zero(probe):
    import torch
    rng = np.random.default_rng(1)
    n = 1 << 20
    odd = np.array([0.0, -0.0, 1e-200, -1e-200, 1e-150, -1e-150, 1e-170, -1e-170, 1e-320, 1e-30, -1.0, 0.5])
    U = np.zeros((17, n))
    U[0] = rng.choice([1.0, 0.7, 2.0 - 2.0 ** -52], n)
    U[1] = rng.uniform(3.0, 9.0, n)
    U[2:11] = rng.choice(odd, (9, n))
    for d in (2, 6, 10):  # mostly a distortion near the identity, whose determinant is positive
        keep = rng.random(n) < 0.8
        U[d] = np.where(keep, rng.choice([1.0, 1.1, 0.9], n), U[d])
    U[11:17] = rng.choice(odd, (6, n))
    prm = np.zeros(48)  # the device's parameter block, its last slot 1 / (gamma - 1)
    p = np.asarray(wl.hpr_params(), dtype=np.float64)
    prm[:len(p)] = p
    prm[47] = 1.0 / (p[0] - 1.0)
    dev = [torch.from_numpy(x).cuda() for x in (U, prm)]
    out = torch.empty((3, 51, n), dtype=torch.float64, device="cuda")
    ok = torch.empty(n, dtype=torch.uint8, device="cuda")
    ptr = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    assert probe.probe_forms(ptr(dev[0]), ptr(dev[1]), ctypes.c_long(n), ptr(out), ptr(ok)) == 0
    g, plain, shared = out.cpu().numpy()
    ok = ok.cpu().numpy() == 1
    assert ok.mean() > 0.005
    same = lambda x, y: (x == y) | (np.isnan(x) & np.isnan(y))  # noqa: E731
    assert same(g, plain).all(0).all(), np.flatnonzero(~same(g, plain).all(1))
    assert same(g, shared).all(0)[ok].all()
