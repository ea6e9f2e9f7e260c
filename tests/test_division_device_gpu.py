"""The division of exact_div.cuh on the device, quotient by quotient, against the host's IEEE division: random pairs, dividends
next to the midpoints between two quotients, divisors just below 2, the edges of the range flags, and operands outside them."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")


@pytest.fixture(scope="module")
def probe(gpu, tmp_path_factory):
    so = tmp_path_factory.mktemp("probe") / "division_probe.so"
    env = {k: v for k, v in os.environ.items() if k not in ("CXX", "CC")}
    # the flags of the exact form's units (vanguard_b200/build.py)
    subprocess.run([NVCC, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-fmad=false", "-shared",
                    "-Xcompiler", "-fPIC", "-ccbin", "g++", "-o", str(so), os.path.join(HERE, "device", "division_probe.cu")],
                   check=True, env=env)
    return ctypes.CDLL(str(so))


def _call(f, inputs, outputs):
    """f(inputs..., n, outputs...) on device arrays; outputs: dtypes.  Returns host arrays."""
    import torch
    n = len(inputs[0])
    ins = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in inputs]
    outs = [torch.empty(n, dtype=torch.uint8 if d is np.uint8 else torch.float64, device="cuda") for d in outputs]
    p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    assert f(*[p(t) for t in ins], ctypes.c_long(n), *[p(t) for t in outs]) == 0
    return [t.cpu().numpy() for t in outs]


def _same(x, y):
    """Equal bits, the sign of a zero included; any NaN equals any NaN."""
    return (x.view(np.int64) == y.view(np.int64)) | (np.isnan(x) & np.isnan(y))


def _check(probe, a, b, inside):
    with np.errstate(all="ignore"):
        q = a / b
    shared, ieee, ok = _call(probe.probe_quotients, (a, b), (np.float64, np.float64, np.uint8))
    assert _same(ieee, q).all()
    assert _same(shared, q)[ok == 1].all()
    if inside is not None:
        assert (ok == inside).all()


def _significands(rng, n):
    """In [1, 2), a quarter of them next to 1 or 2."""
    m = rng.integers(0, 2 ** 52, n)
    k = n // 8
    m[:k] = rng.integers(0, 2 ** 12, k)
    m[k:2 * k] = 2 ** 52 - 1 - rng.integers(0, 2 ** 12, k)
    rng.shuffle(m)
    return (m + 2 ** 52) * 2.0 ** -52


@pytest.mark.parametrize("seed", range(8))
def test_random_pairs(probe, seed):
    rng = np.random.default_rng(seed)
    n = 1 << 23
    b = np.ldexp(_significands(rng, n), rng.integers(-255, 257, n))
    a = np.ldexp(_significands(rng, n), rng.integers(-764, 513, n)) * rng.choice([-1.0, 1.0], n)
    a[::101] = 0.0
    a[1::101] = -0.0
    _check(probe, a, b, 1)


def _next_to_midpoints(rng, b):
    """For divisors in [1, 2): dividends next to b times a midpoint of two neighbouring quotients."""
    m = rng.integers(2 ** 52, 2 ** 53, len(b))  # the lower neighbour, in units of its last place
    twice = m.astype(object) * 2 + 1
    ib = np.ldexp(b, 52).astype(np.int64).astype(object)
    prod = twice * ib  # exact: b * midpoint * 2^105
    lo = np.array([int(p) >> (int(p).bit_length() - 53) for p in prod], dtype=np.int64)
    return lo * 2.0 ** -52


@pytest.mark.parametrize("seed", range(2))
def test_dividends_next_to_midpoints(probe, seed):
    rng = np.random.default_rng(100 + seed)
    n = 1 << 18
    b = _significands(rng, n)
    a = _next_to_midpoints(rng, b)
    bits = a.view(np.int64)
    for d in (-1, 0, 1, 2):
        _check(probe, (bits + d).view(np.float64).copy(), b, 1)


def test_divisors_just_below_two(probe):
    rng = np.random.default_rng(7)
    k = np.arange(1, (1 << 24) + 1)
    b = 2.0 - k * 2.0 ** -52
    for _ in range(2):
        _check(probe, _significands(rng, len(k)), b, 1)
    _, y = _call(probe.probe_reciprocals, (b,), (np.float64, np.float64))
    assert (y == 1.0 / b).all()
    n = 1 << 17  # the divisors for which 1 / b is closest to a midpoint, with the hardest dividends
    a = _next_to_midpoints(rng, b[:n])
    for d in (-1, 0, 1, 2):
        _check(probe, (a.view(np.int64) + d).view(np.float64).copy(), b[:n], 1)


def test_reciprocal(probe):
    """The approximation over every upper word of a binade, and Newton's result within 2^-53 (1 + 2^-25) of 1 / b."""
    hi = np.arange(1 << 20, dtype=np.int64)
    worst = 0.0
    for low in (0, 0xffffffff, 0x5a5a5a5a):
        b = ((hi + 0x3ff00000) << 32 | low).view(np.float64)
        r, y = _call(probe.probe_reciprocals, (b,), (np.float64, np.float64))
        bl = b.astype(np.longdouble)
        assert np.abs(1 - bl * r.astype(np.longdouble)).max() < 2.0 ** -19.9
        # b y - 1 in integers: b, y < 2^53 units of 2^-52 and 2^-53 (1 / b in (1/2, 1])
        ib = np.ldexp(b, 52).astype(np.int64)
        iy = np.ldexp(y, 53).astype(np.int64)
        e = [abs(int(p) * int(q) - (1 << 105)) / int(p) for p, q in zip(ib[::37], iy[::37])]  # |y - 1 / b| in units of 2^-53
        worst = max(worst, max(e))
    assert worst <= 0.5 * (1 + 2.0 ** -25)


def test_third(probe):
    rng = np.random.default_rng(3)
    n = 1 << 22
    a = np.ldexp(_significands(rng, n), rng.integers(-764, 513, n)) * rng.choice([-1.0, 1.0], n)
    a[:4] = [0.0, -0.0, 2.0 ** -764, np.nextafter(2.0 ** 513, 0)]
    shared, ok = _call(probe.probe_thirds, (a,), (np.float64, np.uint8))
    assert ok.all() and _same(shared, a / 3.0).all()


def test_quotients_of_the_limiters(probe):
    """Slope ratios (magnitudes from 1e-5 to 2^513) and 2 r / (1 + r), 2 / (1 + r) over the ratios that come of them."""
    rng = np.random.default_rng(4)
    n = 1 << 22
    floor = 10.0 ** -5
    pick = lambda: np.maximum(np.ldexp(_significands(rng, n), rng.choice([rng.integers(-17, 513, n), rng.integers(-17, 3, n)])),  # noqa: E731
                              floor) * rng.choice([-1.0, 1.0], n)
    num, den = pick(), pick()
    num[:1000], den[500:1500] = floor, floor
    r, = _call(probe.probe_knowns, (num, den), (np.float64,))
    assert _same(r, num / den).all()
    r = r[r >= 0]
    for x, y in ((np.full(len(r), 2.0), 1.0 + r), (2.0 * r, 1.0 + r), (np.full(len(r), 2.0), 0.7 + 1.3 * r)):
        q, = _call(probe.probe_knowns, (x, y), (np.float64,))
        assert _same(q, x / y).all()


def test_range_flags(probe):
    """The flags are raised by everything outside the proven ranges and by nothing inside them."""
    tiny, huge = np.nextafter, np.inf
    divisors = {1: [2.0 ** -255, 1.0, 3.0, tiny(2.0 ** 257, 0)],
                0: [tiny(2.0 ** -255, 0), 2.0 ** 257, 0.0, -0.0, -1.0, 5e-324, huge, -huge, np.nan]}
    dividends = {1: [0.0, -0.0, 2.0 ** -764, -(2.0 ** -764), 1.0, tiny(2.0 ** 513, 0), -tiny(2.0 ** 513, 0)],
                 0: [tiny(2.0 ** -764, 0), -tiny(2.0 ** -764, 0), 1e-240, 1e-310, 5e-324, -5e-324, 2.0 ** 513, -(2.0 ** 513),
                     huge, -huge, np.nan]}
    for bi, bs in divisors.items():
        for ai, as_ in dividends.items():
            a, b = (x.ravel().copy() for x in np.meshgrid(np.array(as_), np.array(bs)))
            _check(probe, a, b, bi and ai)
    positive = {1: divisors[1], 0: divisors[0]}
    for ai, as_ in positive.items():
        a = np.array(as_)
        q, ok, below = _call(probe.probe_positives, (a, np.ones(len(a))), (np.float64, np.uint8, np.uint8))
        assert (ok == ai).all() and _same(q, a)[ok == 1].all()
    a = np.array([0.0, -0.0, 5e-324, 1e-310, -1.0, tiny(2.0 ** 513, 0), 2.0 ** 513, -(2.0 ** 513), huge, -huge, np.nan])
    _, _, below = _call(probe.probe_positives, (a, np.ones(len(a))), (np.float64, np.uint8, np.uint8))
    assert list(below) == [1] * 6 + [0] * 5
