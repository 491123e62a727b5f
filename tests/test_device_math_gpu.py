"""The device forms of the transforms' square roots and of the packed fp32 Box-Muller, run by
themselves (tests/devapi/math_check.cu): on the host these headers use other operations (std::sqrt,
scalar fma), so the host checks do not see the approximate reciprocal roots or the packed ones.

sqrt_mid (fp32) must be the rounded root on every float of its range.  sqrt_inner (fp64) is within
2^-103 of the root before its one rounding (derived in precise_math.cuh), so it must be the rounded
root wherever the root is further than that from a midpoint between two doubles, and never another
number than a neighbour of it.  The Box-Muller bounds are those of tests/test_normal_math.py."""

import ctypes
import os
from ctypes import c_size_t, c_uint32, c_void_p

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def dev():
    import torch
    torch.cuda.init()
    return ctypes.CDLL(os.path.join(HERE, "devapi", "libdevmath_b200.so"))


def _ptr(t):
    return c_void_p(t.data_ptr())


def test_sqrt_mid_equals_rounded_root(dev):
    import torch
    differ = torch.zeros(1, dtype=torch.int64, device="cuda")
    low, high = (np.array([v], dtype=np.float32).view(np.uint32)[0] for v in (2.0 ** -26, 2.0 ** 10))
    assert dev.math_sqrt_mid(c_uint32(int(low)), c_uint32(int(high - low)), _ptr(differ)) == 0
    assert dev.math_sqrt_mid(c_uint32(0), c_uint32(1), _ptr(differ)) == 0  # and 0
    assert int(differ[0]) == 0


def _sqrt_inner(dev, t):
    import torch
    x = torch.from_numpy(t).cuda()
    out = [torch.empty_like(x) for _ in range(3)]
    assert dev.math_sqrt_inner(_ptr(x), c_size_t(x.numel()), *(_ptr(o) for o in out)) == 0
    return [o.cpu().numpy() for o in out]


def test_sqrt_inner_equals_rounded_root(dev):
    rng = np.random.default_rng(3)
    n = 1 << 22
    m = 1.0 + rng.random(n)
    k = np.floor(rng.random(n) * 2.0 ** 26) + 1.0
    squares = k * k
    parts = [np.ldexp(m, rng.integers(-200, 200, n)),               # the whole range
             -2.0 * np.log(rng.random(n) + 2.0 ** -54),              # radii of Box-Muller
             -2.0 * np.log1p(-np.ldexp(rng.random(n), -rng.integers(0, 52, n))),  # of uniforms next to 1
             squares, np.nextafter(squares, 0.0), np.nextafter(squares, np.inf),
             np.array([0.0, -0.0, 2.0 ** -200, 2.0 ** 200, 1.0, 2.0, np.nextafter(1.0, 0.0), np.nextafter(4.0, 0.0)])]
    t = np.concatenate([p[(p == 0) | (p >= 2.0 ** -200)] for p in parts])
    ours, rounded, seed = _sqrt_inner(dev, t)
    assert np.array_equal(rounded.view(np.uint64), np.sqrt(t).view(np.uint64))
    assert np.array_equal(ours.view(np.uint64), rounded.view(np.uint64))
    # the seed the derivation starts from
    pos = t > 0
    assert np.max(np.abs(seed[pos] * rounded[pos] - 1.0)) < 2.0 ** -19


def _nearly_halfway(gap):
    """t with sqrt(t) just below the midpoint m = 1 + x 2^-53 (x odd): m^2 - t = gap 2^-106, by lifting
    x^2 = gap (mod 2^54) bit by bit."""
    x = 1
    for k in range(3, 54):
        if (x * x - gap) % (1 << (k + 1)):
            x += 1 << (k - 1)
    found = []
    for y in (x, (1 << 54) - x, x + (1 << 53), (1 << 53) - x):
        y %= 1 << 54
        if 0 < y < (1 << 53) and (y * y - gap) % (1 << 54) == 0:
            ulps = (1 << 52) + y + ((y * y - gap) >> 54)  # t in units of 2^-52
            if ulps < (1 << 53) or ulps % 2 == 0:
                found.append(float(ulps) * 2.0 ** -52)
    return found


def test_sqrt_inner_next_to_midpoints(dev):
    near, far = [], []
    for gap in range(1, 40001, 8):
        for t in _nearly_halfway(gap):
            # sqrt(t) is gap 2^-107 / m from the midpoint, of t's own size: against 2^-103
            (far if gap >= 64 else near).extend((t, t * 2.0 ** 20, t * 2.0 ** -20))
    assert len(near) >= 10 and len(far) >= 1000
    ours, rounded, _ = _sqrt_inner(dev, np.array(far))
    assert np.array_equal(ours.view(np.uint64), rounded.view(np.uint64))
    ours, rounded, _ = _sqrt_inner(dev, np.array(near))
    assert np.max(np.abs(ours.view(np.int64) - rounded.view(np.int64))) <= 1


def test_box_muller_accuracy(dev):
    import torch
    rng = np.random.default_rng(7)
    n = 1 << 22
    x = rng.integers(0, 1 << 32, n, dtype=np.uint64)
    y = rng.integers(0, 1 << 32, n, dtype=np.uint64)
    kind = np.arange(n) % 16
    sub = (np.arange(n) // 16).astype(np.uint64)
    x = np.where(kind == 0, np.uint64(0xffffffff) - (x >> (np.uint64(8) + sub % np.uint64(24))), x)  # near 1
    x = np.where(kind == 1, x >> (sub % np.uint64(32)), x)  # small
    # the kernels' own steps: fma(x, 2^-32, 2^-32) rounds once (exact in double), y 2^-32 2 pi twice
    u = (x.astype(np.float32).astype(np.float64) * 2.0 ** -32 + 2.0 ** -32).astype(np.float32)
    scale = np.float32(1.46291807e-09)
    a = (scale + y.astype(np.float32) * scale).astype(np.float32)
    half_pis = np.array([1.5707964, 3.1415927, 4.712389, 6.2831855], dtype=np.float32)[(sub % np.uint64(4)).astype(int)]
    a = np.where(kind == 2, np.nextafter(half_pis, np.float32(0.0)), np.where(kind == 3, half_pis, a)).astype(np.float32)
    u[:4], a[:4] = 1.0, [1.0, 4.0, 2.0, 6.0]
    ins = [torch.from_numpy(np.ascontiguousarray(v)).cuda() for v in (u, a)]
    out = [torch.empty(n, dtype=torch.float32, device="cuda") for _ in range(3)]
    assert dev.math_box_muller(*(_ptr(t) for t in ins), c_size_t(n // 2), *(_ptr(t) for t in out)) == 0
    l, s, c = (t.cpu().numpy() for t in out)
    u64, a64 = u.astype(np.float64), a.astype(np.float64)
    m = 2.0 * np.log(u64)
    r = np.sqrt(-m)
    want = np.stack([r * np.sin(a64), r * np.cos(a64)])
    got = np.stack([s, c]).astype(np.float64)

    def ulps(g, e):
        return np.abs(g - e) / np.spacing(np.abs(e).astype(np.float32)).astype(np.float64)

    some = m != 0.0
    assert np.max(ulps(l.astype(np.float64), m)[some]) < 1.0
    assert np.max(ulps(got, want)[want != 0.0]) < 4.0
    assert np.linalg.norm(got - want) < 4.7e-8 * np.linalg.norm(want)  # the library functions' error
    assert np.all(got[:, ~some] == 0.0) and not np.all(some)
