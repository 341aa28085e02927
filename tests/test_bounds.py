"""cafe_bounds.h against the double-precision expressions it stands in for (CPU
only): bounds hold, decided classes and quotients are the same."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
D = ctypes.POINTER(ctypes.c_double)
F = ctypes.POINTER(ctypes.c_float)
I = ctypes.POINTER(ctypes.c_int)
U = ctypes.POINTER(ctypes.c_uint)


@pytest.fixture(scope="module")
def bc(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("bc") / "bc.so")
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-fPIC", "-shared",
                    os.path.join(HERE, "native", "bounds_check.cpp"), "-o", so], check=True)
    return ctypes.CDLL(so)


def _p(a, t):
    return a.ctypes.data_as(t)


@pytest.mark.parametrize("dx", [1e-9, 2.5e-6, 1.0, 1e6])
@pytest.mark.parametrize("kind", ["near", "far", "cancelling", "axes"])
def test_numerator_bounds(bc, dx, kind):
    n, g = 40000, np.random.default_rng(7)
    c = g.uniform(-1.2, 1.2, (n, 3)) * dx
    if kind == "far":
        c *= 3.0
    elif kind == "cancelling":  # offsets that meet the neighbour's centre but for 1e-12 .. 1
        c = dx * g.choice([-1.0, 0.0, 1.0], (n, 3)) * (1.0 + g.uniform(-1, 1, (n, 3)) * 10.0 ** g.uniform(-12, 0, (n, 3)))
    elif kind == "axes":
        c *= g.choice([0.0, 1.0, 1e-9], (n, 3))
    q = g.normal(size=(n, 4))
    w, x, y, z = (q / np.linalg.norm(q, axis=1, keepdims=True)).T
    if kind == "axes":
        w, x, y, z = np.ones(n), np.zeros(n), np.zeros(n), np.zeros(n)
    R = np.stack([1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w), 2 * (x * y + z * w),
                  1 - 2 * (x * x + z * z), 2 * (y * z - x * w), 2 * (x * z - y * w), 2 * (y * z + x * w),
                  1 - 2 * (x * x + y * y)], axis=1)
    R, c, d = np.ascontiguousarray(R), np.ascontiguousarray(c), (np.arange(n) % 26).astype(np.int32)
    lo, hi, ex = np.empty(n, np.float32), np.empty(n, np.float32), np.empty(n)
    bc.bc_glb(ctypes.c_long(n), ctypes.c_double(dx), _p(c, D), _p(R, D), _p(d, I), _p(lo, F), _p(hi, F), _p(ex, D))
    assert np.all(lo <= ex) and np.all(ex <= hi)
    c[0, 1], R[1, 4] = np.inf, np.nan  # not finite: no bound
    bc.bc_glb(ctypes.c_long(n), ctypes.c_double(dx), _p(c, D), _p(R, D), _p(d, I), _p(lo, F), _p(hi, F), _p(ex, D))
    assert np.isnan(lo[:2]).all() and np.isnan(hi[:2]).all()


@pytest.mark.parametrize("length", [0.1, 2.0, 5.0, 40.0, 1e6])
def test_numerator_bounds_of_axes_of_any_length(bc, length):
    """cTheta as a host program uploads it need not hold a unit axis: the matrix that
    SampleOrientation's formula makes of it is then no rotation, its entries up to length^2."""
    n, g, dx = 40000, np.random.default_rng(9), 2.5e-6
    a = g.normal(size=(n, 3))
    a *= length / np.linalg.norm(a, axis=1, keepdims=True)
    w = g.uniform(0, np.pi, n)
    K = np.zeros((n, 3, 3))
    K[:, 0, 1], K[:, 0, 2], K[:, 1, 2] = -a[:, 2], a[:, 1], -a[:, 0]
    K -= K.transpose(0, 2, 1)
    R = (np.cos(w)[:, None, None] * np.eye(3) + (1 - np.cos(w))[:, None, None] * a[:, :, None] * a[:, None, :] +
         np.sin(w)[:, None, None] * K)
    # the numerator in the direction that cancels most: a neighbour's offset that R^T nearly loses
    c = g.uniform(-1.0, 1.0, (n, 3)) * dx
    d = (np.arange(n) % 26).astype(np.int32)
    d27 = np.where(d < 13, d, d + 1)
    off = np.stack([d27 % 3 - 1, d27 // 3 % 3 - 1, d27 // 9 - 1], axis=1) * dx
    k = n // 2
    c[:k] = a[:k] / length * g.uniform(-1, 1, (k, 1)) * 1e-3 * dx + np.cross(a[:k] / length, g.normal(size=(k, 3))) * dx - off[:k]
    R, c = np.ascontiguousarray(R.reshape(n, 9)), np.ascontiguousarray(c)
    lo, hi, ex = np.empty(n, np.float32), np.empty(n, np.float32), np.empty(n)
    bc.bc_glb(ctypes.c_long(n), ctypes.c_double(dx), _p(c, D), _p(R, D), _p(d, I), _p(lo, F), _p(hi, F), _p(ex, D))
    assert np.all(lo <= ex) and np.all(ex <= hi)


@pytest.mark.parametrize("theta", [0.0, 0.7, np.pi / 2, -2.0])
@pytest.mark.parametrize("dirp", [1.0, -1.0, 0.0, 1e-250])
@pytest.mark.parametrize("n", [1, 31, 33, 257])
def test_decided_classes(bc, theta, dirp, n):
    g = np.random.default_rng(n)
    decided = total = 0
    for _ in range(200):
        dx = 2.5e-6
        a1 = np.array([40e-6, g.uniform(5e-6, 60e-6), g.uniform(5e-6, 60e-6), 90e-6, 30e-6, 28e-6])
        h = dx * n / 2
        z = g.uniform(-30e-6, 2e-6)
        s = np.array([np.cos(theta), np.sin(theta), h, h, g.uniform(0, 2 * h), g.uniform(0, 2 * h), 0.0, dirp, dx,
                      g.uniform(0, 2 * h), z])
        fast, exact = np.empty(n, np.int32), np.empty(n, np.int32)
        bc.bc_class(n, _p(s, D), _p(a1, D), ctypes.c_double(a1[0]), 0, _p(fast, I), _p(exact, I))
        assert np.all((fast == -1) | (fast == exact))
        decided += int((fast >= 0).sum())
        total += n
    if abs(dirp) != 1e-250:  # (the product's sign may be lost: left to the exact test)
        assert decided > 0.9 * total


def test_division_by_reciprocal(bc):
    n, g = 400000, np.random.default_rng(3)
    a = g.uniform(1, 2, n) * 2.0 ** g.integers(-1000, 1000, n) * g.choice([-1, 1], n)
    v = g.uniform(1, 2, n) * 2.0 ** g.integers(-300, 300, n)
    k = n // 4  # mantissas at the ends, zeros, infinities, NaN
    v[:k] = (2.0 - g.integers(0, 4, k) * 2.0 ** -52) * 2.0 ** g.integers(-40, 40, k)
    a[:k] = (1.0 + g.integers(0, 4, k) * 2.0 ** -52) * 2.0 ** g.integers(-40, 40, k)
    a[:5] = [0.0, -0.0, np.inf, -np.inf, np.nan]
    q = np.empty(n)
    bc.bc_div(ctypes.c_long(n), _p(a, D), _p(v, D), _p(q, D))
    with np.errstate(all="ignore"):
        assert np.array_equal(q.view(np.int64)[5:], (a / v).view(np.int64)[5:])
        assert np.array_equal(q[:5], (a / v)[:5], equal_nan=True)


@pytest.mark.parametrize("V", [1e-60, 3e-39, 1e-9, 1.0, 7e3, 1e30])
@pytest.mark.parametrize("time", [0, 1])
def test_window_limit(bc, V, time):
    n, g = 100000, np.random.default_rng(11)
    lim = g.uniform(1, 2, n) * 2.0 ** g.integers(-60, 19, n) * g.choice([-1, 1], n)
    lim[:3] = [0.0, -0.0, -1e300]
    key, at, below = (np.empty(n, np.uint32) for _ in range(3))
    with np.errstate(all="ignore"):
        bc.bc_limit(ctypes.c_long(n), _p(lim, D), ctypes.c_double(V), time, _p(key, U), _p(at, U), _p(below, U))
    sign = lim != 0.0  # (the key of a zero depends on its sign: one apart)
    assert np.all(key[sign] <= at[sign])
    if time or 1e-9 <= V <= 7e3:  # in single precision's range no looser than a relative 2^-16
        assert np.all(key[3:] >= below[3:])
