"""cafe_intmath.h (exp, atan2, cos, sin, division, square root in integers) returns the bits of the
floating-point functions, inside its ranges and outside, and cafe_crmath.h's fast
paths those of its double-double paths (CPU only)."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
D = ctypes.POINTER(ctypes.c_double)


@pytest.fixture(scope="module")
def ic(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("ic") / "ic.so")
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-fPIC", "-shared",
                    os.path.join(HERE, "native", "intmath_check.cpp"), "-o", so], check=True)
    return ctypes.CDLL(so)


def _same(ic, fn, x, y=None):
    x = np.ascontiguousarray(x, np.float64)
    y = x if y is None else np.ascontiguousarray(y, np.float64)
    got, want = np.empty_like(x), np.empty_like(x)
    ic.ic_eval(fn, ctypes.c_long(len(x)), *(a.ctypes.data_as(D) for a in (x, y, got, want)))
    bad = (got.view(np.int64) != want.view(np.int64)) & ~(np.isnan(got) & np.isnan(want))
    assert not bad.any(), (x[bad][:4], y[bad][:4], got[bad][:4], want[bad][:4])


EDGES = np.array([0.0, np.inf, np.nan, 5e-324, 2.2250738585072014e-308, 1.7976931348623157e308, 1.0, 2.0, 0.5,
                  np.nextafter(1.0, 0), np.nextafter(1.0, 2), np.nextafter(2.0, 0), 4.0, np.nextafter(4.0, 0)])


def _around(v, n=40):
    out = [v]
    for s in (-np.inf, np.inf):
        w = v
        for _ in range(n):
            w = np.nextafter(w, s)
            out.append(w)
    return np.array(out)


@pytest.mark.parametrize("kind", ["uniform", "scales", "steps", "limits"])
def test_exp(ic, kind):
    g, n = np.random.default_rng(5), 300000
    if kind == "uniform":
        x = -g.uniform(0, 760, n)
    elif kind == "scales":
        x = -(2.0 ** g.uniform(-60, 11, n))
    elif kind == "steps":  # at and beside the table's steps and the powers of two
        k = g.integers(1, 128 * 1020, n) * (np.log(2) / 128)
        x = -k * (1 + g.integers(-3, 4, n) * 2.0 ** -52)
    else:
        x = np.concatenate([_around(-v) for v in (707.0, 745.2, 2.0 ** -40, 1.0, np.log(2), 708.4, 709.8)] +
                           [EDGES, -EDGES, g.uniform(0, 720, 1000)])
    _same(ic, 0, x)


def _numbers(g, n, emax):
    m = 1 + g.integers(0, 2 ** 52, n) * 2.0 ** -52
    k = n // 3  # significands near the ends
    m[:k] = np.where(g.integers(0, 2, k), 1 + g.integers(0, 4, k) * 2.0 ** -52, 2 - g.integers(1, 5, k) * 2.0 ** -52)
    g.shuffle(m)
    with np.errstate(all="ignore"):
        return m * 2.0 ** g.integers(-emax, emax, n).astype(float)


@pytest.mark.parametrize("fn", [1, 2])
@pytest.mark.parametrize("emax", [3, 400, 1020])
def test_division(ic, fn, emax):
    g, n = np.random.default_rng(emax), 300000
    a, b = _numbers(g, n, emax) * g.choice([-1, 1], n), _numbers(g, n, emax)
    b[::97] *= -1
    _same(ic, fn, a, b)
    e = np.concatenate([EDGES, -EDGES])
    _same(ic, fn, np.repeat(e, len(e)), np.tile(e, len(e)))


@pytest.mark.parametrize("emax", [3, 400, 1020])
def test_sqrt(ic, emax):
    g, n = np.random.default_rng(emax), 300000
    x = _numbers(g, n, emax)
    _same(ic, 3, x)
    with np.errstate(all="ignore"):  # squares and their neighbours
        s = (x * 2.0 ** 26 % 2 ** 26) ** 2
    _same(ic, 3, np.concatenate([s, np.nextafter(s, 0), np.nextafter(s, np.inf), EDGES, -EDGES]))


@pytest.mark.parametrize("off", [-2.0 ** -21, -2.0 ** -22, 0.0, 2.0 ** -22, 2.0 ** -21])
def test_sqrt_of_any_allowed_seed(ic, off):
    """The device's 1/sqrt is not the host's: the root is right for any that is good to 2^-21."""
    g, n = np.random.default_rng(4), 400000
    x = g.uniform(1, 4, n)
    x[: n // 4] = 4.0 - np.arange(1, n // 4 + 1) * 2.0 ** -51  # the largest remainders: just below powers of four
    x[n // 4: n // 2] = 1.0 + np.arange(n // 4) * 2.0 ** -52
    x = x * 4.0 ** g.integers(-500, 500, n)
    got = np.empty(n)
    ic.ic_root(ctypes.c_long(n), ctypes.c_double(off * (1 - 2.0 ** -2)), x.ctypes.data_as(D), got.ctypes.data_as(D))
    assert np.array_equal(got, np.sqrt(x))
    # the whole allowance, the rounding of f to single precision (2^-24) included
    ic.ic_root(ctypes.c_long(n), ctypes.c_double(off + np.sign(-off) * 2.0 ** -24), x.ctypes.data_as(D), got.ctypes.data_as(D))
    assert np.array_equal(got, np.sqrt(x))


@pytest.mark.parametrize("kind", ["uniform", "scales", "midpoints"])
def test_fast_paths(ic, kind):
    """arctangent, sine and cosine at arguments where the series' terms are largest"""
    g, n = np.random.default_rng(2), 400000
    y, x = g.uniform(0, 1, n), g.uniform(0, 1, n)
    t = g.uniform(0, np.pi / 2, n)
    if kind == "scales":
        y *= 2.0 ** g.uniform(-60, 0, n)
        t = np.where(g.integers(0, 2, n), np.pi / 2 - t * 2.0 ** g.uniform(-50, 0, n), t * 2.0 ** g.uniform(-50, 0, n))
    elif kind == "midpoints":  # between the tables' points
        y = x * (g.integers(0, 64, n) + 0.5) / 64 * (1 + g.uniform(-1, 1, n) * 1e-3)
        t = (g.integers(0, 201, n) + 0.5) / 128 * (1 + g.uniform(-1, 1, n) * 1e-3)
    _same(ic, 4, y, x)
    _same(ic, 4, x, y)
    _same(ic, 5, t)
    _same(ic, 6, t)


@pytest.mark.parametrize("kind", ["uniform", "scales", "steps", "exponents", "edges"])
def test_angles(ic, kind):
    """atan2 of non-negative arguments, cos on [0, pi/4] and sin on [pi/4, pi/2], and beyond"""
    g, n = np.random.default_rng(8), 300000
    y, x, t = g.uniform(0, 1, n), g.uniform(0, 1, n), g.uniform(0, np.pi / 4, n)
    if kind == "scales":
        y *= 2.0 ** g.uniform(-60, 0, n)
        t *= 2.0 ** g.uniform(-50, 0, n)
    elif kind == "steps":  # at, beside and between the tables' points
        d = 1 + g.integers(-2, 3, n) * 2.0 ** -52
        y = x * (g.integers(0, 129, n) / 128) * d
        t = g.integers(0, 202, n) / 256 * d
    elif kind == "exponents":
        e = g.integers(-1000, 1000, n).astype(float)
        y, x = y * 2.0 ** e, x * 2.0 ** (e + g.integers(-8, 9, n))
    elif kind == "edges":
        e = np.concatenate([EDGES, _around(1 / 128), _around(2.0 ** -37)])
        y, x = np.repeat(e, len(e)), np.tile(e, len(e))
        t = np.concatenate([EDGES, -EDGES, _around(np.pi / 4), _around(2.0 ** -27), np.pi / 2 - _around(np.pi / 4)])
    _same(ic, 7, y, x)
    _same(ic, 7, x, y)
    _same(ic, 8, t)
    _same(ic, 9, t)
    _same(ic, 9, np.pi / 2 - t)
    _same(ic, 10, np.concatenate([y, -y]))
