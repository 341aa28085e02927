"""cafe_intmath.h on the device, whose single-precision starting values are not the
host's, returns the bits of the floating-point functions."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))
D = ctypes.POINTER(ctypes.c_double)
N = 1 << 22


@pytest.fixture(scope="module")
def ic(tmp_path_factory):
    from amcafe_gb300 import build as b

    so = str(tmp_path_factory.mktemp("icg") / "ic.so")
    subprocess.run([b._nvcc()] + b.NVCC_FLAGS + [os.path.join(HERE, "native", "intmath_check.cu"), "-o", so], check=True)
    return ctypes.CDLL(so)


def _same(ic, fn, x, y=None):
    x = np.ascontiguousarray(x, np.float64)
    y = x if y is None else np.ascontiguousarray(y, np.float64)
    got, want = np.empty_like(x), np.empty_like(x)
    assert ic.ic_gpu(fn, ctypes.c_long(len(x)), *(a.ctypes.data_as(D) for a in (x, y, got, want))) == 0
    bad = (got.view(np.int64) != want.view(np.int64)) & ~(np.isnan(got) & np.isnan(want))
    assert not bad.any(), (bad.sum(), x[bad][:4], y[bad][:4], got[bad][:4], want[bad][:4])


def _near(powers, n):
    """n doubles below and n from each power on, the significands one unit apart and wider."""
    s = np.arange(n)
    s = np.concatenate([s[: n // 2], (s[n // 2:] * 1e7).astype(np.int64)]).astype(float)
    return np.concatenate([np.concatenate([p - (s + 1) * p * 2.0 ** -53, p + s * p * 2.0 ** -52]) for p in powers])


@pytest.mark.parametrize("fn", [0, 1, 2, 3, 4, 5, 6])
def test_device_bits(ic, fn):
    g = np.random.default_rng(fn)
    m = 1 + g.random(N)
    if fn == 3:
        _same(ic, 3, np.concatenate([m, 2 * m, m * 4.0 ** g.integers(-500, 500, N), _near([1.0, 2.0, 4.0, 2.0 ** -40], N // 8)]))
    elif fn == 0:
        _same(ic, 0, np.concatenate([-g.uniform(0, 760, N), -(2.0 ** g.uniform(-60, 11, N))]))
    elif fn in (1, 2):
        b = np.concatenate([1 + g.random(N), _near([1.0, 2.0], N // 4)])
        _same(ic, fn, np.resize(m, len(b)) * g.choice([-1.0, 1.0], len(b)), b)
    elif fn == 4:
        y, x = g.random(N), g.random(N)
        _same(ic, 4, y, x)
        _same(ic, 4, y * 2.0 ** g.uniform(-50, 0, N), x)
        _same(ic, 4, x, y * 2.0 ** g.uniform(-50, 0, N))
    else:
        _same(ic, fn, g.uniform(0, np.pi / 2, N))
