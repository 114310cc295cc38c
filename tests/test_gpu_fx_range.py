"""The FP64 form's transforms at both ends of FP64's range: results between
2^1023 and the largest value, and subnormal ones."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(8, 8, 8), (64, 16, 128), (16, 512, 16), (256, 16, 32), (16, 8, 512)]


def _params(fipi, shape):
    nx, ny, nz = shape
    return fipi.workload("t32").with_(name="fx", nx=nx, ny=ny, nz=nz, lx=float(nx), ly=float(ny), lz=float(nz),
                                      n_p=0).params()


def _half(x, shape):
    nx, ny, nz = shape
    return np.ascontiguousarray(np.fft.rfftn(x.reshape(nz, ny, nx)).transpose(0, 2, 1)).ravel()


@pytest.mark.parametrize("shape", SHAPES)
def test_largest_results(fipi, shape):
    nx, ny, nz = shape
    A = 1.5e308
    x = np.zeros((nz, ny, nx))
    x[nz // 8, ny // 4, nx // 8] = 1.0  # phases of eighths of a turn: both components reach A cos(pi / 4) > 2^1023
    unit = _half(x, shape)
    with fipi.Simulation(_params(fipi, shape), "fp64") as s:
        X = s.fft_r2c(x.ravel() * A)
        one = np.zeros(s.SH, np.complex128)
        one[0] = A
        mean = s.fft_c2r(one)
    assert np.abs(X.real).max() >= 2.0 ** 1023 and np.abs(X.imag).max() >= 2.0 ** 1023
    assert np.isfinite(X.view(np.float64)).all()
    # a few 2^-53 of the row's norm per axis
    assert np.abs(X.view(np.float64) / A - unit.view(np.float64)).max() < 4e-15
    assert np.abs(mean / (A / x.size) - 1.0).max() < 4e-15


@pytest.mark.parametrize("shape", SHAPES)
def test_subnormal_results(fipi, shape):
    nx, ny, nz = shape
    x = np.random.default_rng(nx).standard_normal(nx * ny * nz) * 2.0 ** -1040
    exact = _half(x * 2.0 ** 500, shape).view(np.float64)
    with fipi.Simulation(_params(fipi, shape), "fp64") as s:
        got = s.fft_r2c(x).view(np.float64) * 2.0 ** 500  # exact
    # every pass rounds to at most half a unit of 2^-1074; the passes after it
    # add up the errors of ny nz and nz values
    unit = 2.0 ** (-1074 + 500)
    bar = 0.5 * unit * (np.sqrt(ny * nz) + np.sqrt(nz) + 1.0)
    assert np.sqrt(np.mean((got - exact) ** 2)) <= bar
