"""The FP64 form's block fixed-point transforms against numpy: every axis
length's plan, rows of very different content and magnitude, rows that are
not finite."""
from __future__ import annotations

import numpy as np
import pytest
from conftest import rel_l2

pytestmark = pytest.mark.gpu

SHAPES = [(8, 8, 8), (16, 8, 32), (32, 64, 8), (64, 16, 128), (128, 32, 16), (256, 8, 16), (512, 16, 8), (8, 512, 16),
          (16, 128, 256), (8, 256, 64), (16, 8, 512)]


def _params(fipi, shape):
    nx, ny, nz = shape
    return fipi.workload("t32").with_(name="fx", nx=nx, ny=ny, nz=nz, lx=float(nx), ly=float(ny), lz=float(nz),
                                      n_p=0).params()


def _half(x, shape):
    nx, ny, nz = shape
    return np.ascontiguousarray(np.fft.rfftn(x.reshape(nz, ny, nx)).transpose(0, 2, 1)).ravel()


@pytest.mark.parametrize("shape", SHAPES)
def test_transforms_of_unlike_rows(fipi, shape):
    nx, ny, nz = shape
    V = nx * ny * nz
    rng = np.random.default_rng(V)
    noise = rng.standard_normal(V)
    fields = {
        "noise": noise,
        "offset": 1e6 + noise,                                     # one dominant mode
        "spike": 1e-4 * noise + (np.arange(V) == V // 3) * 1e3,    # few large values in a row
        "rows": noise * 10.0 ** rng.integers(-12, 12, V // nx).repeat(nx),
        "sparse": noise * (rng.random(V) < 0.02),                  # rows of zeros
        "large": noise * 1e290,
        "small": noise * 1e-299,                                   # below 2^-959: scaled rows
    }
    # FP64 (numpy's, the bar's other side) and the fixed-point rows err by a
    # few 2^-53 of the norm per axis
    bar = 2e-15
    with fipi.Simulation(_params(fipi, shape), "fp64") as s:
        for name, x in fields.items():
            X = _half(x, shape)
            assert rel_l2(s.fft_r2c(x).view(np.float64) / np.abs(x).max(), X.view(np.float64) / np.abs(x).max()) < bar, name
            if name != "large":  # its spectrum times numpy's own normalisation overflows
                assert rel_l2(s.fft_c2r(X) / np.abs(x).max(), x / np.abs(x).max()) < bar, name
        assert not s.fft_r2c(np.zeros(V)).any()
        assert np.isfinite(s.fft_r2c(np.full(V, 5e-324)).view(np.float64)).all()


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("shape", [(8, 8, 8), (64, 16, 128), (16, 512, 16)])
def test_non_finite_values_reach_every_output(fipi, shape, bad):
    V = shape[0] * shape[1] * shape[2]
    x = np.random.default_rng(1).standard_normal(V)
    with fipi.Simulation(_params(fipi, shape), "fp64") as s:
        X = _half(x, shape)
        x[V // 2 + 3] = bad
        assert not np.isfinite(s.fft_r2c(x).view(np.float64)).reshape(-1, 2).all(axis=1).any()
        X[len(X) // 2 + 1] = bad
        assert not np.isfinite(s.fft_c2r(X)).any()
        # the context is as good as new
        y = np.random.default_rng(2).standard_normal(V)
        assert rel_l2(s.fft_r2c(y).view(np.float64), _half(y, shape).view(np.float64)) < 2e-15
