"""The FP64 form's block fixed-point transforms against extended precision."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(64, 32, 32), (128, 64, 8), (512, 16, 8), (8, 512, 16), (8, 16, 512), (32, 256, 8)]


def _fields(shape):
    nx, ny, nz = shape
    rng = np.random.default_rng(nx + 3 * ny)
    z, y, x = np.meshgrid(np.arange(nz) / nz, np.arange(ny) / ny, np.arange(nx) / nx, indexing="ij")
    noise = rng.uniform(-1.0, 1.0, (nz, ny, nx))
    spike = 1e-6 * noise
    spike[nz // 3, ny // 5, nx // 7] = 1.0
    return {"noise": noise, "offset": 1.0 + 0.05 * noise, "spike": spike,
            "interface": np.tanh(12.0 * (np.sqrt((x - 0.5) ** 2 + (y - 0.5) ** 2 + (z - 0.5) ** 2) - 0.3)),
            "mode": np.cos(2.0 * np.pi * (x + 2.0 * y + 3.0 * z))}


@pytest.mark.parametrize("shape", SHAPES)
def test_errors_are_those_of_rounding(fipi, shape):
    """An FP64 transform of some 2^16 values in radix-8 stages rounds some
    dozen times on the way to a result, by half a unit at most: 1 to 2 units
    of 2^-53 of the norm.  Four units allow no lost bits."""
    fft = pytest.importorskip("scipy.fft")
    nx, ny, nz = shape
    P = fipi.workload("t32").with_(name="fx", nx=nx, ny=ny, nz=nz, lx=float(nx), ly=float(ny), lz=float(nz),
                                   n_p=0).params()
    bar = 4.0 * 2.0 ** -53
    with fipi.Simulation(P, "fp64") as s:
        for name, x in _fields(shape).items():
            X = fft.rfftn(x.astype(np.longdouble))
            got = s.fft_r2c(x.ravel()).reshape(nz, nx // 2 + 1, ny).transpose(0, 2, 1)
            err = np.sqrt(np.sum(np.abs(got - X) ** 2) / np.sum(np.abs(X) ** 2))
            # the inverse of the rounded spectrum (modes that are their own mirror image: real parts)
            Y = X.astype(np.complex128)
            y = fft.irfftn(Y.astype(np.clongdouble), s=x.shape)
            back = s.fft_c2r(np.ascontiguousarray(Y.transpose(0, 2, 1)).ravel()).reshape(x.shape)
            rre = np.sqrt(np.sum((back - y) ** 2) / np.sum(y ** 2))
            print(shape, name, float(err), float(rre))
            assert err <= bar and rre <= bar, (name, float(err / 2.0 ** -53), float(rre / 2.0 ** -53))
