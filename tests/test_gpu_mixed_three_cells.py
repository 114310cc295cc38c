"""Mixed-form contact forces with 3 cells on an axis: full warps of selected
candidates (k_f_pp_warp) against one lane per home particle (k_f_pp) bit for
bit, packing energies to rounding.  A margin that changes no cell takes the latter."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("seed", range(3))
@pytest.mark.parametrize("N, r_p, n", [((32, 32, 32), 2.1, 1), ((32, 32, 32), 2.1, 33), ((32, 32, 32), 2.1, 700),
                                       ((32, 32, 64), 2.1, 300), ((64, 32, 128), 2.1, 900)])
def test_forces_are_the_plain_kernels(fipi, N, r_p, n, seed):
    nx, ny, nz = N
    w = fipi.workload("t32").with_(name="three", nx=nx, ny=ny, nz=nz, lx=float(nx), ly=float(ny), lz=float(nz),
                                   n_p=n, r_p=r_p)
    assert fipi.cell_geometry(w.params())[0].min() == 3
    rng = np.random.default_rng(seed)
    p = (rng.uniform(0.0, 1.0, (n, 3)) * [nx, ny, nz]).ravel()
    f_pi = rng.standard_normal(3 * n)
    res = []
    for margin in (0.0, 1e-300):
        P = w.params()
        P.margin = margin
        with fipi.Simulation(P, "mixed") as s:
            res.append(s.f_pp(p, 5, f_pi))
    (f, t), (g, u) = res
    assert np.array_equal(f, g)
    assert abs(t - u) <= 1e-12 * max(1.0, abs(u))
