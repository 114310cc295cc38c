"""Contact forces (cluster.cpp:174-275) against the oracle where the kernels'
rules change: 3 cells on an axis, more candidates than one staging round,
coincident particles, a contact range wider than a cell, one particle per
cell and none."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# name: (grid, n_p, r_p, r_eq / r_c)
CASES = {
    "cells3": ((64, 64, 64), 256, 4.0, 1.0),       # 3 x 3 x 3 cells
    "cells3_5": ((64, 128, 64), 301, 4.0, 1.0),    # 3 x 6 x 3
    "dense": ((16, 16, 16), 1700, 1.0, 1.0),       # 3^3 cells, 1700 candidates: three staging rounds
    "crowded": ((32, 32, 32), 2500, 1.2, 1.0),     # 5^3 cells, 540 candidates a cell and more
    "wide": ((64, 64, 64), 200, 4.0, 1.2),         # 3 cells, r_eq > d_cell: the general path
    "wide5": ((64, 64, 64), 200, 2.0, 1.3),        # 6 cells, r_eq > d_cell
    "sparse": ((64, 64, 64), 5, 1.0, 1.0),         # 12^3 cells, almost all empty
    "one": ((16, 16, 16), 1, 1.0, 1.0),
}


@pytest.mark.parametrize("name", CASES)
@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_contact_forces_match_oracle(fipi, oracle_mod, name, prec):
    (nx, ny, nz), n, r_p, wide = CASES[name]
    w = fipi.workload("t32").with_(name=name, nx=nx, ny=ny, nz=nz, lx=float(nx), ly=float(ny), lz=float(nz), n_p=n,
                                   r_p=r_p)
    P = w.params()
    P.r_eq = wide * P.r_c
    rng = np.random.default_rng(n)
    p = rng.uniform(0.0, 1.0, (n, 3)) * [nx, ny, nz]
    if n > 4:
        p[0] = p[n - 1]        # coincident
        p[1, 0] = 0.0          # on a cell face and the box face
        p[2] = p[3] + [1e-7, 0.0, 0.0] if p[3, 0] < nx - 1 else p[3] - [1e-7, 0.0, 0.0]
    p = p.ravel()
    f_pi = rng.standard_normal(3 * n)
    with fipi.Simulation(P, prec) as s:
        f, tau = s.f_pp(p, 3, f_pi)
        f0, _ = s.f_pp(p, 3)
    assert np.array_equal(f, f0)
    st, g, tau2, pairs = oracle_mod.f_pp(P, p, 3, f_pi, want_pairs=True)
    assert st == 0
    # every pair's force is at most r_eq k_n ramp; a particle sums up to m of
    # them, each off by a few units of rounding of that (positions: L eps)
    m = np.bincount(pairs.ravel(), minlength=n).max() if len(pairs) else 0
    unit = P.r_eq * P.k_n * min(1.0, 3 / (0.2 * P.t_end))
    eps = 2.0 ** -53 if prec == "fp64" else 2.0 ** -24
    # coincident to FP32 positions: the direction of the 1e-7 pair is not resolved in the mixed form
    near = np.zeros(n, bool)
    if n > 4 and prec == "mixed":
        near[[2, 3]] = True
    bar = 64 * eps * (m + 1) * unit + np.repeat(near, 3) * 4 * unit
    assert np.all(np.abs(f - g) <= bar)
    # tau sums 0.5 f . d over the pairs (k_f_pp_fast gives the 1e-7 pair, coincident
    # in FP32, the hashed separation of a coincident pair: FP64 form only)
    if prec == "fp64":
        assert abs(tau - tau2) <= 64 * eps * (len(pairs) + 1) * unit * P.r_eq
