"""Grids with far more cells than particles: lists and contact forces against the
oracle, and the time of a list."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _params(fipi, r_p, n, N=32):
    return fipi.workload("t32").with_(name="cells", nx=N, ny=N, nz=N, lx=float(N), ly=float(N), lz=float(N), n_p=n,
                                      r_p=r_p).params()


def _clusters(n, L, r_eq, seed):
    """Groups of a few within reach of one another, across the faces too."""
    rng = np.random.default_rng(seed)
    site = rng.choice([0.0, 0.3, 0.61, 1.0], (max(1, n // 4), 3)) * L
    p = np.mod(site[rng.integers(0, len(site), n)] + rng.uniform(-0.7, 0.7, (n, 3)) * r_eq, L)
    return np.where(p >= L, 0.0, p).ravel()


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("r_p, n", [(0.2, 5), (0.3, 33), (0.3, 1500), (0.45, 64), (0.6, 7)])  # 32^3 to 10^3 cells
def test_lists_of_sparse_cells(fipi, oracle_mod, prec, r_p, n):
    P = _params(fipi, r_p, n)
    with fipi.Simulation(P, prec) as s:
        for seed in range(3):  # the counts are left at zero
            p = _clusters(n, 32.0, P.r_eq, seed)
            got = s.cells_build(p)
            st, keys, srt, off = oracle_mod.sorting(P, p)[:4]
            assert st == 0
            for a, b in zip(got, (keys, srt, off)):
                assert np.array_equal(a, b)


def _ms(fipi, P, prec, p, name):
    with fipi.Simulation(P, prec) as s:
        s.f_pp(p, 3)
        s.set_kernel_timing(True)
        s.f_pp(p, 3)
        return sum(k["ms"] for k in s.kernel_stats() if k["name"] == name)


def test_time_of_the_offsets(fipi):
    """614,000 cells: 0.70 ms, and 1.16 with the counts zeroed in the same pass."""
    P = _params(fipi, 0.6, 1000, 256)
    ms = _ms(fipi, P, "fp64", np.random.default_rng(1).uniform(0.0, 256.0, 3000), "cell offsets")
    assert 0.0 < ms < 0.95
