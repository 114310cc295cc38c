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
    assert 0.0 < ms < 1.1


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("r_p, n", [(0.2, 5), (0.3, 33), (0.3, 1500), (0.45, 64), (0.6, 7)])
def test_forces_in_sparse_cells(fipi, oracle_mod, prec, r_p, n):
    P = _params(fipi, r_p, n)
    p = _clusters(n, 32.0, P.r_eq, n)
    with fipi.Simulation(P, prec) as s:
        f, _ = s.f_pp(p, 3)
    st, g, _, pairs = oracle_mod.f_pp(P, p, 3, want_pairs=True)
    assert st == 0 and len(pairs) > 0
    # at most m terms of up to r_eq k_n ramp a particle, each off by a few units of rounding (positions: L eps)
    m = np.bincount(pairs.ravel(), minlength=n).max()
    unit = P.r_eq * P.k_n * min(1.0, 3 / (0.2 * P.t_end))
    eps = 2.0 ** -53 if prec == "fp64" else 2.0 ** -24
    assert np.abs(f - g).max() <= 64 * eps * (m + 1) * unit * (32.0 / P.r_eq if prec == "fp64" else 1.0)


@pytest.mark.parametrize("r_p, n", [(0.2, 6), (0.3, 40)])
def test_gradient_in_sparse_cells(fipi, r_p, n):
    steps, h = 2, 1e-6
    P = _params(fipi, r_p, n)
    c = fipi.seed_phase(P, 3, 0.0, 0.05)
    rng = np.random.default_rng(n)
    p = np.clip(_clusters(n, 32.0, P.r_eq, n), 1e-3, 32.0 - 1e-3)
    w, d = rng.standard_normal(3 * n), rng.standard_normal(3 * n)

    def loss(q, grad=False):
        with fipi.Simulation(P, "fp64") as s:
            s.set_phase(c)
            s.set_particles(q)
            if not grad:
                s.step(steps)
                return np.dot(w, s.get_particles()[1])
            s.trajectory_forward(steps, steps)
            s.trajectory_backward(np.zeros(c.size), np.zeros(3 * c.size), np.zeros(3 * n), w)
            return s.adjoint_get()[2]

    fd = (loss(p + h * d) - loss(p - h * d)) / (2 * h)
    ad = float(loss(p, True) @ d)
    assert abs(ad - fd) <= 1e-5 * abs(fd), (ad, fd)


@pytest.mark.parametrize("prec, most", [("fp64", 0.25), ("mixed", 1.4)])
def test_time_of_the_forces(fipi, prec, most):
    """1000 particles in 614,000 cells, in ms: one warp or block looking at every
    cell's neighbours took `most` or a little less, a block starting for every cell more."""
    P = _params(fipi, 0.6, 1000, 256)
    ms = _ms(fipi, P, prec, np.random.default_rng(1).uniform(0.0, 256.0, 3000), "contact forces")
    assert 0.0 < ms < most
