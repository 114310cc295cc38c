"""Contact forces where the reference's cells do not tile the box: L / r_c that
rounds up to a whole number (d_cell = fmod(L, r_c) / n + r_c then reaches one
r_c beyond L, cluster.cpp:26-32) and margin != 0.  The minimum image
shifts by L all the same."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_adjoint import _linear_loss

pytestmark = pytest.mark.gpu

# name: (box, r_c, margin)
CASES = {"five": (32.0, 6.4, 0.0), "thirteen": (32.0, 32.0 / 13, 0.0), "three": (10.0, 10.0 / 3, 0.0),
         "margin": (32.0, 5.0, 0.7), "margin_up": (32.0, 6.4, 0.25), "plain": (32.0, 5.0, 0.0)}


def _params(fipi, box, r_c, margin, n):
    w = fipi.workload("t32").with_(name="cells", lx=box, ly=box, lz=box, n_p=n, r_p=r_c / 5)
    P = w.params()
    P.r_c = P.r_eq = r_c
    P.margin = margin
    return P


def _positions(box, n, seed):
    """Half of them near the box's faces."""
    rng = np.random.default_rng(seed)
    p = rng.uniform(0.0, box, (n, 3))
    near = rng.integers(0, 3, n)
    half = np.arange(n) % 2 == 0
    p[half, near[half]] = rng.uniform(-box / 32, box / 32, half.sum()) % box
    return np.where(p >= box, 0.0, p).ravel()


@pytest.mark.parametrize("name", CASES)
@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_forces_match_oracle(fipi, oracle_mod, name, prec):
    box, r_c, margin = CASES[name]
    n = 400
    P = _params(fipi, box, r_c, margin, n)
    nc, dc = fipi.cell_geometry(P)
    if name in ("five", "thirteen", "three"):
        assert (nc * dc > box + 0.9 * r_c).all()
    p = _positions(box, n, 5)
    with fipi.Simulation(P, prec) as s:
        f, _ = s.f_pp(p, 3)
        pairs = s.pairs(p)
    st, g, _, pairs2 = oracle_mod.f_pp(P, p, 3, want_pairs=True)
    assert st == 0 and np.array_equal(pairs, pairs2)
    # at most m terms of up to r_eq k_n ramp a particle, each off by a few units of rounding (positions: L eps)
    m = np.bincount(pairs2.ravel(), minlength=n).max()
    unit = P.r_eq * P.k_n * min(1.0, 3 / (0.2 * P.t_end))
    eps = 2.0 ** -53 if prec == "fp64" else 2.0 ** -24
    assert np.abs(f - g).max() <= 64 * eps * (m + 1) * unit


@pytest.mark.parametrize("name", ["five", "margin"])
def test_gradient_matches_finite_differences(fipi, name):
    box, r_c, margin = CASES[name]
    n, steps, h = 60, 2, 1e-6
    P = _params(fipi, box, r_c, margin, n)
    c = fipi.seed_phase(P, 3, 0.0, 0.05)
    rng = np.random.default_rng(4)
    # clear of the faces by more than the step of the differences, so that no image changes
    p = np.clip(_positions(box, n, 8), 1e-3, box - 1e-3)
    w = {"c": np.zeros(c.size), "u": np.zeros(3 * c.size), "p": rng.standard_normal(3 * n), "f": rng.standard_normal(3 * n)}
    d = rng.standard_normal(3 * n)

    def loss(q, grad=False):
        with fipi.Simulation(P, "fp64") as s:
            s.set_phase(c)
            s.set_particles(q)
            if not grad:
                s.step(steps)
                return _linear_loss(s, w)
            s.trajectory_forward(steps, steps)
            s.trajectory_backward(w["c"], w["u"], w["p"], w["f"])
            return s.adjoint_get()[2]

    fd = (loss(p + h * d) - loss(p - h * d)) / (2 * h)
    ad = float(loss(p, True) @ d)
    assert abs(ad - fd) <= 1e-5 * abs(fd), (ad, fd)
