"""Spreading and its adjoint where particles crowd a node: lists on both sides of
what a thread keeps in registers (8 records) and what a warp ranks in shared
memory (512), and the time of the longest."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_adjoint import _linear_loss

pytestmark = pytest.mark.gpu


def _params(fipi, n):
    return fipi.workload("t32").with_(name="crowd", n_p=n).params()


@pytest.mark.parametrize("n", [7, 8, 9, 31, 32, 33, 64, 65, 511, 512, 513, 545, 3000])
def test_one_cell_is_the_references_sum(fipi, oracle_mod, n):
    P = _params(fipi, n)
    rng = np.random.default_rng(n)
    p = (np.array([31.0, 4.0, 17.0]) + rng.uniform(0.0, 1.0, (n, 3))).ravel()  # n records on each of eight nodes
    f = rng.standard_normal(3 * n)
    with fipi.Simulation(P, "fp64") as s:
        want = oracle_mod.spread(P, p, f)
        assert np.array_equal(s.spread(p, f), want)
        assert np.array_equal(s.spread(p, f), want)  # the lists were left empty


@pytest.mark.parametrize("n", [300, 2500])
def test_lists_of_many_lengths(fipi, oracle_mod, n):
    """A cloud that thins out: lists of one to hundreds of records in a warp."""
    P = _params(fipi, n)
    rng = np.random.default_rng(n)
    p = np.mod(16.0 + rng.standard_normal((n, 3)) * 10.0 ** rng.uniform(-2.0, 0.8, (n, 1)), 32.0)
    p = np.where(p >= 32.0, 0.0, p).ravel()
    f = rng.standard_normal(3 * n)
    with fipi.Simulation(P, "fp64") as s:
        assert np.array_equal(s.spread(p, f), oracle_mod.spread(P, p, f))


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("n", [9, 512, 1000])
def test_sums_of_whole_numbers(fipi, prec, n):
    """Particles on a node and whole forces: exact sums in either form."""
    P = _params(fipi, n)
    f = np.arange(3 * n) % 7 - 2.0
    with fipi.Simulation(P, prec) as s:
        got = s.spread(np.tile([3.0, 5.0, 30.0], n), f).reshape(3, 32, 32, 32)
    want = np.zeros_like(got)
    want[:, 30, 5, 3] = f.reshape(n, 3).sum(0)
    assert np.array_equal(got, want)


@pytest.mark.parametrize("n", [3, 20, 400])  # two records a particle: 6, 40 and 800 on a node
def test_gradient_matches_finite_differences(fipi, n):
    steps, h = 2, 1e-5
    P = _params(fipi, n)
    P.k_n = 1e-3  # contacts of so many spheres in one place would drive them apart
    rng = np.random.default_rng(n)
    c = fipi.seed_phase(P, 3, 0.0, 0.05)
    p = (np.array([7.0, 12.0, 20.0]) + rng.uniform(0.3, 0.7, (n, 3))).ravel()
    w = {"c": np.zeros(c.size), "u": np.zeros(3 * c.size), "p": rng.standard_normal(3 * n), "f": rng.standard_normal(3 * n)}
    d = rng.standard_normal(c.size)

    def loss(x, grad=False):
        with fipi.Simulation(P, "fp64") as s:
            s.set_phase(x)
            s.set_particles(p)
            if not grad:
                s.step(steps)
                return _linear_loss(s, w)
            s.trajectory_forward(steps, steps)
            s.trajectory_backward(w["c"], w["u"], w["p"], w["f"])
            return s.adjoint_get()[0]

    fd = (loss(c + h * d) - loss(c - h * d)) / (2 * h)
    ad = float(loss(c, True) @ d)
    assert abs(ad - fd) <= 1e-5 * abs(fd), (ad, fd)


def test_time_of_a_crowded_cell(fipi):
    """20,000 particles in a cell: a sort of all records and a thread per node
    took 18.6 ms, a merge of links by one thread 150."""
    n = 20000
    P = _params(fipi, n)
    rng = np.random.default_rng(1)
    p = (5.0 + rng.uniform(0.0, 1.0, (n, 3))).ravel()
    with fipi.Simulation(P, "fp64") as s:
        s.spread(p, p)
        s.set_kernel_timing(True)
        s.spread(p, p)
        ms = sum(k["ms"] for k in s.kernel_stats() if k["name"].startswith("spread"))
    assert 0.0 < ms < 18.6
