"""FP64 contact forces of isolated pairs: one term a particle, so the force is the
reference's (cluster.cpp:225-255) bit for bit, for either id order, through the
periodic faces and from nearly touching centres to the contact range."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("box", [64.0, 6.2831852])  # dx = 1 and an odd spacing
def test_isolated_pairs_are_the_references(fipi, oracle_mod, box):
    m = 6  # pairs per axis, 2 r_eq apart and more
    r_eq = box / (2 * m + 1)
    w = fipi.workload("t32").with_(name="pairs", nx=64, ny=64, nz=64, lx=box, ly=box, lz=box, n_p=2 * m ** 3,
                                   r_p=r_eq / 5)
    P = w.params()
    rng = np.random.default_rng(3)
    centre = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3) * (box / m)
    axis = rng.standard_normal(centre.shape)
    axis /= np.linalg.norm(axis, axis=1)[:, None]
    half = 0.5 * P.r_eq * 10.0 ** rng.uniform(-6, 0, len(centre))[:, None]  # separations up to r_eq
    p = np.concatenate([centre + half * axis, centre - half * axis]) % box
    p = np.where(p >= box, 0.0, p)[rng.permutation(w.n_p)].ravel()
    with fipi.Simulation(P, "fp64") as s:
        f, _ = s.f_pp(p, 40)
    st, g, _, pairs = oracle_mod.f_pp(P, p, 40, want_pairs=True)
    assert st == 0 and np.bincount(pairs.ravel(), minlength=w.n_p).max() == 1 and len(pairs) > m ** 3 // 2
    assert np.array_equal(f, g)
