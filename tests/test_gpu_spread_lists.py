"""FP64 spreading by node lists and one-block cell lists against the oracle:
bit for bit, with short lists, lists longer than a thread keeps in registers,
and particle counts on both sides of the one-block limit."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n, extent", [(1, 1.0), (9, 0.4), (300, 1.5), (1500, 3.0), (2500, 32.0)])
def test_spread_is_the_references_sum(fipi, oracle_mod, n, extent):
    """`extent`: the particles lie in a cube of that many nodes (n / extent^3
    of them add up on a node, from 1 to 300)."""
    P = fipi.workload("t32").with_(name="lists", n_p=n).params()
    rng = np.random.default_rng(n)
    p = np.mod(31.0 + rng.uniform(0.0, extent, (n, 3)), 32.0).ravel()  # across the periodic faces
    f = rng.standard_normal(3 * n)
    with fipi.Simulation(P, "fp64") as s:
        assert np.array_equal(s.spread(p, f), oracle_mod.spread(P, p, f))
        assert np.array_equal(s.spread(p, f), oracle_mod.spread(P, p, f))  # the lists were left empty


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("n", [1, 31, 1023, 1024, 1025])
def test_cell_lists_around_the_one_block_limit(fipi, oracle_mod, n, prec):
    P = fipi.workload("t32").with_(name="cells", n_p=n).params()
    p = np.random.default_rng(n).uniform(0.0, 32.0, 3 * n)
    with fipi.Simulation(P, prec) as s:
        got = s.cells_build(p)
    st, keys, srt, off = oracle_mod.sorting(P, p)[:4]
    assert st == 0
    for a, b in zip(got, (keys, srt, off)):
        assert np.array_equal(a, b)
