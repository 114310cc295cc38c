"""Step graphs in each of their layouts (spreading beside the Cahn-Hilliard
part, particle stages beside the projection, one chain, fluid coupling)
against direct launches bit for bit, and graphs kept over a new phase."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (grid, particles, radius): both branches up to 2^18 nodes, particle stages
# only above, one chain for mixed grids above 2^21
SMALL, MIDDLE, LARGE = ((32, 32, 32), 40, 1.2), ((128, 64, 64), 600, 2.0), ((256, 128, 128), 1500, 3.0)


def _start(fipi, s, P, couple, seed):
    c = fipi.seed_phase(P, seed, 0.0, 0.05)
    p, _, _ = fipi.seed_particles(P, seed + 1)
    s.set_phase(c)
    s.set_velocity(np.zeros(3 * c.size))
    s.set_particles(p)
    if couple:  # (a change of the setting drops the graphs)
        s.set_fluid_coupling(True)


def _state(s):
    return (s.get_phase(), s.get_velocity(), *s.get_particles())


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("size, couple", [(SMALL, True), (MIDDLE, False), (MIDDLE, True), (LARGE, False)])
def test_replay_equals_direct_launches(fipi, prec, size, couple):
    (nx, ny, nz), n, r = size
    P = fipi.workload("t32").with_(name="g", nx=nx, ny=ny, nz=nz, lx=float(nx), ly=float(ny), lz=float(nz), n_p=n,
                                   r_p=r, rho2=5e-2).params()
    res = []
    for direct in (False, True):
        with fipi.Simulation(P, prec) as s:
            _start(fipi, s, P, couple, 5)
            s.set_kernel_timing(direct)  # timed launches are direct
            s.step(5)
            res.append(_state(s))
    for a, b in zip(*res):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("steps", [3, 4])  # the buffers' assignment after an odd and an even number
def test_graphs_kept_over_a_new_phase(fipi, prec, steps):
    (nx, ny, nz), n, r = SMALL
    P = fipi.workload("t32").params()
    with fipi.Simulation(P, prec) as s:
        _start(fipi, s, P, False, 5)
        s.step(steps)
        _start(fipi, s, P, False, 9)
        s.step(4)
        again = _state(s)
    with fipi.Simulation(P, prec) as s:
        _start(fipi, s, P, False, 9)
        s.step(4)
        fresh = _state(s)
    for a, b in zip(again, fresh):
        assert np.array_equal(a, b)
