"""fipi_trajectory_backward returns with the context's state in place: the
context stream has nothing left to do, and the state is the one after the
trajectory's first step."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_backward_returns_with_the_state_in_place(fipi):
    torch = pytest.importorskip("torch")
    # states of 0.8 GB: restoring one takes longer than the query below
    w = fipi.workload("t32").with_(name="large", nx=256, ny=256, nz=128, lx=256.0, ly=256.0, lz=128.0, n_p=0)
    P = w.params()
    c = fipi.seed_phase(P, 3, 0.0, 0.05)
    with fipi.Simulation(P, "fp64") as s:
        s.set_phase(c)
        s.step(1)
        first = s.get_phase()
    with fipi.Simulation(P, "fp64") as s:
        stream = torch.cuda.ExternalStream(s.stream())
        s.set_phase(c)
        s.trajectory_forward(2, 2)
        s.trajectory_backward(c)
        idle = stream.query()
        assert idle
        assert np.array_equal(s.get_phase(), first)
