"""Fine-grained spreading between the steps of a running context: the lists it
shares with the step are left as they were, and are allocated once."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_calls_between_steps_change_nothing(fipi, prec):
    P = fipi.workload("t32").params()
    c = fipi.seed_phase(P, 3, 0.0, 0.05)
    p, _, _ = fipi.seed_particles(P, 4)
    rng = np.random.default_rng(5)
    q, f = rng.uniform(0.0, 32.0, p.size), rng.standard_normal(p.size)
    res, calls, held = [], [], []
    for between in (False, True):
        with fipi.Simulation(P, prec) as s:
            s.set_phase(c)
            s.set_particles(p)
            for _ in range(4):
                if between:
                    calls.append(s.spread(q, f))
                    held.append(s.device_bytes())
                s.step(1)
            res.append((s.get_phase(), s.get_velocity(), *s.get_particles()))
    for a, b in zip(*res):
        assert np.array_equal(a, b)
    assert all(np.array_equal(x, calls[0]) for x in calls) and len(set(held)) == 1
