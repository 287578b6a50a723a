"""nb_sim_set_state with masses of the other kind (equal, or one per particle) after the
work lists were planned: every kernel shape then runs its other variant in the scratch
that was made for the first, and gives what a simulation made with those masses gives."""
from __future__ import annotations

import numpy as np
import pytest

import nbody_gb300 as nb
from helpers import disk_case, params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cfg", range(nb.num_kernel_configs()))
@pytest.mark.parametrize("acc", [nb.ACC_PLAIN, nb.ACC_COMPENSATED])
@pytest.mark.parametrize("first", ["own", "equal"])
def test_other_masses_after_planning(cfg, acc, first):
    n = 9001
    pos, vel, m = disk_case(n, seed=3)
    own = (m * np.random.default_rng(1).uniform(0.5, 1.5, n)).astype(np.float32)
    before, after = (own, m) if first == "own" else (m, own)
    with nb.Simulation(params(n, acc=acc), pos, vel, before) as sim:
        sim.set_kernel_config(cfg)
        sim.advance(1)
        sim.set_state(pos, vel, after)
        got = sim.accelerations()
    with nb.Simulation(params(n, acc=acc), pos, vel, after) as sim:
        sim.set_kernel_config(cfg)
        want = sim.accelerations()
    for g, w in zip(got, want):
        scale = np.sqrt(np.mean(np.square(w, dtype=np.float64)))
        assert np.max(np.abs(g - w)) <= 1e-4 * scale
