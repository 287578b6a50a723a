"""The adjoint after a call of it that failed between two of its allocations: the buffers
that are missing are made by the next call."""
from __future__ import annotations

import numpy as np
import pytest

import nbody_gb300 as nb
from helpers import disk_case, params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [300, 5000])       # direct, symmetric
def test_forward_again_after_a_failed_allocation(n):
    pos, vel, m = disk_case(n, seed=17)
    g = np.random.default_rng(4).normal(size=3 * n).astype(np.float32)
    with nb.Simulation(params(n), pos, vel, m) as sim:
        sim.adjoint_forward(5, 2)
        want = sim.adjoint_backward(g)
    failures = 0
    for k in range(1, 60):
        with nb.Simulation(params(n), pos, vel, m) as sim:
            nb.inject_alloc_failure(k)
            try:
                sim.adjoint_forward(5, 2)
                break
            except nb.NbError as e:
                assert e.status == nb.NB_ERR_OUT_OF_MEMORY
            finally:
                nb.inject_alloc_failure(0)
            failures += 1
            sim.set_state(pos, vel)
            sim.adjoint_forward(5, 2)
            got = sim.adjoint_backward(g)
        for a, b in zip(got, want):
            assert np.array_equal(a, b), k
    assert failures >= 12                        # checkpoints, segment, cotangents
