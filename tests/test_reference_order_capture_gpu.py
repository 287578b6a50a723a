"""A captured step allocates nothing: graph capture right after a reference-order shape
was selected, without a step in between."""
from __future__ import annotations

import numpy as np
import pytest

import nbody_gb300 as nb
from helpers import disk_case, params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("method", [nb.BRANCH, nb.PREDICATED])
@pytest.mark.parametrize("shape", [0, 1, 2, 3])
def test_capture_right_after_a_shape_is_selected(shape, method):
    n = 3000                            # its default shape reads the positions themselves
    pos, vel, _ = disk_case(n, seed=11)
    p = params(n, method=method, acc=nb.ACC_REFERENCE_ORDER)
    with nb.Simulation(p, pos, vel, None) as sim:
        sim.set_kernel_config(shape)
        sim.graph_capture(2)
        sim.graph_launch()
        got = sim.get_state()
    with nb.Simulation(p, pos, vel, None) as sim:
        sim.advance(2)
        want = sim.get_state()
    for g, w in zip(got, want):
        assert np.array_equal(g.view(np.uint32), w.view(np.uint32))
