"""PREDICATED on the reference-order kernel's j-pair shape: terms of other particles are
multiplied by zero, so a coincident, infinite or NaN one shows as NaN in the same places
as on the i-pair shape, and nowhere else."""
from __future__ import annotations

import numpy as np
import pytest

import nbody_gb300 as nb
from helpers import disk_case, params

pytestmark = pytest.mark.gpu


# Coincident particles in one warp, in one j-tile of 512 and in two, at block ends.
@pytest.mark.parametrize("n", [66, 200, 1025, 5001])
@pytest.mark.parametrize("what", ["coincident", "infinite", "nan"])
def test_not_a_number_in_the_same_places(n, what):
    pos, vel, _ = disk_case(n, seed=n)
    for a, b in ((1, 33), (5, n - 1), (64, 65), (n // 2, n // 2 + 1)):
        for c in pos:
            c[a] = c[b] if what == "coincident" else c[a]
    if what != "coincident":
        pos[1][n - 1] = np.inf if what == "infinite" else np.nan
    p = params(n, eps=0.0 if what == "coincident" else 1e-3, method=nb.PREDICATED)
    out = []
    for shape in (0, 3):
        with nb.Simulation(p, pos, vel, None) as sim:
            sim.set_kernel_config(shape)
            sim.advance(1)
            out.append(sim.get_state())
    assert any(np.isnan(a).any() for a in out[0])
    for a, b in zip(*out):
        assert np.array_equal(np.isnan(a), np.isnan(b))
        ok = ~np.isnan(a)
        assert np.array_equal(a[ok].view(np.uint32), b[ok].view(np.uint32))
