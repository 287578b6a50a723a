"""Calls that need the symmetric kernels' scratch where it cannot be had in full: per-system
launches run the tuned kernel then, and the adjoint takes more, smaller bands."""
from __future__ import annotations

import numpy as np
import pytest

import nbody_gb300 as nb
import oracle_binding as orc
from helpers import disk_case, displacement_errors, g_eff, params

pytestmark = pytest.mark.gpu

N = 20000


@pytest.fixture
def sim():
    """A simulation that runs the tuned kernel and holds none of the scratch."""
    pos, vel, m = disk_case(N, seed=16)
    with nb.Simulation(params(N, acc=nb.ACC_COMPENSATED), pos, vel, m) as s:
        s.set_kernel_config(3)
        s.case = (pos, vel, m)
        yield s


@pytest.mark.parametrize("k", [1, 2, 3, 4])      # segments, i-tiles, rows, parts
def test_per_system_launches(sim, k):
    pos, vel, m = sim.case
    nb.inject_alloc_failure(k)
    try:
        sim.advance_per_system(2)
    finally:
        nb.inject_alloc_failure(0)
    got = sim.get_state()
    ref = orc.run_fp32(pos, vel, None, g_eff(1.0, m[0]), 1e-3, 0.999, 1e-3, iters=2)
    rms, mx = displacement_errors(got[:3], ref[:3], pos)
    assert rms <= 1e-4 and mx <= 1e-2, (rms, mx)


def test_adjoint(sim):
    g = np.random.default_rng(3).normal(size=3 * N).astype(np.float32)
    pos, vel, m = sim.case
    sim.adjoint_forward(2, 1)
    want = sim.adjoint_backward(g)
    failures = 0
    for k in range(1, 20):
        with nb.Simulation(params(N, acc=nb.ACC_COMPENSATED), pos, vel, m) as again:
            again.set_kernel_config(3)
            nb.inject_alloc_failure(k)
            try:
                again.adjoint_forward(2, 1)
            except nb.NbError as e:
                assert e.status == nb.NB_ERR_OUT_OF_MEMORY
                failures += 1
                continue
            finally:
                nb.inject_alloc_failure(0)
            got = again.adjoint_backward(g)
        # Other bands add the same terms in another order.
        for a, b in zip(got, want):
            assert np.linalg.norm(a - b) <= 1e-5 * np.linalg.norm(b), k
    assert failures == 9                         # two checkpoints, five work buffers
